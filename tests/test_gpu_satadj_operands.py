"""The saturation adjustment on cells no model holds (infinite energies, squares that overflow,
densities at the ends of FP64's range): the oracle's temperatures, partitions and iteration counts."""
import ctypes

import numpy as np
import pytest

from canoe_b200 import thermo
from canoe_b200._abi import SatOpts, check, load

pytestmark = pytest.mark.gpu

INF = np.inf
CASES = [{}, dict(u0=0.0, u1=0.0, u2=0.0), dict(u7=-1e5), dict(u7=1e300), dict(u0=np.nan),
         dict(u7=INF), dict(u7=-INF), dict(u4=1e200), dict(u4=INF), dict(u1=INF),
         dict(u0=1e300, u7=1e300), dict(u0=1e308, u7=1e308), dict(u0=-1.0), dict(u1=-0.5),
         dict(u7=1e7), dict(u0=0.0)]


def test_adjustment_at_the_ends_of_the_range():
    import torch
    from oracle import oracle
    th = thermo.earth_moist()
    base = np.array([1.1, 0.01, 1e-4, 0.0, 3.0, 2.0, 1.0, 0.0])
    base[7] = 7.0 + 1.1 * 718 * 290 + 0.01 * 2.5e6
    u = np.repeat(base[:, None], len(CASES), axis=1)
    for i, c in enumerate(CASES):
        for k, v in c.items():
            u[int(k[1:]), i] = v
    n = u.shape[1]
    d = torch.from_numpy(u).cuda()
    t = torch.zeros(n, dtype=torch.float64, device="cuda")
    it = torch.zeros(n, dtype=torch.int32, device="cuda")
    o = SatOpts(1e-8, 30, 0)
    check(load().canoe_saturation_adjust(ctypes.byref(th), ctypes.byref(o), d.data_ptr(), n, None,
                                         t.data_ptr(), it.data_ptr(), None, None))
    torch.cuda.synchronize()
    want = u.copy()
    wt, wi, _ = oracle.satadj(th, want)
    assert it.cpu().numpy().tolist() == wi.tolist()
    # both converge a Newton step beyond 1e-8 K
    np.testing.assert_allclose(t.cpu().numpy(), wt, rtol=1e-9, atol=0.0)
    np.testing.assert_allclose(d.cpu().numpy(), want, rtol=1e-9, atol=1e-12)
