"""The pointwise Riemann entry points on states at the ends of FP64's range, where the kernels'
branch-free division does not serve: the oracle's IEEE fluxes."""
import ctypes

import numpy as np
import pytest

from canoe_b200 import thermo
from canoe_b200._abi import RS_HLLC, RS_LMARS, check, load

pytestmark = pytest.mark.gpu


def _flux(rs, th, ivx, wl, wr):
    import torch
    dl, dr = torch.from_numpy(wl).cuda(), torch.from_numpy(wr).cuda()
    df = torch.zeros_like(dl)
    fn = load().canoe_riemann_lmars if rs == RS_LMARS else load().canoe_riemann_hllc
    check(fn(ctypes.byref(th), ivx, dl.data_ptr(), dr.data_ptr(), df.data_ptr(), wl.shape[1], None))
    torch.cuda.synchronize()
    return df.cpu().numpy()


# subnormal densities of 44 bits (2^-1030): a few dozen roundings of 2^-44; densities whose
# reciprocal is subnormal (2^1022, slow sound, so that HLLC's products stay in range): roundings of
# 2^-53, 1e-13 as tests/test_gpu_parity.py
@pytest.mark.parametrize("lo,hi,p,v,tol", [(1.0, 1.9, 1e5, 100.0, 64 * 2.0 ** -44),
                                           (1.1, 1.9, 2.0 ** -800, 2.0 ** -402, 1e-13)])
@pytest.mark.parametrize("rs", [RS_LMARS, RS_HLLC])
@pytest.mark.parametrize("moist", [0, 1])
def test_fluxes_at_the_ends_of_the_range(lo, hi, p, v, tol, rs, moist):
    from oracle import oracle
    th = thermo.earth_moist() if moist else thermo.dry()
    scale = 2.0 ** -1030 if p > 1 else 2.0 ** 1022
    rng = np.random.Generator(np.random.PCG64(5))
    n, ny = 257, th.ny

    def side():
        w = np.zeros((5 + ny, n))
        w[0] = rng.uniform(lo, hi, n) * scale
        w[1:1 + ny] = rng.uniform(0, 0.01, (ny, n))
        w[1 + ny:4 + ny] = v * rng.uniform(-1, 1, (3, n))
        w[4 + ny] = p * rng.uniform(0.9, 1.1, n) * scale
        return w

    wl, wr = side(), side()
    ref = oracle.riemann(rs, th, 1 + ny, wl, wr)
    got = _flux(rs, th, 1 + ny, wl, wr)
    assert np.isfinite(ref).all() and np.isfinite(got).all()
    s = np.abs(ref).max(axis=1, keepdims=True)
    assert (np.abs(got - ref) <= tol * s).all()
