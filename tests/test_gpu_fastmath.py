"""The kernels' branch-free division and square root (csrc/physics.cuh) against the correctly
rounded results: at most one unit in the last place over the normal range."""
import numpy as np
import pytest

from canoe_b200._abi import check, load

pytestmark = pytest.mark.gpu


def _run(fp32, a, b=None):
    out = np.empty_like(a)
    check(load().canoe_selftest_fastmath(fp32, a.ctypes.data, None if b is None else b.ctypes.data,
                                         out.ctypes.data, len(a)), "selftest_fastmath")
    return out


def _ulps(got, want, dt):
    got, want = got.astype(dt), want.astype(dt)
    return np.abs((got.astype(np.longdouble) - want.astype(np.longdouble)) /
                  np.spacing(np.abs(want)).astype(np.longdouble)).max()


@pytest.mark.parametrize("fp32,dt,span", [(0, np.float64, 100.0), (1, np.float32, 17.0)])
def test_division_and_root_within_one_ulp(fp32, dt, span):
    # magnitudes 10^-span .. 10^span (quotients stay normal), mantissas at random and close to
    # powers of two, where a residual correction that is off by one shows
    rng = np.random.Generator(np.random.PCG64(3))
    n = 1 << 20
    edge = 1.0 + np.finfo(dt).eps * rng.integers(-8, 9, n // 4)
    m = np.concatenate([rng.uniform(1.0, 2.0, n - len(edge)), edge])
    a = (m * 10.0 ** rng.uniform(-span, span, n)).astype(dt).astype(np.float64)
    b = (rng.permutation(m) * 10.0 ** rng.uniform(-span, span, n)).astype(dt).astype(np.float64)
    a[::3] *= -1.0
    assert _ulps(_run(fp32, a, b), a.astype(dt) / b.astype(dt), dt) <= 1.0
    assert _ulps(_run(fp32, np.abs(b)), np.sqrt(np.abs(b).astype(dt)), dt) <= 1.0


@pytest.mark.parametrize("fp32", [0, 1])
def test_special_operands(fp32):
    z = np.array([0.0, -0.0, np.nan, np.inf])
    r = _run(fp32, z)
    assert r[0] == 0.0 and r[1] == 0.0 and np.isnan(r[2]) and np.isinf(r[3])
    assert np.isnan(_run(fp32, np.array([-1.0]))[0])
    q = _run(fp32, np.array([0.0, np.nan, 1.0, 3.0]), np.array([2.0, 2.0, np.nan, 1.5]))
    assert q[0] == 0.0 and np.isnan(q[1]) and np.isnan(q[2]) and q[3] == 2.0
