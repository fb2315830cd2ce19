"""The 5x5 block solve of the column march (csrc/march.cuh): elimination without pivoting where no
pivot cancels, with pivoting where one does."""
import numpy as np
import pytest

from canoe_b200._abi import check, load

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _solve(a, rhs):
    n = len(a)
    a, rhs = np.ascontiguousarray(a), np.ascontiguousarray(rhs)
    x, piv = np.empty_like(rhs), np.empty(n, dtype=np.int32)
    check(load().canoe_selftest_block_solve(a.ctypes.data, rhs.ctypes.data, x.ctypes.data,
                                            piv.ctypes.data, n), "selftest_block_solve")
    return x, piv


def _backward(a, rhs, x):
    """largest componentwise backward error, in units of the last place"""
    r = np.abs(a @ x - rhs) / (np.abs(a) @ np.abs(x) + np.abs(rhs))
    return (r / EPS).max()


# Elimination of a 5x5 system: each entry of L U and of the two sweeps sums at most five products, so
# |A x - b| <= 3 * 5 eps |L| |U| |x| (Higham, theorem 9.4), and |L| |U| <= g |A| with g <= 160 where the
# pivots stay within a factor of 8 or 16 of the diagonal; without cancellation g is about 5
def test_dominant_diagonals_need_no_pivoting():
    rng = np.random.Generator(np.random.PCG64(1))
    n = 4000
    a = np.eye(5) * 4.0 + rng.uniform(-1, 1, (n, 5, 5))
    s = 10.0 ** rng.uniform(-6, 6, (n, 5))
    a = a * s[:, :, None] / s[:, None, :]  # units: no largest entry to go by
    rhs = rng.uniform(-1, 1, (n, 5, 6)) * s[:, :, None]
    x, piv = _solve(a, rhs)
    assert piv.sum() <= n // 100
    assert _backward(a[piv == 0], rhs[piv == 0], x[piv == 0]) < 15 * 160


@pytest.mark.parametrize("small", [0.0, 1e-300, 1e-12, 1e-3])
@pytest.mark.parametrize("at", range(4))
def test_vanishing_pivots_are_pivoted(small, at):
    rng = np.random.Generator(np.random.PCG64(2))
    n = 500
    # well-conditioned, with a leading minor of `at` + 1 rows that (nearly) vanishes
    q = np.linalg.qr(rng.standard_normal((n, 5, 5)))[0]
    lead = q[:, :at, :at]
    d = np.zeros(n)
    if at:
        d = np.einsum("ni,ni->n", q[:, at, :at],
                      np.linalg.solve(lead, q[:, :at, at][:, :, None])[:, :, 0])
    q[:, at, at] = d + small
    ok = np.linalg.cond(q) < 1e3
    if at:
        ok &= np.linalg.cond(lead) < 1e2
    q = q[ok]
    rhs = rng.uniform(-1, 1, (len(q), 5, 6))
    x, piv = _solve(q, rhs)
    assert piv.all()
    # partial pivoting: |A x - b| <= 15 eps g |A| |x| with growth g <= 16
    assert _backward(q, rhs, x) < 15 * 16 * 5
