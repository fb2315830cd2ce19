"""The column march (csrc/march.cuh) when one of its bounded waits gives up: the error bit is set,
the state stays what the stage found, and the next step of the same block is unharmed.  The waits
give up by themselves here (no poll is made) while their copies arrive as always."""
import numpy as np
import pytest

from canoe_b200 import MeshBlock, problems, thermo
from canoe_b200._abi import FP32_PERTURBATION, check, load

pytestmark = pytest.mark.gpu

EBIT_TIMEOUT = 32
POLLS = 1 << 18  # the default


def _problem(nx1, nx2, nx3, f32, flag, ny):
    p = problems.moist3d(nx1=nx1, nx2=nx2, nx3=nx3, x1max=250.0 * nx1, x2max=250.0 * nx2,
                         x3max=250.0 * nx3, th=thermo.earth_moist() if ny else thermo.dry(),
                         satadj=0, implicit_flag=flag)
    if f32:
        p.cfg.precision = FP32_PERTURBATION
    return p


# columns of even and odd numbers of levels, chunks of four and eight levels, both block sizes
@pytest.mark.parametrize("nx1,nx2,nx3,f32,flag,ny", [
    (18, 71, 62, 0, 1, 3), (13, 71, 62, 0, 1, 3), (18, 71, 62, 1, 1, 3), (13, 71, 62, 1, 1, 0),
    (18, 40, 33, 0, 9, 3), (13, 40, 33, 1, 9, 0)])
@pytest.mark.parametrize("way", ["down", "up"])
def test_timed_out_stage_leaves_the_state(nx1, nx2, nx3, f32, flag, ny, way):
    p = _problem(nx1, nx2, nx3, f32, flag, ny)
    lib = load()
    a, b = MeshBlock(p), MeshBlock(p)
    u0 = a.conserved()
    check(lib.canoe_selftest_march_wait(a.h, *((0, POLLS) if way == "down" else (POLLS, 0))))
    a.step(0.2)
    assert a.error_word() & EBIT_TIMEOUT
    assert np.array_equal(p.interior(a.conserved()), p.interior(u0))
    check(lib.canoe_selftest_march_wait(a.h, POLLS, POLLS))
    a.step(0.2)
    b.step(0.2)
    assert a.error_word() == 0 and b.error_word() == 0
    assert np.array_equal(a.conserved(), b.conserved())


def test_wait_limits_are_checked():
    p = _problem(18, 8, 8, 0, 1, 3)
    b = MeshBlock(p)
    lib = load()
    assert lib.canoe_selftest_march_wait(None, 1, 1) != 0
    assert lib.canoe_selftest_march_wait(b.h, -1, 1) != 0
    assert lib.canoe_selftest_march_wait(b.h, 1, POLLS + 1) != 0
