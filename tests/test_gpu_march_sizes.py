"""The column march (csrc/march.cuh) at the sizes where its forms have edges, each case checked to
march: 5x5 blocks on Cartesian columns, and FP32 chunks of eight and of four levels, even and odd
columns, whole chunks and every remainder, both reconstructions and solvers, and the shell."""
import numpy as np
import pytest

from canoe_b200 import MeshBlock, Shell, problems, thermo
from canoe_b200._abi import FP32_PERTURBATION, RECON_PLM, RECON_PPM, RS_HLLC, RS_LMARS
from test_gpu_march import _perturbed, _rel

pytestmark = pytest.mark.gpu

THERMO = {0: thermo.dry, 2: lambda: thermo.moist(("H2O",), ice=False), 3: thermo.earth_moist,
          6: thermo.earth_water_ammonia}


def _problem(nx1, nx2, nx3, recon, rs, ny, **kw):
    p = problems.moist3d(nx1=nx1, nx2=nx2, nx3=nx3, x1max=250.0 * nx1, x2max=250.0 * nx2,
                         x3max=250.0 * nx3, th=THERMO[ny](), recon=recon, rsolver=rs, satadj=0, **kw)
    return _perturbed(p, 31)


def _step(p, dt=0.2):
    b = MeshBlock(p)
    assert b.marches()
    b.step(dt)
    assert b.error_word() == 0
    return b.conserved()


# bounds as tests/test_gpu_march.py: FP64 5e-11 (3x3) and 1e-10 (5x5) of the oracle, FP32 fluxes 1e-5

@pytest.mark.parametrize("nx1,nx2,nx3", [(4, 36, 37), (7, 39, 35), (34, 37, 36), (61, 1301, 1)])
@pytest.mark.parametrize("recon,rs,ny", [(RECON_PPM, RS_HLLC, 3), (RECON_PLM, RS_LMARS, 0),
                                         (RECON_PPM, RS_HLLC, 6)])
def test_full_correction(nx1, nx2, nx3, recon, rs, ny):
    from oracle import oracle
    p = _problem(nx1, nx2, nx3, recon, rs, ny, implicit_flag=9)
    o = oracle.OracleBlock(p, roundtrip=False)
    o.step(0.2)
    assert _rel(p, _step(p), o.conserved(), 0.2) < 1e-10
    p.cfg.precision = FP32_PERTURBATION
    assert _rel(p, _step(p), o.conserved(), 0.2) < 1e-5


# nc1 = nx1 + 6 levels: remainders 0 to 7 of eight, with ragged tiles
@pytest.mark.parametrize("nx1,nx2,nx3", [(4, 62, 63), (5, 64, 64), (18, 62, 63), (19, 63, 62),
                                         (20, 62, 64), (21, 61, 64), (22, 3601, 1), (23, 64, 63),
                                         (33, 62, 63)])
@pytest.mark.parametrize("recon,rs,ny", [(RECON_PPM, RS_HLLC, 0), (RECON_PLM, RS_LMARS, 2),
                                         (RECON_PLM, RS_HLLC, 3), (RECON_PPM, RS_LMARS, 0)])
def test_fp32_partial_correction(nx1, nx2, nx3, recon, rs, ny):
    from oracle import oracle
    p = _problem(nx1, nx2, nx3, recon, rs, ny)
    o = oracle.OracleBlock(p, roundtrip=False)
    o.step(0.2)
    p.cfg.precision = FP32_PERTURBATION
    assert _rel(p, _step(p), o.conserved(), 0.2) < 1e-5


@pytest.mark.parametrize("f32,nx1,nx2,nx3", [(0, 65, 64, 74), (1, 64, 62, 63), (1, 33, 64, 74)])
def test_six_species(f32, nx1, nx2, nx3):
    from oracle import oracle
    p = _problem(nx1, nx2, nx3, RECON_PPM, RS_HLLC, 6)
    o = oracle.OracleBlock(p, roundtrip=False)
    o.step(0.2)
    if f32:
        p.cfg.precision = FP32_PERTURBATION
    assert _rel(p, _step(p), o.conserved(), 0.2) < (1e-5 if f32 else 5e-11)


@pytest.mark.parametrize("nx1,nside,flag,f32", [(15, 16, 9, 0), (15, 16, 9, 1), (12, 16, 9, 1),
                                                (10, 32, 1, 1), (13, 24, 1, 1), (11, 28, 1, 0)])
def test_shell(nx1, nside, flag, f32):
    from oracle import oracle
    p = problems.shell_c3(nx1=nx1, nside=nside, implicit_flag=flag)
    o = oracle.OracleShell(p)
    o.step(30.0)
    if f32:
        p.cfg.precision = FP32_PERTURBATION
    g = Shell(p)
    assert g.marches()
    g.step(30.0)
    a, b = p.interior(g.conserved()), p.interior(o.conserved())
    tol = 1e-5 if f32 else (5e-11 if flag == 1 else 1e-10)
    for n in range(5):
        s = np.linalg.norm(b[:, n])
        if 1 <= n <= 3:
            s = max(s, 30.0 * 24.79 * np.linalg.norm(b[:, 0]))
        assert np.linalg.norm(a[:, n] - b[:, n]) <= tol * s
