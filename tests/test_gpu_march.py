"""The column march (csrc/march.cuh), which steps blocks of many columns, against the oracle at
the sizes where its chunks of four levels and tiles of 32 columns have edges."""
import numpy as np
import pytest

from canoe_b200 import MeshBlock, Shell, problems, thermo
from canoe_b200._abi import (BC_OUTFLOW, BC_REFLECT, FP32_PERTURBATION, RECON_PLM, RECON_PPM,
                             RS_HLLC, RS_LMARS)

pytestmark = pytest.mark.gpu


def _rel(p, a, b, dt):
    """largest per-variable relative L2 difference of two interior states; momentum is held to
    the larger of its norm and the gravity impulse dt rho g, of which it is the small net"""
    a, b = p.interior(a), p.interior(b)
    ivx = 1 + p.ny
    imp = dt * abs(p.cfg.thermo.grav) * np.linalg.norm(b[0])
    out = 0.0
    for n in range(len(b)):
        s = np.linalg.norm(b[n])
        if ivx <= n < ivx + 3:
            s = max(s, imp)
        d = np.linalg.norm(a[n] - b[n])
        out = max(out, d / s if s > 0 else d)
    return out


def _perturbed(p, seed):
    """seeded winds and condensate on top of the configuration's state, so that every slot and
    every flux is exercised"""
    rng = np.random.Generator(np.random.PCG64(seed))
    w = p.interior(p.w).copy()
    ny = p.ny
    if ny:
        w[1] *= 1.0 + 0.1 * rng.uniform(-1, 1, w[1].shape)
        w[2:1 + ny] = 1e-4 * rng.uniform(0, 1, w[2:1 + ny].shape)
    w[1 + ny:4 + ny] = 5.0 * rng.uniform(-1, 1, w[1 + ny:4 + ny].shape)
    w[4 + ny] *= 1.0 + 1e-3 * rng.uniform(-1, 1, w[0].shape)
    p.interior(p.u)[...] = thermo.prim_to_cons(p.cfg.thermo, w)
    return p


# levels: below, at and off the chunk of four, even rows (16-byte copies) and odd ones (8-byte);
# columns: whole tiles and a ragged last one
@pytest.mark.parametrize("nx1,nx2,nx3", [(4, 80, 80), (5, 63, 96), (7, 99, 61), (8, 6007, 1),
                                         (33, 78, 77), (34, 77, 79)])
@pytest.mark.parametrize("recon,rs,ny", [(RECON_PPM, RS_HLLC, 3), (RECON_PLM, RS_LMARS, 0),
                                         (RECON_PLM, RS_HLLC, 2), (RECON_PPM, RS_LMARS, 6)])
def test_march_step_matches_oracle(nx1, nx2, nx3, recon, rs, ny):
    from oracle import oracle
    th = {0: thermo.dry, 2: lambda: thermo.moist(("H2O",), ice=False), 3: thermo.earth_moist,
          6: thermo.earth_water_ammonia}[ny]()
    p = problems.moist3d(nx1=nx1, nx2=nx2, nx3=nx3, x1max=250.0 * nx1, x2max=250.0 * nx2,
                         x3max=250.0 * nx3, th=th, recon=recon, rsolver=rs, satadj=0)
    _perturbed(p, 7)
    g, o = MeshBlock(p), oracle.OracleBlock(p, roundtrip=False)
    dt = 0.2
    g.step(dt)
    o.step(dt)
    # as tests/test_gpu_parity.py: 5e-11 per variable and step
    assert _rel(p, g.conserved(), o.conserved(), dt) < 5e-11
    assert g.error_word() == 0


# the 5x5 correction: 1e-10 as its pin to the reference's own code (tests/test_ref_pin.py), whose
# two Gauss-Jordan inverses already differ by 1e-11
@pytest.mark.parametrize("nx1,nx2,nx3", [(4, 32, 33), (7, 35, 30), (34, 33, 34), (61, 1031, 1)])
@pytest.mark.parametrize("recon,rs,ny", [(RECON_PPM, RS_HLLC, 3), (RECON_PLM, RS_LMARS, 0)])
def test_march_full_correction_matches_oracle(nx1, nx2, nx3, recon, rs, ny):
    from oracle import oracle
    th = thermo.earth_moist() if ny else thermo.dry()
    p = problems.moist3d(nx1=nx1, nx2=nx2, nx3=nx3, x1max=250.0 * nx1, x2max=250.0 * nx2,
                         x3max=250.0 * nx3, th=th, recon=recon, rsolver=rs, satadj=0,
                         implicit_flag=9)
    _perturbed(p, 8)
    g, o = MeshBlock(p), oracle.OracleBlock(p, roundtrip=False)
    g.step(0.2)
    o.step(0.2)
    assert _rel(p, g.conserved(), o.conserved(), 0.2) < 1e-10
    p.cfg.precision = FP32_PERTURBATION
    m = MeshBlock(p)
    m.step(0.2)
    assert _rel(p, m.conserved(), o.conserved(), 0.2) < 1e-5


@pytest.mark.parametrize("bc", [(BC_OUTFLOW, BC_OUTFLOW), (BC_REFLECT, BC_OUTFLOW),
                                (BC_OUTFLOW, BC_REFLECT)])
def test_march_outflow_walls(bc):
    from oracle import oracle
    p = problems.moist3d(nx1=18, nx2=80, nx3=78, x1max=4500.0, x2max=20000.0, x3max=19500.0,
                         satadj=0)
    p.cfg.bc[0], p.cfg.bc[1] = bc
    _perturbed(p, 9)
    g, o = MeshBlock(p), oracle.OracleBlock(p, roundtrip=False)
    g.step(0.2)
    o.step(0.2)
    assert _rel(p, g.conserved(), o.conserved(), 0.2) < 5e-11


@pytest.mark.parametrize("nx1", [18, 19])
def test_march_fp32_fluxes_close_to_fp64(nx1):
    p = problems.moist3d(nx1=nx1, nx2=79, nx3=78, x1max=250.0 * nx1, x2max=19750.0, x3max=19500.0,
                         satadj=0)
    _perturbed(p, 11)
    a = MeshBlock(p)
    p.cfg.precision = FP32_PERTURBATION
    b = MeshBlock(p)
    for _ in range(2):
        a.step(0.2)
        b.step(0.2)
    # FP32 fluxes: 1e-5 of the flux (tests/test_gpu_mixed.py), times dt over dx, two steps
    assert _rel(p, b.conserved(), a.conserved(), 0.4) < 1e-5


def test_march_by_stages_on_a_stream_and_by_graph():
    """stage by stage, on a caller's stream and through a graph: the same bits"""
    import torch
    from canoe_b200._abi import check
    p = problems.moist3d(nx1=20, nx2=78, nx3=77, x1max=5000.0, x2max=19500.0, x3max=19250.0)
    _perturbed(p, 13)
    a, b = MeshBlock(p), MeshBlock(p, graph=True)
    s = torch.cuda.Stream()
    check(a.lib.canoe_block_set_stream(a.h, s.cuda_stream))
    a.set_fixed_dt(0.2)
    b.set_fixed_dt(0.2)
    for _ in range(2):
        for st in range(3):
            check(a.lib.canoe_block_stage(a.h, st, 0.2 if st == 0 else -1.0))
        b.step()
    assert np.array_equal(a.conserved(), b.conserved())


@pytest.mark.parametrize("nx1,nside,flag", [(10, 32, 1), (13, 34, 1), (12, 16, 9), (15, 14, 9)])
def test_march_shell_matches_oracle(nx1, nside, flag):
    from oracle import oracle
    p = problems.shell_c3(nx1=nx1, nside=nside, implicit_flag=flag)
    g, o = Shell(p), oracle.OracleShell(p)
    g.step(30.0)
    o.step(30.0)
    a, b = p.interior(g.conserved()), p.interior(o.conserved())
    for n in range(5):
        s = np.linalg.norm(b[:, n])
        if 1 <= n <= 3:
            s = max(s, 30.0 * 24.79 * np.linalg.norm(b[:, 0]))
        assert np.linalg.norm(a[:, n] - b[:, n]) <= (5e-11 if flag == 1 else 1e-10) * s
