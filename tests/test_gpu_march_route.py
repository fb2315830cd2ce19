"""Which blocks march down their columns (csrc/march.cuh) and what that costs and changes: scratch
that gives way to other blocks, the setting and the query, the kernel without scratch, equal bits
among blocks of one route and roundoff across."""
import ctypes

import numpy as np
import pytest

from canoe_b200 import Batch, CanoeError, Mesh, MeshBlock, Shell, problems, thermo
from canoe_b200._abi import FP32_PERTURBATION, check, load
from test_gpu_march import _perturbed, _rel

pytestmark = pytest.mark.gpu


def _p(nx1=12, nx2=72, nx3=62, **kw):
    p = problems.moist3d(nx1=nx1, nx2=nx2, nx3=nx3, x1max=250.0 * nx1, x2max=250.0 * nx2,
                         x3max=250.0 * nx3, satadj=0, **kw)
    return _perturbed(p, 21)


def _free():
    import gc
    import torch
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # what earlier tests left in torch's pool
    return torch.cuda.mem_get_info()[0]


def _ballast(nbytes):
    import torch
    return torch.empty(nbytes, dtype=torch.uint8, device="cuda")


def _drop():
    import torch
    torch.cuda.empty_cache()


def test_scratch_gives_way_to_a_block_until_the_first_step():
    MeshBlock(_p(8, 8, 8)).step(0.1)  # the library's own memory
    p = _p(60, 100, 100)
    arrays = 4 * p.u.nbytes  # u, w, u1, du
    scratch = 60 * 100 * 100 * 18 * 8
    f0 = _free()
    a = MeshBlock(p)
    assert f0 - _free() >= arrays + scratch
    ballast = _ballast(_free() - arrays + scratch // 2)
    b = MeshBlock(p)  # fits without a's scratch
    assert not a.marches() and not b.marches()
    del ballast
    _drop()
    a.step(0.2)
    b.step(0.2)
    assert np.array_equal(a.conserved(), b.conserved())
    a.close()
    b.close()
    assert abs(f0 - _free()) <= 16 << 20


def test_scratch_waits_for_the_first_step_where_memory_is_scarce():
    p = _p(60, 100, 100)
    a = MeshBlock(p)
    ballast = _ballast(int(0.7 * _free()))
    f0 = _free()
    b = MeshBlock(p)
    assert f0 - _free() <= 4 * p.u.nbytes + (16 << 20)
    assert b.marches()
    a.step(0.2)
    b.step(0.2)
    del ballast
    _drop()
    assert np.array_equal(a.conserved(), b.conserved())


def test_setting_and_query():
    p = _p()
    a, b, c = MeshBlock(p), MeshBlock(p), MeshBlock(p)
    b.set_march(False)
    assert a.marches() and not b.marches()
    c.step(0.2)
    for x in (a, c):
        with pytest.raises(CanoeError):
            x.set_march(False)
    a.step(0.2)
    b.step(0.2)
    assert np.array_equal(a.conserved(), c.conserved())
    # each form is held to 5e-11 of the oracle
    assert _rel(p, a.conserved(), b.conserved(), 0.2) < 1e-10
    assert not MeshBlock(_p(12, 16, 12)).marches()
    assert load().canoe_block_marches(None, ctypes.byref(ctypes.c_int())) != 0
    assert load().canoe_block_set_march(None, 1) != 0


def test_shell_setting_and_query():
    p = problems.shell_c3(nx1=10, nside=32)
    a, b = Shell(p), Shell(p)
    b.set_march(False)
    assert a.marches() and not b.marches()
    with pytest.raises(CanoeError):
        a.set_march(False)
    a.step(30.0)
    b.step(30.0)
    x, y = p.interior(a.conserved()), p.interior(b.conserved())
    for n in range(5):
        s = np.linalg.norm(y[:, n])
        if 1 <= n <= 3:  # the gravity impulse, as tests/test_gpu_march.py
            s = max(s, 30.0 * 24.79 * np.linalg.norm(y[:, 0]))
        assert np.linalg.norm(x[:, n] - y[:, n]) <= 1e-10 * s


def test_block_without_room_for_scratch():
    import torch
    p = _p()
    b = MeshBlock(p)
    b.set_march(False)
    free, total = torch.cuda.mem_get_info()
    ballast = _ballast(free - total // 32)
    a = MeshBlock(p)
    assert not a.marches()
    del ballast
    _drop()
    a.step(0.2)
    b.step(0.2)
    assert not a.marches()
    assert np.array_equal(a.conserved(), b.conserved())


def test_caller_allocated_step_has_the_bits_of_a_block_that_does_not_march():
    import torch
    p = _p(16, 72, 60)
    a, b = MeshBlock(p), MeshBlock(p)
    b.set_march(False)
    assert a.marches()
    u = torch.from_numpy(p.u).cuda()
    w = torch.empty_like(u)
    check(load().canoe_block_step_noalloc(ctypes.byref(p.cfg), u.data_ptr(), w.data_ptr(), None,
                                          0.2, None))
    torch.cuda.synchronize()
    a.step(0.2)
    b.step(0.2)
    got = p.interior(u.cpu().numpy())
    assert np.array_equal(got, p.interior(b.conserved()))
    assert _rel(p, u.cpu().numpy(), a.conserved(), 0.2) < 1e-10


@pytest.mark.parametrize("graph", [False, True])
def test_mesh_of_marching_blocks_has_the_single_blocks_bits(graph):
    p = _p(12, 96, 92)
    one, m = MeshBlock(p), Mesh(p, 2, 1, graph=graph)
    assert one.marches() and all(b.marches() for b in m.blocks)
    for _ in range(2):
        one.step()
        m.step()
    assert np.array_equal(p.interior(one.conserved()), p.interior(m.conserved()))


def test_mesh_across_the_threshold():
    p = _p(12, 72, 62)
    one, off, m = MeshBlock(p), MeshBlock(p), Mesh(p, 2, 1)
    off.set_march(False)
    assert one.marches() and not any(b.marches() for b in m.blocks)
    for _ in range(2):
        for x in (one, off, m):
            x.step(0.2)
    assert np.array_equal(p.interior(off.conserved()), p.interior(m.conserved()))
    assert _rel(p, m.conserved(), one.conserved(), 0.4) < 1e-10


def test_first_step_inside_a_callers_capture():
    import torch
    p = _p()
    a, b = MeshBlock(p), MeshBlock(p)
    a.step(0.2)
    s = torch.cuda.Stream()
    check(b.lib.canoe_block_set_stream(b.h, s.cuda_stream))
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        b.step(0.2)
    with torch.cuda.stream(s):
        g.replay()
    torch.cuda.synchronize()
    assert b.marches()
    assert np.array_equal(a.conserved(), b.conserved())


def test_autotuner_leaves_marching_blocks_alone():
    blocks = [MeshBlock(_p()), MeshBlock(_p(12, 16, 12))]
    ref = [b.conserved() for b in blocks]
    bt = Batch(blocks)
    choice = bt.autotune()
    assert choice[0] == 0 and choice[1] in (64, 96, 128, 160, 192, 256)
    assert [t for t, _ in bt.shapes()] == list(choice)
    for b, r in zip(blocks, ref):
        assert np.array_equal(b.conserved(), r)


# one tile on an SM (six species, FP64 and odd FP32 columns): rounds of 148 tiles; two: FP64 columns
# of 32 to 150 levels in more than 148 tiles
@pytest.mark.parametrize("ny,f32,nx1,nx2,nx3,marches", [
    (6, 0, 65, 69, 70, False), (6, 0, 65, 64, 74, True), (6, 0, 16, 69, 70, True),
    (6, 0, 160, 64, 100, True), (6, 1, 65, 69, 70, False), (6, 1, 64, 69, 70, True),
    (3, 0, 128, 65, 67, False), (3, 0, 128, 69, 70, True), (3, 0, 16, 65, 67, True),
    (3, 0, 160, 65, 67, True), (3, 1, 128, 58, 59, True), (3, 0, 330, 64, 100, True)])
def test_rule(ny, f32, nx1, nx2, nx3, marches):
    th = thermo.earth_water_ammonia() if ny == 6 else thermo.earth_moist()
    p = problems.moist3d(nx1=nx1, nx2=nx2, nx3=nx3, x1max=100.0 * nx1, x2max=250.0 * nx2,
                         x3max=250.0 * nx3, th=th, satadj=0)
    if f32:
        p.cfg.precision = FP32_PERTURBATION
    assert MeshBlock(p).marches() == marches
