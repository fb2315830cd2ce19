"""Performance cases of the dynamical core: the work a host model has this
library do, through its public entry points, over the range of sizes, physics
and precisions of the configurations in ``problems`` and ``bench.py``.

A case is a dict of plain values.  Its ``kind`` picks the entry point:

block    one time step of a MeshBlock (``MeshBlock.step``, CFL step computed on
         the device, replayed as a CUDA graph as the benchmark does)
batch    one step of a batch of uneven blocks (``Batch.step``)
shell    an output interval of the cubed-sphere shell: a few steps, then the
         state read into the model's pinned output buffer
satadj   the saturation adjustment of a field of cells (the C ABI operator)
mlp      inference of the warm-start network (the C ABI operator)

``exact`` restates what a pass computes in plain torch, in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

from canoe_b200 import Batch, MeshBlock, Shell, learned, problems, thermo
from canoe_b200._abi import (BC_OUTFLOW, BC_PERIODIC, BC_REFLECT, FP32_PERTURBATION, FP64, NGHOST,
                             RECON_PLM, RECON_PPM, RS_HLLC, RS_LMARS, SatOpts, check, load)

RECON = {"plm": RECON_PLM, "ppm": RECON_PPM}
RSOLVER = {"lmars": RS_LMARS, "hllc": RS_HLLC}
SHELL_DT = 60.0


def _block(name, nx1, nx2, nx3, moist, recon, rsolver, implicit, mixed, learned_start=False,
           rh=0.8):
    return dict(name=name, kind="block", nx1=nx1, nx2=nx2, nx3=nx3, moist=moist, recon=recon,
                rsolver=rsolver, implicit=implicit, mixed=mixed, learned=learned_start, rh=rh)


def listed():
    return [
        # the 2-D dry rising bubble, the smallest run a user makes: launches
        # and latency count
        _block("bubble-150x100", 150, 100, 1, False, "plm", "lmars", 0, False),
        # a 2-D moist bubble domain (the size of the moist regression run),
        # saturated so that the adjustment condenses
        _block("moist2d-200x400", 200, 400, 1, True, "ppm", "lmars", 0, False, rh=1.0),
        # a small 3-D column block, the low end of the batch's sizes
        _block("column-32x16x16", 32, 16, 16, True, "ppm", "hllc", 1, True, True),
        # the moist-convection benchmark in its fast form
        _block("moist-128x256x256", 128, 256, 256, True, "ppm", "hllc", 1, True, True),
        # the same physics in plain FP64 on a quarter of the area
        _block("moist-fp64-128x128x128", 128, 128, 128, True, "ppm", "hllc", 1, False),
        # ragged sizes, the second-order scheme
        _block("ragged-77x83x61", 77, 83, 61, True, "plm", "lmars", 1, True),
        # the full 5x5 vertical correction
        _block("full5x5-64x96x96", 64, 96, 96, True, "ppm", "hllc", 9, True),
        # a dry 3-D bubble-like block without the implicit solve, FP64
        _block("dry-explicit-100x100x100", 100, 100, 100, False, "ppm", "hllc", 0, False),
        # the giant-planet shell: five steps and an output
        dict(name="shell-64x96", kind="shell", nx1=64, nside=96, mixed=True, steps=5),
        # uneven blocks stepped together
        dict(name="batch-12", kind="batch", nblocks=12, nz0=32, nz1=160, nh0=16, nh1=96,
             mixed=True),
        # the adjustment alone on perturbed moist cells
        dict(name="satadj-4M", kind="satadj", ncells=1 << 22, ammonia=False, warm=0),
        # the network's inference alone
        dict(name="mlp-4M", kind="mlp", n=1 << 22),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["block3", "block2", "shell", "batch", "satadj", "mlp"],
                       [50, 20, 10, 8, 7, 5])[0]
    if kind == "block3":
        implicit = rng.choices([1, 0, 9], [70, 10, 20])[0]
        nx1 = _logint(rng, 32, 200)
        cells = (1.0e6 if implicit == 9 else 4.0e6) / nx1
        nx2 = _logint(rng, 16, 256)
        nx3 = max(8, min(_logint(rng, 16, 256), int(cells / nx2)))
        c = _block("", nx1, nx2, nx3, rng.random() < 0.7, rng.choice(["plm", "ppm", "ppm"]),
                   rng.choice(["lmars", "hllc", "hllc"]), implicit, rng.random() < 0.6,
                   rh=rng.choice([0.8, 1.0]))
        c["learned"] = c["moist"] and c["mixed"] and rng.random() < 0.5
    elif kind == "block2":
        c = _block("", _logint(rng, 48, 400), _logint(rng, 48, 600), 1, rng.random() < 0.4,
                   rng.choice(["plm", "ppm"]), "lmars", rng.choice([0, 0, 1]),
                   rng.random() < 0.3, rh=rng.choice([0.8, 1.0]))
    elif kind == "shell":
        c = dict(kind="shell", nx1=_logint(rng, 24, 80), nside=2 * _logint(rng, 12, 48),
                 mixed=rng.random() < 0.6, steps=rng.randint(3, 6))
    elif kind == "batch":
        c = dict(kind="batch", nblocks=rng.randint(4, 16), nz0=32, nz1=rng.randint(64, 160),
                 nh0=16, nh1=rng.randint(32, 96), mixed=rng.random() < 0.7)
    elif kind == "satadj":
        c = dict(kind="satadj", ncells=_logint(rng, 1 << 16, 1 << 23), ammonia=rng.random() < 0.3,
                 warm=rng.choice([0, 0, 2]))
    else:
        c = dict(kind="mlp", n=_logint(rng, 1 << 16, 1 << 24))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs

def _problem(case, seed):
    """The block's configuration and seeded initial state."""
    rng = np.random.Generator(np.random.PCG64(seed))
    nx1, nx2, nx3 = case["nx1"], case["nx2"], case["nx3"]
    if nx3 == 1 and not case["moist"]:
        # the bubble at a seeded place, at the 10 m spacing of its run
        p = problems.bubble2d(nx1=nx1, nx2=nx2, x1max=10.0 * nx1, x2max=10.0 * nx2,
                              dT=rng.uniform(0.4, 0.6), xc=10.0 * nx2 * rng.uniform(0.4, 0.6),
                              zc=260.0, recon=RECON[case["recon"]],
                              rsolver=RSOLVER[case["rsolver"]])
        p.cfg.implicit_flag = case["implicit"]
    else:
        dx = 250.0
        th = thermo.earth_moist() if case["moist"] else thermo.dry()
        p = problems.moist3d(nx1=nx1, nx2=nx2, nx3=nx3, x2max=dx * nx2, x3max=dx * nx3,
                             seed=seed, implicit_flag=case["implicit"],
                             recon=RECON[case["recon"]], rsolver=RSOLVER[case["rsolver"]],
                             satadj=1 if case["moist"] else 0, th=th, rh=case["rh"])
        # without the implicit solve sound also limits the vertical direction
        p.cfg.cfl = 0.4 if case["implicit"] else 0.3
    p.cfg.precision = FP32_PERTURBATION if case["mixed"] else FP64
    return p


def _batch_problems(case, seed):
    ps = problems.batch_c5(case["nblocks"], seed=20240605, nz=(case["nz0"], case["nz1"]),
                           nh=(case["nh0"], case["nh1"]))
    for b, p in enumerate(ps):  # sizes are the case's, the noise the seed's
        c = p.cfg
        q = problems.moist3d(nx1=c.nx1, nx2=c.nx2, nx3=c.nx3, x2max=c.dx2 * c.nx2,
                             x3max=c.dx3 * c.nx3, seed=seed * 131 + b)
        p.u, p.w = q.u, q.w
        c.precision = FP32_PERTURBATION if case["mixed"] else FP64
    return ps


def _shell_problem(case, seed):
    p = problems.shell_c3(nx1=case["nx1"], nside=case["nside"], seed=seed)
    p.cfg.precision = FP32_PERTURBATION if case["mixed"] else FP64
    return p


def _satadj_cells(case, seed):
    th = thermo.earth_water_ammonia() if case["ammonia"] else thermo.earth_moist()
    return th, learned.perturbed_states(th, case["ncells"], seed)


def _mlp_inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.randn(case["n"], 4, device="cuda", dtype=torch.float32, generator=gen)


class _View:
    """A device array of the block, for torch.as_tensor; the tensor holds this
    object, and so the block that owns the memory."""

    def __init__(self, blk, ptr, shape):
        self.owner = blk
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f8", data=(ptr, False),
                                             version=3, strides=None)


def _device_state(blk):
    return [torch.as_tensor(_View(blk, p, blk.shape), device="cuda") for p in blk.device_ptrs()]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "block":
        blk = MeshBlock(_problem(case, seed), graph=True)
        if case["learned"]:
            blk.set_mlp(learned.default_net())
        return dict(kind=kind, blk=blk, out=_device_state(blk))
    if kind == "batch":
        net = learned.default_net() if case["mixed"] else None
        blocks = [MeshBlock(p) for p in _batch_problems(case, seed)]
        for b in blocks:
            b.set_mlp(net)
        return dict(kind=kind, batch=Batch(blocks), blocks=blocks,
                    out=[_device_state(b) for b in blocks])
    if kind == "shell":
        sh = Shell(_shell_problem(case, seed))
        return dict(kind=kind, shell=sh, steps=case["steps"],
                    out=torch.zeros(sh.shape, dtype=torch.float64, pin_memory=True))
    if kind == "satadj":
        th, u = _satadj_cells(case, seed)
        src = torch.from_numpy(u).cuda()
        return dict(kind=kind, lib=load(), th=th, opts=SatOpts(1e-8, 30, case["warm"]), src=src,
                    u=torch.empty_like(src),
                    t=torch.empty(case["ncells"], dtype=torch.float64, device="cuda"),
                    net=learned.default_net() if case["warm"] else None)
    x = _mlp_inputs(case, seed)
    return dict(kind=kind, lib=load(), net=learned.default_net(), x=x,
                y=torch.empty(case["n"], dtype=torch.float32, device="cuda"))


# ---------------------------------------------------------------------------
# one pass

def run(s):
    kind = s["kind"]
    if kind == "block":
        s["blk"].step()
        return s["out"]
    if kind == "batch":
        s["batch"].step()
        return s["out"]
    if kind == "shell":
        sh = s["shell"]
        for _ in range(s["steps"]):
            sh.step(SHELL_DT)
        check(sh.lib.canoe_shell_get_conserved(sh.h, s["out"].data_ptr()), "get_conserved")
        return s["out"]
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "satadj":
        # the dynamics hand the adjustment a new state every step
        s["u"].copy_(s["src"])
        n = s["u"].shape[1]
        if s["net"] is None:
            check(s["lib"].canoe_saturation_adjust(
                ctypes.byref(s["th"]), ctypes.byref(s["opts"]), s["u"].data_ptr(), n, None,
                s["t"].data_ptr(), None, None, st), "saturation_adjust")
        else:
            check(s["lib"].canoe_saturation_adjust_learned(
                ctypes.byref(s["th"]), ctypes.byref(s["opts"]), s["net"].h, s["u"].data_ptr(), n,
                s["t"].data_ptr(), None, None, None, st), "saturation_adjust_learned")
        return s["u"], s["t"]
    check(s["lib"].canoe_mlp_forward(s["net"].h, s["x"].data_ptr(), s["y"].data_ptr(),
                                     s["y"].numel(), 1, st), "mlp_forward")
    return s["y"]


def _block_work(nx1, nx2, nx3, ny, implicit):
    nv, cells = 5 + ny, nx1 * nx2 * nx3
    dims = 1 + (nx2 > 1) + (nx3 > 1)
    # a stage: reconstruction and Riemann problem per direction, the update,
    # the block rows and their elimination (multiply-adds of 3x3 / 5x5
    # blocks), cons -> prim
    solve = {0: 0, 1: 700, 9: 2600}[implicit]
    flops = 3 * cells * (dims * (30 * nv + 170) + 12 * nv + solve)
    # the conserved state read and written, the primitive state written
    return cells * nv * 8 * 3, flops


def work(case):
    kind = case["kind"]
    if kind == "block":
        b, f = _block_work(case["nx1"], case["nx2"], case["nx3"], 3 if case["moist"] else 0,
                           case["implicit"])
        return {"bytes": b, "flops": f}
    if kind == "batch":
        rng = np.random.Generator(np.random.PCG64(20240605))
        b = f = 0
        for _ in range(case["nblocks"]):  # the sizes problems.batch_c5 draws
            n1 = int(round(math.exp(rng.uniform(math.log(case["nz0"]), math.log(case["nz1"])))))
            n2 = int(round(math.exp(rng.uniform(math.log(case["nh0"]), math.log(case["nh1"])))))
            x, y = _block_work(n1, n2, n2, 3, 1)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    if kind == "shell":
        b, f = _block_work(case["nx1"], case["nside"], 6 * case["nside"], 0, 1)
        return {"bytes": case["steps"] * b, "flops": case["steps"] * f}
    if kind == "satadj":
        nv = 11 if case["ammonia"] else 8
        # the cells in and out (and the copy that hands them over), T out
        return {"bytes": case["ncells"] * 8 * (4 * nv + 1), "flops": case["ncells"] * 400}
    return {"bytes": case["n"] * 20, "flops": case["n"] * 2 * (4 * 64 + 64 * 64 + 64)}


# ---------------------------------------------------------------------------
# exact: the pass in plain torch, in 64 bits

class _Thermo:
    """Mixture relations of canoe_thermo_t on (NV, ...) tensors."""

    def __init__(self, th):
        self.ny, self.nvap = th.ny, th.nvapor
        self.rd, self.gammad, self.grav = th.rd, th.gammad, th.grav
        self.cvr = [th.cv_ratio_m1[n] for n in range(th.ny)]
        self.imr = [th.inv_mu_ratio_m1[n] for n in range(th.ny)]
        self.u0 = [th.u0[n] for n in range(th.ny)]
        self.fam = [dict(vap=1 + v, liq=th.liq_slot[v], ice=th.ice_slot[v], t3=th.t3[v],
                         p3=th.p3[v], beta=(th.beta_l[v], th.beta_s[v]),
                         delta=(th.delta_l[v], th.delta_s[v])) for v in range(th.nvapor)]
        self.ivx, self.ipr, self.nv = 1 + th.ny, 4 + th.ny, 5 + th.ny

    def gamma(self, w):
        fsig = torch.ones_like(w[0])
        feps = torch.ones_like(w[0])
        for n in range(1, self.ny + 1):
            fsig = fsig + w[n] * self.cvr[n - 1]
            feps = feps + w[n] * self.imr[n - 1] if n <= self.nvap else feps - w[n]
        return 1.0 + (self.gammad - 1.0) * feps / fsig

    def prim(self, u):
        w = torch.empty_like(u)
        rho = u[:1 + self.ny].sum(0)
        w[0] = rho
        w[1:self.ipr] = u[1:self.ipr] / rho
        ke = 0.5 * (u[self.ivx:self.ipr] * w[self.ivx:self.ipr]).sum(0)
        lat = sum((u[n] * self.u0[n - 1] for n in range(self.nvap + 1, self.ny + 1)),
                  torch.zeros_like(rho))
        w[self.ipr] = (self.gamma(w) - 1.0) * (u[self.ipr] - ke - lat)
        return w

    def sound(self, w):
        return torch.sqrt(self.gamma(w) * w[self.ipr] / w[0])


def _ppm(q):
    """Face values (lower, upper) of the cells 2 .. n-3 along the last axis."""
    a, b = q[..., 1:-1] - q[..., :-2], q[..., 2:] - q[..., 1:-1]
    c = 0.5 * (q[..., 2:] - q[..., :-2])
    s = torch.minimum(c.abs(), 2.0 * torch.minimum(a.abs(), b.abs()))
    s = torch.where(a * b > 0.0, torch.copysign(s, c), torch.zeros_like(c))  # cells 1 .. n-2
    m = q[..., 1:-1]
    f = 0.5 * (m[..., :-1] + m[..., 1:]) - (s[..., 1:] - s[..., :-1]) / 6.0  # above cells 1 .. n-3
    q0, lo, hi = q[..., 2:-2], f[..., :-1], f[..., 1:]
    d, m6 = hi - lo, 6.0 * (q0 - 0.5 * (lo + hi))
    flat = (hi - q0) * (q0 - lo) <= 0.0
    lo2 = torch.where(d * m6 > d * d, 3.0 * q0 - 2.0 * hi, lo)
    hi2 = torch.where((-d * d > d * m6) & ~(d * m6 > d * d), 3.0 * q0 - 2.0 * lo, hi)
    return torch.where(flat, q0, lo2), torch.where(flat, q0, hi2)


def _plm(q):
    """As _ppm with van Leer's slope, uniform spacing."""
    a, b = q[..., 2:-2] - q[..., 1:-3], q[..., 3:-1] - q[..., 2:-2]
    p = a * b
    s = torch.where(p > 0.0, p / torch.where(p > 0.0, a + b, torch.ones_like(a)), torch.zeros_like(a))
    return q[..., 2:-2] - s, q[..., 2:-2] + s


def _riemann(T, solver, d, wl, wr):
    """Fluxes of the faces between states wl and wr along direction d."""
    vx = T.ivx + d
    tr = [T.ivx + (d + 1) % 3, T.ivx + (d + 2) % 3]
    pl, pr, rl, rr = wl[T.ipr], wr[T.ipr], wl[0], wr[0]
    ul, ur = wl[vx], wr[vx]
    gl, gr = T.gamma(wl), T.gamma(wr)
    kl, kr = 1.0 / (gl - 1.0), 1.0 / (gr - 1.0)
    kel = 0.5 * (wl[T.ivx:T.ipr] ** 2).sum(0)
    ker = 0.5 * (wr[T.ivx:T.ipr] ** 2).sum(0)
    dl = 1.0 - wl[1:1 + T.ny].sum(0)
    dr = 1.0 - wr[1:1 + T.ny].sum(0)
    f = torch.empty_like(wl)
    if solver == RS_LMARS:
        hl, hr = pl / rl * (kl + 1.0) + kel, pr / rr * (kr + 1.0) + ker
        rb = 0.5 * (rl + rr)
        cb = torch.sqrt(0.5 * (1.0 + 0.5 * (1.0 / kr + 1.0 / kl)) * (pl + pr) / rb)
        pb = 0.5 * (pl + pr) + 0.5 * rb * cb * (ul - ur)
        ub = 0.5 * (ul + ur) + 0.5 / (rb * cb) * (pl - pr)
        up = ub > 0.0
        m = ub * torch.where(up, rl, rr)
        f[0] = m * torch.where(up, dl, dr)
        for n in list(range(1, T.ny + 1)) + tr + [vx]:
            f[n] = m * torch.where(up, wl[n], wr[n])
        f[vx] += pb
        f[T.ipr] = m * torch.where(up, hl, hr)
        return f
    cl, cr = torch.sqrt(gl * pl / rl), torch.sqrt(gr * pr / rr)
    el, er = pl * kl + rl * kel, pr * kr + rr * ker
    pm = 0.5 * (pl + pr + (ul - ur) * 0.5 * (rl + rr) * 0.5 * (cl + cr))
    one = torch.ones_like(pm)
    ql = torch.where(pm <= pl, one, torch.sqrt(
        (1.0 + (gl + 1.0) / (2.0 * gl) * (pm / pl - 1.0)).clamp_min(0.0)))
    qr = torch.where(pm <= pr, one, torch.sqrt(
        (1.0 + (gr + 1.0) / (2.0 * gr) * (pm / pr - 1.0)).clamp_min(0.0)))
    al, ar = ul - cl * ql, ur + cr * qr
    bp, bm = ar.clamp_min(1.0e-20), al.clamp_max(-1.0e-20)
    tl, tr_ = pl + (ul - al) * rl * ul, pr + (ur - ar) * rr * ur
    ml, mr = rl * (ul - al), -rr * (ur - ar)
    am = (tl - tr_) / (ml + mr)
    cp = ((ml * tr_ + mr * tl) / (ml + mr)).clamp_min(0.0)
    xl, xr = ul - bm, ur - bp
    pos = am >= 0.0
    zero = torch.zeros_like(am)
    sl = torch.where(pos, am / (am - bm), zero)
    sr = torch.where(pos, zero, -am / (bp - am))
    sm = torch.where(pos, -bm / (am - bm), bp / (bp - am))
    f[0] = sl * rl * xl * dl + sr * rr * xr * dr
    for n in list(range(1, T.ny + 1)) + tr + [vx]:
        f[n] = sl * rl * wl[n] * xl + sr * rr * wr[n] * xr
    f[vx] += sl * pl + sr * pr + sm * cp
    f[T.ipr] = sl * (el * xl + pl * ul) + sr * (er * xr + pr * ur) + sm * cp * am
    return f


class _Exact:
    """One block: configuration, geometry and the state (NV, k, j, i)."""

    def __init__(self, p):
        c = self.c = p.cfg
        self.T = _Thermo(c.thermo)
        self.n = (c.nx1, c.nx2, c.nx3)
        g = NGHOST
        self.own = (slice(None),) + tuple(
            slice(g, g + m) if m > 1 else slice(0, 1) for m in (c.nx3, c.nx2)) + (slice(g, g + c.nx1),)
        self.u = torch.from_numpy(p.u).cuda()
        f = np.asarray(p.x1f)
        dx = np.diff(f)
        self.dx1 = torch.from_numpy(np.concatenate([dx[g - 1::-1], dx, dx[:-g - 1:-1]])).cuda()
        self.h = (None, c.dx2, c.dx3)
        self.fill()

    def fill(self):
        """cons -> prim with the physical boundaries."""
        T, w = self.T, self.T.prim(self.u[self.own])
        for d in range(3):
            m, axis = self.n[d], 3 - d
            if d > 0 and m == 1:
                continue
            i = torch.arange(-NGHOST, m + NGHOST, device=w.device)
            flip = torch.zeros_like(i, dtype=torch.bool)
            for side, out in ((2 * d, i < 0), (2 * d + 1, i >= m)):
                bc = self.c.bc[side]
                if bc == BC_REFLECT:
                    i = torch.where(out, (-1 - i) if side % 2 == 0 else (2 * m - 1 - i), i)
                    flip |= out
                elif bc == BC_PERIODIC:
                    i = torch.where(out, i % m, i)
                else:
                    i = torch.where(out, i.clamp(0, m - 1), i)
            w = w.index_select(axis, i)
            v = w[T.ivx + d].movedim(axis - 1, -1)
            v[..., flip] = -v[..., flip]
        self.w = w

    def new_dt(self):
        T, c, w = self.T, self.c, self.w[self.own]
        cs = T.sound(w)
        best = math.inf
        for d in range(3):
            if d > 0 and self.n[d] == 1:
                continue
            dx = self.dx1[NGHOST:-NGHOST] if d == 0 else self.h[d]
            v = w[T.ivx + d].abs()
            imp = c.implicit_flag >> d & 1 and (d > 0 or self.n[1] > 1)
            best = min(best, float((dx / (c.cfl * v if imp else v + cs)).min()))
        return c.cfl * best

    def faces(self, q):
        """(left, right) states of the interior faces along the last axis of q,
        which holds NGHOST ghost cells at both ends."""
        lo, hi = (_ppm if self.c.recon == RECON_PPM else _plm)(q[..., 0:])
        # cells 2 .. n-3: the first ghost layer to the last
        return hi[..., :-1], lo[..., 1:]

    def div(self, d):
        """Flux divergence along direction d over the interior."""
        T, axis = self.T, 3 - d
        sl = list(self.own)
        sl[axis] = slice(None)
        q = self.w[tuple(sl)].movedim(axis, -1)
        wl, wr = self.faces(q)
        f = _riemann(T, self.c.rsolver, d, wl, wr)
        return ((f[..., 1:] - f[..., :-1]) / self.h[d]).movedim(-1, axis)

    def div1(self):
        """The vertical divergence through the hydrostatic decomposition."""
        T, c, g = self.T, self.c, NGHOST
        sl = list(self.own)
        sl[3] = slice(None)
        w = self.w[tuple(sl)]
        rho, p, dx, n = w[0], w[T.ipr], self.dx1, c.nx1
        grav, ie = T.grav, NGHOST + n - 1
        if grav == 0.0:
            wl, wr = self.faces(w)
            f = _riemann(T, c.rsolver, 0, wl, wr)
            return (f[..., 1:] - f[..., :-1]) / dx[g:-g]
        psf = torch.empty(rho.shape[:-1] + (n + 2 * g + 1,), dtype=rho.dtype, device=rho.device)
        psf[..., ie + 1] = p[..., ie] * torch.exp(grav * dx[ie] / (2.0 * p[..., ie] / rho[..., ie]))
        for i in range(ie, -1, -1):
            gi = -grav if i < g and c.bc[0] == BC_REFLECT else grav
            psf[..., i] = psf[..., i + 1] - gi * rho[..., i] * dx[i]
        gt = -grav if c.bc[1] == BC_REFLECT else grav
        for i in range(ie + 1, n + 2 * g):
            psf[..., i + 1] = psf[..., i] + gt * rho[..., i] * dx[i]
        a, b = psf[..., :-1], psf[..., 1:]
        near = (a - b).abs() < 1.0e-6
        psv = torch.where(near, 0.5 * (a + b), (a - b) / torch.log(torch.where(near, 2.0 * b, a) / b))
        feps = torch.ones_like(rho)
        for m in range(1, T.nvap + 1):
            feps = feps + w[m] * T.imr[m - 1]
        rov = T.rd * feps
        q = w.clone()
        q[0] = p / (rho * rov)
        q[T.ipr] = p - psv
        for m in (0, T.ipr):
            if c.bc[0] == BC_OUTFLOW:
                q[m][..., :g] = q[m][..., g:g + 1]
            if c.bc[1] == BC_OUTFLOW:
                q[m][..., ie + 1:] = q[m][..., ie:ie + 1]
        wl, wr = (x.clone() for x in self.faces(q))
        pf = psf[..., g:ie + 2]
        r = torch.sqrt(rov[..., g:ie + 2] * rov[..., g - 1:ie + 1])
        for x in (wl, wr):
            t = x[T.ipr] + pf
            x[T.ipr] = torch.where(t < 0.0, pf, t)
            x[0] = x[T.ipr] / (x[0] * r)
        f = _riemann(T, c.rsolver, 0, wl, wr)
        return (f[..., 1:] - f[..., :-1]) / dx[g:-g]

    def roe(self, N, wl, wr):
        """|A| between cell states wl and wr, (..., N, N)."""
        T = self.T
        gm1 = T.gammad - 1.0
        sl, sr = torch.sqrt(wl[0]), torch.sqrt(wr[0])
        m = (sl * wl + sr * wr) / (sl + sr)
        m[0] = sl * sr
        e = [x[T.ipr] / gm1 + 0.5 * x[0] * (x[T.ivx:T.ipr] ** 2).sum(0) for x in (wl, wr)]
        hb = ((e[0] + wl[T.ipr]) / sl + (e[1] + wr[T.ipr]) / sr) / (sl + sr)
        u, v, w = m[T.ivx], m[T.ivx + 1], m[T.ivx + 2]
        ke = 0.5 * (u * u + v * v + w * w)
        m[T.ipr] = (hb - ke) * gm1 / (gm1 + 1.0) * m[0]
        cs = T.sound(m)
        hp = (gm1 + 1.0) / gm1 * m[T.ipr] / m[0]
        h, o, z = hp + ke, torch.ones_like(u), torch.zeros_like(u)
        R = [[o, o, o, z, z], [u - cs, u, u + cs, z, z], [v, v, v, o, z], [w, w, w, z, o],
             [h - u * cs, ke, h + u * cs, v, w]]
        Ri = [[(cs * ke + u * hp) / (2 * cs * hp), (-hp - cs * u) / (2 * cs * hp), -v / (2 * hp),
               -w / (2 * hp), o / (2 * hp)],
              [(hp - ke) / hp, u / hp, v / hp, w / hp, -o / hp],
              [(cs * ke - u * hp) / (2 * cs * hp), (hp - cs * u) / (2 * cs * hp), -v / (2 * hp),
               -w / (2 * hp), o / (2 * hp)],
              [-v, z, o, z, z], [-w, z, z, o, z]]
        lam = [(u - cs).abs(), u.abs(), (u + cs).abs(), u.abs(), u.abs()]
        pick = (0, 1, 4) if N == 3 else range(5)
        return torch.stack([torch.stack([sum(R[a][k] * lam[k] * Ri[k][b] for k in range(5))
                                         for b in pick], -1) for a in pick], -2)

    def jac(self, N, x):
        T = self.T
        gm1 = T.gammad - 1.0
        a, b, c = x[T.ivx], x[T.ivx + 1], x[T.ivx + 2]
        s2, t = a * a + b * b + c * c, (gm1 + 1.0) / gm1 * x[T.ipr] / x[0]
        o, z = torch.ones_like(a), torch.zeros_like(a)
        J = [[z, o, z, z, z], [gm1 * s2 / 2 - a * a, (2 - gm1) * a, -gm1 * b, -gm1 * c, gm1 * o],
             [-a * b, b, a, z, z], [-a * c, c, z, a, z],
             [((gm1 - 1) * s2 / 2 - t) * a, t + s2 / 2 - gm1 * a * a, -gm1 * b * a, -gm1 * c * a,
              (gm1 + 1) * a]]
        pick = (0, 1, 4) if N == 3 else range(5)
        return torch.stack([torch.stack([J[r][k] for k in pick], -1) for r in pick], -2)

    def solve(self, du, dt):
        """The implicit x1 correction of du (interior), in place."""
        T, c, g = self.T, self.c, NGHOST
        N = 5 if c.implicit_flag & 8 else 3
        sl = list(self.own)
        sl[3] = slice(None)
        w = self.w[tuple(sl)]
        A = self.roe(N, w[..., g - 1:-g], w[..., g:w.shape[-1] - g + 1])
        J = self.jac(N, w[..., g - 1:w.shape[-1] - g + 1])
        n, eye = c.nx1, torch.eye(N, dtype=w.dtype, device=w.device)
        Phi = torch.zeros_like(eye)
        Phi[1, 0] = Phi[N - 1, 1] = T.grav
        flip = torch.ones(N, dtype=w.dtype, device=w.device)
        flip[1] = -1.0
        idx = [T.ivx, T.ipr] if N == 3 else [T.ivx, T.ivx + 1, T.ivx + 2, T.ipr]
        rhs = torch.stack([du[:1 + T.ny].sum(0)] + [du[m] for m in idx], -1) / dt
        D = [None] * n
        G = [None] * n
        for i in range(n):
            hh = 0.5 / self.dx1[g + i]
            a = (A[..., i, :, :] + A[..., i + 1, :, :]) * hh + eye / dt - Phi
            b = -(A[..., i, :, :] + J[..., i, :, :]) * hh
            cc = -(A[..., i + 1, :, :] - J[..., i + 2, :, :]) * hh
            r = rhs[..., i, :]
            if i == 0:
                a = a + b * flip
            else:
                a = a - b @ D[i - 1]
                r = r - (b @ G[i - 1][..., None])[..., 0]
            if i == n - 1:
                a = a + cc * flip
            x = torch.linalg.solve(a, torch.cat([cc, r[..., None]], -1))
            D[i], G[i] = x[..., :N], x[..., N]
        for i in range(n - 2, -1, -1):
            G[i] = G[i] - (D[i] @ G[i + 1][..., None])[..., 0]
        x = torch.stack(G, -1).movedim(-2, 0)
        dens = x[0] - du[:1 + T.ny].sum(0)
        for m in range(1, T.ny + 1):
            du[m] += dens * w[m][..., g:-g]
        for m, q in enumerate(idx):
            du[q] = x[1 + m]
        du[0] = x[0] - du[1:1 + T.ny].sum(0)

    def step(self):
        T, c, dt = self.T, self.c, self.new_dt()
        u1 = self.u[self.own].clone()
        for g1, g2, beta in ((0.0, 1.0, 1.0), (0.25, 0.75, 0.25), (2.0 / 3.0, 1.0 / 3.0, 2.0 / 3.0)):
            h = beta * dt
            w = self.w[self.own]
            du = -h * self.div1()
            for d in (1, 2):
                if self.n[d] > 1:
                    du -= h * self.div(d)
            src = h * w[0] * T.grav
            du[T.ivx] += src
            du[T.ipr] += src * w[T.ivx]
            if c.implicit_flag & 1:
                self.solve(du, h)
            self.u[self.own] = g1 * self.u[self.own] + g2 * u1 + du
            if beta == 2.0 / 3.0 and c.satadj:
                self.u[self.own] = _saturate(T, self.u[self.own])[0]
            self.fill()
        return [self.u, self.w]


def _saturate(T, u):
    """Saturation adjustment of conserved cells (NV, ...): (u, T)."""
    cvd = T.rd / (T.gammad - 1.0)
    rho = u[:1 + T.ny].sum(0)
    ie = u[T.ipr] - 0.5 * (u[T.ivx:T.ipr] ** 2).sum(0) / rho
    q = u[1:1 + T.ny] / rho
    qd = 1.0 - q.sum(0)
    tot = [sum(q[f[s] - 1] for s in ("vap", "liq", "ice") if f[s] > 0) for f in T.fam]

    def state(t, force=None):
        """energy residual, its slope and the mass fractions at t"""
        out = torch.zeros_like(q)
        cvs, lat, dlat = qd.clone(), torch.zeros_like(t), torch.zeros_like(t)
        for f, qt in zip(T.fam, tot):
            liq = t >= f["t3"] if force is None or force[0] is not f else torch.full_like(t, force[1], dtype=torch.bool)
            if f["ice"] < 0:
                liq = torch.ones_like(liq)
            cv = [1.0 + T.cvr[f[s] - 1] for s in ("vap", "liq", "ice")]
            beta = torch.where(liq, *(x * torch.ones_like(t) for x in f["beta"]))
            delta = torch.where(liq, *(x * torch.ones_like(t) for x in f["delta"]))
            rv = T.rd * (1.0 + T.imr[f["vap"] - 1])
            qs = f["p3"] * torch.exp(beta * (1.0 - f["t3"] / t) - delta * torch.log(t / f["t3"])) / (rho * rv * t)
            wet = qs < qt
            qv = torch.where(wet, qs, qt)
            qc = qt - qv
            dq = torch.where(wet, qs * (beta * f["t3"] / (t * t) - (delta + 1.0) / t), torch.zeros_like(t))
            cvc = torch.where(liq, cv[1], cv[2])
            uc = torch.where(liq, T.u0[f["liq"] - 1], T.u0[f["ice"] - 1])
            out[f["vap"] - 1] = qv
            out[f["liq"] - 1] = torch.where(liq, qc, torch.zeros_like(qc))
            if f["ice"] > 0:
                out[f["ice"] - 1] = torch.where(liq, torch.zeros_like(qc), qc)
            cvs = cvs + qv * cv[0] + qc * cvc
            lat = lat + qc * uc
            dlat = dlat + dq * (cvd * (cv[0] - cvc) * t - uc)
        return rho * (cvd * cvs * t + lat) - ie, rho * (cvd * cvs + dlat), out

    lo, hi = torch.full_like(rho, 20.0), torch.full_like(rho, 2000.0)
    for _ in range(60):
        t = 0.5 * (lo + hi)
        up = state(t)[0] > 0.0
        lo, hi = torch.where(up, lo, t), torch.where(up, t, hi)
    t = 0.5 * (lo + hi)
    for _ in range(2):
        f, fp, _ = state(t)
        n = t - f / fp
        t = torch.where((n - t).abs() < 1.0e-9, n, t)
    out = state(t)[2]
    for fam in T.fam:  # a root on the liquid / ice jump: both phases at t3
        if fam["ice"] < 0:
            continue
        t3 = torch.full_like(t, fam["t3"])
        fl, _, ql = state(t3, (fam, True))
        fs = state(t3, (fam, False))[0]
        on = ((t - t3).abs() < 1.0e-3) & ((fl > 0.0) != (fs > 0.0))
        x = -fs / torch.where(on, fl - fs, torch.ones_like(fl))
        qc = ql[fam["liq"] - 1].clone()
        ql[fam["liq"] - 1] = x * qc
        ql[fam["ice"] - 1] = qc - x * qc
        out, t = torch.where(on, ql, out), torch.where(on, t3, t)
    v = u.clone()
    v[1:1 + T.ny] = out * rho
    return v, t


def exact(case, seed):
    kind = case["kind"]
    if kind == "block":
        return _Exact(_problem(case, seed)).step()
    if kind == "batch":
        return [_Exact(p).step() for p in _batch_problems(case, seed)]
    if kind == "shell":
        return None  # the panels' exchange and metric have no short restatement
    if kind == "satadj":
        th, u = _satadj_cells(case, seed)
        return _saturate(_Thermo(th), torch.from_numpy(u).cuda())
    p = torch.from_numpy(learned.default_net().params()).cuda().double()
    w1, b1, w2, b2, w3, b3 = torch.split(p, [256, 64, 4096, 64, 64, 1])
    x = _mlp_inputs(case, seed).double()
    y = torch.empty(len(x), dtype=torch.float64, device="cuda")
    for i in range(0, len(x), 1 << 20):
        h = torch.tanh(x[i:i + (1 << 20)] @ w1.view(64, 4).T + b1)
        y[i:i + (1 << 20)] = torch.tanh(h @ w2.view(64, 64).T + b2) @ w3 + b3
    return y
