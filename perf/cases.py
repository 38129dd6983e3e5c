"""The work that programs built on drnum_b200 have it do, as timed cases.

One pass advances a flow by a number of Runge-Kutta steps and reads the state
back into pinned host memory, as an application does between two outputs.
The kinds:

    box      one periodic patch, a vortex and a density pulse on a uniform stream
    channel  one patch with patch-face fluxes: a prescribed inflow and far field
             in x, slip walls in y, z periodic or slip walls, optionally with
             inactive cells
    jet      the eight-patch dual-resolution jet (drnum_b200.workloads)
    sphere   the two-patch level-set sphere wall, by dn_rk_step or, "staged",
             by the stage-by-stage sequence with the wall as a post-operation
             and the output-step diagnostics
    tiled    the uneven grid of many small patches
    stream   a periodic patch whose state comes from the host before the step and
             goes back after it (a coupled program)

precision 32 is the FP32 bulk path (fixed-point storage), 64 the FP64 path.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from drnum_b200 import _lib, cases, workloads
from drnum_b200.api import (AusmPlus, B200CartesianIterator, B200LevelSetObjectBC, CartesianPatch, Roe, RungeKutta,
                            VanLeer)

ALPHAS = (0.25, 0.5, 1.0)
OPS = {"ausm": AusmPlus, "vanleer": VanLeer, "roe": Roe}


def listed():
    return [
        # the headline configuration of bench.py: production runs of one large patch, tuned and graph-replayed
        dict(name="box32_256", kind="box", ni=256, nj=256, nk=256, precision=32, scheme="ausm", steps=32, tuned=True),
        # the smallest calls: a small patch stepped with the defaults, where launches and short CTAs count
        dict(name="box32_32", kind="box", ni=32, nj=32, nk=32, precision=32, scheme="ausm", steps=100, tuned=False),
        # ordinary single patch of odd extents with patch faces and inactive cells, defaults
        dict(name="channel32_odd", kind="channel", ni=125, nj=67, nk=93, precision=32, scheme="ausm", steps=40,
             tuned=False, zper=False, mask=True),
        # multi-patch production workloads of bench.py, tuned and graph-replayed
        dict(name="jet32_full", kind="jet", scale=1.0, precision=32, steps=20, tuned=True),
        dict(name="sphere32_full", kind="sphere", scale=1.0, precision=32, steps=30, tuned=True, staged=False),
        dict(name="tiled32_64", kind="tiled", scale=0.5, precision=32, steps=20, tuned=True),
        # coupled program: state in from the host, a step, state out, every time
        dict(name="stream32_128", kind="stream", ni=128, nj=128, nk=128, precision=32, scheme="ausm", steps=1,
             tuned=True),
        # stage-by-stage sequence with a post-operation and the output-step diagnostics
        dict(name="sphere32_staged", kind="sphere", scale=0.5, precision=32, steps=20, tuned=False, staged=True),
        # the 64^3 FP64 configuration of the parity tests
        dict(name="box64_64", kind="box", ni=64, nj=64, nk=64, precision=64, scheme="ausm", steps=20, tuned=True),
        # FP64 single patch of odd extents with patch faces and inactive cells, defaults
        dict(name="channel64_odd", kind="channel", ni=97, nj=61, nk=83, precision=64, scheme="ausm", steps=10,
             tuned=False, zper=False, mask=True),
        # FP64 multi-patch jet, tuned and graph-replayed
        dict(name="jet64_half", kind="jet", scale=0.5, precision=64, steps=8, tuned=True),
        # the jet application's flux functor (FP64 functor stage)
        dict(name="box64_vanleer", kind="box", ni=96, nj=96, nk=96, precision=64, scheme="vanleer", steps=6,
             tuned=False),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["box", "box", "channel", "channel", "jet", "sphere", "tiled", "stream"])
    precision = rng.choice([32, 32, 64])
    tuned = rng.random() < 0.5
    if kind in ("jet", "sphere", "tiled"):
        top = {"jet": 1.0, "sphere": 1.0, "tiled": 0.5}[kind] if precision == 32 else 0.5
        c = dict(kind=kind, scale=round(rng.uniform(0.25, top), 3), precision=precision, steps=rng.randint(3, 8),
                 tuned=tuned)
        if kind == "sphere":
            c["staged"] = rng.random() < 0.3
        return c
    if kind == "stream":
        n = [_log_int(rng, 24, 160) for _ in range(3)]
        return dict(kind=kind, ni=n[0], nj=n[1], nk=n[2], precision=32, scheme="ausm", steps=rng.randint(1, 3),
                    tuned=tuned)
    n = [_log_int(rng, 12, 240 if precision == 32 else 110) for _ in range(3)]
    cells = n[0] * n[1] * n[2]
    budget = 1.0e8 if precision == 32 else 6.0e6     # cells times steps
    steps = max(2, min(100, int(budget / cells)))
    c = dict(kind=kind, ni=n[0], nj=n[1], nk=n[2], precision=precision, steps=steps, tuned=tuned)
    c["scheme"] = rng.choice(["ausm", "ausm", "vanleer", "roe"]) if precision == 64 else "ausm"
    if kind == "channel":
        c["zper"] = rng.random() < 0.5
        c["mask"] = rng.random() < 0.5
    return c


# ---------------------------------------------------------------- the flows

def _flow(case, seed):
    """Patches, states, walls and time step of a case (host data):
    dict(patches, states, bcs, levelset, dt, periodic, active)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("box", "stream", "channel"):
        n = (case["ni"], case["nj"], case["nk"])
        h = 1.0 / max(n)
        L = tuple(m * h for m in n)
        mach = float(rng.uniform(0.25, 0.4))
        r = 0.15 * min(L[0], L[1])
        U = cases.vortex_pulse(*n, lengths=L, mach=mach, beta=float(rng.uniform(2.0, 4.0)), radius=r,
                               pulse_amp=float(rng.uniform(0.5e-2, 2e-2)), pulse_width=0.15 * min(L),
                               centre=tuple(float(x) * float(rng.uniform(0.4, 0.6)) for x in L))
        # a cross stream, so that every momentum component carries a signal
        p, T, u, v, w = cases.cons_to_prim(U)
        U = cases.prim_to_cons(p, T, u, v, w + 0.05 * mach * cases.A_INF * (p / cases.P_INF))
        dt = 0.4 * h / (1.8 * cases.A_INF)
        patch = dict(n=n, origin=(0.0, 0.0, 0.0), length=L, seek=(0,) * 6)
        bcs, active = {}, None
        periodic = (True, True, True)
        if kind == "channel":
            periodic = (False, False, bool(case["zper"]))
            far = (cases.BC_FARFIELD, (cases.P_INF, cases.T_INF, mach * cases.A_INF, 0.0, 0.05 * mach * cases.A_INF),
                   None)
            t = cases.jet_table(patch, mach * cases.A_INF, cases.T_INF, 0.2 * min(L[1], L[2]),
                                u_far=0.5 * mach * cases.A_INF, noise=1e-3, seed=seed)
            bcs = {0: {0: (cases.BC_INFLOW, None, t), 1: far, 2: (cases.BC_SLIP, None, None),
                       3: (cases.BC_SLIP, None, None)}}
            if not periodic[2]:
                bcs[0][4] = bcs[0][5] = (cases.BC_SLIP, None, None)
            if case["mask"]:
                x, y, z = cases.patch_centres(patch)
                d2 = (x - 0.3 * L[0]) ** 2 + (y - 0.3 * L[1]) ** 2 + (z - 0.6 * L[2]) ** 2
                active = (d2 > (0.12 * min(L)) ** 2).astype(np.uint8)
        return dict(patches=[patch], states=[U], bcs=bcs, levelset=None, dt=dt, periodic=periodic, active=active)
    w = workloads.build(kind, case["scale"])
    w["periodic"], w["active"] = (False, False, False), None
    if kind == "jet":
        mach = float(rng.uniform(0.6, 0.8))
        w["bcs"] = cases.jet_bcs(w["patches"], mach_jet=mach, radius=0.05, noise=1e-3, seed=seed)
        # a slow stream along the jet instead of fluid at rest, so that no patch is still
        w["states"] = cases.uniform_state(w["patches"], mach=float(rng.uniform(0.02, 0.05)))
    elif kind == "sphere":
        mach = float(rng.uniform(0.3, 0.5))
        w["states"] = cases.uniform_state(w["patches"], mach=mach)
        w["bcs"] = cases.outer_farfield_bcs(w["patches"], (cases.P_INF, cases.T_INF, mach * cases.A_INF, 0.0, 0.0))
    else:
        w["states"] = cases.tiled_state(w["patches"], seed=seed % 100000)
    return w


def prepare(case, seed):
    """The iterator with its patches, tables, walls and state on the device,
    the integrator, and pinned host buffers for what is read back (and, for
    a stream, for what is sent)."""
    f = _flow(case, seed)
    f32 = case["precision"] == 32
    if case["kind"] in ("box", "stream", "channel"):
        p = f["patches"][0]
        cp = CartesianPatch(*p["n"], lengths=p["length"], periodic=f["periodic"], num_fields=1)
        cp.setField(0, f["states"][0])
        for side, bc in f["bcs"].get(0, {}).items():
            cp.setBoundary(side, *bc)
        if f["active"] is not None:
            cp.active[...] = f["active"]
        it = B200CartesianIterator(OPS[case["scheme"]](), 0, _lib.DN_FP32 if f32 else _lib.DN_FP64)
        it.addPatch(cp)
        it.updateDevice(fields=(0,))
        objs = [cp]
    else:
        _, objs = workloads.make_grid(f)
        it = workloads.make_iterator(objs, _lib.DN_FP32 if f32 else _lib.DN_FP64)
    for cp in objs:      # the state lives on the device from here on
        cp.data = None
    if case["tuned"]:
        it.setOption(_lib.DN_OPT_GRAPH, 1)
        it.autotune()
    rk = RungeKutta()
    for a in ALPHAS:
        rk.addAlpha(a)
    rk.addIterator(it)
    if case.get("staged"):
        rk.addPostOperation(B200LevelSetObjectBC(it))
    dtype = torch.float32 if f32 else torch.float64
    out = [torch.empty((5,) + tuple(p["n"]), dtype=dtype).pin_memory() for p in f["patches"]]
    send = None
    if case["kind"] == "stream":
        send = torch.from_numpy(np.ascontiguousarray(f["states"][0])).to(dtype).pin_memory()
    return dict(case=case, it=it, rk=rk, dt=f["dt"], out=out, send=send)


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_float if t.dtype == torch.float32 else ctypes.c_double))


def _outputs(fields):
    """One patch: density, momentum and energy; several: each patch's state."""
    if len(fields) == 1:
        return {"density": fields[0][0], "momentum": fields[0][1:4], "energy": fields[0][4]}
    return {"patches": list(fields)}


def run(state):
    case, it = state["case"], state["it"]
    lib, ctx = it.lib, it.ctx
    if state["send"] is not None:
        _lib.check(ctx, lib.dn_patch_upload_f32_async(ctx, 0, 0, _ptr(state["send"])))
    for _ in range(case["steps"]):
        state["rk"](state["dt"])
    down = lib.dn_patch_download_f32_async if case["precision"] == 32 else lib.dn_patch_download_async
    for q, t in enumerate(state["out"]):
        _lib.check(ctx, down(ctx, q, 0, _ptr(t)))
    got = _outputs(state["out"])
    if case.get("staged"):
        got["sums"] = it.conservationSums()
        got["stats"] = np.array(it.flowStats(0, state["dt"]))
    it.sync()            # the host reads the buffers after this
    return got


def _cells(case):
    if case["kind"] in ("box", "stream", "channel"):
        return case["ni"] * case["nj"] * case["nk"]
    s = case["scale"]
    if case["kind"] == "tiled":
        slots = (max(2, int(round(8 * s))),) * 3
        return sum(int(np.prod(p["n"])) for p in cases.tiled_grid(slots=slots))
    if case["kind"] == "jet":
        core = tuple(max(8, int(round(x * s)) // 4 * 4) for x in (192, 96, 96))
        nx, ny = (max(12, int(round(x * s / 4)) * 4) for x in (64, 128))
        box = (2 * (nx - 3), 2 * (ny - 3), 2 * (ny - 3))
        return sum(int(np.prod(p["n"])) for p in cases.jet_grid(core=core, box=box))
    return sum(int(np.prod(p["n"])) for p in
               cases.sphere_group(n=tuple(max(16, int(round(x * s)) // 2 * 2) for x in (256, 128, 128))))


def work(case):
    """Every stage reads f(k-1) and f(n) and writes f(k) (15 words per cell;
    the first stage's f(k-1) is f(n): 10), the read-back writes 5 words; about 900
    operations per cell and stage (three faces)."""
    cells, word = _cells(case), case["precision"] // 8
    words = case["steps"] * (10 + 15 + 15) + 5 + (5 if case["kind"] == "stream" else 0)
    return {"bytes": cells * word * words, "flops": 900.0 * 3 * case["steps"] * cells}


def tolerance(case):
    # FP64: the same operations in another order; FP32 bulk: FP32 fluxes on a state
    # held to about 4e-9 of its scale, read back as float
    if case["precision"] == 64:
        return {"rel": 1e-12, "max": 1e-9}
    return {"rel": 4e-6, "max": 2e-3}


# ------------------------------------------- the same flows in 64 bits, plain torch

R, GAMMA, CV, CP = 287.2, 1.4, 717.5, 1004.5


def _limiter(d1, d2):
    e = torch.full_like(d1, 1e-10)
    r = d2 / torch.where(d1 < 0, torch.minimum(d1, -e), torch.maximum(d1, e))
    return (r * r + r) / (r * r + 1.0)


def _prim(U):
    r = U[0]
    u, v, w = U[1] / r, U[2] / r, U[3] / r
    T = (U[4] / r - 0.5 * (u * u + v * v + w * w)) / CV
    return r, u, v, w, T, r * R * T


def _split(M, s):
    inner = M.abs() < 1.0
    m1 = 0.5 * (M + s * M.abs())
    m2, m2o = 0.25 * s * (M + s) ** 2, -0.25 * s * (M - s) ** 2
    m4 = torch.where(inner, m2 * (1.0 - 2.0 * s * m2o), m1)
    p5 = torch.where(inner, m2 * ((2.0 * s - M) - 3.0 * s * M * m2o), m1 / torch.where(inner, torch.ones_like(M), M))
    return m4, p5


def _ausm(L, Rt, d, A):
    l, r = _prim(L), _prim(Rt)
    al, ar = (GAMMA * R * l[4]).sqrt(), (GAMMA * R * r[4]).sqrt()
    a = 0.5 * (al + ar)
    m4l, p5l = _split(l[1 + d] / a, 1.0)
    m4r, p5r = _split(r[1 + d] / a, -1.0)
    M = m4l + m4r
    f0 = a * A * (l[0] * M.clamp(min=0) + r[0] * M.clamp(max=0))
    up, dn = f0.clamp(min=0), f0.clamp(max=0)
    F = [f0] + [up * l[1 + q] + dn * r[1 + q] for q in range(3)]
    F[1 + d] = F[1 + d] + A * (p5l * l[5] + p5r * r[5])
    F.append(up * (L[4] + l[5]) / l[0] + dn * (Rt[4] + r[5]) / r[0])
    return torch.stack(F)


def _vanleer(L, Rt, d, A):
    F = torch.zeros_like(L)
    for U, s in ((L, 1.0), (Rt, -1.0)):
        r, u, v, w, T, p = _prim(U)
        a = (GAMMA * R * T).sqrt()
        un = (u, v, w)[d]
        M = un / a
        full = [r * un, un * U[1], un * U[2], un * U[3], un * (U[4] + p)]
        full[1 + d] = full[1 + d] + p
        f0 = s * 0.25 * a * r * (M + s) ** 2
        part = [f0, f0 * u, f0 * v, f0 * w, f0 / r * (U[4] + p)]
        part[1 + d] = f0 * (un + p / (a * r) * (-M + 2.0 * s))
        out = M * s >= 1.0
        none = M * s <= -1.0
        F = F + torch.stack([torch.where(out, x, torch.where(none, torch.zeros_like(y), y))
                             for x, y in zip(full, part)])
    return A * F


def _roe(L, Rt, d, A):
    l, r = _prim(L), _prim(Rt)
    g1 = GAMMA - 1.0
    cl, cr = l[0].sqrt(), r[0].sqrt()
    ke = [U[1] ** 2 + U[2] ** 2 + U[3] ** 2 for U in (L, Rt)]
    pl, pr = g1 * (L[4] - 0.5 * ke[0] / l[0]), g1 * (Rt[4] - 0.5 * ke[1] / r[0])
    hl = GAMMA * L[4] / l[0] - 0.5 * g1 * ke[0] / l[0] ** 2
    hr = GAMMA * Rt[4] / r[0] - 0.5 * g1 * ke[1] / r[0] ** 2
    ave = [(cl * l[1 + q] + cr * r[1 + q]) / (cl + cr) for q in range(3)]
    h = (cl * hl + cr * hr) / (cl + cr)
    un, q2 = ave[d], ave[0] ** 2 + ave[1] ** 2 + ave[2] ** 2
    c = (g1 * (h - 0.5 * q2)).clamp(min=1e-6).sqrt()
    dU = Rt - L

    def side(U, s, p):
        F = [U[1 + d]] + [U[1 + d] * s[1 + q] for q in range(3)]
        F[1 + d] = F[1 + d] + p
        return torch.stack(F + [(U[4] + p) * s[1 + d]]) * A

    def acoustic(sg):
        """The flux from one side, corrected by the acoustic wave of sign sg
        (+1: from the right side, with u + c; -1: from the left, with u - c)."""
        ll = (l[1 + d] + sg * (GAMMA * pl / l[0]).sqrt()) * A
        lr = (r[1 + d] + sg * (GAMMA * pr / r[0]).sqrt()) * A
        eig = (un + sg * c) * A
        den = torch.where(lr != ll, lr - ll, torch.ones_like(ll))
        fix = lr * (eig - ll) / den if sg > 0 else ll * (lr - eig) / den
        eig = torch.where((ll < 0) & (lr > 0), fix, eig)
        t = g1 / c
        av = [1.0 / c] + [ave[q] / c for q in range(3)] + [0.5 * q2 / c + 2.5 * c + sg * un]
        av[1 + d] = av[1 + d] + sg
        b = [0.5 * (0.5 * t * q2 - sg * un)] + [-0.5 * t * ave[q] for q in range(3)] + [0.5 * t]
        b[1 + d] = 0.5 * (sg - t * ave[d])
        eig = eig.clamp(min=0) if sg > 0 else eig.clamp(max=0)
        alpha = eig * sum(x * y for x, y in zip(b, dU))
        F = side(Rt, r, pr) if sg > 0 else side(L, l, pl)
        return F - sg * torch.stack([x * alpha for x in av])

    return torch.where(un <= 0, acoustic(1.0), acoustic(-1.0))


FLUX = {"ausm": _ausm, "vanleer": _vanleer, "roe": _roe}


def _wall(U, d, side, A, bc):
    """Flux through a patch face from its cells' states U [5][faces...]."""
    kind, params, table = bc
    r, u, v, w, T, p = _prim(U)
    vel = [u, v, w]
    if kind == cases.BC_SLIP:
        F = torch.zeros_like(U)
        F[1 + d] = A * p
        return F
    if kind == cases.BC_INFLOW:
        t = torch.as_tensor(table, device=U.device).reshape(p.shape + (5,))
        p = torch.where(torch.isnan(t[..., 0]), p, t[..., 0])
        T, vel = t[..., 1], [t[..., 2], t[..., 3], t[..., 4]]
    else:
        p0, T0, u0, v0, w0 = params
        sg = -1.0 if side % 2 else 1.0
        M = 0.5 * sg * ((u0, v0, w0)[d] / math.sqrt(GAMMA * R * T0) + vel[d] / (GAMMA * R * T).sqrt())
        into = M >= 0
        p = torch.where(M >= 1, torch.full_like(p, p0), p)
        T = torch.where(into, torch.full_like(T, T0), T)
        vel = [torch.where(into, torch.full_like(x, x0), x) for x, x0 in zip(vel, (u0, v0, w0))]
    f0 = A * p / (R * T) * vel[d]
    F = [f0] + [f0 * x for x in vel] + [f0 * (CP * T + 0.5 * sum(x * x for x in vel))]
    F[1 + d] = F[1 + d] + A * p
    return torch.stack(F)


def _residual(U, h, periodic, bcs, flux):
    res = torch.zeros_like(U)
    for d in range(3):
        n, ax = U.shape[1 + d], 1 + d
        if n <= 2:
            continue
        A = h[(d + 1) % 3] * h[(d + 2) % 3]
        if periodic[d]:
            m = lambda s: torch.roll(U, s, ax)     # noqa: E731  cell c - s
            um2, um1, u0, up1 = m(2), m(1), U, m(-1)
            d01, d12, d23 = um1 - um2, u0 - um1, up1 - u0
            L = um1 + 0.5 * _limiter(d01, d12) * d01
            Rt = u0 - 0.5 * _limiter(-d23, -d12) * d23
            F = flux(L, Rt, d, A)
            res += F - torch.roll(F, -1, ax)
            continue
        df = U.narrow(ax, 1, n - 1) - U.narrow(ax, 0, n - 1)
        L, Rt = U.narrow(ax, 0, n - 1).clone(), U.narrow(ax, 1, n - 1).clone()
        a, b = df.narrow(ax, 0, n - 2), df.narrow(ax, 1, n - 2)
        L.narrow(ax, 1, n - 2).add_(0.5 * _limiter(a, b) * a)
        Rt.narrow(ax, 0, n - 2).sub_(0.5 * _limiter(-b, -a) * b)
        F = flux(L, Rt, d, A)
        res.narrow(ax, 1, n - 1).add_(F)
        res.narrow(ax, 0, n - 1).sub_(F)
        for s in (2 * d, 2 * d + 1):
            if s in bcs and bcs[s][0] != cases.BC_ZERO:
                i = n - 1 if s % 2 else 0
                res.select(ax, i).add_(_wall(U.select(ax, i), d, s, A, bcs[s]), alpha=-1.0 if s % 2 else 1.0)
    return res


def _axis_weights(rx, dx, a, device):
    """Along axis a: the cells of patch rx whose centres lie in the donor zone
    of dx (its cells but the seek layers), their lower donor cell and weight."""
    hr, hd = rx["length"][a] / rx["n"][a], dx["length"][a] / dx["n"][a]
    first, last = dx["seek"][2 * a], dx["n"][a] - dx["seek"][2 * a + 1]
    s = (rx["origin"][a] - dx["origin"][a] + (0.5 + np.arange(rx["n"][a])) * hr) / hd
    i = np.nonzero((s >= first) & (s < last))[0]
    t = np.clip(s[i] - 0.5, first, last - 1)
    lo = np.clip(np.floor(t + 1e-9).astype(np.int64), first, last - 2)
    return (torch.as_tensor(i, device=device), torch.as_tensor(lo, device=device),
            torch.as_tensor(np.clip(t - lo, 0.0, 1.0), device=device))


def _donor_plan(patches, device):
    """Per receiving patch: the pairs (donor, axis weights), and the share of
    each seek cell's donors (0: the cell keeps its state)."""
    plan = []
    for q, r in enumerate(patches):
        seek = torch.zeros(r["n"], dtype=torch.bool, device=device)
        for a in range(3):
            lo, hi = r["seek"][2 * a], r["seek"][2 * a + 1]
            seek.narrow(a, 0, lo).fill_(True)
            seek.narrow(a, r["n"][a] - hi, hi).fill_(True)
        hits = torch.zeros(r["n"], dtype=torch.float64, device=device)
        pairs = []
        for e, d in enumerate(patches):
            if e == q:
                continue
            w = [_axis_weights(r, d, a, device) for a in range(3)]
            if all(x[0].numel() for x in w):
                box = tuple(slice(int(x[0][0]), int(x[0][-1]) + 1) for x in w)
                if bool(seek[box].any()):
                    hits[box] += 1.0
                    pairs.append((e, w, box))
        plan.append((pairs, seek & (hits > 0), hits))
    return plan


def _donor_copy(Us, plan):
    new = []
    for U, (pairs, cells, hits) in zip(Us, plan):
        got = torch.zeros_like(U)
        for e, w, box in pairs:
            V = Us[e]
            for a, (_, lo, t) in enumerate(w):
                shape = [1, 1, 1, 1]
                shape[1 + a] = -1
                t = t.reshape(shape)
                V = V.index_select(1 + a, lo) * (1.0 - t) + V.index_select(1 + a, lo + 1) * t
            got[(slice(None),) + box] += V
        new.append(torch.where(cells, got / hits.clamp(min=1.0), U))
    return new


def exact(case, seed):
    """The state after the pass in 64 bits, by plain torch.  None for the
    level-set wall: its mirror layers have no short independent form."""
    if case["kind"] == "sphere":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = _flow(case, seed)
    Us = [torch.as_tensor(np.ascontiguousarray(U), dtype=torch.float64, device=dev) for U in f["states"]]
    hs = [[p["length"][a] / p["n"][a] for a in range(3)] for p in f["patches"]]
    act = None if f["active"] is None else torch.as_tensor(f["active"], device=dev).bool()
    plan = _donor_plan(f["patches"], dev) if len(Us) > 1 else None
    flux = FLUX[case.get("scheme", "ausm")]
    for _ in range(case["steps"]):
        if plan:
            Us = _donor_copy(Us, plan)
        U0 = Us
        for a in ALPHAS:
            new = []
            for q, (U, Un, h) in enumerate(zip(Us, U0, hs)):
                V = Un + (a * f["dt"] / (h[0] * h[1] * h[2])) * _residual(U, h, f["periodic"], f["bcs"].get(q, {}), flux)
                new.append(V if act is None else torch.where(act, V, U))
            Us = _donor_copy(new, plan) if plan else new
    return _outputs(Us)
