"""Workloads whose speed matters to users of the framework, each through its public entry points.

A case is a dict of plain values; `kind` names the path:

  mobility   one FCM mobility solve (Fcm.mobility_solve): bead forces and torques in, U and Omega out
  barrier    cell link + collision barrier (LinkedList.link, apply_collision_barrier)
  iteration  the filament half of one Broyden iteration: forces, J0 and its inverse, residual, J0^-1 with history
  steps      implicit time steps of a suspension whose state the caller holds on the host (upload, run_steps)
  ensemble   implicit time steps of several independent boxes advanced together (Ensemble.run)
  mlp        the learned start's network: predictions and the gradients of a training batch

Results of the mixed-precision chain (precision "fp32") are single-precision numbers that the library hands out
in float64 arrays, so they are returned as float32; every other result keeps its type.
"""
import math

import numpy as np
import torch

from filsim_b200 import abi
from filsim_b200.configs import DX, params_for, sediment_params
from filsim_b200.ensemble import Ensemble
from filsim_b200.fcm import Context, Fcm, LinkedList, Simulation
from filsim_b200.learn import WarmStartModel
from filsim_b200.suspension import Suspension, random_suspension

PRECISIONS = {"fp64": abi.FS_PREC_FP64, "fp32": abi.FS_PREC_FP32}
# grid lengths in use: whole 16-point tiles with small prime factors
LENGTHS = (32, 48, 64, 80, 96, 112, 128, 144, 160, 192, 224, 256, 320, 384, 448, 512)
STARTUP = 12  # steps before the steady regime (implicit Euler, then the tension extrapolation's build-up)


def listed():
    return [
        # the smallest configured solve: launches and latency
        dict(name="mobility_64_fp64", kind="mobility", nx=64, ny=64, nz=64, nfil=32, nw=15, ngd=12, precision="fp64"),
        # the 256^3 configuration in both precisions
        dict(name="mobility_256_fp64", kind="mobility", nx=256, ny=256, nz=256, nfil=1024, nw=30, ngd=12,
             precision="fp64"),
        dict(name="mobility_256_fp32", kind="mobility", nx=256, ny=256, nz=256, nfil=1024, nw=30, ngd=12,
             precision="fp32"),
        # the reference's long box (its [4, 1, 1] shape) with its own stencil, 20 points at dx = sigma_dip / 1.5
        dict(name="mobility_384x96x96_ngd20", kind="mobility", nx=384, ny=96, nz=96, nfil=200, nw=15, ngd=20,
             precision="fp64"),
        # a box whose sides are no power of two, with an odd number of long filaments
        dict(name="mobility_ragged_fp32", kind="mobility", nx=160, ny=96, nz=224, nfil=223, nw=37, ngd=12,
             precision="fp32"),
        # the solve of the largest configured suspension
        dict(name="mobility_512_fp32", kind="mobility", nx=512, ny=512, nz=512, nfil=4096, nw=32, ngd=12,
             precision="fp32"),
        # the collision barrier of the largest configured suspension
        dict(name="barrier_512", kind="barrier", n=512, nfil=4096, nw=32),
        # filament mechanics, Jacobian and Broyden correction of the 256^3 suspension
        dict(name="iteration_1024x32", kind="iteration", n=256, nfil=1024, nw=32, columns=6),
        # a small simulation as the reference runs it: FP64, its own start, the host driving every iteration
        dict(name="steps_64_fp64", kind="steps", n=64, nfil=32, nw=15, steps=3, precision="fp64"),
        # the largest simulation with everything that speeds it up: mixed precision, captured steps, improved
        # start, Broyden memory and velocity predictor
        dict(name="steps_512_fp32", kind="steps", n=512, nfil=4096, nw=32, steps=3, precision="fp32"),
        # a parameter sweep of small boxes, two of each grid size of the sweep
        dict(name="ensemble_8_boxes", kind="ensemble", boxes=8, nw=16, fill=0.03, steps=4),
        # the learned start's network at the size the largest suspension trains it
        dict(name="mlp_4096x32", kind="mlp", nw=32, hidden=256, rows=4096),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _filaments(rng, volume):
    """(nfil, nw) for a bead volume fraction between 0.2 % and 4 % of the box."""
    beads = _log_uniform(rng, 0.002, 0.04) * volume / (4.0 / 3.0 * math.pi)
    nw = rng.choice((1, 2, 5, 8, 15, 15, 16, 20, 30, 31, 32, 37, 48))
    return max(1, round(beads / nw)), nw


def _length(rng, lo=32, hi=512):
    x = _log_uniform(rng, lo, hi)
    return min((n for n in LENGTHS if lo <= n <= hi), key=lambda n: abs(math.log(n / x)))


def draw(rng):
    kind = rng.choice(["mobility"] * 8 + ["barrier", "iteration", "steps", "steps"])
    if kind == "mobility":
        if rng.random() < 0.5:
            nx = ny = nz = _length(rng)
        else:
            nx, ny, nz = _length(rng), _length(rng), _length(rng)
        ngd = rng.choice((12, 12, 20))
        nfil, nw = _filaments(rng, nx * ny * nz * _dx(ngd) ** 3)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nfil=nfil, nw=nw, ngd=ngd, precision=rng.choice(("fp64", "fp32")))
    n = _length(rng, 64, 384)
    nfil, nw = _filaments(rng, (n * DX) ** 3)
    nw = min(max(nw, 5), int(1.5 * n * DX / 2.2))  # straight filaments that can still be placed
    nfil = max(1, min(nfil, round(0.03 * (n * DX) ** 3 / (nw * 4.2))))
    if kind == "barrier":
        return dict(kind=kind, n=n, nfil=nfil, nw=nw)
    if kind == "iteration":
        return dict(kind=kind, n=n, nfil=nfil, nw=nw, columns=rng.randrange(0, 16))
    n = _length(rng, 48, 160)
    nw = rng.choice((5, 8, 15, 16, 31))
    nfil = max(1, round(_log_uniform(rng, 0.004, 0.03) * (n * DX) ** 3 / (nw * 4.2)))
    return dict(kind="steps", n=n, nfil=nfil, nw=nw, steps=rng.randrange(1, 5), precision=rng.choice(("fp64", "fp32")))


# ---- inputs ---------------------------------------------------------------------------------------------------


def _dx(ngd):
    """Grid spacing of a stencil width: a / 1.86 in the configurations, sigma_dip / 1.5 with the reference's 20."""
    return DX if ngd == 12 else 1.0 / (36.0 * math.pi) ** (1.0 / 6.0) / 1.5


def _mobility_inputs(case, seed):
    """Straight filaments at random places, positions as assign_filament_data leaves them (fmod(X, L), which keeps
    the sign), forces and torques N(0, 1) per component."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nfil, nw = case["nfil"], case["nw"]
    dx = _dx(case["ngd"])
    box = torch.tensor([case["nx"] * dx, case["ny"] * dx, case["nz"] * dx], dtype=torch.float64, device="cuda")
    c = torch.rand((nfil, 1, 3), generator=g, dtype=torch.float64, device="cuda") * box
    t = torch.randn((nfil, 1, 3), generator=g, dtype=torch.float64, device="cuda")
    t = t / t.norm(dim=2, keepdim=True)
    s = 2.2 * (torch.arange(nw, dtype=torch.float64, device="cuda") - 0.5 * nw).reshape(1, nw, 1)
    y = torch.fmod((c + s * t).reshape(-1, 3), box)
    f = torch.randn((nfil * nw, 3), generator=g, dtype=torch.float64, device="cuda")
    tau = torch.randn((nfil * nw, 3), generator=g, dtype=torch.float64, device="cuda")
    return y, f, tau


def _barrier_inputs(case, seed):
    """A placed suspension whose beads have moved a little, so that some pairs are within the barrier's range."""
    p = params_for(case["n"])
    s = random_suspension(p, case["nfil"], case["nw"], seed)
    rng = np.random.default_rng(seed + 1)
    x = s.X + rng.uniform(-0.3, 0.3, s.X.shape)
    box = np.array([case["n"] * DX] * 3)
    f = rng.standard_normal(s.X.shape)
    dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    return p, dev(x), dev(np.fmod(x, box)), dev(f), dev(s.fil_id), dev(s.seg_id)


def _bent_suspension(case, seed):
    """Filaments bent by a few degrees a link, moving and under tension: a state as a step meets it."""
    p = sediment_params(case["n"])
    s = random_suspension(p, case["nfil"], case["nw"], seed)
    rng = np.random.default_rng(seed + 2)
    turn = np.cumsum(rng.normal(0.0, 0.03, (case["nfil"], case["nw"], 3)), axis=1).reshape(-1, 3)

    def rotated(q, v):  # exp(v / 2) q
        th = np.linalg.norm(v, axis=1, keepdims=True) + 1e-300
        ps, pv = np.cos(th / 2), np.sin(th / 2) / th * v
        qs, qv = q[:, :1], q[:, 1:]
        return np.concatenate([ps * qs - (pv * qv).sum(1, keepdims=True), ps * qv + qs * pv + np.cross(pv, qv)], axis=1)

    s.q[...] = rotated(s.q, turn)
    s.U[...] = rng.normal(0.0, 1e-2, s.U.shape)
    s.Ut[...] = s.U + rng.normal(0.0, 1e-3, s.U.shape)
    s.Us[...] = s.U + rng.normal(0.0, 1e-3, s.U.shape)
    s.qs[...] = rotated(s.q, s.Us)
    drift = rng.normal(0.0, 2e-2, (case["nfil"], 1, 3)) * np.ones((1, case["nw"], 1))
    s.Xt[...] = s.X - drift.reshape(-1, 3)
    s.Xs[...] = s.X + drift.reshape(-1, 3)
    s.lam[...] = rng.normal(0.0, 1.0, s.lam.shape)
    n6 = 6 * s.np
    v = rng.normal(0.0, 0.3, (s.np, 3))
    w = rng.normal(0.0, 0.1, (s.np, 3))
    c = rng.standard_normal((case["columns"], n6)) * 1e-2
    d = rng.standard_normal((case["columns"], n6)) / math.sqrt(n6)
    return p, s, v, w, c, d


def _pinned(s):
    """The suspension's host arrays in pinned memory, where a program that uploads its state keeps them."""
    s.keep = {}
    for k, v in s.arrays.items():
        s.keep[k] = torch.empty(v.shape, dtype=torch.float64, pin_memory=True)
        s.keep[k].numpy()[...] = v
        s.arrays[k] = s.keep[k].numpy()
    return s


def _mlp_weights(dims, seed):
    """Flat parameters [W1 b1 ... W4 b4], uniform in +-1 / sqrt(fan in)."""
    rng = np.random.default_rng(seed + 3)
    out = []
    for fan_in, fan_out in zip(dims[:-1], dims[1:]):
        a = 1.0 / math.sqrt(fan_in)
        out += [rng.uniform(-a, a, fan_out * fan_in), rng.uniform(-a, a, fan_out)]
    return np.concatenate(out).astype(np.float32)


def _mlp_dims(case):
    up = lambda x: -(-x // 128) * 128  # noqa: E731
    nw, h = case["nw"], case["hidden"]
    features, targets = 19 * nw + 9 * (nw - 1) + 1, 12 * nw
    return features, targets, [up(features), h, h, h, up(targets)]


def _mlp_inputs(case, seed):
    features, targets, _ = _mlp_dims(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((case["rows"], features), generator=g, device="cuda")
    t = torch.randn((case["rows"], targets), generator=g, device="cuda")
    return x, t


# ---- what a user's program has in hand ------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mobility":
        y, f, t = _mobility_inputs(case, seed)
        p = params_for((case["nx"], case["ny"], case["nz"]), ngd=case["ngd"], dx=_dx(case["ngd"]))
        ctx = Context(p, max_beads=y.shape[0], max_filaments=case["nfil"])
        ctx.set_precision(PRECISIONS[case["precision"]])
        fcm = Fcm(ctx, y.shape[0])
        fcm.set(y, f, t)
        return dict(kind=kind, ctx=ctx, fcm=fcm, precision=case["precision"])
    if kind == "barrier":
        p, x, y, f, fil, seg = _barrier_inputs(case, seed)
        ctx = Context(p, max_beads=x.shape[0], max_filaments=case["nfil"])
        return dict(kind=kind, ctx=ctx, cells=LinkedList(ctx), x=x, y=y, f0=f, f=torch.empty_like(f), fil=fil, seg=seg)
    if kind == "iteration":
        p, s, v, w, c, d = _bent_suspension(case, seed)
        ctx = Context(p, max_beads=s.np, max_filaments=s.nfil)
        sim = Simulation(ctx, s)
        for i in range(case["columns"]):
            sim.set_cols(c[i], d[i], i)
        dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
        return dict(kind=kind, ctx=ctx, sim=sim, v=dev(v), w=dev(w), columns=case["columns"])
    if kind == "steps":
        p = sediment_params(case["n"])
        s = random_suspension(p, case["nfil"], case["nw"], seed)
        ctx = Context(p, max_beads=s.np, max_filaments=s.nfil)
        ctx.set_precision(PRECISIONS[case["precision"]])
        if case["precision"] == "fp32":
            ctx.set_start_order(2)
            ctx.set_tension_extrapolation(1)
            ctx.set_broyden_memory(16, 4, 8, 30)
            ctx.set_velocity_predictor(0.5)
            abi.check(abi.lib().fs_set_graph_mode(ctx.h, 1), "fs_set_graph_mode")
        sim = Simulation(ctx, s)
        sim.run_steps(1, STARTUP)
        s.set_arrays(sim.download())
        return dict(kind=kind, ctx=ctx, sim=sim, start=_pinned(s), steps=case["steps"], precision=case["precision"])
    if kind == "ensemble":
        grids = (48, 64, 96, 128)
        boxes = []
        for i in range(case["boxes"]):
            n = grids[i % len(grids)]
            nfil = max(1, int(case["fill"] * (n * DX) ** 3 / (case["nw"] * 4.0 / 3.0 * math.pi)))
            p = sediment_params(n, broyden_maxiter=100)
            kb = 0.1 * 100.0 ** ((i + 0.5) / case["boxes"])  # K_B over [0.1, 10]
            boxes.append((n, p, random_suspension(p, nfil, case["nw"], seed=1000 * seed + i, kap=kb), kb))
        e = Ensemble(boxes, start_order=2, tension_order=1, memory=(16, 4, 8, 30), predictor=0.5)
        e.startup(STARTUP)
        start = []
        for sim in e.sims:
            s = sim.susp.copy()
            s.set_arrays(sim.download())
            start.append(_pinned(s))
        return dict(kind=kind, e=e, start=start, steps=case["steps"])
    if kind == "mlp":
        ctx = Context(params_for(32), max_beads=case["nw"], max_filaments=1)
        model = WarmStartModel(ctx, case["nw"], hidden=case["hidden"], batch_capacity=case["rows"])
        _, _, dims = _mlp_dims(case)
        model.set_params(_mlp_weights(dims, seed))
        x, t = _mlp_inputs(case, seed)
        return dict(kind=kind, ctx=ctx, model=model, x=x, t=t)
    raise ValueError(kind)


# ---- one pass -------------------------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "mobility":
        fcm = state["fcm"]
        fcm.mobility_solve()
        if state["precision"] == "fp32":
            return dict(V=fcm.V.float(), W=fcm.W.float())
        return dict(V=fcm.V, W=fcm.W)
    if kind == "barrier":
        state["cells"].link(state["x"])
        f = state["f"].copy_(state["f0"])
        d2 = state["cells"].apply_collision_barrier(state["y"], f, STARTUP + 1, state["fil"], state["seg"])
        return dict(F=f, min_dist2=d2)
    if kind == "iteration":
        sim, nt = state["sim"], STARTUP + 1
        sim.filament_forces(nt)
        sim.build_jacobian(nt)
        err, check = sim.error_check(state["v"], state["w"], nt)
        x = sim.broyden_apply(err, state["columns"])
        np_ = sim.susp.np
        return dict(F=sim.device_array("F", (np_, 3)), TAU=sim.device_array("TAU", (np_, 3)), err=err, x=x, check=check)
    if kind == "steps":
        sim = state["sim"]
        sim.upload(state["start"])
        sim.run_steps(STARTUP + 1, state["steps"])
        s = sim.susp
        out = dict(X=sim.device_array("X", (s.np, 3)), q=sim.device_array("q", (s.np, 4)))
        if state["precision"] == "fp32":  # positions and orientations: what an output row holds
            return {k: v.float() for k, v in out.items()}
        out["U"] = sim.device_array("U", (s.np, 3))
        out["lam"] = sim.device_array("lam", (s.nlink, 3))
        return out
    if kind == "ensemble":
        e = state["e"]
        for sim, s in zip(e.sims, state["start"]):
            sim.upload(s)
        e.run(STARTUP + 1, state["steps"])
        return [dict(X=sim.device_array("X", (sim.susp.np, 3)).float(), q=sim.device_array("q", (sim.susp.np, 4)).float())
                for sim in e.sims]
    if kind == "mlp":
        model = state["model"]
        y = model.forward(state["x"])
        g, loss = model.gradients(state["x"], state["t"])
        return dict(y=y, g=g, loss=loss)
    raise ValueError(kind)


# ---- what a pass cannot do without ----------------------------------------------------------------------------


def _solve_work(n, beads, ngd, size):
    """One mobility solve: the force grid, its spectrum and the velocity grid each written and read once (they are
    larger than the chip's memory in all but the smallest boxes), the bead arrays once; the transforms at
    2.5 N log2 N per real field and direction, the spread's and the interpolation's stencil sums."""
    return {"bytes": 18.0 * size * n + 120.0 * beads,
            "flops": 15.0 * n * math.log2(n) + 15.0 * n + beads * ngd ** 3 * (16.0 + 24.0)}


def _iteration_work(nfil, nw, columns, build):
    """Bead state in and out, S^-1 written and read; the inverse of S at 2 m^3, the matvec and the history."""
    beads, m = nfil * nw, 3.0 * nw
    return {"bytes": beads * 8.0 * (40 + 12 * columns) + nfil * 8.0 * m * m * (2 if build else 1),
            "flops": nfil * ((2.0 * m ** 3 if build else 0.0) + 2.0 * m * m) + beads * (400.0 + 24.0 * columns)}


def work(case):
    kind = case["kind"]
    if kind == "mobility":
        return _solve_work(case["nx"] * case["ny"] * case["nz"], case["nfil"] * case["nw"], case["ngd"],
                           8 if case["precision"] == "fp64" else 4)
    if kind == "barrier":
        beads = case["nfil"] * case["nw"]
        return {"bytes": beads * (4 * 24.0 + 8.0), "flops": beads * 200.0}
    if kind == "iteration":
        return _iteration_work(case["nfil"], case["nw"], case["columns"], True)
    if kind == "steps":
        # iterations a step takes at the tolerance: about 18 from the reference's start, about 4 with everything on
        its, size = (18, 8) if case["precision"] == "fp64" else (4, 4)
        a = _solve_work(case["n"] ** 3, case["nfil"] * case["nw"], 12, size)
        b = _iteration_work(case["nfil"], case["nw"], its // 2, False)
        return {k: case["steps"] * (its + 1) * (a[k] + b[k]) for k in a}
    if kind == "ensemble":
        total = {"bytes": 0.0, "flops": 0.0}
        for i in range(case["boxes"]):
            n = (48, 64, 96, 128)[i % 4]
            a = _solve_work(n ** 3, case["fill"] * (n * DX) ** 3 / 4.2, 12, 4)
            for k in total:
                total[k] += case["steps"] * 2 * a[k]
        return total
    if kind == "mlp":
        _, _, d = _mlp_dims(case)
        pairs = [a * b for a, b in zip(d[:-1], d[1:])]
        return {"bytes": 4.0 * (case["rows"] * (d[0] + 2 * d[-1]) + 2 * sum(pairs)),
                "flops": 2.0 * case["rows"] * (4 * sum(pairs) - pairs[0])}
    raise ValueError(kind)


# ---- the same in 64 bits --------------------------------------------------------------------------------------


def _stencils(case, y):
    """Per axis: grid indices and the monopole weight, dipole weight and -xx / sigma_dip^2 of each stencil point."""
    ngd, dx = case["ngd"], _dx(case["ngd"])
    sig, sd = 1.0 / math.sqrt(math.pi), 1.0 / (36.0 * math.pi) ** (1.0 / 6.0)
    k = torch.arange(ngd, device="cuda")
    out = []
    for a, n in enumerate((case["nx"], case["ny"], case["nz"])):
        xg = torch.trunc(y[:, a] / dx).long()[:, None] - ngd // 2 + 1 + k
        xx = xg.double() * dx - y[:, a:a + 1]
        out.append((xg % n, torch.exp(-xx * xx / (2 * sig ** 2)) / math.sqrt(2 * math.pi * sig ** 2),
                    torch.exp(-xx * xx / (2 * sd ** 2)) / math.sqrt(2 * math.pi * sd ** 2), -xx / sd ** 2))
    return out


def _exact_mobility(case, seed):
    y, f, t = _mobility_inputs(case, seed)
    dims, dx = (case["nx"], case["ny"], case["nz"]), _dx(case["ngd"])
    grid = torch.zeros((3, dims[0] * dims[1] * dims[2]), dtype=torch.float64, device="cuda")

    def chunks():
        for b in range(0, y.shape[0], 4096):
            (ix, gx, dxx, rx), (iy, gy, dy, ry), (iz, gz, dz, rz) = _stencils(case, y[b:b + 4096])
            at = (ix[:, :, None, None] * dims[1] + iy[:, None, :, None]) * dims[2] + iz[:, None, None, :]
            g = gx[:, :, None, None] * gy[:, None, :, None] * gz[:, None, None, :]
            d = dxx[:, :, None, None] * dy[:, None, :, None] * dz[:, None, None, :]
            yield slice(b, b + 4096), at, g, d, rx[:, :, None, None], ry[:, None, :, None], rz[:, None, None, :]

    col = lambda v, a: v[:, a, None, None, None]  # noqa: E731
    for s, at, g, d, rx, ry, rz in chunks():
        h = 0.5 * t[s]
        r = (rx, ry, rz)
        for a in range(3):
            b, c = (a + 1) % 3, (a + 2) % 3
            # F g + (T / 2 x grad) g_dip, grad = -(rx, ry, rz)... written as the rotlet's antisymmetric part
            val = col(f[s], a) * g + (col(h, c) * r[b] - col(h, b) * r[c]) * d
            grid[a].index_add_(0, at.reshape(-1), val.reshape(-1))
    spec = torch.fft.rfftn(grid.reshape(3, *dims), dim=(1, 2, 3))
    q = []
    for a, n in enumerate(dims):
        i = torch.arange(n if a < 2 else n // 2 + 1, device="cuda")
        i = torch.where(i <= n // 2, i, i - n).double() * (2 * math.pi / (n * dx))
        q.append(i.reshape([-1 if a == b else 1 for b in range(3)]))
    inv = 1.0 / (q[0] ** 2 + q[1] ** 2 + q[2] ** 2 + 1e-18)
    along = (q[0] * spec[0] + q[1] * spec[1] + q[2] * spec[2]) * inv
    total = float(dims[0] * dims[1] * dims[2])
    for a in range(3):
        spec[a] = inv * (spec[a] - q[a] * along) / total
    del along, inv
    spec[:, 0, 0, 0] = 0
    spec = torch.fft.ifftn(spec, dim=(1, 2), norm="forward")
    spec[..., 0].imag.zero_()
    spec[..., -1].imag.zero_()
    grid = torch.fft.irfft(spec, n=dims[2], dim=3, norm="forward").reshape(3, -1)
    del spec
    v, w = torch.empty_like(y), torch.empty_like(y)
    for s, at, g, d, rx, ry, rz in chunks():
        u = [grid[a][at] for a in range(3)]
        r = (rx, ry, rz)
        for a in range(3):
            b, c = (a + 1) % 3, (a + 2) % 3
            v[s, a] = (u[a] * g).sum((1, 2, 3)) * dx ** 3
            w[s, a] = -0.5 * ((u[c] * r[b] - u[b] * r[c]) * d).sum((1, 2, 3)) * dx ** 3
    return dict(V=v, W=w)


def _exact_barrier(case, seed):
    _, _, y, f, fil, seg = _barrier_inputs(case, seed)
    box = case["n"] * DX
    reach, near = 1.21 * 4.0, 4.0
    f = f.clone()
    least = 100000.0
    for b in range(0, y.shape[0], 256):
        d = y[b:b + 256, None, :] - y[None, :, :]
        d -= box * torch.floor(d / box + 0.5)
        r2 = (d * d).sum(2)
        skip = (fil[b:b + 256, None] == fil[None]) & ((seg[b:b + 256, None] - seg[None]).abs() <= 1)
        r2[skip] = 100000.0
        least = min(least, float(r2.min()))
        i, j = torch.nonzero(r2 < reach, as_tuple=True)
        e, rr = d[i, j], r2[i, j]
        capped = rr < 4.0  # at the distance cap, 2a, the force stays the contact force
        e = torch.where(capped[:, None], e / rr.sqrt()[:, None] * 2.0, e)
        rr = torch.where(capped, torch.full_like(rr, 4.0), rr)
        f.index_add_(0, b + i, (15 * math.pi * ((reach - rr) / (reach - near)) ** 4)[:, None] * e)
    return dict(F=f, min_dist2=least)


def _exact_iteration(case, seed):
    """Forces, torques and residual; J0^-1 belongs to the framework's approximate Jacobian and has no other value."""
    p, s, v, w, _, _ = _bent_suspension(case, seed)
    nfil, nw, dl, dt = case["nfil"], case["nw"], p.dl, p.dt
    dev = lambda a: torch.as_tensor(np.asarray(a), device="cuda").reshape(nfil, -1, a.shape[-1])  # noqa: E731
    qs, us, lam, x, xt, u, v, w = (dev(a) for a in (s.qs, s.Us, s.lam, s.X, s.Xt, s.U, v, w))
    x0 = dev(s.Xs)[:, :1]
    cross = torch.linalg.cross
    q0, qv = qs[..., :1], qs[..., 1:]
    a, b, c = qv.unbind(-1)
    z = q0[..., 0]
    tan = torch.stack([1 - 2 * b * b - 2 * c * c, 2 * (a * b + z * c), 2 * (a * c - z * b)], -1)
    xs = torch.cat([x0, x0 + torch.cumsum(0.5 * dl * (tan[:, 1:] + tan[:, :-1]), 1)], 1)

    def mul(p0, pv, r0, rv):
        return p0 * r0 - (pv * rv).sum(-1, keepdim=True), p0 * rv + r0 * pv + cross(pv, rv)

    tau = torch.zeros_like(xs)
    f = torch.zeros_like(xs) + torch.tensor([p.gravity[k] for k in range(3)], dtype=torch.float64, device="cuda")
    if nw > 1:
        # the link's frame: halfway along the rotation from bead i to bead i + 1
        r0, rv = mul(q0[:, 1:], qv[:, 1:], q0[:, :-1], -qv[:, :-1])
        h0 = torch.sqrt(0.5 * (r0 + 1))
        m0, mv = mul(h0, rv / (2 * h0), q0[:, :-1], qv[:, :-1])
        # strain twist 2 vec(conj(m) dq / ds), then into the laboratory frame
        _, bend = mul(m0, -mv, (q0[:, 1:] - q0[:, :-1]) / dl, (qv[:, 1:] - qv[:, :-1]) / dl)
        _, bend = mul(*mul(m0, mv, torch.zeros_like(m0), 2 * bend), m0, -mv)
        tau[:, 1:] -= bend
        tau[:, :-1] += bend
        f[:, 1:] += lam
        f[:, :-1] -= lam
        tau[:, 1:] -= 0.5 * dl * cross(tan[:, 1:], lam)
        tau[:, :-1] -= 0.5 * dl * cross(tan[:, :-1], lam)
    th = us.norm(dim=-1, keepdim=True)
    uw = cross(us, w)
    e = w - 0.5 * uw - (0.5 * th / torch.tan(0.5 * th) - 1) / th ** 2 * cross(us, uw)
    e1 = xs - 4.0 / 3.0 * x + xt / 3.0 - 2.0 / 3.0 * dt * v
    e2 = us - u / 3.0 - 2.0 / 3.0 * dt * e
    err = torch.cat([e1.reshape(nfil, -1), e2.reshape(nfil, -1)], 1).reshape(-1)
    return dict(F=f.reshape(-1, 3), TAU=tau.reshape(-1, 3), err=err, x=None, check=bool((err.abs() > p.tol).any()))


def _exact_mlp(case, seed):
    features, targets, dims = _mlp_dims(case)
    x, t = (a.double() for a in _mlp_inputs(case, seed))
    flat = torch.as_tensor(_mlp_weights(dims, seed), device="cuda").double().requires_grad_()
    h = torch.nn.functional.pad(x, (0, dims[0] - features))
    at = 0
    for k, (i, o) in enumerate(zip(dims[:-1], dims[1:])):
        h = h @ flat[at:at + i * o].reshape(o, i).T + flat[at + i * o:at + i * o + o]
        at += i * o + o
        if k < 3:
            h = torch.nn.functional.silu(h)
    y = h[:, :targets]
    loss = ((y - t) ** 2).mean()
    loss.backward()
    return dict(y=y.detach(), g=flat.grad, loss=float(loss))


def exact(case, seed):
    """Whole steps and ensembles have no value of their own: a step stops at the iteration's tolerance."""
    kind = case["kind"]
    if kind == "mobility":
        return _exact_mobility(case, seed)
    if kind == "barrier":
        return _exact_barrier(case, seed)
    if kind == "iteration":
        return _exact_iteration(case, seed)
    if kind == "mlp":
        return _exact_mlp(case, seed)
    return None
