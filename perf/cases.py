"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values: the operation, the model it runs on and how
much of it there is.  The models are the checkerboard OBS experiments of
fmt2d_b200.synth (a water layer over a sinusoidal seafloor, a gradient crust,
a sediment base and an undulating Moho) at the sizes of the repository's
configurations, tests and benchmark; the checkerboard's amplitude, a smooth
velocity perturbation and the OBS positions' shift are drawn from the seed.

Operations:

forward   time fields of every source and phase on an uploaded model
          (Fmt2d.forward), and the terminal-stage fields, which the rays
          start from, as CUDA tensors (torch.ops.fmt2d.field)
batch     the same for several models of uneven size at once (forward_batch)
trace     rays and Frechet rows of the model's picks on solved fields
          (Fmt2d.trace, and the rows through the C ABI's fmt2d_frechet_rows into
          arrays that the program keeps)
times     receiver times alone, as a line search reads them (Fmt2d.trace_times)
gradient  misfit and its gradient with respect to the slowness and the
          interface depths (Fmt2d.misfit_gradient)
lsqr      a damped, smoothed LSQR solve on a sensitivity matrix kept on the
          device (Fmt2d.lsqr), and the matrix's column norms (Fmt2d.gtg_diag)
iterate   one outer iteration of the joint inversion from the starting model
          (Inversion.iteration): forward, rays, selection, LSQR, line search
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from fmt2d_b200 import synth, torch_ops
from fmt2d_b200.api import Fmt2d, fields_of, forward_batch, phase_mask
from fmt2d_b200.inversion import Inversion, InversionParams

# last time field of each phase: where the rays of the phase start
TERMINAL = {1: 1, 2: 3, 3: 5, 4: 8, 5: 12}


def listed():
    return [
        # one OBS on the test suite's small model: launches, host work and latency
        dict(name="forward_121_1obs", op="forward", nx=121, dx=0.25, depth=16.5, obs=1,
             phases="13"),
        # the plain velocity checkerboard: 401x121, 10 OBS, first arrivals
        dict(name="forward_401_10obs_pg", op="forward", nx=401, dx=0.25, depth=30.0, obs=10,
             phases="1"),
        # one OBS at a time on the benchmark model (the un-batched form)
        dict(name="forward_2001_1obs", op="forward", nx=2001, dx=0.1, depth=40.0, obs=1,
             phases="13"),
        # the benchmark: joint velocity + Moho model, 30 OBS, Pg + PmP
        dict(name="forward_2001_30obs", op="forward", nx=2001, dx=0.1, depth=40.0, obs=30,
             phases="13"),
        # the largest grid of the configurations, a few OBS, with the sediment reflection
        dict(name="forward_4001_6obs", op="forward", nx=4001, dx=0.1, depth=60.0, obs=6,
             phases="123"),
        # models of uneven size at once, all five phases (water multiples included)
        dict(name="batch_3_uneven", op="batch", nx=1187, dx=0.13, depth=27.0, obs=9,
             phases="12345", models=3),
        # rays and Frechet rows of every pick of the benchmark model
        dict(name="trace_2001_30obs", op="trace", nx=2001, dx=0.1, depth=40.0, obs=30,
             phases="13"),
        # the line search's receiver times, all five phases
        dict(name="times_401_10obs", op="times", nx=401, dx=0.25, depth=30.0, obs=10,
             phases="12345"),
        # the misfit's gradient on the benchmark model
        dict(name="gradient_2001_30obs", op="gradient", nx=2001, dx=0.1, depth=40.0, obs=30,
             phases="13"),
        # LSQR at the benchmark's matrix size (24k rows, 0.74 M parameters), Laplacian smoothing
        dict(name="lsqr_2001x371", op="lsqr", nx=2001, nz=371, rows=24000, iters=40, smooth=1),
        # LSQR with Gaussian smoothing on a model's own parameters
        dict(name="lsqr_gauss_401", op="lsqr", nx=401, nz=0, rows=3000, iters=30, smooth=2),
        # a whole iteration of the joint inversion
        dict(name="iterate_401_10obs", op="iterate", nx=401, dx=0.25, depth=30.0, obs=10,
             phases="13"),
    ]


def _odd(rng, lo, hi):
    """A whole number of lo..hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["forward", "forward", "forward", "batch", "trace", "times", "gradient",
                     "lsqr", "iterate"])
    if op == "lsqr":
        if rng.random() < 0.3:
            return dict(op=op, nx=_odd(rng, 121, 401), nz=0, rows=_odd(rng, 200, 3000),
                        iters=rng.randint(10, 40), smooth=2)
        return dict(op=op, nx=_odd(rng, 121, 2001), nz=_odd(rng, 30, 371),
                    rows=_odd(rng, 200, 24000), iters=rng.randint(10, 40), smooth=1)
    nx = _odd(rng, 121, 801 if op in ("batch", "iterate") else 2001)
    dx = round(rng.uniform(0.1, 0.25), 3)
    depth = round(rng.uniform(17.0, 40.0), 1)
    obs = _odd(rng, 1, 10 if op in ("batch", "iterate") else 30)
    phases = rng.choice(["1", "13", "13", "123", "12345"])
    if op == "iterate":
        phases, obs = "13", max(obs, 3)
    if op == "batch" or phases == "12345":
        obs, nx = min(obs, 9), min(nx, _odd(rng, 121, 600))
    case = dict(op=op, nx=nx, dx=dx, depth=depth, obs=obs, phases=phases)
    if op == "batch":
        case["models"] = rng.randint(2, 4)
    return case


# ---------------------------------------------------------------- inputs
def _phases(case):
    return tuple(int(c) for c in case["phases"])


def _model(nx, dx, depth, obs, phases, seed):
    """A seeded checkerboard OBS model of nx columns of dx km and about `depth` km."""
    rng = np.random.default_rng([seed, nx, obs])
    zrel = depth - 8.5
    moho = min(20.0, 3.5 + 0.55 * zrel)
    width = (nx - 1) * dx
    m = synth.checkerboard_model(
        nx, dx, zrel, max(16, int(zrel / 0.25) + 1), n_obs=obs, obs_spacing=0.9 * width / obs,
        shot_spacing=0.2 if nx > 1000 else 0.5, lower_crust=True, moho_base=moho,
        moho_amp=0.05 * moho, moho_wavelength=40.0, cb_dx=10.0, cb_dz=5.0,
        cb_amp=float(rng.uniform(0.03, 0.05)), phases=phases,
        max_offset=min(60.0, 0.8 * width), lc_thick=0.35 * moho)
    x, z = m.xpos[None, :], m.zrel[:, None]
    v = m.vel.copy()
    for _ in range(3):
        kx, kz = rng.uniform(15.0, 60.0), rng.uniform(6.0, 20.0)
        v *= 1.0 + 0.006 * np.sin(2 * np.pi * (x / kx + z / kz + rng.uniform()))
    shift = int(rng.integers(-3, 4))
    obs_x = np.clip(m.obs_x + shift * dx, m.xpos[1], m.xpos[-2])
    return dataclasses.replace(m, vel=v, obs_x=obs_x)


def _of(case, seed):
    return _model(case["nx"], case["dx"], case["depth"], case["obs"], _phases(case), seed)


def _picks(m):
    P = m.picks
    return (P[:, 0].astype(np.int32), P[:, 1].astype(np.int32), P[:, 2].copy(), P[:, 3].copy())


def _ray_rows(nx, nz, rows, np_vel, seed):
    """Ray-like rows over an nx x nz node grid numbered row by row: each row a
    parabolic path between two columns, two nodes per column with the path's
    length split between them, and two interface entries on a third of the
    rows.  Returns 1-based (row_ptr, gindx, gval) with ascending columns."""
    g = torch.Generator().manual_seed(seed)
    dev = "cuda"
    a = torch.rand(rows, generator=g, dtype=torch.float64)
    span = torch.clamp((0.02 + 0.28 * torch.rand(rows, generator=g, dtype=torch.float64)) * nx,
                       min=4.0).long()
    first = (a * (nx - 1 - span).double()).long()
    deep = (0.05 + 0.85 * torch.rand(rows, generator=g, dtype=torch.float64)) * (nz - 2)
    refl = torch.rand(rows, generator=g) < 0.33
    w_if = torch.rand(rows, generator=g, dtype=torch.float64)
    span, first, deep, refl, w_if = (t.to(dev) for t in (span, first, deep, refl, w_if))
    start = torch.cumsum(span, 0) - span
    r = torch.repeat_interleave(torch.arange(rows, device=dev), span)
    k = torch.arange(int(span.sum()), device=dev) - start[r]
    t = (k.double() + 0.5) / span[r].double()
    z = deep[r] * 4.0 * t * (1.0 - t)
    iz = z.long().clamp(0, nz - 2)
    w = z - iz
    slope = deep[r] * 4.0 * (1.0 - 2.0 * t) / span[r].double()
    step = 0.1 * torch.sqrt(1.0 + slope * slope)
    c = first[r] + k
    ri = torch.nonzero(refl).ravel()
    ci = np_vel + first[ri] + span[ri] // 2
    row = torch.cat([r, r, ri, ri])
    col = torch.cat([iz * nx + c, (iz + 1) * nx + c, ci, ci + 1])
    val = torch.cat([(1.0 - w) * step, w * step, 0.2 * w_if[ri], 0.2 * (1.0 - w_if[ri])])
    order = torch.argsort(row * (np_vel + nx + 1) + col)
    row, col, val = row[order], col[order], val[order]
    rp = torch.ones(rows + 1, dtype=torch.int64, device=dev)
    rp[1:] += torch.cumsum(torch.bincount(row, minlength=rows), 0)
    return (rp.to(torch.int32).cpu().numpy(), (col + 1).to(torch.int32).cpu().numpy(),
            val.cpu().numpy())


def _lsqr_inputs(case, seed, nvp, nz):
    nx = case["nx"]
    rp, gi, gv = _ray_rows(nx, nz, case["rows"], nvp, seed)
    rng = np.random.default_rng(seed)
    res = rng.normal(0.0, 0.05, case["rows"])
    dms = rng.normal(0.0, 1e-3, nvp + nx)
    gtg_max = float(np.bincount(gi - 1, weights=gv * gv).max())
    par = dict(wdv=1.0, wdv_iface=0.5, w_smooth=10.0, w_smooth_iface=3.0,
               eps_min=max(1e-6, 1e-4 * gtg_max), max_iter=case["iters"],
               smooth_type=case["smooth"])
    return rp, gi, gv, res, dms, par


def prepare(case, seed):
    torch_ops.load()
    op = case["op"]
    if op == "lsqr":
        nx = case["nx"]
        if case["smooth"] == 1:
            # a parameter grid of its own, every node a parameter
            nz = case["nz"]
            nvp = nx * nz
            g = Fmt2d(0).upload(_model(121, 0.25, 16.5, 1, (1,), seed))
            g.set_param_grid(np.arange(1, nvp + 1, dtype=np.int32).reshape(nz, nx), nvp, nx)
            rp, gi, gv, res, dms, par = _lsqr_inputs(case, seed, nvp, nz)
        else:
            # the model's own parameters: a ray's nodes through the model's numbering
            g = Fmt2d(0).upload(_model(nx, 0.25, 17.0, 1, (1,), seed))
            inv, nvp, npar = g.inv_index()
            rp, gi, gv, res, dms, par = _lsqr_inputs(case, seed, nvp, nvp // nx)
            dms = dms[:npar]
            g.set_smoothing(np.ones(npar), 2.0, 1.0, 2.0)
        g.set_frechet(case["rows"], dms.size, rp, gi, gv)
        return dict(op=op, g=g, res=res, dms=dms, par=par)
    ph = _phases(case)
    if op == "batch":
        ms = [_model(int(case["nx"] / (1.0 + 0.37 * k)) + k, case["dx"] * (1.0 + 0.21 * k),
                     case["depth"] - 1.7 * k, max(1, case["obs"] - 2 * k), ph, seed + 1000 * k)
              for k in range(case["models"])]
        return dict(op=op, gs=[Fmt2d(0).upload(m) for m in ms], xs=[m.obs_x for m in ms], ph=ph)
    m = _of(case, seed)
    if op == "forward":
        return dict(op=op, g=Fmt2d(0).upload(m), x=m.obs_x, ph=ph)
    picks = _picks(m)
    if op in ("trace", "times", "gradient"):
        g = Fmt2d(0).upload(m)
        g.forward(m.obs_x, ph)
        s = dict(op=op, g=g, picks=picks)
        if op == "trace":
            # the program's arrays for the rows, with room for every model of this size
            n = picks[0].size
            cap = n * int(3.0 * (0.45 * min(60.0, 0.8 * (m.nx - 1) * m.dx)
                                 + 2.0 * float(m.moho_z.max())) / m.dx)
            s["rows"] = (np.zeros(n + 1, np.int32), np.zeros(cap, np.int32), np.zeros(cap))
        if op == "gradient":
            # observations: computed times with 40 ms noise, as a bench of the inversion has them
            t, valid = g.trace_times(*picks)
            rng = np.random.default_rng(seed)
            s["obs"] = np.where(valid, t + rng.normal(0.0, 0.04, t.size), -1.0)
        return s
    # iterate: observed times of the checkerboard model, started from a smoothed one
    g = Fmt2d(0).upload(m)
    g.forward(m.obs_x, ph)
    t, valid = g.trace_times(*picks)
    rng = np.random.default_rng(seed)
    obs = np.where(valid, t + rng.normal(0.0, 0.04, t.size), -1.0)
    vel = np.repeat(m.vel.mean(axis=1, keepdims=True), m.nx, axis=1)
    start = dataclasses.replace(m, vel=vel, moho_z=np.full_like(m.moho_z, m.moho_z.mean()))
    g.upload(start)
    params = InversionParams(phases=ph, lam_damp=1.0, lam_damp_iface=1.0, lam_smooth=10.0,
                             lam_smooth_iface=10.0, smooth_type=3, corr_x_iface=2.0,
                             lsqr_max_iter=100, alt_inv_mode=0)
    return dict(op=op, g=g, x=m.obs_x, picks=m.picks, obs=obs, params=params,
                v0=g.velocity().copy(), z0=g.interface(4).copy())


# ---------------------------------------------------------------- one pass
def _terminal_fields(g, nsrc, ph):
    """Per phase the terminal fields of every source: (T, dT/dx, dT/dz), a row per source."""
    out = {}
    for p in ph:
        f = [torch.ops.fmt2d.field(torch_ops.handle(g), s, TERMINAL[p]) for s in range(nsrc)]
        out[f"phase{p}"] = [torch.stack([x[k] for x in f]) for k in range(3)]
    return out


def run(state):
    op = state["op"]
    if op == "forward":
        g = state["g"].forward(state["x"], state["ph"])
        return _terminal_fields(g, state["x"].size, state["ph"])
    if op == "batch":
        forward_batch(state["gs"], state["xs"], state["ph"])
        return [_terminal_fields(g, x.size, state["ph"])
                for g, x in zip(state["gs"], state["xs"])]
    g = state["g"]
    if op == "trace":
        t, valid, nnz = g.trace(*state["picks"])
        rp, gi, gv = state["rows"]
        if nnz > gi.size:
            raise RuntimeError(f"{nnz} Frechet entries, room for {gi.size}")
        g._check(g.L.fmt2d_frechet_rows(g.h, rp.ctypes.data, gi.ctypes.data, gv.ctypes.data, 1),
                 "fmt2d_frechet_rows")
        return [t, valid, rp, gi, gv]
    if op == "times":
        return g.trace_times(*state["picks"])
    if op == "gradient":
        r = g.misfit_gradient(*state["picks"], state["obs"], 0.04, want=("slow", "iface"))
        return [r[k] for k in ("misfit", "t_calc", "valid", "grad_slow", "grad_iface")]
    if op == "lsqr":
        gtg = g.gtg_diag()
        return [gtg, *g.lsqr(state["res"], state["dms"], gtg, **state["par"])]
    g.update_model(vel=state["v0"], iface_z=state["z0"])
    inv = Inversion(g, state["x"], state["picks"], state["obs"], state["params"])
    r = inv.iteration()
    return [g.velocity(), g.interface(4), inv.dm_sum, r.rms_orig, r.rms_new, r.step,
            r.ndata, r.forwards]


# ---------------------------------------------------------------- work
# share of the grid's nodes in the region of each time field: the solid below
# the seafloor, the layer above the sediment base, that above the Moho, the water
_SHARE = {1: 0.85, 2: 0.12, 3: 0.12, 4: 0.5, 5: 0.5, 6: 0.1, 7: 0.1, 8: 0.1, 9: 0.1, 10: 0.1,
          11: 0.85, 12: 0.1}


def _field_nodes(nx, dx, depth, obs, ph):
    n = nx * (depth / dx + 1.0)
    return obs * sum(_SHARE[tf] * n for tf in fields_of(phase_mask(ph)))


def work(case):
    op = case["op"]
    if op == "lsqr":
        nx, rows = case["nx"], case["rows"]
        npar = nx * (case["nz"] or 35) + nx
        nnz = rows * 0.32 * nx
        # the matrix once for each of the two products of an iteration, and the
        # vectors u (data, smoothing, damping rows), v, w, dm read and written
        it = case["iters"]
        return {"bytes": it * (2 * 12.0 * nnz + 16.0 * (rows + 5 * npar)),
                "flops": it * (4.0 * nnz + 40.0 * npar)}
    ph = _phases(case)
    if op == "batch":
        n = sum(_field_nodes(int(case["nx"] / (1 + 0.37 * k)), case["dx"] * (1 + 0.21 * k),
                             case["depth"] - 1.7 * k, max(1, case["obs"] - 2 * k), ph)
                for k in range(case["models"]))
        return {"bytes": 32.0 * n, "flops": 200.0 * n}
    n = _field_nodes(case["nx"], case["dx"], case["depth"], case["obs"], ph)
    if op == "forward":
        # velocity read, time and gradient written; a node's update at least once
        return {"bytes": 32.0 * n, "flops": 200.0 * n}
    if op == "iterate":
        return {"bytes": 64.0 * n, "flops": 400.0 * n}
    width = (case["nx"] - 1) * case["dx"]
    picks = case["obs"] * len(ph) * min(width, 0.9 * min(60.0, 0.8 * width) * 2) / (
        0.2 if case["nx"] > 1000 else 0.5)
    # steps of a ray (a twelfth of a grid step at 6 km/s) and its Frechet entries
    points = picks * 0.4 * min(60.0, 0.8 * width) / (0.08 * case["dx"])
    entries = picks * 3.5 * 0.4 * min(60.0, 0.8 * width) / case["dx"]
    read = 24.0 * picks + min(24.0 * n, 64.0 * points)
    if op == "times":
        return {"bytes": read + 12.0 * picks, "flops": 100.0 * points}
    if op == "trace":
        return {"bytes": read + 12.0 * entries, "flops": 120.0 * points}
    # the fields and the velocity read once, an adjoint written per node
    return {"bytes": read + 16.0 * n, "flops": 400.0 * n + 100.0 * points}


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """run_lsqr with the Laplacian layout in 64-bit torch.  The other
    operations have no value a short program could state: the fields are the
    fixed point of the heap fast marching's stencil, rays and gradients read
    them, and the Gaussian layouts need the model's smoothing matrices."""
    if case["op"] != "lsqr" or case["smooth"] != 1:
        return None
    nx, nz, nd = case["nx"], case["nz"], case["rows"]
    nvp = nx * nz
    npar = nvp + nx
    rp, gi, gv, res, dms, par = _lsqr_inputs(case, seed, nvp, nz)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    row = torch.repeat_interleave(torch.arange(nd, device=dev),
                                  torch.as_tensor(np.diff(rp), device=dev).long())
    col = torch.as_tensor(gi - 1, device=dev).long()
    val = torch.as_tensor(gv, **f64)
    res, dms = torch.as_tensor(res, **f64), torch.as_tensor(dms, **f64)

    def ax(x):
        return torch.zeros(nd, **f64).index_add_(0, row, val * x[col])

    def atx(u):
        return torch.zeros(npar, **f64).index_add_(0, col, val * u[row])

    def lap(x):
        v = x[:nvp].reshape(nz, nx)
        out, k = torch.zeros_like(v), torch.zeros_like(v)
        for dst, src in (((slice(None), slice(1, None)), (slice(None), slice(0, -1))),
                         ((slice(0, -1), slice(None)), (slice(1, None), slice(None)))):
            out[dst] += v[src]
            k[dst] += 1
            out[src] += v[dst]
            k[src] += 1
        i = x[nvp:]
        li = torch.zeros_like(i)
        li[1:-1] = i[:-2] + i[2:] - 2.0 * i[1:-1]
        li[0] = i[1] - i[0]
        li[-1] = i[-2] - i[-1]
        return torch.cat([(out - k * v).ravel(), li])

    gtg = torch.zeros(npar, **f64).index_add_(0, col, val * val)
    keep = torch.ones(npar, dtype=torch.bool, device=dev)
    keep[:nvp] = ~(gtg[:nvp] < par["eps_min"] * 0.01)
    ws = torch.full((npar,), par["w_smooth"], **f64)
    wd = torch.full((npar,), par["wdv"], **f64)
    ws[nvp:], wd[nvp:] = par["w_smooth_iface"], par["wdv_iface"]
    ws, wd = ws * keep, wd * keep

    def fwd(v):
        return ax(v), ws * lap(v), wd * v

    def adj(u):
        return (atx(u[0]) + ws * lap(u[1]) + wd * u[2]) * keep

    def norm(u):
        return torch.sqrt(sum((x * x).sum() for x in u))

    u = (res, -(ws * lap(dms)), -(wd * dms))
    bnorm = beta = norm(u)
    u = tuple(x / beta for x in u)
    v = adj(u)
    alpha = norm((v,))
    v = v / alpha
    w, dm = v.clone(), torch.zeros(npar, **f64)
    phibar, rhobar, anorm2 = beta, alpha, alpha * alpha + beta * beta
    iters, rnorm, test2 = par["max_iter"] + 1, beta, torch.zeros((), **f64)
    for k in range(1, par["max_iter"] + 1):
        u = tuple(a - alpha * b for a, b in zip(fwd(v), u))
        beta = norm(u)
        u = tuple(x / beta for x in u)
        v = adj(u) - beta * v
        alpha = norm((v,))
        v = v / alpha
        anorm2 = anorm2 + alpha * alpha + beta * beta
        rho = torch.sqrt(rhobar * rhobar + beta * beta)
        c, s = rhobar / rho, beta / rho
        theta, rhobar = s * alpha, -c * alpha
        phi, phibar = c * phibar, s * phibar
        dm = dm + (phi / rho) * w
        w = v - (theta / rho) * w
        rnorm = torch.abs(phibar)
        test2 = phibar * alpha * torch.abs(c) / (torch.sqrt(anorm2) * rnorm + 1e-30)
        if float(test2) < 1e-4:
            iters = k
            break
    return [gtg.cpu().numpy(), dm.cpu().numpy(), iters, float(rnorm), float(bnorm), float(test2)]
