"""The work that users of this framework have it do, as cases that can be measured.

A case is one pass through the public entry points at one size: a plain FP64 Stokes solve, the mixed-precision
solve of one problem or of a batch, the marker deposit, the marker advection, the rebinning, or a whole timestep.
The sizes are those of this repository's configurations, tests and benchmark (20 x 26 points up to 4096 points
per side, 9 to 25 markers per cell), with odd and ragged ones among them.  Iteration counts are fixed, so a pass
is the same work every time; a solve keeps its residual checks and dt updates where its schedule has them.

``exact`` gives a pass's results from plain torch in 64 bits, written from the finite-difference scheme and the
bilinear marker interpolation.
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "stokesflow.jl_b200"))

G_Y = 9.81
MAXDISP = 0.5
EPS = 1e-30      # never reached: a pass runs its fixed number of iterations
MOST_POINT_ITERATIONS = 2048 * 2048 * 1500   # of one solve
MOST_MARKERS = 67_043_344                    # 2047 x 2047 cells with 16 markers each


def listed():
    return [
        # the reference's own 20 x 26 test grid: the smallest solve, where every launch counts
        dict(name="solve_20x26", kind="solve", Nx=20, Ny=26, iters=3100, stab=True, work=True),
        # a small served request, 127 cells per side
        dict(name="solve_128", kind="solve", Nx=128, Ny=128, iters=5120, stab=True, work=False),
        # a ragged grid (odd, not square, no power of two) of the middle of the batching range
        dict(name="solve_511x385", kind="solve", Nx=511, Ny=385, iters=4000, stab=True, work=False),
        # 1023 cells per side, the largest grid of the serving and batching range; a plain solve without the
        # free-surface stabilisation
        dict(name="solve_1024", kind="solve", Nx=1024, Ny=1024, iters=4000, stab=False, work=False),
        # the benchmark's grid, 2047 cells per side
        dict(name="solve_2048", kind="solve", Nx=2048, Ny=2048, iters=1500, stab=True, work=False),
        # a large ragged grid, up to the precision form's 4095 cells per side
        dict(name="solve_4001x3003", kind="solve", Nx=4001, Ny=3003, iters=400, stab=True, work=False),
        # the precision form: FP32 sweeps with FP64 defect correction of one 1023-cell problem
        dict(name="mixed_1024", kind="mixed", Nx=1024, Ny=1024, iters=4000),
        # the batching form: uneven instances, 127 to 511 cells per side
        dict(name="batch_16", kind="batch", n=16, lo=128, hi=512, iters=2000),
        # the three deposits of a timestep of a small request, 9 markers per cell
        dict(name="deposit_128", kind="deposit", Nx=128, Ny=128, md=3),
        # the three deposits of a benchmark timestep: 67 million markers that have moved
        dict(name="deposit_2048", kind="deposit", Nx=2048, Ny=2048, md=4),
        # the marker half of a timestep after the solve: RK4 advection and rebinning, 1023 cells, 25 markers per cell
        dict(name="move_1024", kind="move", Nx=1024, Ny=1024, md=5),
        # a whole timestep through the driver: deposit, solve, advection, rebin
        dict(name="timestep_256", kind="timestep", Nx=256, Ny=256, md=4, iters=2560),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "mixed", "batch", "deposit", "deposit", "move", "timestep"])
    if kind == "solve":
        Nx = _log_int(rng, 20, 4096)
        Ny = min(4096, max(20, int(Nx * math.exp(rng.uniform(-0.7, 0.7)))))
        most = MOST_POINT_ITERATIONS // (Nx * Ny)
        return dict(kind=kind, Nx=Nx, Ny=Ny, iters=max(50, min(_log_int(rng, 500, 5000), most)),
                    stab=rng.random() < 0.75, work=rng.random() < 0.3)
    if kind == "mixed":
        Nx = _log_int(rng, 64, 2048)
        Ny = min(2048, max(64, int(Nx * math.exp(rng.uniform(-0.5, 0.5)))))
        return dict(kind=kind, Nx=Nx, Ny=Ny, iters=max(400, min(4000, MOST_POINT_ITERATIONS // (Nx * Ny))))
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(4, 24), lo=rng.randint(64, 160), hi=rng.randint(300, 600),
                    iters=rng.randint(800, 1600))
    if kind == "timestep":
        Nx = _log_int(rng, 40, 700)
        Ny = max(40, int(Nx * math.exp(rng.uniform(-0.4, 0.4))))
        return dict(kind=kind, Nx=Nx, Ny=Ny, md=rng.randint(3, 5), iters=rng.randint(800, 2600))
    md = rng.randint(3, 5)
    Nx = _log_int(rng, 40, 2048)
    Ny = max(40, int(Nx * math.exp(rng.uniform(-0.5, 0.5))))
    while md * md * Nx * Ny > MOST_MARKERS:
        Nx, Ny = Nx // 2, Ny // 2
    return dict(kind=kind, Nx=Nx, Ny=Ny, md=md)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _spacing(case):
    """The domain is the unit square on any grid, so dx and dy differ where Nx and Ny do."""
    return 1.0 / (case["Nx"] - 1), 1.0 / (case["Ny"] - 1)


def _model(seed):
    """A matrix of density and viscosity 1 under a sticky-air layer, with one to three light circular bodies that touch
    only the matrix: the materials of the batching and serving workloads."""
    r = random.Random("model %d" % seed)
    bodies = []
    for _ in range(r.randint(1, 3)):
        rad, rho, mu = r.uniform(0.05, 0.2), r.uniform(0.75, 0.9), 10.0 ** r.uniform(-1.0, 0.5)
        for _ in range(50):
            cx, cy = r.uniform(0.25, 0.75), r.uniform(0.2 + rad, 0.95 - rad)
            if all(math.hypot(cx - x, cy - y) >= rad + q + 0.03 for x, y, q, _, _ in bodies):
                bodies.append((cx, cy, rad, rho, mu))
                break
    return dict(air=0.1, rho_air=1e-3, mu_air=2e-2, bodies=bodies)


def _materials(m, x, y, h):
    """(rho, mu) at positions x, y; h > 0 blends a body's edge over a cell, as averaging markers onto nodes does."""
    def mix(old, new, f):
        return old + (new - old) * f
    rho, mu = torch.ones_like(x), torch.ones_like(x)
    for cx, cy, rad, r, v in m["bodies"]:
        d = rad - torch.sqrt((x - cx) ** 2 + (y - cy) ** 2)
        f = (d / h + 0.5).clamp(0, 1) if h > 0 else (d > 0).to(x.dtype)
        rho, mu = mix(rho, torch.full_like(x, r), f), mix(mu, torch.full_like(x, v), f)
    d = m["air"] - y
    f = (d / h + 0.5).clamp(0, 1) if h > 0 else (d > 0).to(x.dtype)
    return mix(rho, torch.full_like(x, m["rho_air"]), f), mix(mu, torch.full_like(x, m["mu_air"]), f)


def _nodes(nx, ny, x0, y0, dx, dy, dev):
    x = x0 + dx * torch.arange(nx, dtype=torch.float64, device=dev)
    y = y0 + dy * torch.arange(ny, dtype=torch.float64, device=dev)
    return x[None, :].expand(ny, nx), y[:, None].expand(ny, nx)


def _stokes_inputs(Nx, Ny, dx, dy, seed, dev):
    """rho_vy, mu_b, mu_p, and a smooth velocity and pressure to warm-start from, as (ny, nx) row-major tensors
    (the transposes are the framework's column-major (nx, ny) arrays), and the dt of that velocity."""
    m, h = _model(seed), max(dx, dy)
    rho = _materials(m, *_nodes(Nx + 1, Ny, -0.5 * dx, 0.0, dx, dy, dev), h)[0]
    mub = _materials(m, *_nodes(Nx, Ny, 0.0, 0.0, dx, dy, dev), h)[1]
    mup = _materials(m, *_nodes(Nx - 1, Ny - 1, 0.5 * dx, 0.5 * dy, dx, dy, dev), h)[1]
    r = random.Random("flow %d" % seed)
    vx = torch.zeros(Ny + 1, Nx, dtype=torch.float64, device=dev)
    vy = torch.zeros(Ny, Nx + 1, dtype=torch.float64, device=dev)
    for k, l in ((1, 1), (2, 1), (1, 2)):   # free-slip modes of a stream function: no flow through the sides
        a = 0.01 * r.uniform(-1, 1)
        x, y = _nodes(Nx, Ny + 1, 0.0, -0.5 * dy, dx, dy, dev)
        vx += a * l * torch.sin(math.pi * k * x) * torch.cos(math.pi * l * y)
        x, y = _nodes(Nx + 1, Ny, -0.5 * dx, 0.0, dx, dy, dev)
        vy -= a * k * torch.cos(math.pi * k * x) * torch.sin(math.pi * l * y)
    vx[:, 0] = 0.0
    vx[:, -1] = 0.0
    vy[0] = 0.0
    vy[-1] = 0.0
    _, yp = _nodes(Nx - 1, Ny - 1, 0.5 * dx, 0.5 * dy, dx, dy, dev)
    P = (0.9 * G_Y * (yp - m["air"]).clamp(min=0.0)).contiguous()
    dt = 0.5 * MAXDISP * min(dx / float(vx.abs().max()), dy / float(vy.abs().max()))
    return dict(rho_vy=rho.contiguous(), mu_b=mub.contiguous(), mu_p=mup.contiguous(), Vx_s=vx, Vy_s=vy, P=P), dt


def _markers(case, seed, dev, moved=True):
    """md x md markers per cell, jittered, and moved along by a flow over several cells (a run's markers leave
    their initial order); rho and mu of the material that they carry."""
    Nx, Ny, md = case["Nx"], case["Ny"], case["md"]
    dx, dy = _spacing(case)
    nx, ny = md * (Nx - 1), md * (Ny - 1)
    g = torch.Generator(device=dev).manual_seed(int(seed))
    x = ((torch.arange(nx, dtype=torch.float64) + 0.5) * (dx / md)).to(dev)[:, None].expand(nx, ny).reshape(-1)
    y = ((torch.arange(ny, dtype=torch.float64) + 0.5) * (dy / md)).to(dev)[None, :].expand(nx, ny).reshape(-1)
    x = x + (torch.rand(nx * ny, dtype=torch.float64, generator=g, device=dev) - 0.5) * (0.5 * dx / md)
    y = y + (torch.rand(nx * ny, dtype=torch.float64, generator=g, device=dev) - 0.5) * (0.5 * dy / md)
    rho, mu = _materials(_model(seed), x, y, 0.0)
    if moved:
        s = 4.0 * max(dx, dy)
        x, y = (x + s * torch.sin(math.pi * x) * torch.cos(2 * math.pi * y),
                y - 0.5 * s * torch.cos(math.pi * x) * torch.sin(2 * math.pi * y))
        x, y = x.clamp(0.0, 1.0), y.clamp(0.0, 1.0)
    return x.contiguous(), y.contiguous(), rho.contiguous(), mu.contiguous()


def _velocity(case, seed, dev):
    """Padded Vx (Nx+2, Ny+1) and Vy (Nx+1, Ny+2) of a circulating flow, as row-major tensors."""
    Nx, Ny = case["Nx"], case["Ny"]
    dx, dy = _spacing(case)
    r = random.Random("velocity %d" % seed)
    x, y = _nodes(Nx + 2, Ny + 1, -dx, -0.5 * dy, dx, dy, dev)
    vx = torch.zeros_like(x, memory_format=torch.contiguous_format)
    xv, yv = _nodes(Nx + 1, Ny + 2, -0.5 * dx, -dy, dx, dy, dev)
    vy = torch.zeros_like(xv, memory_format=torch.contiguous_format)
    for k, l in ((1, 1), (2, 3)):
        a = r.uniform(0.5, 1.0)
        vx += a * l * torch.sin(math.pi * k * x) * torch.cos(math.pi * l * y)
        vy -= a * k * torch.cos(math.pi * k * xv) * torch.sin(math.pi * l * yv)
    dt = MAXDISP * min(dx / float(vx.abs().max()), dy / float(vy.abs().max()))
    return vx, vy, dt


STATE = ("P", "Vx_s", "Vy_s")


def _batch_sizes(case, seed):
    r = random.Random("batch %d %d %d" % (case["n"], case["lo"], case["hi"]))   # the sizes belong to the case
    return [(_log_int(r, case["lo"], case["hi"]), _log_int(r, case["lo"], case["hi"]), seed * 1000 + k)
            for k in range(case["n"])]


def _problem_state(sf, Nx, Ny, seed, dev):
    """One Stokes problem as a program holds it: parameter arrays, state arrays and the values they start from."""
    dx, dy = 1.0 / (Nx - 1), 1.0 / (Ny - 1)
    inp, dt = _stokes_inputs(Nx, Ny, dx, dy, seed, dev)
    a = dict(rho_vy=inp["rho_vy"].t(), mu_b=inp["mu_b"].t(), mu_p=inp["mu_p"].t())
    for k in STATE:
        a[k] = inp[k].clone().t()
    a["Vx_pad"], a["Vy_pad"] = sf.zeros(Nx + 2, Ny + 1), sf.zeros(Nx + 1, Ny + 2)
    a["dVxdt"], a["dVydt"] = sf.zeros(Nx - 2, Ny - 1), sf.zeros(Nx - 1, Ny - 2)
    return dict(Nx=Nx, Ny=Ny, dx=dx, dy=dy, dt=dt, a=a, start={k: inp[k].t() for k in STATE})


def _restart(p):
    """The state back to where this pass's solve starts."""
    for k, v in p["start"].items():
        p["a"][k].copy_(v)
    p["a"]["dVxdt"].zero_()
    p["a"]["dVydt"].zero_()


SOLVE_OUT = ("P", "Vx_pad", "Vy_pad", "dVxdt", "dVydt", "Vx_s", "Vy_s")
WORK = ("txx", "tyy", "txy", "divV", "dtPt", "Rx", "Ry", "dtVx", "dtVy")


def prepare(case, seed):
    import stokesflow_b200 as sf
    dev = torch.device("cuda")
    kind = case["kind"]
    st = dict(case=case, kind=kind, sf=sf)
    if kind in ("solve", "mixed"):
        Nx, Ny = case["Nx"], case["Ny"]
        st["p"] = p = _problem_state(sf, Nx, Ny, seed, dev)
        if kind == "solve":
            shapes = dict(txx=(Nx - 1, Ny - 1), tyy=(Nx - 1, Ny - 1), txy=(Nx, Ny), divV=(Nx - 1, Ny - 1),
                          dtPt=(Nx - 1, Ny - 1), Rx=(Nx - 2, Ny - 1), Ry=(Nx - 1, Ny - 2), dtVx=(Nx - 2, Ny - 1),
                          dtVy=(Nx - 1, Ny - 2))
            p["work"] = {k: sf.zeros(*shapes[k]) if case["work"] else None for k in WORK}
    elif kind == "batch":
        st["ps"] = [_problem_state(sf, Nx, Ny, s, dev) for Nx, Ny, s in _batch_sizes(case, seed)]
    elif kind == "deposit":
        Nx, Ny = case["Nx"], case["Ny"]
        st["m"] = _markers(case, seed, dev)
        st["grids"] = [sf.zeros(Nx + 1, Ny), sf.zeros(Nx, Ny), sf.zeros(Nx - 1, Ny - 1)]
    elif kind == "move":
        x, y, _, _ = _markers(case, seed, dev)
        vx, vy, dt = _velocity(case, seed, dev)
        st.update(x=x.clone(), y=y.clone(), x0=x, y0=y, Vx=vx.t(), Vy=vy.t(), dt=dt)
    else:
        Nx, Ny = case["Nx"], case["Ny"]
        model = sf.plume_model_unit_square()
        s = sf.StokesFlow2D(Nx, Ny, 1.0, 1.0, model, marker_density=case["md"], stokes_eps=EPS,
                            iter_max=case["iters"], rebin=True)
        x, y, rho, mu = _markers(case, seed, dev)
        s.rho_m.copy_(rho)
        s.mu_m.copy_(mu)
        inp, dt = _stokes_inputs(Nx, Ny, s.dx, s.dy, seed, dev)
        st.update(s=s, x0=x, y0=y, dt=dt, start={k: inp[k].t() for k in STATE})
    return st


def run(st):
    sf, case, kind = st["sf"], st["case"], st["kind"]
    if kind == "solve":
        p, w = st["p"], st["p"]["work"]
        a = p["a"]
        _restart(p)
        info = sf.solve_stokes_info(a["P"], a["Vx_pad"], a["Vy_pad"], a["rho_vy"], a["mu_b"], a["mu_p"], w["txx"],
                                    w["tyy"], w["txy"], w["divV"], w["dtPt"], w["Rx"], w["Ry"], a["dVxdt"], a["dVydt"],
                                    w["dtVx"], w["dtVy"], a["Vx_s"], a["Vy_s"], G_Y, p["dx"], p["dy"], p["Nx"],
                                    p["Ny"], p["dt"], MAXDISP, use_free_surface_stabilization=case["stab"], eps=EPS,
                                    iter_max=case["iters"])
        out = {k: a[k] for k in SOLVE_OUT}
        out.update({k: v for k, v in w.items() if v is not None})
        out.update(dt=float(info["dt"]), err=float(info["err"]), iters=int(info["iters"]))
        return out
    if kind in ("mixed", "batch"):
        ps = st["ps"] if kind == "batch" else [st["p"]]
        for p in ps:
            _restart(p)
        problems = [sf.MixedProblem(p["a"]["P"], p["a"]["Vx_pad"], p["a"]["Vy_pad"], p["a"]["rho_vy"], p["a"]["mu_b"],
                                    p["a"]["mu_p"], p["a"]["Vx_s"], p["a"]["Vy_s"], G_Y, p["dx"], p["dy"], p["Nx"],
                                    p["Ny"], p["dt"], MAXDISP, eps=EPS, dVxdt=p["a"]["dVxdt"], dVydt=p["a"]["dVydt"])
                    for p in ps]
        res = sf.solve_stokes_batch_mixed(problems, options=sf.mixed_options(max_sweeps=case["iters"]))
        names = SOLVE_OUT if kind == "mixed" else ("P", "Vx_pad", "Vy_pad")
        outs = [dict({k: p["a"][k] for k in names}, iters=int(r["inner_iters"])) for p, r in zip(ps, res)]
        # a batch's outputs whole, one array for each of its kinds
        return outs[0] if kind == "mixed" else _batch_out(outs)
    if kind == "deposit":
        dx, dy = _spacing(case)
        x, y, rho, mu = st["m"]
        g = st["grids"]
        sf.bilinear_marker_to_grids([(-0.5 * dx, 0.0, g[0], rho), (0.0, 0.0, g[1], mu), (0.5 * dx, 0.5 * dy, g[2], mu)],
                                    x, y, dx, dy)
        return dict(rho_vy=g[0], mu_b=g[1], mu_p=g[2])
    if kind == "move":
        dx, dy = _spacing(case)
        st["x"].copy_(st["x0"])
        st["y"].copy_(st["y0"])
        sf.move_markers_rk4(st["x"], st["y"], st["Vx"], st["Vy"], -dx, -0.5 * dy, -0.5 * dx, -dy, st["dt"], 1.0, 1.0, dx,
                            dy)
        counts, offsets, perm = sf.rebin_markers(st["x"], st["y"], 0.0, 0.0, dx, dy, case["Nx"], case["Ny"])
        return dict(x=st["x"], y=st["y"], counts=counts, offsets=offsets, perm=perm)
    s = st["s"]
    s.x_m.copy_(st["x0"])
    s.y_m.copy_(st["y0"])
    for k, v in st["start"].items():
        getattr(s, k).copy_(v)
    s.dVxdt.zero_()
    s.dVydt.zero_()
    s.dt = st["dt"]
    rec = s.step()
    return dict(P=s.P, Vx=s.Vx, Vy=s.Vy, rho_vy=s.rho_vy, mu_b=s.mu_b, mu_p=s.mu_p, x=s.x_m, y=s.y_m, counts=s.counts,
                dt=float(rec["dt"]), iters=int(rec["info"]["iters"]))


def _batch_out(outs):
    out = {k: torch.cat([o[k].t().reshape(-1) for o in outs]) for k in outs[0] if k != "iters"}
    out["iters"] = sum(o["iters"] for o in outs)
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
SOLVE_FLOPS = 62     # FP64 operations of one pseudo-transient iteration per point


def work(case):
    kind = case["kind"]
    if kind == "batch":
        pts = sum(nx * ny for nx, ny, _ in _batch_sizes(case, 0))
        return dict(bytes=8 * 9 * pts, flops=SOLVE_FLOPS * pts * case["iters"])
    pts = case["Nx"] * case["Ny"]
    if kind in ("solve", "mixed"):
        # in: P, Vx, Vy, rho, mu_b, mu_p, 2 rates; out: P, Vx, Vy, their padded copies, 2 rates
        return dict(bytes=8 * (15 + (9 if case.get("work") else 0)) * pts, flops=SOLVE_FLOPS * pts * case["iters"])
    nm = case["md"] ** 2 * (case["Nx"] - 1) * (case["Ny"] - 1)
    if kind == "deposit":
        return dict(bytes=4 * 8 * nm + 3 * 8 * pts, flops=3 * 24 * nm)
    if kind == "move":
        return dict(bytes=(4 * 8 + 4) * nm + (2 * 8 + 2 * 4) * pts, flops=480 * nm)
    return dict(bytes=6 * 8 * nm + 8 * 15 * pts, flops=SOLVE_FLOPS * pts * case["iters"] + (3 * 24 + 480) * nm)


# ---------------------------------------------------------------------------
# the same results in plain torch
# ---------------------------------------------------------------------------
def _exact_solve(inp, dt, Nx, Ny, dx, dy, iters, stab, want_work=False):
    """`iters` damped pseudo-transient iterations of the staggered-grid Stokes equations with free-slip sides, on
    row-major (y, x) arrays."""
    rho, mub, mup = inp["rho_vy"], inp["mu_b"], inp["mu_p"]
    P, Vx, Vy = inp["P"].clone(), inp["Vx_s"].clone(), inp["Vy_s"].clone()
    dev = P.device
    dVx = torch.zeros(Ny - 1, Nx - 2, dtype=torch.float64, device=dev)
    dVy = torch.zeros(Ny - 2, Nx - 1, dtype=torch.float64, device=dev)
    h2, nmax, nmin = min(dx, dy) ** 2, max(Nx, Ny), min(Nx, Ny)
    dtP = 0.5 * 4.1 * mup / nmax
    dtVx = 0.45 * h2 / (0.5 * (mup[:, 1:] + mup[:, :-1])) / 4.1
    dtVy = 0.45 * h2 / (0.5 * (mup[1:] + mup[:-1])) / 4.1
    ncheck, ndt = min(5 * nmin, 2000), 10 * nmin
    dt = dt if stab else 0.0
    drx = 0.5 / dx * (rho[1:-1, 2:] - rho[1:-1, :-2])
    dry = 0.5 / dy * (rho[2:, 1:-1] - rho[:-2, 1:-1])
    err, w = 0.0, {}

    def cfl():
        return MAXDISP * min(dx / float(Vx.abs().max()), dy / float(Vy.abs().max()))

    def residual_y(tyy, txy, P, Vx, Vy, dt):
        r = (tyy[1:] - tyy[:-1] - P[1:] + P[:-1]) / dy + (txy[1:-1, 1:] - txy[1:-1, :-1]) / dx
        if dt != 0.0:
            av = 0.25 * (Vx[1:-2, :-1] + Vx[1:-2, 1:] + Vx[2:-1, :-1] + Vx[2:-1, 1:])
            return r + G_Y * (rho[1:-1, 1:-1] - dt * (av * drx + Vy[1:-1, 1:-1] * dry))
        return r + G_Y * rho[1:-1, 1:-1]

    for it in range(1, iters + 1):
        ex = (Vx[1:-1, 1:] - Vx[1:-1, :-1]) / dx
        ey = (Vy[1:, 1:-1] - Vy[:-1, 1:-1]) / dy
        div = ex + ey
        P = P - dtP * div
        txx, tyy = 2.0 * mup * (ex - div / 3.0), 2.0 * mup * (ey - div / 3.0)
        txy = mub * ((Vx[1:] - Vx[:-1]) / dy + (Vy[:, 1:] - Vy[:, :-1]) / dx)
        sx = txx - P
        Rx = (sx[:, 1:] - sx[:, :-1]) / dx + (txy[1:, 1:-1] - txy[:-1, 1:-1]) / dy
        Ry = residual_y(tyy, txy, P, Vx, Vy, dt)
        dVx = (1.0 - 4.0 / Nx) * dVx + Rx
        dVy = (1.0 - 4.0 / Ny) * dVy + Ry
        Vx, Vy = Vx.clone(), Vy.clone()
        Vx[1:-1, 1:-1] += dtVx * dVx
        Vy[1:-1, 1:-1] += dtVy * dVy
        Vx[:, 0] = 0.0
        Vx[:, -1] = 0.0
        Vy[0] = 0.0
        Vy[-1] = 0.0
        Vx[0], Vx[-1] = Vx[1], Vx[-2]
        Vy[:, 0], Vy[:, -1] = Vy[:, 1], Vy[:, -2]
        if stab and it % ndt == 0:
            dt = cfl()
        if it % ncheck == 0:
            Ry = residual_y(tyy, txy, P, Vx, Vy, cfl() if stab else 0.0)
            err = max(float(t.abs().mean()) for t in (Rx, Ry, div))
            w = dict(Rx=Rx, Ry=Ry)
        if it == iters:
            w.update(txx=txx, tyy=tyy, txy=txy, divV=div)
    Vx_pad = torch.cat([-Vx[:, 1:2], Vx, -Vx[:, -2:-1]], dim=1)
    Vy_pad = torch.cat([-Vy[1:2], Vy, -Vy[-2:-1]], dim=0)
    out = dict(P=P, Vx_pad=Vx_pad, Vy_pad=Vy_pad, dVxdt=dVx, dVydt=dVy, Vx_s=Vx, Vy_s=Vy)
    if want_work:
        out.update(w, dtPt=dtP, dtVx=dtVx, dtVy=dtVy)
    out = {k: v.t() for k, v in out.items()}
    return out, cfl(), err


def _exact_deposit(x, y, val, x0, y0, dx, dy, nx, ny):
    qx, qy = torch.floor((x - x0) / dx), torch.floor((y - y0) / dy)
    ok = (qx >= -1) & (qx <= nx - 1) & (qy >= -1) & (qy <= ny - 1)
    fx, fy = (x - (x0 + qx * dx)) / dx, (y - (y0 + qy * dy)) / dy
    ix, iy = qx.long() + 1, qy.long() + 1          # padded by one node on the low sides
    s = torch.zeros((ny + 2) * (nx + 2), dtype=torch.float64, device=x.device)
    w = torch.zeros_like(s)
    for a in (0, 1):
        for b in (0, 1):
            wt = (fx if a else 1 - fx) * (fy if b else 1 - fy) * ok
            k = ((iy + b) * (nx + 2) + ix + a).clamp(0, s.numel() - 1)
            w.index_add_(0, k, wt)
            s.index_add_(0, k, wt * val)
    s, w = s.view(ny + 2, nx + 2)[1:-1, 1:-1], w.view(ny + 2, nx + 2)[1:-1, 1:-1]
    return torch.where(w != 0, s / torch.where(w != 0, w, torch.ones_like(w)), torch.zeros_like(s))


def _exact_interp(V, x, y, x0, y0, dx, dy, along_x):
    """Bilinear interpolation of row-major V with the quadratic continuity correction along the component's axis."""
    ny, nx = V.shape
    i, j = torch.floor((x - x0) / dx), torch.floor((y - y0) / dy)
    fx, fy = (x - (x0 + i * dx)) / dx, (y - (y0 + j * dy)) / dy
    i, j = i.long(), j.long()

    def at(a, b):
        return V[j + b, i + a]
    v = (1 - fx) * (1 - fy) * at(0, 0) + fx * (1 - fy) * at(1, 0) + (1 - fx) * fy * at(0, 1) + fx * fy * at(1, 1)
    f, g = (fx, fy) if along_x else (fy, fx)
    s = torch.where(f >= 0.5, 1, 0)      # centre of the second difference: this node or the next

    def bend(side):
        if along_x:
            return V[j + side, i + s - 1] - 2 * V[j + side, i + s] + V[j + side, i + s + 1]
        return V[j + s - 1, i + side] - 2 * V[j + s, i + side] + V[j + s + 1, i + side]
    return v + 0.5 * (f - 0.5) ** 2 * ((1 - g) * bend(0) + g * bend(1))


def _exact_move(x, y, Vx, Vy, dt, dx, dy):
    out_x, out_y = torch.empty_like(x), torch.empty_like(y)
    for c in range(0, x.numel(), 1 << 22):
        xs, ys = x[c:c + (1 << 22)], y[c:c + (1 << 22)]
        ex = ey = kx = ky = torch.zeros_like(xs)
        for a, b in ((0.0, 1 / 6), (0.5, 1 / 3), (0.5, 1 / 3), (1.0, 1 / 6)):
            px, py = xs + a * dt * kx, ys + a * dt * ky
            kx = _exact_interp(Vx, px, py, -dx, -0.5 * dy, dx, dy, True)
            ky = _exact_interp(Vy, px, py, -0.5 * dx, -dy, dx, dy, False)
            ex, ey = ex + b * kx, ey + b * ky
        out_x[c:c + (1 << 22)] = (xs + ex * dt).clamp(0.0, 1.0)
        out_y[c:c + (1 << 22)] = (ys + ey * dt).clamp(0.0, 1.0)
    return out_x, out_y


def exact(case, seed):
    dev, kind = _device(), case["kind"]
    if kind == "batch":
        if case["n"] * case["iters"] > 33_000 or dev.type == "cpu":
            return None
    elif kind != "deposit" and kind != "move":
        # point iterations that plain torch does within the time this may take
        if case["Nx"] * case["Ny"] * case["iters"] > (9e9 if dev.type == "cuda" else 1.5e8):
            return None
    if kind in ("solve", "mixed"):
        Nx, Ny = case["Nx"], case["Ny"]
        dx, dy = _spacing(case)
        inp, dt = _stokes_inputs(Nx, Ny, dx, dy, seed, dev)
        out, dt, err = _exact_solve(inp, dt, Nx, Ny, dx, dy, case["iters"], case.get("stab", True),
                                    case.get("work", False))
        return dict(out, iters=None) if kind == "mixed" else dict(out, dt=dt, err=err, iters=None)
    if kind == "batch":
        outs = []
        for Nx, Ny, s in _batch_sizes(case, seed):
            dx, dy = 1.0 / (Nx - 1), 1.0 / (Ny - 1)
            inp, dt = _stokes_inputs(Nx, Ny, dx, dy, s, dev)
            o = _exact_solve(inp, dt, Nx, Ny, dx, dy, case["iters"], True)[0]
            outs.append(dict(P=o["P"], Vx_pad=o["Vx_pad"], Vy_pad=o["Vy_pad"], iters=0))
        return dict(_batch_out(outs), iters=None)
    dx, dy = _spacing(case)
    Nx, Ny = case["Nx"], case["Ny"]
    x, y, rho, mu = _markers(case, seed, dev)
    if kind == "move":
        vx, vy, dt = _velocity(case, seed, dev)
        x, y = _exact_move(x, y, vx, vy, dt, dx, dy)
        return dict(x=x, y=y, counts=None, offsets=None, perm=None)
    g = [_exact_deposit(x, y, rho, -0.5 * dx, 0.0, dx, dy, Nx + 1, Ny),
         _exact_deposit(x, y, mu, 0.0, 0.0, dx, dy, Nx, Ny),
         _exact_deposit(x, y, mu, 0.5 * dx, 0.5 * dy, dx, dy, Nx - 1, Ny - 1)]
    if kind == "deposit":
        return dict(rho_vy=g[0].t(), mu_b=g[1].t(), mu_p=g[2].t())
    inp, dt = _stokes_inputs(Nx, Ny, dx, dy, seed, dev)
    inp.update(rho_vy=g[0], mu_b=g[1], mu_p=g[2])
    out, dt, _ = _exact_solve(inp, dt, Nx, Ny, dx, dy, case["iters"], True)
    x, y = _exact_move(x, y, out["Vx_pad"].t(), out["Vy_pad"].t(), dt, dx, dy)
    return dict(P=out["P"], Vx=out["Vx_pad"], Vy=out["Vy_pad"], rho_vy=g[0].t(), mu_b=g[1].t(), mu_p=g[2].t(), x=x, y=y,
                counts=None, dt=dt, iters=None)
