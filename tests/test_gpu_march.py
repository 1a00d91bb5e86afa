"""Several PT iterations per launch against the oracle, bit for bit.  No tolerance: every expression is evaluated in
the reference's order.

* resident iterations (sf_resident.cu): the smallest grids, clusters of 1 to 16 tiles in rows, columns and blocks, both
  sides of the cluster's limit, ragged last tiles; the exchange through L2 with one to four points per thread, thin tiles
  with more halo slots than threads, the largest grid;
* the march (sf_march.cu), on grids beyond that, at the sizes where its split into strips of columns and segments of rows
  changes: the narrowest grids (one strip), odd strip widths, short and long segments, and iteration counts that leave one
  and two iterations over (the first ten and chunks of up to three iterations run on every grid)."""
import numpy as np
import pytest

from fields import random_fields
from test_gpu_parity import NAMES, dev, gpu_solve, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny,iters,stab", [
    # resident
    (7, 6, 61, True), (10, 9, 93, False), (4, 61, 61, True), (18, 33, 185, True), (85, 85, 851, True), (86, 86, 861, True),
    (100, 101, 501, True), (109, 108, 545, False), (110, 111, 551, True), (200, 50, 251, True), (9, 800, 91, True),
    (170, 40, 403, True), (6, 900, 62, False), (70, 5, 104, True), (1000, 5, 51, True), (1400, 4, 61, True),
    (4, 4, 60, True), (5, 9, 61, True), (9, 5, 62, False), (27, 31, 300, True), (28, 31, 301, True), (59, 22, 231, True),
    (61, 4, 61, True), (114, 31, 321, True), (20, 700, 260, True), (3000, 20, 230, True), (233, 129, 700, True),
    (300, 301, 500, False), (330, 330, 97, True), (511, 385, 94, True), (521, 520, 65, True),
    (522, 533, 61, True), (700, 400, 63, False), (550, 552, 61, True),
    # march
    (552, 551, 62, True), (58, 5400, 63, True), (59, 5400, 64, True), (60, 5300, 65, True), (5400, 60, 66, True),
    (20000, 17, 187, True), (801, 903, 94, False), (1023, 1101, 41, True)])
def test_march_bitexact(sf, oracle_lib, Nx, Ny, iters, stab):
    O = oracle_lib
    dx, dy = 1.0 / (Nx - 1), 1.2 / (Ny - 1)
    a = O.stokes_arrays(Nx, Ny)
    a["rho_vy"][:], a["mu_b"][:], a["mu_p"][:] = random_fields(Nx, Ny, seed=Nx + Ny, contrast=5.0)
    rng = np.random.default_rng(Nx * Ny)
    for k in ("P", "Vx_s", "Vy_s", "dVxdt", "dVydt"):   # the boundary entries of V among them
        a[k][:] = 1e-3 * rng.normal(size=a[k].shape)
    b, info = gpu_solve(sf, {k: v.copy(order="F") for k, v in a.items()}, 9.81, dx, dy, Nx, Ny, 1e-3, 0.5, stab, 1e-300,
                        iters)
    r = O.solve_stokes(a, 9.81, dx, dy, Nx, Ny, 1e-3, 0.5, stab, 1e-300, iters)
    assert info["iters"] == r.iters == iters
    assert info["dt"] == r.dt
    for k in NAMES:
        assert np.array_equal(b[k], a[k], equal_nan=True), f"{k} differs from the oracle"


@pytest.mark.parametrize("Nx,Ny,bad", [(20, 26, False), (150, 131, False), (20, 26, True), (150, 131, True)])
def test_resident_stops_where_the_loop_does(sf, oracle_lib, Nx, Ny, bad):
    """The iterations behind a check are launched before its result is known: a solve that converges there (or meets a
    NaN) ends with that check's state, and the same holds for the solve after it in the same context."""
    O = oracle_lib
    dx, dy = 1.0 / (Nx - 1), 1.0 / (Ny - 1)
    args = (9.81, dx, dy, Nx, Ny, 1e-3, 0.5, True)
    ncheck = 5 * min(Nx, Ny)
    a0 = O.stokes_arrays(Nx, Ny)
    a0["rho_vy"][:], a0["mu_b"][:], a0["mu_p"][:] = random_fields(Nx, Ny, seed=5, contrast=2.0)
    copy = lambda: {k: v.copy(order="F") for k, v in a0.items()}
    if bad:
        a0["rho_vy"][Nx // 2, Ny // 2] = np.nan
        eps, stop = 1e-300, ncheck
    else:
        eps, stop = O.solve_stokes(copy(), *args, 1e-300, 3 * ncheck).err * (1 + 1e-9), 3 * ncheck
    for iter_max in (10 * ncheck, 3 * ncheck + 7):
        a = copy()
        r = O.solve_stokes(a, *args, eps, iter_max)
        if bad:   # reported as an error; the state is in the arrays
            t = {k: dev(v) for k, v in copy().items()}
            with pytest.raises(sf.StokesFlowError, match="not finite"):
                sf.solve_stokes_info(*[t[k] for k in NAMES], *args[:7], eps=eps, iter_max=iter_max)
            b, iters = {k: host(v) for k, v in t.items()}, stop
        else:
            b, info = gpu_solve(sf, copy(), *args, eps, iter_max)
            iters = info["iters"]
            assert info["dt"] == r.dt
        assert iters == r.iters == stop
        for k in NAMES:
            assert np.array_equal(b[k], a[k], equal_nan=True), f"{k} differs from the oracle"


def test_solve_where_only_the_compact_layout_fits(sf):
    """Memory for 17 fields of the grid's size but not for 23: single iterations, the same results."""
    import torch

    Nx, Ny, iters = 1500, 1100, 25
    dx, dy = 1.0 / (Nx - 1), 1.0 / (Ny - 1)
    rho, mu_b, mu_p = random_fields(Nx, Ny, seed=11, contrast=5.0)
    shape = dict(P=(Nx - 1, Ny - 1), Vx=(Nx + 2, Ny + 1), Vy=(Nx + 1, Ny + 2), dVxdt=(Nx - 2, Ny - 1),
                 dVydt=(Nx - 1, Ny - 2), Vx_s=(Nx, Ny + 1), Vy_s=(Nx + 1, Ny))
    par, res = [dev(rho), dev(mu_b), dev(mu_p)], []
    held = None
    for short in (False, True):
        t, ctx = {k: sf.zeros(*v) for k, v in shape.items()}, sf.Context(0)
        if short:
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            field = ((Nx + 2 + 31) // 32 * 32) * (Ny + 5) * 8
            held = torch.empty(torch.cuda.mem_get_info()[0] - 20 * field, dtype=torch.uint8, device="cuda")
        sf.solve_stokes_info(t["P"], t["Vx"], t["Vy"], *par, *[None] * 7, t["dVxdt"], t["dVydt"], None, None, t["Vx_s"],
                             t["Vy_s"], 9.81, dx, dy, Nx, Ny, 1e-3, 0.5, eps=1e-300, iter_max=iters, ctx=ctx)
        scratch = ctx.scratch_bytes()
        del held
        held = None
        res.append(({k: host(v) for k, v in t.items()}, scratch))
        ctx = None
        torch.cuda.empty_cache()
    assert res[1][1] < 0.8 * res[0][1]
    for k in shape:
        assert np.array_equal(res[0][0][k], res[1][0][k]), f"{k} differs"


def test_concurrent_solves_bitexact(sf, oracle_lib):
    """Solves of several threads at once, contexts and streams of their own, more of them than the device has room for
    resident tiles (the rest marches), some of them small enough for a cluster: each equals the oracle."""
    import threading

    import torch

    O = oracle_lib
    n = 8
    shape = lambda k: (61, 47, 600) if k % 3 == 1 else (300, 260, 150)
    want, got = [], [None] * n
    for k in range(n):
        Nx, Ny, iters = shape(k)
        a = O.stokes_arrays(Nx, Ny)
        a["rho_vy"][:], a["mu_b"][:], a["mu_p"][:] = random_fields(Nx, Ny, seed=k, contrast=5.0)
        want.append(a)

    def one(k, a):
        Nx, Ny, iters = shape(k)
        dx, dy = 1.0 / (Nx - 1), 1.0 / (Ny - 1)
        with torch.cuda.stream(torch.cuda.Stream()):
            t = {q: dev(v) for q, v in a.items()}
            sf.solve_stokes_info(*[t[q] for q in NAMES], 9.81, dx, dy, Nx, Ny, 1e-3, 0.5, eps=1e-300, iter_max=iters,
                                 ctx=sf.Context(0))
            got[k] = {q: host(v) for q, v in t.items()}

    threads = [threading.Thread(target=one, args=(k, {q: v.copy(order="F") for q, v in a.items()}))
               for k, a in enumerate(want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, a in enumerate(want):
        Nx, Ny, iters = shape(k)
        dx, dy = 1.0 / (Nx - 1), 1.0 / (Ny - 1)
        O.solve_stokes(a, 9.81, dx, dy, Nx, Ny, 1e-3, 0.5, True, 1e-300, iters)
        for q in NAMES:
            assert np.array_equal(got[k][q], a[q]), f"solve {k}: {q} differs from the oracle"
