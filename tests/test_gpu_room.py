"""Resident tiles that fill the device give way to other work, in the middle of a solve too, and come back after it; the
results are those of a solve by itself.  Where a solve ran shows in its launches of iterations: one per hundreds of them
with tiles, one per two or three without."""
import threading
import time

import numpy as np
import pytest

from fields import random_fields

pytestmark = pytest.mark.gpu

STATE = {"P": (-1, -1), "Vx": (2, 1), "Vy": (1, 2), "dVxdt": (-2, -1), "dVydt": (-1, -2), "Vx_s": (0, 1), "Vy_s": (1, 0)}


class Solve:
    def __init__(self, sf, Nx, Ny):
        import torch

        from test_gpu_parity import dev
        self.sf, self.Nx, self.Ny, self.ctx, self.stream = sf, Nx, Ny, sf.Context(0), torch.cuda.Stream()
        self.par = [dev(a) for a in random_fields(Nx, Ny, seed=Nx, contrast=5.0)]
        torch.cuda.synchronize()

    def __call__(self, iters):
        import torch

        sf, Nx, Ny = self.sf, self.Nx, self.Ny
        with torch.cuda.stream(self.stream):
            t = {k: sf.zeros(Nx + a, Ny + b) for k, (a, b) in STATE.items()}
            info = sf.solve_stokes_info(t["P"], t["Vx"], t["Vy"], *self.par, *[None] * 7, t["dVxdt"], t["dVydt"], None, None,
                                        t["Vx_s"], t["Vy_s"], 9.81, 1 / (Nx - 1), 1 / (Ny - 1), Nx, Ny, 1e-3, 0.5, eps=1e-300,
                                        iter_max=iters, ctx=self.ctx)
            return {k: v.cpu().numpy() for k, v in t.items()}, info["fused_launches"]


def mixed(sf, n, sweeps):
    from test_gpu_parity import dev
    par = [dev(a) for a in random_fields(n, n, seed=n, contrast=5.0)]
    z = {k: sf.zeros(n + a, n + b) for k, (a, b) in STATE.items()}
    p = sf.MixedProblem(z["P"], z["Vx"], z["Vy"], *par, z["Vx_s"], z["Vy_s"], 9.81, 1 / (n - 1), 1 / (n - 1), n, n, 1e-3, 0.5,
                        eps=1e-300, dVxdt=z["dVxdt"], dVydt=z["dVydt"])
    return p, sf.mixed_options(max_sweeps=sweeps)


@pytest.mark.parametrize("beside", ["batch", "engine", "rebin", "deposit_noalloc", "decomposed"])
def test_tiles_give_way_to_other_work(sf, beside):
    import torch

    from stokesflow_b200 import domains
    from test_gpu_parity import dev

    main = Solve(sf, 250, 240)               # tiles of whole SMs
    n = 20 * 1200                            # twenty checks
    want, alone = main(n)
    assert alone < n / 100
    stop, begun = threading.Event(), threading.Event()
    ctx = sf.Context(0)

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            if beside in ("rebin", "deposit_noalloc"):
                x = torch.rand(200_000, dtype=torch.float64, device="cuda")
                out = sf.zeros(100, 100)

                def call():
                    if beside == "rebin":
                        sf.rebin_markers(x, x, 0.0, 0.0, 0.01, 0.01, 101, 101, ctx=ctx)
                    else:
                        sf.bilinear_marker_to_grid_noalloc(0.0, 0.0, out, x, x, x, 0.01, 0.01)
                    torch.cuda.current_stream().synchronize()
            elif beside == "decomposed":
                nloc = domains.local_size(2, 128)
                glob = {k: sf.zeros(128 + a, 100 + b) for k, (a, b) in domains.ARRAYS.items()}
                for k, a in zip(("rho_vy", "mu_b", "mu_p"), random_fields(128, 100, seed=1, contrast=5.0)):
                    glob[k] = dev(a)
                ranks = domains.split(glob, (2, 1), nloc, 100)
                ctxs = {c: sf.Context(0) for c in ranks}
                call = lambda: domains.solve_stokes_decomposed(  # noqa: E731
                    ranks, (2, 1), nloc, 100, 9.81, 1 / 127, 1 / 99, 1e-4, 0.5, eps=1e-300, iter_max=600, contexts=ctxs)
            else:
                p, opt = mixed(sf, 200, 3000)
                if beside == "batch":
                    call = lambda: sf.solve_stokes_batch_mixed([p], options=opt, ctx=ctx)  # noqa: E731
                else:
                    eng = sf.Engine(sf.Engine.instance_bytes(200, 200) + (1 << 20), 4, options=opt, ctx=ctx)

                    def call():
                        assert eng.submit(p) is not None
                        while eng.active:
                            eng.step()
            call()
            begun.set()
            while not stop.is_set():
                call()

    th = threading.Thread(target=work)
    th.start()
    try:
        assert begun.wait(60)
        got, shared = main(n)
    finally:
        stop.set()
        th.join()
    # two iterations per launch; at some checks the other thread may be between two calls
    assert shared > n / 4, "the tiles did not give way"
    time.sleep(0.02)
    again, after = main(n)
    assert after == alone, "the tiles did not come back"
    for k in want:
        assert np.array_equal(got[k], want[k]) and np.array_equal(again[k], want[k]), k


def test_tiles_give_way_in_the_middle_of_a_solve(sf):
    """A solve with whole-SM tiles, another plain solve during a part of it."""
    main, other = Solve(sf, 250, 240), Solve(sf, 64, 64)
    n = 240 * 5 * 60
    want, alone = main(n)
    small, _ = other(640)
    got, fails = [], []

    def beside():
        for _ in range(12):
            r, _ = other(640)
            if not all(np.array_equal(r[k], small[k]) for k in r):
                fails.append(r)

    th = threading.Thread(target=lambda: got.append(main(n)))
    th.start()
    time.sleep(0.02)
    b = threading.Thread(target=beside)
    b.start()
    b.join()
    th.join()
    state, launches = got[0]
    assert not fails
    for k in want:
        assert np.array_equal(state[k], want[k]), k
    assert alone + 100 < launches < n / 4, (alone, launches)   # a part of it with tiles, a part without
