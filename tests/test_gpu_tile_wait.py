"""Resident tiles (sf_resident.cu) whose waits for one another run out: the solve begins again without them, from the
caller's arrays, and ends as if nothing had been.  The first launch goes without its last tile, so that the waits for it
give up after a short budget (tiles of a cluster: the launch counts as given up); nothing faults."""
import time

import numpy as np
import pytest

from fields import random_fields
from test_gpu_parity import NAMES, gpu_solve

pytestmark = pytest.mark.gpu


# one cluster, tiles of two quarters of an SM and of whole SMs; the last iteration with a check and without one
@pytest.mark.parametrize("Nx,Ny,iters", [(20, 26, 300), (20, 26, 257), (150, 131, 1310), (150, 131, 900), (400, 390, 500)])
def test_solve_begins_again_without_tiles(sf, oracle_lib, Nx, Ny, iters):
    O = oracle_lib
    dx, dy = 1.0 / (Nx - 1), 1.2 / (Ny - 1)
    a0 = O.stokes_arrays(Nx, Ny)
    a0["rho_vy"][:], a0["mu_b"][:], a0["mu_p"][:] = random_fields(Nx, Ny, seed=Nx, contrast=5.0)
    args = (9.81, dx, dy, Nx, Ny, 1e-3, 0.5, True, 1e-300, iters)
    copy = lambda: {k: v.copy(order="F") for k, v in a0.items()}
    want = copy()
    r = O.solve_stokes(want, *args)
    launches = []
    for lost in (False, True, False):
        if lost:
            sf.selftest_tile_wait(20_000_000)
        t0 = time.perf_counter()
        got, info = gpu_solve(sf, copy(), *args)
        assert not lost or time.perf_counter() - t0 < 1.9   # the product's budget is 2 s
        launches.append(info["fused_launches"])
        assert (info["iters"], info["dt"]) == (r.iters, r.dt)
        for k in NAMES:
            assert np.array_equal(got[k], want[k], equal_nan=True), f"{k} differs from the oracle (lost {lost})"
    # few launches of many iterations; where the tiles were lost, launches of at most three
    assert launches[0] == launches[2] < iters / 10 and launches[1] >= iters / 3


def test_budget_is_checked(sf):
    for bad in (0, 3_000_000_000):
        with pytest.raises(sf.StokesFlowError):
            sf.selftest_tile_wait(bad)
