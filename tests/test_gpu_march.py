"""Several PT iterations per launch (sf_march.cu) against the oracle, bit for bit, at the sizes where its split into
strips of columns and segments of rows changes: the smallest grids, the widest grid of one strip (59 points) and its
neighbours, odd strip widths, several strips, segments of two rows and of many, and iteration counts that leave one
and two iterations over.  No tolerance: every expression is evaluated in the reference's order."""
import numpy as np
import pytest

from fields import random_fields
from test_gpu_parity import NAMES, gpu_solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny,iters,stab", [
    (4, 4, 60, True), (5, 9, 61, True), (9, 5, 62, False), (58, 21, 230, True), (59, 22, 231, True), (60, 23, 232, True),
    (61, 4, 61, True), (113, 30, 320, True), (114, 31, 321, True), (171, 7, 150, True), (20, 700, 260, True),
    (233, 129, 700, True), (300, 301, 500, False), (700, 61, 700, True), (801, 903, 94, True)])
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
