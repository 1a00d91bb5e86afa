"""RK4 advection where its code path changes: markers on and around cell edges, in the outermost cells (index failsafes),
outside the domain, NaN and infinite, closer to a node than 2^-895, and spacings that the constant division does not take.
Against the oracle, bit for bit, with the failsafe count.  Markers that are not finite have no reference (Julia's
floor(Int, x) throws, C leaves the conversion undefined): they are compared with the same call on coordinates and
velocities times 2^70 or 2^-70, which takes the general code and scales every result exactly."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny,scale", [(4, 4, 1.0), (37, 21, 1.0), (64, 80, 3.7e5), (33, 33, 2.0 ** -70), (20, 26, 2.0 ** 70)])
def test_advection_edges(sf, oracle_lib, Nx, Ny, scale):
    O = oracle_lib
    rng = np.random.default_rng(Nx * Ny)
    Lx, Ly = scale, 1.3 * scale
    dx, dy = Lx / (Nx - 1), Ly / (Ny - 1)
    Vx = np.asfortranarray(rng.normal(size=(Nx + 2, Ny + 1)))
    Vy = np.asfortranarray(rng.normal(size=(Nx + 1, Ny + 2)))
    k = np.arange(-2, 2 * Nx + 3) * 0.5 * dx
    edges = np.concatenate([k, np.nextafter(k, -np.inf), np.nextafter(k, np.inf)])
    x = np.concatenate([rng.random(5000) * Lx, edges, [0.0, Lx, 1e-300, 2.0 ** -1000, -0.0, 1e300, -1e300]])
    y = np.concatenate([rng.random(x.size - 9) * Ly, [0.0, Ly, 1e-300, -0.0, Ly / 2, 0.5 * dy, 1.5 * dy, 1e300, -1e300]])
    bad = np.array([np.nan, np.inf, -np.inf, 0.3 * Lx, 0.3 * Lx, 0.3 * Lx])
    x, y = np.concatenate([x, bad]), np.concatenate([y, bad[::-1]])
    dt = 0.4 * min(dx, dy) / np.abs(Vx).max()
    o = O.node_origins(dx, dy)
    args = (o["x_vx"], o["y_vx"], o["x_vy"], o["y_vy"], dt, Lx, Ly, dx, dy)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda().t()  # noqa: E731

    def move(s, x, y):
        tx, ty = torch.from_numpy(x * s).cuda(), torch.from_numpy(y * s).cuda()
        sf.get_warnings(reset=True)
        sf.move_markers_rk4(tx, ty, dev(Vx * s), dev(Vy * s), *(a if i == 4 else a * s for i, a in enumerate(args)))
        return tx.cpu().numpy(), ty.cpu().numpy(), sf.get_warnings(reset=True)["interp_failsafe"]

    finite = np.isfinite(x) & np.isfinite(y)
    gx, gy, _ = move(1.0, x, y)
    s = 2.0 ** -70 if scale > 1e10 else 2.0 ** 70
    if 1e-10 < scale < 1e10:
        sx, sy, _ = move(s, x[~finite], y[~finite])
        assert np.array_equal(gx[~finite] * s, sx, equal_nan=True) and np.array_equal(gy[~finite] * s, sy, equal_nan=True)
    fx, fy, fails = move(1.0, x[finite], y[finite])
    ox, oy = x[finite].copy(), y[finite].copy()
    n = O.move_markers_rk4(ox, oy, Vx, Vy, *args)
    assert np.array_equal(fx, ox) and np.array_equal(fy, oy) and fails == n
    assert np.array_equal(gx[finite], fx) and np.array_equal(gy[finite], fy)
