"""Which kernels a plain solve's iterations run: every rule that chooses falls back to another kernel with the same bits,
so the other tests would pass without the one they are meant for.  Launches of iterations (fused_launches): resident tiles
take all iterations up to the next check, dt update or 512 / 20000 of them; the march two or three, single ones where a
check follows; the compact layout one.  Memory: tiles that exchange through L2 have halo slots in the context's scratch,
tiles of one cluster have none."""
import pytest
import torch

from fields import random_fields
from test_gpu_parity import dev

pytestmark = pytest.mark.gpu

STATE = {"P": (-1, -1), "Vx": (2, 1), "Vy": (1, 2), "dVxdt": (-2, -1), "dVydt": (-1, -2), "Vx_s": (0, 1), "Vy_s": (1, 0)}
MB = 1 << 20


def launches(sf, Nx, Ny, iters):
    z = {k: sf.zeros(Nx + a, Ny + b) for k, (a, b) in STATE.items()}
    par = [dev(a) for a in random_fields(Nx, Ny, seed=1, contrast=5.0)]
    ctx = sf.Context(0)
    torch.cuda.synchronize()
    info = sf.solve_stokes_info(z["P"], z["Vx"], z["Vy"], *par, *[None] * 7, z["dVxdt"], z["dVydt"], None, None, z["Vx_s"],
                                z["Vy_s"], 9.81, 1 / (Nx - 1), 1 / (Ny - 1), Nx, Ny, 1e-3, 0.5, eps=1e-300, iter_max=iters,
                                ctx=ctx)
    fields = 23 * ((Nx + 2 + 31) // 32 * 32) * (Ny + 5) * 8
    extra = ctx.scratch_bytes() - (fields + MB - 1) // MB * MB - MB    # beyond the fields and the partial sums
    return info["fused_launches"], extra


def expected(n, per_launch, ncheck, ndt, resident):
    """Launches for n iterations: cut after iteration 10, at checks and dt updates; the march leaves the iteration before a
    check (or the end) to a launch of its own."""
    count, it = 0, 1
    while it <= n:
        last = min(((it - 1) // ncheck + 1) * ncheck, n)
        stop = min(last, ((it - 1) // ndt + 1) * ndt, 10 if it < 11 else n)
        if resident and stop - it + 1 >= 4:
            k = min(stop - it + 1, per_launch)
        elif it < last:
            k = min(3 if resident else per_launch, min(stop, last - 1) - it + 1)
        else:
            k = 1
        it += k
        count += 1
    return count


@pytest.mark.parametrize("Nx,Ny,kind,per_launch", [
    (4, 4, "cluster", 20000), (20, 26, "cluster", 20000), (85, 85, "cluster", 20000), (108, 108, "cluster", 20000),
    (170, 40, "cluster", 20000), (120, 120, "L2", 20000), (200, 150, "L2", 20000), (300, 301, "L2", 20000),
    (240, 240, "L2", 512), (511, 385, "L2", 512), (529, 529, "L2", 512),
    (601, 605, "march", 3), (58, 6400, "march", 3), (58, 5400, "march", 3), (551, 551, "march", 3), (1023, 1101, "march", 3), (20000, 18, "march", 3)])
def test_path_of_a_solve(sf, Nx, Ny, kind, per_launch):
    ncheck, ndt = min(5 * min(Nx, Ny), 2000), 10 * min(Nx, Ny)
    n = min(2 * ncheck + 17, 1200)
    got, extra = launches(sf, Nx, Ny, n)
    assert got == expected(n, per_launch, ncheck, ndt, kind != "march")
    assert (extra > 0) == (kind == "L2")


@pytest.mark.parametrize("Nx,Ny,per_launch", [(235, 230, 3), (250, 240, 2), (395, 400, 2), (402, 400, 3)])
def test_iterations_per_launch_where_tiles_are_lost(sf, Nx, Ny, per_launch):
    """The march of grids that have tiles: two iterations per launch between 240^2 and 400^2 points."""
    sf.selftest_tile_wait(1_000_000, ctx=sf.default_context())
    z = {k: sf.zeros(Nx + a, Ny + b) for k, (a, b) in STATE.items()}
    par = [dev(a) for a in random_fields(Nx, Ny, seed=1, contrast=5.0)]
    info = sf.solve_stokes_info(z["P"], z["Vx"], z["Vy"], *par, *[None] * 7, z["dVxdt"], z["dVydt"], None, None, z["Vx_s"],
                                z["Vy_s"], 9.81, 1 / (Nx - 1), 1 / (Ny - 1), Nx, Ny, 1e-3, 0.5, eps=1e-300, iter_max=200)
    assert info["fused_launches"] == expected(200, per_launch, 2000, 10 * min(Nx, Ny), False)
