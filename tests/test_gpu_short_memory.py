"""Solves for which only the smaller of two layouts finds memory: a second one keeps the first one's memory, instead of
freeing it to find out again (another allocator could take it in between)."""
import numpy as np
import pytest
import torch

from fields import random_fields
from test_gpu_parity import dev

pytestmark = pytest.mark.gpu

STATE = {"P": (-1, -1), "Vx": (2, 1), "Vy": (1, 2), "dVxdt": (-2, -1), "dVydt": (-1, -2), "Vx_s": (0, 1), "Vy_s": (1, 0)}


def waits_for_the_device(call):
    """Whether call() waits for a kernel of another stream, as freeing device memory does."""
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda._sleep(1_000_000_000)    # half a second, one thread
        done = torch.cuda.Event()
        done.record()
    call()
    waited = done.query()
    done.synchronize()
    return waited


@pytest.mark.parametrize("form", ["plain", "mixed"])
def test_second_solve_keeps_its_memory(sf, form):
    Nx, Ny = 3000, 2200
    LD, rows = (Nx + 2 + 31) // 32 * 32, Ny + 5
    z = {k: sf.zeros(Nx + a, Ny + b) for k, (a, b) in STATE.items()}
    par = [dev(a) for a in random_fields(Nx, Ny, seed=1, contrast=5.0)]
    ctx = sf.Context(0)
    args = (9.81, 1 / (Nx - 1), 1 / (Ny - 1), Nx, Ny, 1e-3, 0.5)

    def mixed(z, par, n, m):
        p = sf.MixedProblem(z["P"], z["Vx"], z["Vy"], *par, z["Vx_s"], z["Vy_s"], 9.81, 1 / (n - 1), 1 / (m - 1), n, m, 1e-3,
                            0.5, eps=1e-300, dVxdt=z["dVxdt"], dVydt=z["dVydt"])
        sf.solve_stokes_batch_mixed([p], options=sf.mixed_options(max_sweeps=60), ctx=ctx)

    if form == "plain":
        small, large = 17 * LD * rows * 8, 23 * LD * rows * 8
        call = lambda: sf.solve_stokes_info(z["P"], z["Vx"], z["Vy"], *par, *[None] * 7, z["dVxdt"], z["dVydt"], None,  # noqa: E731
                                            None, z["Vx_s"], z["Vy_s"], *args, eps=1e-300, iter_max=30, ctx=ctx)
    else:
        small = sf.Engine.instance_bytes(Nx, Ny)
        large = small + 2 * 4 * ((Nx + 4 + 31) // 32 * 32) * (Ny + 3)
        # the engine and its tables, before memory is short
        mixed({k: sf.zeros(20 + a, 20 + b) for k, (a, b) in STATE.items()}, [dev(a) for a in random_fields(20, 20, seed=1)], 20, 20)
        call = lambda: mixed(z, par, Nx, Ny)  # noqa: E731
    waits_for_the_device(lambda: None)   # (its streams and module, too, before memory is short)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (small + large) // 2, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(3):   # (the batched solve's sweeps are timed and captured first)
            call()
        assert torch.cuda.mem_get_info()[0] < large - small
        scratch = ctx.scratch_bytes()
        assert not waits_for_the_device(call), "the scratch was freed"
        assert ctx.scratch_bytes() == scratch
    finally:
        del held
        torch.cuda.empty_cache()
    assert np.isfinite(z["Vx_s"].cpu().numpy()).all()
