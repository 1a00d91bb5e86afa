"""Three FP32 sweeps per launch (sf_mixed_march.cuh) against one per launch in fixed tiles (k_pt32), bit for bit: every
point's arithmetic is the same.  Sizes at the edges of the strips (58 columns fit one; 56 each beyond) and of the
segments, folds that leave one and two sweeps over, odd sweep counts, checks inside, rates in and out, both pseudo-step
rules, and more strips than warps.  A first solve times the workload class, the second one marches from its start."""
import numpy as np
import pytest

from fields import random_fields

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (20, 26), (58, 40), (59, 61), (60, 33), (113, 70), (114, 131), (300, 17), (17, 300), (171, 173)]


def solve(sf, ctx, sizes, **opts):
    import torch

    from test_gpu_parity import dev
    probs = []
    for k, (Nx, Ny) in enumerate(sizes):
        dx, dy = 1.0 / (Nx - 1), 1.2 / (Ny - 1)
        rng = np.random.default_rng(k)
        rho, mub, mup = (dev(a) for a in random_fields(Nx, Ny, seed=k, contrast=5.0))
        r = lambda *s: dev(1e-3 * rng.normal(size=s))  # noqa: E731
        probs.append(sf.MixedProblem(r(Nx - 1, Ny - 1), sf.zeros(Nx + 2, Ny + 1), sf.zeros(Nx + 1, Ny + 2), rho, mub, mup,
                                     r(Nx, Ny + 1), r(Nx + 1, Ny), 9.81, dx, dy, Nx, Ny, 1e-3, 0.5, eps=1e-30,
                                     use_free_surface_stabilization=k % 3 != 0, dVxdt=r(Nx - 2, Ny - 1),
                                     dVydt=r(Nx - 1, Ny - 2)))
    res = sf.solve_stokes_batch_mixed(probs, options=sf.mixed_options(**opts), ctx=ctx)
    torch.cuda.synchronize()
    return [{q: a.cpu().numpy() for q, a in p.arrays.items()} for p in probs], res


@pytest.mark.parametrize("sizes,opts", [
    (SIZES, dict(max_sweeps=700, fold_every=50)), (SIZES, dict(max_sweeps=333, fold_every=400)),
    (SIZES, dict(max_sweeps=251, fold_every=2)), (SIZES, dict(max_sweeps=430, fold_every=52, use_graphs=False)),
    (SIZES, dict(max_sweeps=430, fold_every=100, dtau_local_max=True)), ([(20, 26)], dict(max_sweeps=1200, fold_every=400)),
    ([(1024, 900)], dict(max_sweeps=211, fold_every=100)), ([(700, 690)] * 60, dict(max_sweeps=60, fold_every=50))])
def test_march32_bitexact(sf, sizes, opts):
    ref, res_ref = solve(sf, sf.Context(0), sizes, tile_rows=16, **opts)
    ctx = sf.Context(0)
    for turn in range(2):
        got, res = solve(sf, ctx, sizes, **opts)
        assert [r["inner_iters"] for r in res] == [r["inner_iters"] for r in res_ref]
        assert [r["dt_out"] for r in res] == [r["dt_out"] for r in res_ref]
        for (Nx, Ny), a, b in zip(sizes, got, ref):
            for q in b:
                assert np.array_equal(a[q], b[q], equal_nan=True), f"{Nx} x {Ny}: {q} differs (turn {turn})"
