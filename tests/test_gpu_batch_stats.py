"""The stats of a batched solve name what its sweeps ran: three per launch once the workload class is measured, one in
fixed tiles; and the launches are as many as that makes."""
import pytest

from test_gpu_march32 import solve

pytestmark = pytest.mark.gpu


def test_sweeps_per_launch(sf):
    sizes, opts = [(60, 33), (114, 131)], dict(max_sweeps=600, fold_every=50)
    counts = {}
    for rows in (16, 0):
        ctx = sf.Context(0)
        solve(sf, ctx, sizes, tile_rows=rows, **opts)       # (with rows 0: measures the class)
        n = ctx.launch_count()
        solve(sf, ctx, sizes, tile_rows=rows, **opts)
        counts[rows] = ctx.launch_count() - n
        st = sf.batch_stats(ctx)
        assert st["sweeps_per_launch"] == (1 if rows else 3)
        if not rows:
            assert st["tune_state"] == "cached"
    # the rounds' other kernels are the same; of 600 sweeps' launches at least half go
    assert counts[0] < counts[16] - 300, counts
    with sf.Engine(arena_bytes=64 << 20) as eng:
        assert eng.stats()["sweeps_per_launch"] == 0
