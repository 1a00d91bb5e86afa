"""The marker sort and the deposit where their launches change: cell counts around one scan tile (8192), more tiles than a block adds up
itself (2048), long cells on a tile's edge, and several grids in one launch or one after the other (4 Mi markers).
Against numpy's stable sort, the fused deposit against one call per grid, and the deposit against the oracle where the
marker runs, the values' arrays or the division by dx and dy are unusual; exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rebin_numpy(x, y, dx, dy, nx, ny):
    key = (np.floor(x / dx) + 1 + (np.floor(y / dy) + 1) * (nx + 1)).astype(np.int64)
    return np.bincount(key, minlength=(nx + 1) * (ny + 1)), np.argsort(key, kind="stable")


@pytest.mark.parametrize("nx,ny,nm", [(63, 127, 30000), (8190, 1, 9000), (8191, 1, 9000), (89, 91, 0), (4200, 4010, 5000),
                                      (64, 127, 1), (127, 127, 3_000_000)])
def test_rebin_edges(sf, nx, ny, nm):
    rng = np.random.default_rng(nx + nm)
    dx, dy = 1.0, 0.5
    x, y = rng.random(nm) * (nx - 1) * dx, rng.random(nm) * max(ny - 1, 1) * dy * 0.999
    x[: nm // 8] = (nx - 1) * dx * 0.5      # long cells
    y[: nm // 8] = 0.1
    counts, offsets, perm = sf.rebin_markers(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), 0.0, 0.0, dx, dy, nx, ny)
    want, order = rebin_numpy(x, y, dx, dy, nx, ny)
    assert np.array_equal(counts.cpu().numpy(), want)
    assert np.array_equal(offsets.cpu().numpy(), np.concatenate([[0], np.cumsum(want)]))
    assert np.array_equal(perm.cpu().numpy(), order)


@pytest.mark.parametrize("nm", [50_000, (1 << 22) - 1, (1 << 22) + 1])
def test_grids_together_or_in_turn(sf, nm):
    g = torch.Generator(device="cuda").manual_seed(nm)
    x, y, a, b = (torch.rand(nm, dtype=torch.float64, device="cuda", generator=g) for _ in range(4))
    N, h = 301, 1.0 / 300
    # four grids over three value arrays: two groups
    specs = [(-0.5 * h, 0.0, N + 1, N, a), (0.0, 0.0, N, N, b), (0.5 * h, 0.5 * h, N - 1, N - 1, x), (0.1, 0.2, 40, 30, a)]
    one = [sf.zeros(s[2], s[3]) for s in specs]
    for (x0, y0, _, _, v), out in zip(specs, one):
        sf.bilinear_marker_to_grid(x0, y0, out, x, y, v, h, h)
    fused = [sf.zeros(s[2], s[3]) for s in specs]
    sf.bilinear_marker_to_grids([(s[0], s[1], out, s[4]) for s, out in zip(specs, fused)], x, y, h, h)
    for p, q in zip(one, fused):
        assert torch.equal(p, q)


def test_grids_that_share_an_output(sf):
    """Two grids of a call that write the same array: the second deposit's values, as one call after the other."""
    g = torch.Generator(device="cuda").manual_seed(5)
    x, y, a, b = (torch.rand(20_000, dtype=torch.float64, device="cuda", generator=g) for _ in range(4))
    one, both = sf.zeros(60, 60), sf.zeros(60, 60)
    for v in (a, b):
        sf.bilinear_marker_to_grid(0.0, 0.0, one, x, y, v, 1 / 59, 1 / 59)
    sf.bilinear_marker_to_grids([(0.0, 0.0, both, a), (0.0, 0.0, both, b)], x, y, 1 / 59, 1 / 59)
    assert torch.equal(one, both)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -70, 2.0 ** 70])
@pytest.mark.parametrize("order", ["runs", "shuffled", "one cell", "tiny"])
def test_deposit_runs_match_the_oracle(sf, oracle_lib, scale, order):
    """Runs of 1 to 32 markers and beyond a warp, markers outside (which break runs), a cell with thousands of runs,
    distances from a cell's corner below 2^-895, and spacings beyond the constant division's."""
    O = oracle_lib
    rng = np.random.default_rng(11)
    nx, ny, nm = 23, 17, 20_011
    dx, dy = scale / (nx - 1), scale / (ny - 1)
    x, y, v = rng.random(nm) * 1.2 - 0.1, rng.random(nm) * 1.2 - 0.1, rng.random(nm)
    if order == "runs":
        i = np.argsort(np.floor(x * (nx - 1)) * 100 + np.floor(y * (ny - 1)), kind="stable")
        x, y = x[i], y[i]
        x[::41], y[100:140] = -3.0, 7.0
    elif order == "one cell":
        x[::2], y[::2] = 0.51 + 1e-3 * x[::2], 0.51 + 1e-3 * y[::2]
    elif order == "tiny":
        x[:7], y[:7] = [1e-300, 2.0 ** -1000, 5e-324, 0.0, 1e-310, 2.0 ** -900, 1e-280], 0.4
    x, y = x * scale, y * scale
    got, want = sf.zeros(nx, ny), O.zeros(nx, ny)
    t = [torch.from_numpy(a.copy()).cuda() for a in (x, y, v)]
    sf.bilinear_marker_to_grid(0.0, 0.0, got, *t, dx, dy)
    O.bilinear_marker_to_grid(0.0, 0.0, want, x, y, v, dx, dy, O.zeros(nx, ny), O.zeros(nx, ny))
    assert np.array_equal(got.cpu().numpy(), want)
