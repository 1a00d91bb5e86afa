"""The scan of the marker sort (sf_deposit.cu) where its split changes: cell counts around one tile (2048) and around the
tiles that a block adds up itself (4096), and the allocation-free deposit's largest grid.  Exact: against numpy's stable
sort, and the regular deposit against the allocation-free one.  And the place it needs: blocks that fit beside resident
tiles."""
import numpy as np
import pytest
import torch

from test_gpu_sort_edges import rebin_numpy


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(88, 22), (1023, 1), (682, 2), (2047, 4095), (2048, 4095)])
def test_rebin_around_a_tile(sf, nx, ny):
    nm = 20_000
    rng = np.random.default_rng(nx)
    x, y = rng.random(nm) * (nx - 1), rng.random(nm) * max(ny - 1, 1) * 0.999
    x[: nm // 8], y[: nm // 8] = nx - 1.5, 0.1     # a long cell
    counts, offsets, perm = sf.rebin_markers(torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), 0.0, 0.0, 1.0, 1.0, nx, ny)
    want, order = rebin_numpy(x, y, 1.0, 1.0, nx, ny)
    assert np.array_equal(counts.cpu().numpy(), want)
    assert np.array_equal(offsets.cpu().numpy(), np.concatenate([[0], np.cumsum(want)]))
    assert np.array_equal(perm.cpu().numpy(), order)


@pytest.mark.gpu
def test_noalloc_largest_grid(sf):
    n, h = 511, 1.0 / 510
    g = torch.Generator(device="cuda").manual_seed(1)
    x, y, v = (torch.rand(400_000, dtype=torch.float64, device="cuda", generator=g) for _ in range(3))
    a, b = sf.zeros(n, n), sf.zeros(n, n)
    sf.bilinear_marker_to_grid_noalloc(0.0, 0.0, a, x, y, v, h, h)
    sf.bilinear_marker_to_grid(0.0, 0.0, b, x, y, v, h, h)
    assert torch.equal(a, b)


def test_blocks_fit_beside_resident_tiles():
    """A quarter of an SM: 512 of its 2048 threads."""
    import pathlib
    import re

    src = pathlib.Path(__file__).parents[1] / "stokesflow.jl_b200" / "csrc"
    consts = dict(re.findall(r"\b(\w+_THREADS) = (\d+)", (src / "sf_deposit.cu").read_text()))
    assert {"DEP_THREADS", "SORT_THREADS", "SCAN_THREADS"} <= set(consts)
    assert all(int(n) <= 512 for n in consts.values()), consts
