// sf_deposit.cu -- marker->grid deposit (scripts/MarkerToGrid.jl:18-172) and
// marker->cell rebinning for libstokesflow_b200.so.
//
// Design: the reference scatters 8 floating-point adds per marker (serial on
// the CPU, CUDA.@atomic on the GPU, MarkerToGrid.jl:58-155).  Here the adds
// become a gather with no floating-point atomics: a node visits the markers of
// its four adjacent cells in ascending marker index, the reference CPU loop's
// order, so its sums are bit-identical to it.  Markers keep much of their
// initial lattice order, so a cell's markers are a few runs of consecutive
// indices; the deposit sorts runs, not markers:
//   1. k_cell_runs     cell (ix, iy) of every marker for each grid, exactly
//                      topleftIndexRelDist (common.jl:22-33); runs of
//                      consecutive markers of one cell (within a warp's 32),
//                      counted per cell, their last markers as a bit mask; and
//                      the markers' x, y and values as records of 32 bytes.
//   2. k_scan_*        exclusive scan of the counts -> cell offsets (and the
//                      list of long cells).
//   3. k_scatter_runs  the runs' first markers into their cell's segment (in
//                      no particular order inside it).
//   4. segment sort    every segment ascending: k_sort_long sorts the cells
//                      holding more than SORT_LONG entries in place (a
//                      block-wide LSD radix sort per cell, stable, linear in
//                      the cell's count, so a cell where markers pile up costs
//                      no more than its size); k_sort_cells sorts the others
//                      in shared memory, a window of consecutive cells at a
//                      time.
//   5. k_gather_runs   one thread per node merges the four adjacent cells'
//                      runs (they are disjoint intervals, so a run is taken
//                      whole, its records loaded several at a time),
//                      accumulates w and w*val, and divides (safeDivision,
//                      :164-172).
// The rebin (sf_rebin_markers) sorts markers the same way: k_cell_keys,
// k_scan_*, k_scatter, segment sort; the allocation-free deposit gathers from
// that.
//
// The grids of a timestep go through each kernel together (8 launches instead of
// 32): small deposits were bound by their launches.
#include <algorithm>

#include "sf_internal.cuh"

namespace sf {

constexpr int DEP_THREADS = 256;
constexpr int SORT_THREADS = 256;
constexpr int SORT_CPB = 256;     // cells per block of k_sort_cells
constexpr int SORT_CAP = 4096;    // entries of a k_sort_cells window in shared memory
constexpr int SORT_LONG = 64;     // cells with more markers are sorted by k_sort_long
// markers up to which the grids of a deposit go through each kernel in one launch, every grid in scratch of its own (4
// bytes per marker and grid).  Against one grid after the other, 145 k markers: 228 -> 84 us; 1.4 M: 443 -> 315; 4.2 M:
// 920 -> 714.  Beyond, launches no longer count (26 M markers: 4.10 ms either way) and one grid's scratch serves all.
constexpr int64_t DEPOSIT_TOGETHER = 1 << 22;

// What the gather reads of a marker: its position and its values in up to two arrays.  32 bytes: one sector.
struct __align__(32) Record {
    double x, y, v0, v1;
};

// One grid of a sort: what its kernels read and write.  Several grids over the same markers (the deposits of a timestep)
// go through each kernel together, blockIdx.y choosing the grid.
struct SortGrid {
    double xmin, ymin;
    int64_t nx, ny, ncells;    // nodes, cells (nx + 1) * (ny + 1)
    int32_t* keys;             // cell of each marker (-1: none); spent after the scatter, then the radix sort's buffer
    int32_t* counts;           // markers of each cell
    int32_t* offsets;          // [ncells + 1]
    int32_t* cursor;           // next place in each cell's segment (scatter)
    int32_t* tiles;            // sums of the scan's tiles
    int32_t* n_list;           // the cells holding more than SORT_LONG markers: their number ...
    int32_t* list;             // ... and the cells
    int32_t* perm;             // sorted markers, or (deposit) first markers of runs
    uint32_t* ends;            // (deposit) bit m & 31 of word m / 32: marker m is the last of its run
    int32_t* general;          // (deposit) not 0: some distance is out of div_const's range
    int second;                // (deposit) the grid's values are the records' v1
    const double* val;
    double *val_grid, *val_wt_sum, *wt_sum;
    int64_t ld_sum;
};
struct SortGrids {
    SortGrid g[SF_MAX_GRIDS];
    int n;
    const double *val0, *val1; // (deposit) the records' values
    Record* rec;
};

// 1 for the rebin and the allocation-free deposit: cell key of every marker; counts[key]++ (warp-aggregated).  (Keeping the
// counters' old values as the markers' places, so that the scatter needs no atomics, costs more here, 87 us per grid and
// 26 M markers, than the 25 us it saves there.)
__global__ void k_cell_keys(const double* __restrict__ x, const double* __restrict__ y, int64_t nm, double dx, double dy,
                            const __grid_constant__ SortGrids s, unsigned long long* __restrict__ bad_counter) {
    const SortGrid& g = s.g[0];
    const int lane = threadIdx.x & 31;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < nm; base += stride) {
        int64_t m = base + threadIdx.x;
        int32_t key = -1;
        if (m < nm) {
            TopLeft t = topleft(g.xmin, g.ymin, x[m], y[m], dx, dy);
            // MarkerToGrid.jl:66: accept iff 0 <= ix <= Nx && 0 <= iy <= Ny (ix = qx + 1)
            if (t.qx >= -1.0 && t.qx <= (double)(g.nx - 1) && t.qy >= -1.0 && t.qy <= (double)(g.ny - 1))
                key = (int32_t)((int64_t)t.qx + 1 + ((int64_t)t.qy + 1) * (g.nx + 1));
            g.keys[m] = key;
        }
        unsigned active = __ballot_sync(0xffffffffu, m < nm);
        if (m < nm) {
            unsigned peers = __match_any_sync(active, key);
            if (lane == __ffs(peers) - 1) {
                int n = __popc(peers);
                if (key >= 0)
                    atomicAdd(&g.counts[key], n);
                else if (bad_counter)
                    atomicAdd(bad_counter, (unsigned long long)n);
            }
        }
    }
}

// 1 for a deposit: the runs of consecutive markers that share a cell, and the records.
template <int MOST>
__global__ void k_cell_runs(const double* __restrict__ x, const double* __restrict__ y, int64_t nm, double dx, double dy,
                            const __grid_constant__ SortGrids s, unsigned long long* __restrict__ bad_counter) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < nm; base += stride) {
        const int64_t m = base + threadIdx.x;
        const bool live = m < nm;
        const double xm = live ? x[m] : 0.0, ym = live ? y[m] : 0.0;
        if (live) {
            Record r;
            r.x = xm;
            r.y = ym;
            r.v0 = s.val0[m];
            r.v1 = s.val1 ? s.val1[m] : 0.0;
            s.rec[m] = r;
        }
#pragma unroll
        for (int k = 0; k < MOST; ++k) {
            if (MOST > 1 && k >= s.n) break;
            const SortGrid& g = s.g[k];
            int32_t key = -1;
            const TopLeft t = topleft(g.xmin, g.ymin, xm, ym, dx, dy);
            // MarkerToGrid.jl:66: accept iff 0 <= ix <= Nx && 0 <= iy <= Ny (ix = qx + 1)
            if (t.qx >= -1.0 && t.qx <= (double)(g.nx - 1) && t.qy >= -1.0 && t.qy <= (double)(g.ny - 1))
                key = (int32_t)((int64_t)t.qx + 1 + ((int64_t)t.qy + 1) * (g.nx + 1));
            const int32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
            const bool start = !live || lane == 0 || prev != key;
            const unsigned starts = __ballot_sync(0xffffffffu, start);
            const unsigned bad = __ballot_sync(0xffffffffu, live && key < 0);
            if (live) {
                g.keys[m] = key;
                if (start && key >= 0) atomicAdd(&g.counts[key], 1);
            }
            // the gather divides these by dx, dy (topleft's dxij, dyij)
            const bool odd = live && key >= 0 &&
                             !(div_const_takes_a(xm - (g.xmin + t.qx * dx)) && div_const_takes_a(ym - (g.ymin + t.qy * dy)));
            if (__any_sync(0xffffffffu, odd) && lane == 0) *g.general = 1;
            if (lane == 0 && live) {
                g.ends[m >> 5] = starts >> 1 | 0x80000000u;
                if (bad && bad_counter) atomicAdd(bad_counter, (unsigned long long)__popc(bad));
            }
        }
    }
}

// 2. exclusive scan of the counts -> offsets, in tiles of SCAN_TILE cells: the tiles' sums, then every tile with the sum
// of the tiles before it, which a block adds up itself (or, of more than SCAN_DIRECT tiles, finds scanned already).
// The second pass also lists the long cells.  Blocks of 256 threads find a place beside the resident tiles of a solve on
// another stream, which leave a quarter of an SM; 1024 threads waited for a launch of those to end.  A rebin of 0.6 M
// markers beside 180^2: 203 -> 137 - 164 us, beside 300^2 245 -> 193; by itself, with more blocks, 82 -> 75, three deposits of
// 128^2 with the host's time 102 -> 95.
constexpr int SCAN_THREADS = 256, SCAN_ITEMS = 8, SCAN_TILE = SCAN_THREADS * SCAN_ITEMS, SCAN_DIRECT = 4096;

__device__ __forceinline__ int32_t block_exclusive_scan(int32_t v, int32_t* warp_sums, int32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int32_t w = (lane < (int)(blockDim.x >> 5)) ? warp_sums[lane] : 0;
        int32_t s = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s - w;  // exclusive warp offsets
        if (lane == 31) *total = s;
    }
    __syncthreads();
    int32_t r = warp_sums[warp] + x - v;
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tile_sums(const __grid_constant__ SortGrids s) {
    __shared__ int32_t warp_sums[32];
    __shared__ int32_t total;
    const SortGrid& g = s.g[blockIdx.y];
    if ((int64_t)blockIdx.x * SCAN_TILE >= g.ncells) return;
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
    int32_t sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k)
        if (base + k < g.ncells) sum += g.counts[base + k];
    block_exclusive_scan(sum, warp_sums, &total);
    if (threadIdx.x == 0) g.tiles[blockIdx.x] = total;
}

// single block per grid: exclusive scan of the tile sums in place
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tile_offsets(const __grid_constant__ SortGrids s) {
    __shared__ int32_t warp_sums[32];
    __shared__ int32_t total;
    const SortGrid& g = s.g[blockIdx.y];
    const int64_t ntiles = (g.ncells + SCAN_TILE - 1) / SCAN_TILE;
    int32_t carry = 0;
    for (int64_t b0 = 0; b0 < ntiles; b0 += SCAN_THREADS) {
        int64_t i = b0 + threadIdx.x;
        int32_t v = (i < ntiles) ? g.tiles[i] : 0;
        int32_t e = block_exclusive_scan(v, warp_sums, &total);
        if (i < ntiles) g.tiles[i] = carry + e;
        carry += total;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(const __grid_constant__ SortGrids s, int scanned) {
    __shared__ int32_t warp_sums[32];
    __shared__ int32_t total;
    const SortGrid& g = s.g[blockIdx.y];
    if ((int64_t)blockIdx.x * SCAN_TILE >= g.ncells) return;
    int32_t before = 0;
    if (scanned) {
        before = g.tiles[blockIdx.x];
    } else {
        for (int t = threadIdx.x; t < (int)blockIdx.x; t += SCAN_THREADS) before += g.tiles[t];
        block_exclusive_scan(before, warp_sums, &total);
        before = total;
        __syncthreads();
    }
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
    int32_t v[SCAN_ITEMS];
    int32_t sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = (base + k < g.ncells) ? g.counts[base + k] : 0;
        sum += v[k];
    }
    int32_t e = block_exclusive_scan(sum, warp_sums, &total) + before;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (base + k < g.ncells) g.offsets[base + k] = g.cursor[base + k] = e;
        e += v[k];
        if (base + k == g.ncells - 1) g.offsets[g.ncells] = e;
        if (v[k] > SORT_LONG) g.list[atomicAdd(g.n_list, 1)] = (int32_t)(base + k);
    }
}

// 3. scatter marker indices into their cells (order within a cell arbitrary).
__global__ void k_scatter(const __grid_constant__ SortGrids s, int64_t nm) {
    const SortGrid& g = s.g[blockIdx.y];
    const int lane = threadIdx.x & 31;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < nm; base += stride) {
        int64_t m = base + threadIdx.x;
        int32_t key = (m < nm) ? g.keys[m] : -1;
        unsigned active = __ballot_sync(0xffffffffu, key >= 0);
        if (key >= 0) {
            unsigned peers = __match_any_sync(active, key);
            int leader = __ffs(peers) - 1;
            int32_t pos0 = 0;
            if (lane == leader) pos0 = atomicAdd(&g.cursor[key], __popc(peers));
            pos0 = __shfl_sync(peers, pos0, leader);
            g.perm[pos0 + __popc(peers & ((1u << lane) - 1u))] = (int32_t)m;
        }
    }
}

// 3 for a deposit: the runs' first markers.
__global__ void k_scatter_runs(const __grid_constant__ SortGrids s, int64_t nm) {
    const SortGrid& g = s.g[blockIdx.y];
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < nm; m += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(m & 31);
        if (q != 0 && !(g.ends[m >> 5] >> (q - 1) & 1u)) continue;
        const int32_t key = g.keys[m];
        if (key >= 0) g.perm[atomicAdd(&g.cursor[key], 1)] = (int32_t)m;
    }
}

// The allocation-free deposit's per-cell sort of short segments (one thread per cell; its long segments are
// sorted by k_sort_long first, and are skipped here).
__global__ void k_sort_segments(const int32_t* __restrict__ offsets, int64_t ncells, int32_t* __restrict__ perm) {
    int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    int32_t b = offsets[c], e = offsets[c + 1];
    if (e - b > SORT_LONG) return;
    for (int32_t i = b + 1; i < e; ++i) {
        int32_t v = perm[i];
        int32_t j = i - 1;
        if (perm[j] <= v) continue;
        while (j >= b && perm[j] > v) {
            perm[j + 1] = perm[j];
            --j;
        }
        perm[j + 1] = v;
    }
}

// 4a. each long cell's segment sorted ascending in place by a block-wide LSD radix sort on 8-bit digits of the
// marker index (indices are non-negative 31-bit values: 4 digits), stable, through `tmp` at the same offsets.
// A digit on which the whole segment agrees moves nothing and is skipped.  Tiles of SORT_THREADS entries are
// ranked in order: lanes within a warp by __match_any_sync, warps by their per-digit counts.
__global__ void __launch_bounds__(SORT_THREADS) k_sort_long(const __grid_constant__ SortGrids s) {
    constexpr int NW = SORT_THREADS / 32;
    __shared__ int hist[256];
    __shared__ int base[256];
    __shared__ int wcnt[NW][256];
    __shared__ int skip;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SortGrid& g = s.g[blockIdx.y];
    const int32_t* offsets = g.offsets;
    int32_t *perm = g.perm, *tmp = g.keys;
    const int n_long = *g.n_list;
    for (int li = blockIdx.x; li < n_long; li += gridDim.x) {
        const int c = g.list[li];
        const int32_t b = offsets[c], n = offsets[c + 1] - b;
        int32_t* src = perm + b;
        int32_t* dst = tmp + b;
        for (int shift = 0; shift < 32; shift += 8) {
            hist[tid] = 0;
            __syncthreads();
            for (int i = tid; i < n; i += SORT_THREADS) atomicAdd(&hist[(src[i] >> shift) & 255], 1);
            __syncthreads();
            if (tid == 0) {
                int run = 0, same = 0;
                for (int d = 0; d < 256; ++d) {
                    base[d] = run;
                    run += hist[d];
                    same |= (hist[d] == n);
                }
                skip = same;
            }
            __syncthreads();
            if (skip) continue;
            for (int t0 = 0; t0 < n; t0 += SORT_THREADS) {
                for (int k = tid; k < NW * 256; k += SORT_THREADS) (&wcnt[0][0])[k] = 0;
                __syncthreads();
                const int i = t0 + tid;
                const bool valid = i < n;
                const int32_t v = valid ? src[i] : 0;
                const int d = (v >> shift) & 255;
                const unsigned act = __ballot_sync(0xffffffffu, valid);
                int rank = 0;
                if (valid) {
                    const unsigned peers = __match_any_sync(act, d);
                    rank = __popc(peers & ((1u << lane) - 1u));
                    if (lane == __ffs(peers) - 1) wcnt[warp][d] = __popc(peers);
                }
                __syncthreads();
                if (valid) {
                    int off = base[d] + rank;
                    for (int w = 0; w < warp; ++w) off += wcnt[w][d];
                    dst[off] = v;
                }
                __syncthreads();
                int sum = 0;
                for (int w = 0; w < NW; ++w) sum += wcnt[w][tid];
                base[tid] += sum;
                __syncthreads();
            }
            int32_t* t = src;
            src = dst;
            dst = t;
        }
        if (src != perm + b)
            for (int i = tid; i < n; i += SORT_THREADS) perm[b + i] = src[i];
        __syncthreads();
    }
}

// 4b. every short segment sorted ascending, in place; long segments are sorted already (k_sort_long).  A block takes
// SORT_CPB consecutive cells and works through them in windows of consecutive cells holding at most SORT_CAP entries:
// it loads a window's entries into shared memory, ranks each within its cell by counting the smaller ones there, and
// writes it to its sorted place.
__global__ void __launch_bounds__(SORT_THREADS) k_sort_cells(const __grid_constant__ SortGrids s) {
    __shared__ int32_t soff[SORT_CPB + 1];
    __shared__ int32_t sm[SORT_CAP];
    const int tid = threadIdx.x;
    const SortGrid& g = s.g[blockIdx.y];
    const int64_t ncells = g.ncells;
    const int32_t* __restrict__ offsets = g.offsets;
    int32_t* perm = g.perm;
    const int64_t c0 = (int64_t)blockIdx.x * SORT_CPB;
    if (c0 >= ncells) return;
    const int nc = (int)min((int64_t)SORT_CPB, ncells - c0);
    for (int i = tid; i <= nc; i += SORT_THREADS) soff[i] = offsets[c0 + i];
    __syncthreads();
    int w0 = 0;
    while (w0 < nc) {
        // the largest w1 with soff[w1] - soff[w0] <= SORT_CAP (w1 == w0: cell w0 alone holds more)
        int lo = w0, hi = nc;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (soff[mid] - soff[w0] <= SORT_CAP) lo = mid; else hi = mid - 1;
        }
        const int w1 = lo;
        if (w1 == w0) {  // a long cell
            ++w0;
            continue;
        }
        const int32_t e0 = soff[w0];
        const int ne = soff[w1] - e0;
        for (int i = tid; i < ne; i += SORT_THREADS) sm[i] = perm[e0 + i];
        __syncthreads();
        for (int i = tid; i < ne; i += SORT_THREADS) {
            // the entry's cell k: the last one in [w0, w1) starting at or before it
            int a = w0, z = w1 - 1;
            while (a < z) {
                const int mid = (a + z + 1) >> 1;
                if (soff[mid] - e0 <= i) a = mid; else z = mid - 1;
            }
            const int cb = soff[a] - e0, ce = soff[a + 1] - e0;
            if (ce - cb <= SORT_LONG) {
                const int32_t v = sm[i];
                int rank = 0;
                for (int j = cb; j < ce; ++j) rank += (sm[j] < v) ? 1 : 0;
                perm[e0 + cb + rank] = v;
            }
        }
        __syncthreads();
        w0 = w1;
    }
}

// 5. per-node gather over the sorted runs.  Node (I, J), 1-based.  A marker in cell (ix, iy) contributes to
// node (ix, iy) with (1-dx)(1-dy), (ix+1, iy) with dx(1-dy), (ix, iy+1) with (1-dx)dy and (ix+1, iy+1) with dx*dy
// (MarkerToGrid.jl:124-151), so node (I, J) merges the cells (I,J), (I-1,J), (I,J-1), (I-1,J-1), whose runs are sorted by
// marker index: taking the run with the smallest first marker each time visits the node's markers in ascending index
// order, the reference's serial order.  The next run's start is loaded while the taken run's records are, GT_AHEAD of
// them at once, so a node waits for memory once per run, not once per marker.
//
// What bounds it: the latency of those loads (27 warps per SM) and half the L1 rate: each of 32 lanes reads a line of its
// own.  Three grids over 67 M markers: 9.07 -> 7.73 ms against sorting the markers themselves into 32-byte records per
// grid (sort 0.95, gather 1.14 ms per grid); 26 M with 25 per cell 3.9 -> 3.03 ms; the same in random order 10.3 -> 6.1.
// Four records ahead with 5 blocks per SM: 9.5 ms, one ahead 10.4; three 7.9 - 8.1; 10 blocks 8.7; dividing with a range
// test per record instead of once per deposit (SortGrid::general) 8.5.
constexpr int GT_NONE = 0x7fffffff;   // start of an exhausted list
// nodes of a block, and of a warp along x.  Neighbours read the same records, in both directions: compact warps and blocks
// find more of them in L1 (33% of the sectors before) and L2.  Against rows of 32 nodes in blocks of 4, 67 M markers: 7.73
// -> 7.48 ms; 26 M 3.04 -> 2.92, after a strong swirl 5.03 -> 4.62, shuffled in their cells 4.16 -> 4.10, sorted by cell
// 3.30 -> 3.31, in rows along x 2.79 -> 2.83.  Warps of 4 x 8 nodes: 7.51, of 1 x 32 7.71 and 5.37 after the swirl.
constexpr int GT_X = 16, GT_Y = 8, GT_LX = 8, GT_LY = 32 / GT_LX;
constexpr int GT_AHEAD = 2;           // records of a run loaded at once
constexpr int GT_BLOCKS = 8;          // blocks per SM (64 registers)

// FAST: every marker's distances from its cell's corner are within div_const's range (and dx, dy too).
template <bool FAST>
__device__ __forceinline__ void gather_node(const SortGrids& s, const SortGrid& g, double dx, double dy, double rdx,
                                            double rdy, unsigned long long* __restrict__ empty_counter) {
    const Record* __restrict__ rec = s.rec;
    const int32_t* __restrict__ offsets = g.offsets;
    const int32_t* __restrict__ runs = g.perm;
    const uint32_t* __restrict__ ends = g.ends;
    const int64_t nx = g.nx, ny = g.ny;
    const int64_t ntx = (nx + GT_X - 1) / GT_X;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t I = (int64_t)(blockIdx.x % ntx) * GT_X + (warp % (GT_X / GT_LX)) * GT_LX + lane % GT_LX + 1;
    const int64_t J = (int64_t)(blockIdx.x / ntx) * GT_Y + (warp / (GT_X / GT_LX)) * GT_LY + lane / GT_LX + 1;
    if (I > nx || J > ny) return;
    const int64_t ldc = nx + 1;
    const bool second = g.second != 0;
    // corner k: 0 = marker's top-left node (cell I,J), 1 = top-right (cell I-1,J),
    //           2 = bottom-left (cell I,J-1), 3 = bottom-right (cell I-1,J-1)
    int32_t cur[4], end[4], hm[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int64_t key = (I - (k & 1)) + (J - (k >> 1)) * ldc;
        cur[k] = offsets[key];
        end[k] = offsets[key + 1];
        hm[k] = cur[k] < end[k] ? runs[cur[k]] : GT_NONE;
    }
    // topleftIndexRelDist's node coordinate x_grid_min + (ix - 1) * dx of the cells ix = I and I - 1 (likewise y)
    const double xr = g.xmin + (double)(I - 1) * dx, xl = g.xmin + (double)(I - 2) * dx;
    const double yr = g.ymin + (double)(J - 1) * dy, yl = g.ymin + (double)(J - 2) * dy;
    double ws = 0.0, vs = 0.0;
    while (true) {
        int kb = 0;
        int32_t m = hm[0];
#pragma unroll
        for (int k = 1; k < 4; ++k)
            if (hm[k] < m) {
                m = hm[k];
                kb = k;
            }
        if (m == GT_NONE) break;
        const int stop = m + __ffs(ends[m >> 5] >> (m & 31));
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k == kb) {
                ++cur[k];
                hm[k] = cur[k] < end[k] ? runs[cur[k]] : GT_NONE;
            }
        const bool fx = kb & 1, fy = kb >> 1;
        const double xc = fx ? xl : xr, yc = fy ? yl : yr;
        for (; m < stop; m += GT_AHEAD) {
            Record r[GT_AHEAD];
#pragma unroll
            for (int q = 0; q < GT_AHEAD; ++q)
                if (m + q < stop) r[q] = rec[m + q];
#pragma unroll
            for (int q = 0; q < GT_AHEAD; ++q)
                if (m + q < stop) {
                    const double rx = r[q].x - xc, ry = r[q].y - yc;
                    const double px = FAST ? div_const(rx, dx, rdx) : rx / dx, py = FAST ? div_const(ry, dy, rdy) : ry / dy;
                    const double wx = fx ? px : (1.0 - px);
                    const double wy = fy ? py : (1.0 - py);
                    const double w = wx * wy;
                    ws = ws + w;
                    vs = vs + w * (second ? r[q].v1 : r[q].v0);
                }
        }
    }
    if (g.wt_sum) {
        g.wt_sum[(I - 1) + (J - 1) * g.ld_sum] = ws;
        g.val_wt_sum[(I - 1) + (J - 1) * g.ld_sum] = vs;
    }
    if (ws != 0.0)
        g.val_grid[(I - 1) + (J - 1) * nx] = vs / ws;   // safeDivision (MarkerToGrid.jl:164-172)
    else if (empty_counter)
        atomicAdd(empty_counter, 1ull);
}

__global__ void __launch_bounds__(GT_X * GT_Y, GT_BLOCKS) k_gather_runs(const __grid_constant__ SortGrids s, double dx,
                                                                      double dy, double rdx, double rdy,
                                                                      unsigned long long* __restrict__ empty_counter) {
    const SortGrid& g = s.g[blockIdx.y];
    if (*g.general == 0)
        gather_node<true>(s, g, dx, dy, rdx, rdy, empty_counter);
    else
        gather_node<false>(s, g, dx, dy, rdx, rdy, empty_counter);
}

// The allocation-free deposit's gather (its scratch holds no payload): the same merge of node (I, J)'s cells
// (I,J), (I-1,J), (I,J-1), (I-1,J-1) in ascending marker index, reading each marker's position and value
// through the sorted permutation.
__global__ void k_gather(const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ val,
                         const int32_t* __restrict__ offsets, const int32_t* __restrict__ perm, int64_t nx,
                         int64_t ny, double xmin, double ymin, double dx, double dy, double* __restrict__ val_grid,
                         double* __restrict__ val_wt_sum, double* __restrict__ wt_sum, int64_t ld_sum,
                         unsigned long long* __restrict__ empty_counter) {
    int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t nnodes = nx * ny;
    bool live = n < nnodes;
    int64_t I = live ? n % nx + 1 : 1, J = live ? n / nx + 1 : 1;
    int32_t cur[4], end[4];
    const int64_t ldc = nx + 1;
    // corner k: 0 = marker's top-left node (cell I,J), 1 = top-right (cell I-1,J),
    //           2 = bottom-left (cell I,J-1), 3 = bottom-right (cell I-1,J-1)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        int64_t ci = I - (k & 1), cj = J - (k >> 1);
        int64_t key = ci + cj * ldc;
        cur[k] = live ? offsets[key] : 0;
        end[k] = live ? offsets[key + 1] : 0;
    }
    double ws = 0.0, vs = 0.0;
    while (true) {
        int32_t best = 0x7fffffff;
        int kb = -1;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (cur[k] < end[k]) {
                int32_t m = perm[cur[k]];
                if (m < best) { best = m; kb = k; }
            }
        }
        if (kb < 0) break;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k == kb) ++cur[k];
        TopLeft t = topleft(xmin, ymin, x[best], y[best], dx, dy);
        double wx = (kb & 1) ? t.dxij : (1.0 - t.dxij);
        double wy = (kb >> 1) ? t.dyij : (1.0 - t.dyij);
        double w = wx * wy;
        ws = ws + w;
        vs = vs + w * val[best];
    }
    if (!live) return;
    if (wt_sum) {
        wt_sum[(I - 1) + (J - 1) * ld_sum] = ws;
        val_wt_sum[(I - 1) + (J - 1) * ld_sum] = vs;
    }
    if (ws != 0.0)
        val_grid[(I - 1) + (J - 1) * nx] = vs / ws;
    else if (empty_counter)
        atomicAdd(empty_counter, 1ull);
}

static unsigned grid_for(sf_ctx* ctx, int64_t n, int threads) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, threads), (int64_t)ctx->num_sms * 32));
}

// Step 1 for all grids of s: markers, or (records) runs
static int launch_keys(sf_ctx* ctx, const SortGrids& s, const double* x, const double* y, int64_t nm, double dx, double dy,
                       unsigned long long* bad_counter, cudaStream_t st) {
    if (nm == 0) return SF_OK;
    const unsigned blocks = grid_for(ctx, nm, DEP_THREADS);
    if (!s.rec)
        k_cell_keys<<<blocks, DEP_THREADS, 0, st>>>(x, y, nm, dx, dy, s, bad_counter);
    else if (s.n == 1)
        k_cell_runs<1><<<blocks, DEP_THREADS, 0, st>>>(x, y, nm, dx, dy, s, bad_counter);
    else
        k_cell_runs<SF_MAX_GRIDS><<<blocks, DEP_THREADS, 0, st>>>(x, y, nm, dx, dy, s, bad_counter);
    SF_LAUNCHED(ctx);
    return SF_OK;
}

// Step 2 for the grids of s, blockIdx.y each; no context (the allocation-free deposit), *launches: kernels launched
static int launch_scan(const SortGrids& s, cudaStream_t st, int* launches) {
    int64_t tiles = 0;
    for (int k = 0; k < s.n; ++k) tiles = std::max(tiles, ceil_div(s.g[k].ncells, SCAN_TILE));
    const dim3 grid((unsigned)tiles, (unsigned)s.n);
    const int scanned = tiles > SCAN_DIRECT;
    k_scan_tile_sums<<<grid, SCAN_THREADS, 0, st>>>(s);
    SF_CHECK_LAUNCH();
    if (scanned) {
        k_scan_tile_offsets<<<dim3(1, (unsigned)s.n), SCAN_THREADS, 0, st>>>(s);
        SF_CHECK_LAUNCH();
    }
    k_scan_tiles<<<grid, SCAN_THREADS, 0, st>>>(s, scanned);
    SF_CHECK_LAUNCH();
    *launches = 2 + scanned;
    return SF_OK;
}

// Steps 2-4 for the grids of s: the markers (or the first markers of the runs) in cell order, ascending in each cell,
// that is a stable counting sort.
static int launch_sort(sf_ctx* ctx, const SortGrids& s, int64_t nm, cudaStream_t st) {
    int n = 0;
    int rc = launch_scan(s, st, &n);
    ctx->launches += n;
    if (rc || nm == 0) return rc;
    int64_t cells = 0;
    for (int k = 0; k < s.n; ++k) cells = std::max(cells, s.g[k].ncells);
    const dim3 blocks(grid_for(ctx, nm, DEP_THREADS), (unsigned)s.n);
    if (s.rec)
        k_scatter_runs<<<blocks, DEP_THREADS, 0, st>>>(s, nm);
    else
        k_scatter<<<blocks, DEP_THREADS, 0, st>>>(s, nm);
    SF_LAUNCHED(ctx);
    k_sort_long<<<dim3((unsigned)ctx->num_sms * 2, (unsigned)s.n), SORT_THREADS, 0, st>>>(s);
    SF_LAUNCHED(ctx);
    k_sort_cells<<<dim3((unsigned)ceil_div(cells, SORT_CPB), (unsigned)s.n), SORT_THREADS, 0, st>>>(s);
    SF_LAUNCHED(ctx);
    return SF_OK;
}

// Scratch of a sort over the grids of s (xmin .. ncells set): what all grids need at once (records, keys, run ends and
// counts come from one pass over the markers) and, `together`, offsets, cursors and permutation of each grid, else those
// of one.  The counts and list lengths are one block, zeroed here.
static int sort_scratch(sf_ctx* ctx, SortGrids& s, int64_t nm, bool together, bool records, cudaStream_t st) {
    const int64_t nmk = std::max<int64_t>(nm, 1), per = round_up(nmk, 64), nlist = nm / (SORT_LONG + 1) + 1;
    int64_t cells = 0, most = 0, tiles = 0;
    for (int k = 0; k < s.n; ++k) {
        cells += s.g[k].ncells + 1;
        most = std::max(most, s.g[k].ncells + 1);
        tiles += ceil_div(s.g[k].ncells, SCAN_TILE);
    }
    const int n = together ? s.n : 1;
    int rc;
    if ((rc = ensure(ctx, ctx->keys, (size_t)(s.n * (per + per / 32)) * 4))) return rc;   // keys, run ends
    if ((rc = ensure(ctx, ctx->counts, (size_t)(cells + 2 * s.n) * 4))) return rc;        // counts, list lengths, general
    if ((rc = ensure(ctx, ctx->offsets, (size_t)(2 * n * most) * 4))) return rc;          // offsets, cursors
    if ((rc = ensure(ctx, ctx->scan_tmp, (size_t)tiles * 4))) return rc;
    if ((rc = ensure(ctx, ctx->longs, (size_t)(n * nlist) * 4))) return rc;
    if ((rc = ensure(ctx, ctx->perm, (size_t)(n * per) * 4))) return rc;
    if (records && (rc = ensure(ctx, ctx->records, (size_t)nmk * sizeof(Record)))) return rc;
    SF_CUDA(cudaMemsetAsync(ctx->counts.ptr, 0, (size_t)(cells + 2 * s.n) * 4, st));
    s.rec = records ? (Record*)ctx->records.ptr : nullptr;
    int32_t* counts = (int32_t*)ctx->counts.ptr;
    int32_t* tile = (int32_t*)ctx->scan_tmp.ptr;
    int64_t at = 0;
    for (int k = 0; k < s.n; ++k) {
        SortGrid& g = s.g[k];
        const int64_t q = together ? k : 0;
        g.keys = (int32_t*)ctx->keys.ptr + k * per;
        g.ends = (uint32_t*)ctx->keys.ptr + s.n * per + k * (per / 32);
        g.counts = counts + at;
        g.n_list = counts + cells + k;
        g.general = counts + cells + s.n + k;
        g.offsets = (int32_t*)ctx->offsets.ptr + 2 * q * most;
        g.cursor = g.offsets + most;
        g.tiles = tile;
        g.list = (int32_t*)ctx->longs.ptr + q * nlist;
        g.perm = (int32_t*)ctx->perm.ptr + q * per;
        at += g.ncells + 1;
        tile += ceil_div(g.ncells, SCAN_TILE);
    }
    return SF_OK;
}

static int launch_gather(sf_ctx* ctx, const SortGrids& s, double dx, double dy, cudaStream_t st) {
    int64_t blocks = 0;
    for (int k = 0; k < s.n; ++k) blocks = std::max(blocks, ceil_div(s.g[k].nx, GT_X) * ceil_div(s.g[k].ny, GT_Y));
    k_gather_runs<<<dim3((unsigned)blocks, (unsigned)s.n), GT_X * GT_Y, 0, st>>>(
        s, dx, dy, 1.0 / dx, 1.0 / dy, ctx->d_counters + CNT_EMPTY_NODES);
    SF_LAUNCHED(ctx);
    return SF_OK;
}

// whether two of the arrays that the deposits of s write overlap
static bool outputs_overlap(const SortGrids& s, int64_t n_sum) {
    struct Range { const double *b, *e; } r[SF_MAX_GRIDS + 2];
    int n = 0;
    for (int k = 0; k < s.n; ++k) {
        r[n++] = Range{s.g[k].val_grid, s.g[k].val_grid + s.g[k].nx * s.g[k].ny};
        if (s.g[k].wt_sum) {
            r[n++] = Range{s.g[k].wt_sum, s.g[k].wt_sum + n_sum};
            r[n++] = Range{s.g[k].val_wt_sum, s.g[k].val_wt_sum + n_sum};
        }
    }
    for (int i = 0; i < n; ++i)
        for (int j = i + 1; j < n; ++j)
            if (r[i].b < r[j].e && r[j].b < r[i].e) return true;
    return false;
}

// The deposits of s's grids over the same markers (only the last one's sums are kept), whose values come from at most
// two arrays.  Up to DEPOSIT_TOGETHER markers all grids go through each kernel in one launch; beyond, or where they
// write the same places, one grid after the other, in the scratch of one.
static int deposit_group(sf_ctx* ctx, SortGrids& s, const double* x, const double* y, int64_t nm, double dx, double dy,
                         int64_t n_sum, cudaStream_t st) {
    const bool together = s.n > 1 && nm <= DEPOSIT_TOGETHER && !outputs_overlap(s, n_sum);
    int rc;
    if ((rc = sort_scratch(ctx, s, nm, together, true, st))) return rc;
    s.val0 = s.g[0].val;
    s.val1 = nullptr;
    for (int k = 0; k < s.n; ++k) {
        s.g[k].second = s.g[k].val != s.val0;
        if (s.g[k].second) s.val1 = s.g[k].val;
    }
    if (!(div_const_takes(dx) && div_const_takes(dy)))
        SF_CUDA(cudaMemsetAsync(s.g[0].general, 1, (size_t)s.n * 4, st));
    if ((rc = launch_keys(ctx, s, x, y, nm, dx, dy, ctx->d_counters + CNT_BAD_MARKERS, st))) return rc;
    const SortGrid& last = s.g[s.n - 1];
    for (int k = 0; k < (together ? 1 : s.n); ++k) {
        SortGrids one = s;
        one.g[0] = s.g[k];
        one.n = 1;
        const SortGrids& pass = together ? s : one;
        if ((rc = launch_sort(ctx, pass, nm, st))) return rc;
        if (last.wt_sum && (together || k == s.n - 1)) {
            SF_CUDA(cudaMemsetAsync(last.wt_sum, 0, (size_t)n_sum * 8, st));
            SF_CUDA(cudaMemsetAsync(last.val_wt_sum, 0, (size_t)n_sum * 8, st));
        }
        if ((rc = launch_gather(ctx, pass, dx, dy, st))) return rc;
    }
    return SF_OK;
}

// any grids: in order, in groups whose values come from at most two arrays
static int deposit(sf_ctx* ctx, const SortGrids& all, const double* x, const double* y, int64_t nm, double dx, double dy,
                   int64_t n_sum, cudaStream_t st) {
    for (int k = 0; k < all.n;) {
        SortGrids s{};
        const double* second = nullptr;
        for (; k < all.n; ++k) {
            const double* v = all.g[k].val;
            if (s.n > 0 && v != s.g[0].val) {
                if (second && v != second) break;
                second = v;
            }
            s.g[s.n++] = all.g[k];
        }
        const int rc = deposit_group(ctx, s, x, y, nm, dx, dy, n_sum, st);
        if (rc) return rc;
    }
    return SF_OK;
}

}  // namespace sf

using namespace sf;

extern "C" {

int sf_bilinear_marker_to_grid(sf_ctx* ctx, double x_grid_min, double y_grid_min, double* val_grid, int64_t nx,
                               int64_t ny, const double* x_m, const double* y_m, const double* val_m, int64_t nm,
                               double dx, double dy, double* val_wt_sum, double* wt_sum, int64_t ld_sum,
                               int64_t n_sum, void* stream) {
    SF_REQUIRE(ctx, "sf_bilinear_marker_to_grid: ctx is NULL");
    SF_REQUIRE(val_grid && nx >= 1 && ny >= 1, "sf_bilinear_marker_to_grid: bad grid");
    SF_REQUIRE(nm >= 0 && (nm == 0 || (x_m && y_m && val_m)), "sf_bilinear_marker_to_grid: bad markers");
    SF_REQUIRE(nm < (int64_t)INT32_MAX, "sf_bilinear_marker_to_grid: more than 2^31-1 markers");
    SF_REQUIRE((nx + 1) * (ny + 1) < (int64_t)INT32_MAX, "sf_bilinear_marker_to_grid: grid too large");
    SF_REQUIRE(dx > 0.0 && dy > 0.0, "sf_bilinear_marker_to_grid: dx, dy must be positive");
    SF_REQUIRE((val_wt_sum == nullptr) == (wt_sum == nullptr), "sf_bilinear_marker_to_grid: give both sum arrays or neither");
    if (wt_sum) SF_REQUIRE(ld_sum >= nx && n_sum >= ld_sum * (ny - 1) + nx, "sf_bilinear_marker_to_grid: sum arrays too small");
    int rc = set_device(ctx);
    if (rc) return rc;
    markers_launched(ctx, ctx->device, nm);
    cudaStream_t s = as_stream(stream);
    SortGrids sg{};
    sg.n = 1;
    SortGrid& g = sg.g[0];
    g.xmin = x_grid_min;
    g.ymin = y_grid_min;
    g.nx = nx;
    g.ny = ny;
    g.ncells = (nx + 1) * (ny + 1);
    g.val = val_m;
    g.val_grid = val_grid;
    g.val_wt_sum = val_wt_sum;
    g.wt_sum = wt_sum;
    g.ld_sum = ld_sum;
    return deposit(ctx, sg, x_m, y_m, nm, dx, dy, n_sum, s);
}

int sf_bilinear_marker_to_grids(sf_ctx* ctx, const sf_deposit_grid* grids, int n_grids, const double* x_m,
                                const double* y_m, int64_t nm, double dx, double dy, double* val_wt_sum,
                                double* wt_sum, int64_t ld_sum, int64_t n_sum, void* stream) {
    SF_REQUIRE(ctx, "sf_bilinear_marker_to_grids: ctx is NULL");
    SF_REQUIRE(grids && n_grids >= 1 && n_grids <= SF_MAX_GRIDS, "sf_bilinear_marker_to_grids: 1 to SF_MAX_GRIDS grids");
    SF_REQUIRE(nm >= 0 && (nm == 0 || (x_m && y_m)), "sf_bilinear_marker_to_grids: bad markers");
    SF_REQUIRE(nm < (int64_t)INT32_MAX, "sf_bilinear_marker_to_grids: more than 2^31-1 markers");
    SF_REQUIRE(dx > 0.0 && dy > 0.0, "sf_bilinear_marker_to_grids: dx, dy must be positive");
    SF_REQUIRE((val_wt_sum == nullptr) == (wt_sum == nullptr), "sf_bilinear_marker_to_grids: give both sum arrays or neither");
    for (int g = 0; g < n_grids; ++g) {
        const sf_deposit_grid& d = grids[g];
        SF_REQUIRE(d.val_grid && d.nx >= 1 && d.ny >= 1, "sf_bilinear_marker_to_grids: bad grid");
        SF_REQUIRE(nm == 0 || d.val_m, "sf_bilinear_marker_to_grids: bad marker values");
        SF_REQUIRE((d.nx + 1) * (d.ny + 1) < (int64_t)INT32_MAX, "sf_bilinear_marker_to_grids: grid too large");
        if (wt_sum)
            SF_REQUIRE(ld_sum >= d.nx && n_sum >= ld_sum * (d.ny - 1) + d.nx,
                       "sf_bilinear_marker_to_grids: sum arrays too small");
    }
    int rc = set_device(ctx);
    if (rc) return rc;
    markers_launched(ctx, ctx->device, nm);
    cudaStream_t s = as_stream(stream);
    SortGrids sg{};
    sg.n = n_grids;
    for (int k = 0; k < n_grids; ++k) {
        const sf_deposit_grid& d = grids[k];
        SortGrid& g = sg.g[k];
        g.xmin = d.x_grid_min;
        g.ymin = d.y_grid_min;
        g.nx = d.nx;
        g.ny = d.ny;
        g.ncells = (d.nx + 1) * (d.ny + 1);
        g.val = d.val_m;
        g.val_grid = d.val_grid;
        // as after one call per grid in order: the sum arrays hold the last grid's sums
        g.val_wt_sum = k == n_grids - 1 ? val_wt_sum : nullptr;
        g.wt_sum = k == n_grids - 1 ? wt_sum : nullptr;
        g.ld_sum = ld_sum;
    }
    return deposit(ctx, sg, x_m, y_m, nm, dx, dy, n_sum, s);
}

int sf_rebin_markers(sf_ctx* ctx, const double* x_m, const double* y_m, int64_t nm, double x_grid_min,
                     double y_grid_min, double dx, double dy, int64_t nx, int64_t ny, int32_t* counts,
                     int32_t* offsets, int32_t* perm, void* stream) {
    SF_REQUIRE(ctx, "sf_rebin_markers: ctx is NULL");
    SF_REQUIRE(nx >= 1 && ny >= 1 && dx > 0.0 && dy > 0.0, "sf_rebin_markers: bad grid");
    SF_REQUIRE(nm >= 0 && (nm == 0 || (x_m && y_m)), "sf_rebin_markers: bad markers");
    SF_REQUIRE(nm < (int64_t)INT32_MAX && (nx + 1) * (ny + 1) < (int64_t)INT32_MAX, "sf_rebin_markers: too large");
    int rc = set_device(ctx);
    if (rc) return rc;
    markers_launched(ctx, ctx->device, nm);
    cudaStream_t s = as_stream(stream);
    SortGrids sg{};
    sg.n = 1;
    SortGrid& g = sg.g[0];
    g.xmin = x_grid_min;
    g.ymin = y_grid_min;
    g.nx = nx;
    g.ny = ny;
    g.ncells = (nx + 1) * (ny + 1);
    if ((rc = sort_scratch(ctx, sg, nm, false, false, s))) return rc;
    // the caller's arrays, where given, are the sort's own
    if (counts) {
        SF_CUDA(cudaMemsetAsync(counts, 0, (size_t)g.ncells * 4, s));
        g.counts = counts;
    }
    if (offsets) g.offsets = offsets;
    if (perm && nm > 0) g.perm = perm;
    if ((rc = launch_keys(ctx, sg, x_m, y_m, nm, dx, dy, ctx->d_counters + CNT_OUTSIDE, s))) return rc;
    return launch_sort(ctx, sg, nm, s);
}

}  // extern "C"

// ==========================================================================
// Allocation-free deposit
// ==========================================================================
// Some callers cannot let a library call cudaMalloc / cudaFree: hosts whose
// runtime owns the device memory through its own pool (for example Julia's
// CUDA.jl or PyTorch with the rest of the GPU reserved), where an allocation
// outside the pool fails or forces an eviction; latency-critical stream loops,
// where cudaMalloc / cudaFree synchronise the whole device and stall the other
// streams; and processes held to a fixed memory budget after start-up.  For
// them sf_bilinear_marker_to_grid_noalloc runs the same deposit with all of
// its scratch in the file-scope array below, which every GPU that loads the
// library holds (about 11 MB) until the process exits.
#include <mutex>

namespace sf {

constexpr int64_t NA_MAX_MARKERS = SF_NOALLOC_MAX_MARKERS;
constexpr int64_t NA_MAX_CELLS = SF_NOALLOC_MAX_CELLS;          // (nx + 1) * (ny + 1)
constexpr int64_t NA_SCAN_TILES = (NA_MAX_CELLS + SCAN_TILE - 1) / SCAN_TILE;
// layout (bytes): keys | perm | offsets | counts | cursors | scan tiles | long cells | counters
constexpr size_t NA_OFF_KEYS = 0;
constexpr size_t NA_OFF_PERM = NA_OFF_KEYS + 4 * NA_MAX_MARKERS;
constexpr size_t NA_OFF_OFFSETS = NA_OFF_PERM + 4 * NA_MAX_MARKERS;
constexpr size_t NA_OFF_COUNTS = NA_OFF_OFFSETS + 4 * (NA_MAX_CELLS + 64);
constexpr size_t NA_OFF_CURSOR = NA_OFF_COUNTS + 4 * (NA_MAX_CELLS + 64);
constexpr size_t NA_OFF_TILES = NA_OFF_CURSOR + 4 * (NA_MAX_CELLS + 64);
constexpr size_t NA_OFF_LIST = NA_OFF_TILES + 4 * ((NA_SCAN_TILES + 63) / 64 * 64);
constexpr size_t NA_OFF_COUNTERS = NA_OFF_LIST + 4 * ((NA_MAX_MARKERS / (SORT_LONG + 1) + 64) / 64 * 64);
constexpr size_t NA_BYTES = NA_OFF_COUNTERS + 4 * sizeof(unsigned long long);   // 2 counters, the long-cell count

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];

constexpr int NA_MAX_DEVICES = 64;
static unsigned char* g_noalloc_ptr[NA_MAX_DEVICES] = {};
static int g_noalloc_sms[NA_MAX_DEVICES] = {};
static std::mutex g_noalloc_mutex;

// Device address of g_noalloc_scratch and the SM count of the current device.
// In host code the array's name is only a host-side stand-in, so the address
// is looked up once per device (with that device current) and cached, with
// the SM count that sizes the marker kernels' grids.  A device reset
// invalidates the cache (documented at the declaration).
static int noalloc_scratch(unsigned char** out, int* num_sms, int* device) {
    int dev = 0;
    SF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NA_MAX_DEVICES) return fail(SF_ERR_NO_DEVICE, "noalloc deposit: device index too large");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        int sms = 0;
        SF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            (void)cudaGetLastError();
            return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
        }
        g_noalloc_sms[dev] = std::max(1, sms);
        g_noalloc_ptr[dev] = (unsigned char*)p;
    }
    *out = g_noalloc_ptr[dev];
    *device = dev;
    *num_sms = g_noalloc_sms[dev];
    return SF_OK;
}

}  // namespace sf

extern "C" int sf_bilinear_marker_to_grid_noalloc(double x_grid_min, double y_grid_min, double* val_grid, int64_t nx,
                                                  int64_t ny, const double* x_m, const double* y_m, const double* val_m,
                                                  int64_t nm, double dx, double dy, void* stream) {
    SF_REQUIRE(val_grid && nx >= 1 && ny >= 1, "sf_bilinear_marker_to_grid_noalloc: bad grid");
    SF_REQUIRE(nm >= 0 && (nm == 0 || (x_m && y_m && val_m)), "sf_bilinear_marker_to_grid_noalloc: bad markers");
    SF_REQUIRE(dx > 0.0 && dy > 0.0, "sf_bilinear_marker_to_grid_noalloc: dx, dy must be positive");
    if (nm > NA_MAX_MARKERS)
        return fail(SF_ERR_TOO_LARGE, "sf_bilinear_marker_to_grid_noalloc: " + std::to_string(nm) +
                                          " markers exceed the fixed scratch (at most " +
                                          std::to_string(NA_MAX_MARKERS) + ")");
    if (nx > NA_MAX_CELLS || ny > NA_MAX_CELLS || (nx + 1) * (ny + 1) > NA_MAX_CELLS)
        return fail(SF_ERR_TOO_LARGE, "sf_bilinear_marker_to_grid_noalloc: a " + std::to_string(nx) + " x " +
                                          std::to_string(ny) + " grid exceeds the fixed scratch (at most " +
                                          std::to_string(NA_MAX_CELLS) + " cells (nx+1)*(ny+1))");
    unsigned char* base = nullptr;
    int num_sms = 0, device = 0;
    int rc = noalloc_scratch(&base, &num_sms, &device);
    if (rc) return rc;
    markers_launched(nullptr, device, nm);
    cudaStream_t s = as_stream(stream);
    unsigned long long* counters = (unsigned long long*)(base + NA_OFF_COUNTERS);
    const int64_t ncells = (nx + 1) * (ny + 1);
    SortGrids sg{};
    sg.n = 1;
    SortGrid& g = sg.g[0];
    g.xmin = x_grid_min;
    g.ymin = y_grid_min;
    g.nx = nx;
    g.ny = ny;
    g.ncells = ncells;
    g.keys = (int32_t*)(base + NA_OFF_KEYS);
    g.perm = (int32_t*)(base + NA_OFF_PERM);
    g.offsets = (int32_t*)(base + NA_OFF_OFFSETS);
    g.counts = (int32_t*)(base + NA_OFF_COUNTS);
    g.cursor = (int32_t*)(base + NA_OFF_CURSOR);
    g.tiles = (int32_t*)(base + NA_OFF_TILES);
    g.list = (int32_t*)(base + NA_OFF_LIST);
    g.n_list = (int32_t*)(counters + 2);
    int32_t *offsets = g.offsets, *perm = g.perm;
    // the array keeps the previous call's contents: clear what must start at zero
    SF_CUDA(cudaMemsetAsync(g.counts, 0, (size_t)ncells * 4, s));
    SF_CUDA(cudaMemsetAsync(counters, 0, 4 * sizeof(unsigned long long), s));
    // grid-stride marker kernels: up to 32 blocks per SM of this device
    const unsigned blocks =
        (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(nm, DEP_THREADS), (int64_t)num_sms * 32));
    if (nm > 0) {
        k_cell_keys<<<blocks, DEP_THREADS, 0, s>>>(x_m, y_m, nm, dx, dy, sg, counters + 0);
        SF_CHECK_LAUNCH();
    }
    int n = 0;
    if ((rc = launch_scan(sg, s, &n))) return rc;
    if (nm > 0) {
        k_scatter<<<blocks, DEP_THREADS, 0, s>>>(sg, nm);
        SF_CHECK_LAUNCH();
        // long segments by the radix sort (the spent keys are its buffer), the others one thread per cell
        k_sort_long<<<(unsigned)num_sms * 2, SORT_THREADS, 0, s>>>(sg);
        SF_CHECK_LAUNCH();
    }
    k_sort_segments<<<(unsigned)ceil_div(ncells, 128), 128, 0, s>>>(offsets, ncells, perm);
    SF_CHECK_LAUNCH();
    k_gather<<<(unsigned)ceil_div(nx * ny, DEP_THREADS), DEP_THREADS, 0, s>>>(
        x_m, y_m, val_m, offsets, perm, nx, ny, x_grid_min, y_grid_min, dx, dy, val_grid, nullptr, nullptr, 0,
        counters + 1);
    SF_CHECK_LAUNCH();
    return SF_OK;
}
