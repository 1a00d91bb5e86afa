// sf_resident.cu -- many pseudo-transient iterations (StokesSolver_multixpu.jl:48-57) of a small grid in one launch.
//
// On a small grid an iteration's arithmetic takes less than launching a kernel for it.  Here the state stays on
// the chip for as many iterations as the reference's loop runs without an event (a residual check, a dt update):
//
//   * the grid is cut into at most one tile per SM; a thread owns the same points in every iteration and keeps their
//     P, rates and parameters in registers: up to four, one above the other, which share what they read (at 511 x 385
//     17 accesses to shared memory per point and iteration; points of their own 25, and 2.82 us instead of 2.60).
//     Vx, Vy and the stage-1 results of a tile (P, tau_xx, tau_yy, tau_xy) are in shared memory.  An iteration is the
//     two stages of k_pt_iter, a barrier after each, and the exchange of the velocities on the tiles' borders, one of:
//   * the tiles are the blocks of one cluster (up to 16): a thread stores a border point's velocities also into the
//     neighbours' shared memory (st.async), counted there on an mbarrier that the neighbour waits for.  Velocities and
//     mbarriers are double-buffered: a neighbour's border may come in while the old ones are still read, but it cannot
//     be two iterations ahead;
//   * through L2: every value travels in a 16-byte slot as two 8-byte words {half, tag}, the tag being the iteration's
//     number, so that a reader that sees its tag has the value: one store and one load instead of data, fence and flag.
//     Slots are double-buffered by parity; a tile cannot be two iterations ahead of one that it exchanges with, so a
//     slot is never overwritten unread.  The launch is cooperative (all tiles resident), and every wait has a
//     wall-clock budget.
//
// A tile's halo column and row of P and tau are computed by both neighbours from the same values.  Every expression
// keeps the reference's order of operations (compiled without contraction): bit-identical to single iterations.
//
// What bounds it: latency.  A cluster's iteration takes 0.67 us at 20 x 26 and 0.74 at 64^2, checks included
// (k_pt_iter, one launch each: 4.5 and 4.4): the two stages' dependent FP64 chains, two barriers and the neighbours.
// Through L2, 128^2 (104 tiles of 16 x 10 points, 6 warps) takes 1.4 us, about half of it the exchange, against 5.2; at
// 511 x 385 (1450 points per SM) 2.6 us, there barriers and shared memory (16 warps, issue 40%), against 8.3.  Testing every point's flags and
// sending borders to L2 from the update itself took 905 instructions per warp and iteration at 511 x 385 and 4.2 us.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include "sf_resident.cuh"
#include "sf_tma.cuh"

namespace sf {
namespace {

constexpr uint64_t RES_WAIT_NS = 2000000000ull;
constexpr int RES_MAX_K = 4;

// slots of a tile: from the left and right neighbour H of each component, from below and above W of each, and two
// corners (Vx of the upper left, Vy of the lower right one: the only diagonal entries that an iteration reads)
__host__ __device__ __forceinline__ int slots_of(int W, int H) { return 4 * (W + H) + 2; }

__device__ __forceinline__ void put(ulonglong2* slot, double v, uint32_t tag) {
    const uint64_t b = (uint64_t)__double_as_longlong(v), t = (uint64_t)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(slot), "l"(t | (b & 0xffffffffull)),
                 "l"(t | (b >> 32))
                 : "memory");
}

__device__ __forceinline__ bool get(const ulonglong2* slot, uint32_t tag, double* v) {
    uint64_t a, b;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(slot) : "memory");
    if ((uint32_t)(a >> 32) != tag || (uint32_t)(b >> 32) != tag) return false;
    *v = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
    return true;
}

// the address of this block's shared-memory entry p in the block of the given rank of the cluster
__device__ __forceinline__ uint32_t in_block(const void* p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
// v to addr in another block of the cluster, counted (8 bytes) on the barrier bar of that block
__device__ __forceinline__ void put_in_block(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
// whether phase `parity` of the barrier is over, and with it what other blocks put here for it is seen
__device__ __forceinline__ bool all_in(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// every thread of the cluster: earlier shared-memory writes, remote ones too, are seen by all afterwards
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// rows of points of a tile, its halo row included, in whole groups of K
__host__ __device__ __forceinline__ int rows_of(int H, int K) { return (H + K) / K * K; }

// what a thread's point is: one whose Vx / Vy it updates (the others' are boundary entries, zero), one of the tile (not
// of its halo column or row), and the sides of the domain that it lies on
enum { PT_X = 1, PT_Y = 2, PT_OWN = 4, PT_I0 = 8, PT_I1 = 16, PT_J0 = 32, PT_J1 = 64, PT_DX = 128,
       PT_BOUND = PT_I0 | PT_I1 | PT_J0 | PT_J1 };

// K points per thread.  CLUSTER: the tiles are the blocks of one cluster (or there is one tile)
template <int K, bool CLUSTER>
__global__ void __launch_bounds__(512, 1) k_pt_resident(const __grid_constant__ ResidentParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int gave_up;
    __shared__ __align__(8) uint64_t bar[2];   // CLUSTER: halo entries come in, by parity of the iteration
    __shared__ unsigned long long max_v[2];
    // An earlier launch's tiles were lost (a block that starts after one of this launch gave up may leave, too)
    const int lost_before = *(const volatile int*)p.err_flag;
    if (p.err && !goes_on(p.err, p.eps)) return;   // (all blocks)
    if (lost_before) return;
    const int W = p.W, H = p.H, pitch = W + 2;
    const int rows = rows_of(H, K);                               // of points that threads have
    const int comp1 = (rows + 1) * pitch;                         // from an entry of Vx to that of Vy
    double* sVx = reinterpret_cast<double*>(smem_raw);            // (rows + 1) x (W + 2): entry (0, 0) is Vx(i0, j0)
    double* sVy = sVx + comp1;
    // CLUSTER: a second pair, written while the first is read (a neighbour's border may come in at any time)
    double* sVx_n = CLUSTER ? sVy + comp1 : sVx;
    double* sVy_n = sVx_n + comp1;
    double* const sTxx = sVy_n + comp1;                           // `rows` rows of the same pitch
    double* const sTyy = sTxx + rows * pitch;
    double* const sPn = sTyy + rows * pitch;
    double* const sTxy = sPn + rows * pitch;
    const int tid = threadIdx.x, NT = blockDim.x;
    const int bx = blockIdx.x % p.ntx, by = blockIdx.x / p.ntx;
    const int i0 = bx * W, j0 = by * H;
    const int Nx = p.Nx, Ny = p.Ny;
    const int64_t LD = p.LD;
    const double _dx = p._dx, _dy = p._dy;
    const bool has_l = bx > 0, has_r = bx + 1 < p.ntx, has_b = by > 0, has_t = by + 1 < p.nty;

    // ---- state and parameters onto the chip ----
    for (int n = tid; n < comp1; n += NT) {
        const int b = n / pitch, a = n - b * pitch;
        // (the domain's corners are read by nothing but the last iteration's tau_xy, which finds them zero)
        const int i = i0 + a, j = j0 + b;
        const bool in = i <= Nx && j <= Ny && !(i == 0 && (j == 0 || j == Ny)) && !(i == Nx && j == 0);
        const int64_t o = i + (int64_t)j * LD;
        sVx[n] = in ? p.Vx_in[o] : 0.0;
        sVy[n] = in ? p.Vy_in[o] : 0.0;
        if (CLUSTER) sVx_n[n] = sVy_n[n] = 0.0;
    }
    if (tid < 2) max_v[tid] = 0;   // (barriers follow)
    double P[K], dvx[K], dvy[K], tp[K], mu2[K], mb[K], tx[K], ty[K], rho[K], gx[K], gy[K];
    // the thread's points: K of a column a <= W, from row b0 on (b <= H: the tile and one more column and row)
    const bool live = tid < (W + 1) * (rows / K);   // (the other threads compute on the first points and store nothing)
    const int b0 = live ? tid / (W + 1) * K : 0, a = live ? tid % (W + 1) : 0;
    const int o0 = b0 * pitch + a;
    int kind[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int b = b0 + k;
        const int i = i0 + a, j = j0 + b;
        kind[k] = 0;
        P[k] = dvx[k] = dvy[k] = tp[k] = mu2[k] = mb[k] = tx[k] = ty[k] = rho[k] = gx[k] = gy[k] = 0.0;
        if (!live || b > H) continue;
        const int64_t o = i + (int64_t)j * LD;
        const bool own = a < W && b < H && i < Nx - 1 && j < Ny - 1;
        if (own)
            kind[k] |= PT_OWN | (i == 0 ? PT_I0 : 0) | (i == Nx - 2 ? PT_I1 : 0) | (j == 0 ? PT_J0 : 0) |
                       (j == Ny - 2 ? PT_J1 : 0);
        if (i < Nx - 1 && j < Ny - 1) {
            P[k] = p.P_in[o];
            tp[k] = p.dtp[o];
            mu2[k] = p.mup2[o];
        }
        if (i < Nx && j < Ny) mb[k] = p.mub[o];
        if (own && i < Nx - 2) {
            kind[k] |= PT_X;
            dvx[k] = p.dVx_in[o];
            tx[k] = p.dtx[o];
        }
        if (own && j < Ny - 2) {
            kind[k] |= PT_Y;
            dvy[k] = p.dVy_in[o];
            ty[k] = p.dty[o];
            rho[k] = p.rho[o + 1 + LD];
            gx[k] = p.rho[o + 2 + LD] - p.rho[o + LD];
            gy[k] = p.rho[o + 1 + 2 * LD] - p.rho[o + 1];
        }
    }
    const double dt = *p.dt_ptr, g_y = p.g_y, dampX = p.dampX, dampY = p.dampY;

    // The tile's halo slots, and the border entries that fill its neighbours' ones.  Slots: [from left: Vx, Vy][from
    // right][from below][from above][Vx of the upper left tile, Vy of the lower right one].  The last tiles of a row or
    // column may hold fewer points than W x H.
    const int nslots = slots_of(W, H), tiles = p.ntx * p.nty;
    const int hv = min(H, Ny - 1 - j0), wv = min(W, Nx - 1 - i0);
    // slot n: where its value goes in this tile (an offset from sVx), which entry of this tile fills the slot of the
    // same kind of the neighbour on the other side, and that neighbour (as a difference of tile numbers); -1: nobody's
    auto halo = [&](int n, int& to, int& from, int& peer) {
        to = from = -1;
        peer = 0;
        if (n < 4 * H) {                 // from the left or right; filled for the right or left
            const int side = n / (2 * H), m = n - side * 2 * H, comp = m / H, b = m - comp * H;
            if ((side ? has_r : has_l) && b < hv) to = comp * comp1 + (b + 1) * pitch + (side ? W + 1 : 0);
            if ((side ? has_l : has_r) && b < hv) from = comp * comp1 + (b + 1) * pitch + (side ? 1 : W);
            peer = side ? -1 : 1;
        } else if (n < 4 * (H + W)) {    // from below or above; filled for the one above or below
            const int q = n - 4 * H, side = q / (2 * W), m = q - side * 2 * W, comp = m / W, a = m - comp * W;
            if ((side ? has_t : has_b) && a < wv) to = comp * comp1 + (side ? H + 1 : 0) * pitch + a + 1;
            if ((side ? has_b : has_t) && a < wv) from = comp * comp1 + (side ? 1 : H) * pitch + a + 1;
            peer = side ? -p.ntx : p.ntx;
        } else if (n == 4 * (H + W)) {   // Vx of the upper left tile; filled for the lower right one
            if (has_l && has_t) to = (H + 1) * pitch;
            if (has_r && has_b) from = pitch + W;
            peer = 1 - p.ntx;
        } else if (n < nslots) {         // Vy of the lower right tile; filled for the upper left one
            if (has_r && has_b) to = comp1 + W + 1;
            if (has_l && has_t) from = comp1 + H * pitch + 1;
            peer = p.ntx - 1;
        }
    };
    int to0 = -1, from0 = -1, peer0 = 0;
    // CLUSTER: where a border point's Vx goes in the neighbour to its left or right, in the one below or above, and (a
    // corner's Vx or Vy) in the diagonal one; 0: nowhere.  Vy lies behind Vx, the other pair of buffers `other` further
    uint32_t at_x[K], at_y[K], at_d[K], bar_x[K], bar_y[K], bar_d[K];
    uint32_t other = (uint32_t)(2 * comp1 * 8);
    // bytes that come in per iteration
    const uint32_t expected = 8u * (2 * (has_l + has_r) * hv + 2 * (has_b + has_t) * wv + (has_l && has_t) + (has_r && has_b));
    bool lost = false;
    if (CLUSTER) {
        if (tid == 0) {
            mbar_init(&bar[0], 1);
            mbar_init(&bar[1], 1);
            fence_mbar_init();
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            at_x[k] = at_y[k] = at_d[k] = bar_x[k] = bar_y[k] = bar_d[k] = 0;
            if (!(kind[k] & PT_OWN)) continue;
            const int b = b0 + k, t = blockIdx.x;
            if ((a == 0 && has_l) || (a == W - 1 && has_r)) bar_x[k] = in_block(bar, a == 0 && has_l ? t - 1 : t + 1);
            if ((b == 0 && has_b) || (b == H - 1 && has_t)) bar_y[k] = in_block(bar, b == 0 && has_b ? t - p.ntx : t + p.ntx);
            if (a == 0 && has_l) at_x[k] = in_block(sVx_n + (b + 1) * pitch + W + 1, t - 1);
            if (a == W - 1 && has_r) at_x[k] = in_block(sVx_n + (b + 1) * pitch, t + 1);
            if (b == 0 && has_b) at_y[k] = in_block(sVx_n + (H + 1) * pitch + a + 1, t - p.ntx);
            if (b == H - 1 && has_t) at_y[k] = in_block(sVx_n + a + 1, t + p.ntx);
            if (a == W - 1 && b == 0 && has_r && has_b) {
                at_d[k] = in_block(sVx_n + (H + 1) * pitch, t + 1 - p.ntx);
                bar_d[k] = in_block(bar, t + 1 - p.ntx);
                kind[k] |= PT_DX;
            }
            if (a == 0 && b == H - 1 && has_l && has_t) {
                at_d[k] = in_block(sVy_n + W + 1, t - 1 + p.ntx);
                bar_d[k] = in_block(bar, t - 1 + p.ntx);
            }
        }
        cluster_sync();
    } else {
        halo(tid, to0, from0, peer0);
        if (tid == 0) gave_up = 0;
        __syncthreads();
    }

    for (int it = 0; it < p.iters; ++it) {
        // ---- stage 1: compute_P_tau! (:140-169) on the tile and one more column and row.  Evaluated at every point
        // (outside the domain on whatever is there; nothing that is kept depends on it) ----
        if (CLUSTER && tid == 0 && expected && it + 1 < p.iters) mbar_arrive_expect_tx(&bar[it & 1], expected);
        double sterm[K], txx[K], tyy[K], txy[K];
        {
            // (every entry once: points of a column share theirs)
            double vx0 = sVx[o0], vx1 = sVx[o0 + pitch], vx1r = sVx[o0 + pitch + 1], vy0r = sVy[o0 + 1];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int o = o0 + k * pitch;
                const double vx2 = sVx[o + 2 * pitch], vx2r = sVx[o + 2 * pitch + 1];
                const double vy0 = sVy[o], vy1r = sVy[o + pitch + 1];
                const double dVx_dy = (vx1 - vx0) * _dy;
                const double dVy_dx = (vy0r - vy0) * _dx;
                txy[k] = mb[k] * (dVx_dy + dVy_dx);
                const double dVx_dx = (vx1r - vx1) * _dx;
                const double dVy_dy = (vy1r - vy0r) * _dy;
                const double div = dVx_dx + dVy_dy;
                P[k] = P[k] - tp[k] * div;
                const double third = 1.0 / 3.0 * div;
                txx[k] = mu2[k] * (dVx_dx - third);
                tyy[k] = mu2[k] * (dVy_dy - third);
                if (p.divV && it + 1 == p.iters && (kind[k] & PT_OWN)) {
                    const int64_t q = i0 + a + (int64_t)(j0 + b0 + k) * LD;
                    p.divV[q] = div;
                    p.txx[q] = txx[k];
                    p.tyy[q] = tyy[k];
                }
                // the gravity term of compute_ResY (:189-202), from the old velocities
                const double av = 0.25 * (vx1 + vx1r + vx2 + vx2r);
                sterm[k] = g_y * (rho[k] - dt * (av * gx[k] * 0.5 * _dx + vy1r * gy[k] * 0.5 * _dy));
                if (live) {
                    sTxy[o] = txy[k];
                    sPn[o] = P[k];
                    sTxx[o] = txx[k];
                    if (k == 0) sTyy[o] = tyy[k];   // (the other rows' are read by their thread alone)
                }
                vx0 = vx1;
                vx1 = vx2;
                vx1r = vx2r;
                vy0r = vy1r;
            }
        }
        __syncthreads();
        // ---- stage 2: compute_dV!, compute_V! (:209-234), the boundary kernels (:53-56) ----
        double txy01 = sTxy[o0 + 1];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int o = o0 + k * pitch;
            const bool top = k + 1 == K;    // the point above is another thread's
            const int up = top ? k : k + 1;
            const double txy10 = top ? sTxy[o + pitch] : txy[up], tyy10 = top ? sTyy[o + pitch] : tyy[up];
            const double P10 = top ? sPn[o + pitch] : P[up];
            const double txy11 = sTxy[o + pitch + 1];
            const double Rx = (sTxx[o + 1] - txx[k]) * _dx + (txy11 - txy01) * _dy - (sPn[o + 1] - P[k]) * _dx;
            const double Ry = (tyy10 - tyy[k]) * _dy + (txy11 - txy10) * _dx - (P10 - P[k]) * _dy + sterm[k];
            txy01 = txy11;
            dvx[k] = dampX * dvx[k] + Rx;
            dvy[k] = dampY * dvy[k] + Ry;
            // Vx(Nx-1) and Vy(Ny-1) are the zero entries of the boundary
            const double xn = (kind[k] & PT_X) ? sVx[o + pitch + 1] + tx[k] * dvx[k] : 0.0;
            const double yn = (kind[k] & PT_Y) ? sVy[o + pitch + 1] + ty[k] * dvy[k] : 0.0;
            if (kind[k] & PT_OWN) {
                sVx_n[o + pitch + 1] = xn;
                sVy_n[o + pitch + 1] = yn;
            }
            if (kind[k] & PT_BOUND) {
                if (kind[k] & PT_I0) {
                    sVx_n[o + pitch] = 0.0;
                    sVy_n[o + pitch] = yn;
                }
                if (kind[k] & PT_I1) sVy_n[o + pitch + 2] = yn;
                if (kind[k] & PT_J0) {
                    sVx_n[o + 1] = xn;
                    sVy_n[o + 1] = 0.0;
                }
                if (kind[k] & PT_J1) sVx_n[o + 2 * pitch + 1] = xn;
            }
            if (CLUSTER && it + 1 < p.iters) {
                const uint32_t q = (it & 1) * 8;
                if (at_x[k]) {
                    put_in_block(at_x[k], xn, bar_x[k] + q);
                    put_in_block(at_x[k] + comp1 * 8, yn, bar_x[k] + q);
                }
                if (at_y[k]) {
                    put_in_block(at_y[k], xn, bar_y[k] + q);
                    put_in_block(at_y[k] + comp1 * 8, yn, bar_y[k] + q);
                }
                if (at_d[k]) put_in_block(at_d[k], (kind[k] & PT_DX) ? xn : yn, bar_d[k] + q);
                at_x[k] = at_x[k] ? at_x[k] - other : 0;
                at_y[k] = at_y[k] ? at_y[k] - other : 0;
                at_d[k] = at_d[k] ? at_d[k] - other : 0;
            }
        }
        if (CLUSTER) {
            // corners whose owner is a boundary entry of a neighbour's column or row: zero from the first iteration on
            // (the second pair of buffers is zero there from the start)
            if (it == 1 && tid == 0) {
                if (!has_l && has_t) sVx_n[(H + 1) * pitch] = 0.0;
                if (!has_b && has_r) sVy_n[W + 1] = 0.0;
            }
            other = 0u - other;
            double* t = sVx;
            sVx = sVx_n;
            sVx_n = t;
            t = sVy;
            sVy = sVy_n;
            sVy_n = t;
            __syncthreads();
            // the neighbours' entries (after a wait in vain: no more waits, and nothing of this launch is used).  Theirs of
            // the iteration after the next cannot come before this tile has sent its own of the next.
            if (expected && it + 1 < p.iters && !lost && !all_in(&bar[it & 1], (it >> 1) & 1)) {
                const uint64_t t0 = global_timer_ns();
                for (uint32_t q = 1; !all_in(&bar[it & 1], (it >> 1) & 1); ++q)
                    if ((q & 63u) == 0u && global_timer_ns() - t0 > p.wait_ns) {
                        lost = true;
                        break;
                    }
            }
            continue;
        }
        __syncthreads();
        if (it + 1 == p.iters) continue;
        // ---- this tile's borders to the neighbours, theirs into the halo ----
        const uint32_t tag = p.tag0 + (uint32_t)it;
        ulonglong2* const mine = p.comm + ((int64_t)(it & 1) * tiles + blockIdx.x) * nslots;
        int to = to0, from = from0, peer = peer0;
        for (int n = tid; n < nslots; n += NT) {
            if (n != tid) halo(n, to, from, peer);
            if (from >= 0) put(mine + (int64_t)peer * nslots + n, sVx[from], tag);
        }
        for (int n = tid; n < nslots; n += NT) {
            if (nslots > NT) halo(n, to, from, peer);
            if (to < 0) continue;
            double v = 0.0;
            if (!get(mine + n, tag, &v)) {
                const uint64_t t0 = global_timer_ns();
                for (uint32_t q = 1; !get(mine + n, tag, &v); ++q)
                    if ((q & 63u) == 0u && global_timer_ns() - t0 > p.wait_ns) {
                        gave_up = 1;
                        break;
                    }
            }
            sVx[to] = v;
        }
        // corners whose owner is a boundary entry of a neighbour's column or row: zero from the first iteration on
        if (tid == 0) {
            if (!has_l && has_t) sVx[(H + 1) * pitch] = 0.0;
            if (!has_b && has_r) sVy[W + 1] = 0.0;
        }
        __syncthreads();
        if (gave_up) {   // a neighbour's border never came: nothing of this launch is used
            if (tid == 0) atomicExch(p.err_flag, 1);
            return;
        }
    }

    if (CLUSTER) {
        if (lost) atomicExch(p.err_flag, 1);
        cluster_sync();   // (no block leaves while others might still write to it)
    }
    // ---- tau_xy of the last iteration: the tile's points as new velocities see them, one further in x and y, and the
    // domain's first column and row ----
    if (p.txy) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int b = b0 + k, i = i0 + a, j = j0 + b;
            if (live && b <= H && i < Nx && j < Ny && (a || !has_l) && (b || !has_b))
                p.txy[i + (int64_t)j * LD] = sTxy[o0 + k * pitch];
        }
    }
    if (p.max_bits) {   // max|V| over the tile; the boundary entries are copies or zero
        unsigned long long mx = 0, my = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (!(kind[k] & PT_OWN)) continue;
            const int o = o0 + (k + 1) * pitch + 1;
            mx = max(mx, (unsigned long long)__double_as_longlong(fabs(sVx[o])));
            my = max(my, (unsigned long long)__double_as_longlong(fabs(sVy[o])));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            my = max(my, __shfl_xor_sync(0xffffffffu, my, o));
        }
        if ((tid & 31) == 0) {
            atomicMax(&max_v[0], mx);
            atomicMax(&max_v[1], my);
        }
        __syncthreads();
        if (tid < 2) atomicMax(&p.max_bits[tid], max_v[tid]);
    }
    // ---- the state back, with the boundary entries ----
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (!(kind[k] & PT_OWN)) continue;
        const int o = o0 + k * pitch, b = b0 + k;
        const int i = i0 + a, j = j0 + b;
        const int64_t q = i + (int64_t)j * LD;
        const double xn = sVx[o + pitch + 1], yn = sVy[o + pitch + 1];
        p.P_out[q] = P[k];
        if (kind[k] & PT_X) p.dVx_out[q] = dvx[k];
        if (kind[k] & PT_Y) p.dVy_out[q] = dvy[k];
        p.Vx_out[q + 1 + LD] = xn;
        p.Vy_out[q + 1 + LD] = yn;
        if (i == 0) {
            p.Vx_out[q + LD] = 0.0;
            p.Vy_out[q + LD] = yn;
            if (j == 0) p.Vx_out[q] = p.Vy_out[q] = 0.0;
            if (j == Ny - 2) p.Vx_out[q + 2 * LD] = 0.0;
        }
        if (i == Nx - 2) {
            p.Vy_out[q + 2 + LD] = yn;
            if (j == 0) p.Vy_out[q + 2] = 0.0;
        }
        if (j == 0) {
            p.Vx_out[q + 1] = xn;
            p.Vy_out[q + 1] = 0.0;
        }
        if (j == Ny - 2) p.Vx_out[q + 1 + 2 * LD] = xn;
    }
}

typedef void (*ResKernel)(const ResidentParams);
const ResKernel kKernels[] = {k_pt_resident<1, false>, k_pt_resident<2, false>, k_pt_resident<3, false>,
                              k_pt_resident<4, false>, k_pt_resident<1, true>,  k_pt_resident<2, true>};
constexpr int RES_KERNELS = sizeof(kKernels) / sizeof(kKernels[0]);
int kernel_of(const ResidentPlan& p) { return p.k - 1 + (p.cluster ? RES_MAX_K : 0); }
constexpr int CLUSTER_MAX_K = 2;
constexpr int CLUSTER_MAX = 16;
constexpr int CLUSTER_PTS = 800;     // of a tile with its halo column and row
constexpr int RES_SMEM = 200 * 1024;
constexpr int CLUSTER_SMEM = 72 * 1024;   // more than any tile of CLUSTER_PTS points takes

// the last array is one row longer: stage 2 reads a row above its points, those of the halo row too
int smem_of(int W, int rows, bool cluster) { return ((cluster ? 4 : 2) * (rows + 1) + 4 * rows + 1) * (W + 2) * 8; }

// threads and points per thread of a tile; false if they do not fit
bool threads_for(int64_t W, int64_t H, ResidentPlan& p) {
    for (p.k = 1; p.k <= RES_MAX_K; ++p.k) {
        const int64_t n = (W + 1) * (rows_of((int)H, p.k) / p.k);
        p.threads = (int)round_up(n, 32);
        if (n <= 512) return true;
    }
    return false;
}

// What a tile takes, for the choice of its shape; fitted to measured ones (microseconds per iteration of the one taken and
// of others, exchange through L2): its points, idle threads included; a warp across the end of a tile's row meets bank
// conflicts, which wide tiles have fewer of; spills with 4 points per thread; the border.  330^2: 47 x 16 points 2.01,
// 37 x 21 2.07, 83 x 9 2.10, 16 x 47 (the fewest points) 2.24; 511 x 385: 43 x 32 2.61, 73 x 19 with 4 points per thread
// 2.81; 300^2: 43 x 15 1.91, 25 x 25 1.96; 128^2: 16 x 10 1.40, 10 x 16 1.46.
double tile_cost(int64_t W, int64_t H, const ResidentPlan& p) {
    return p.threads * p.k * (1.0 + 4.0 / (W + 1) + (p.k == RES_MAX_K ? 0.1 : 0.0)) + 3.2 * (W + H);
}

void set_tiles(ResidentPlan& p, int64_t cols, int64_t rows, int64_t W, int64_t H) {
    p.fits = true;
    p.ntx = (int)ceil_div(cols, W);
    p.nty = (int)ceil_div(rows, H);
    p.W = (int)W;
    p.H = (int)H;
    p.smem = smem_of(p.W, rows_of(p.H, p.k), p.cluster);
}

// the largest cluster that the device places at all (one in a partition of the device may have fewer SMs together)
int cluster_limit(int device) {
    static std::mutex m;
    static int limit[MAX_DEVICES] = {};
    if (device < 0 || device >= MAX_DEVICES) return 1;
    std::lock_guard<std::mutex> lock(m);
    int& have = limit[device];
    if (have) return have;
    have = 1;
    for (int k = 0; k < CLUSTER_MAX_K; ++k)
        if (cudaFuncSetAttribute((const void*)kKernels[RES_MAX_K + k], cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                cudaSuccess ||
            cudaFuncSetAttribute((const void*)kKernels[RES_MAX_K + k], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 RES_SMEM) != cudaSuccess) {
            cudaGetLastError();
            return have;
        }
    for (int c = CLUSTER_MAX; c > 1 && have == 1; c /= 2) {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)c;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)c);
        cfg.blockDim = dim3(512);
        cfg.dynamicSmemBytes = CLUSTER_SMEM;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kKernels[RES_MAX_K + CLUSTER_MAX_K - 1], &cfg) == cudaSuccess && n > 0)
            have = c;
        else
            cudaGetLastError();
    }
    return have;
}

}  // namespace

// The tiles as one cluster, for grids of which 16 tiles hold at most 800 points each, halo column and row included (up to
// about 108^2).  Writing a border into the neighbour's shared memory takes less than a store to L2 and a load from it;
// beyond, 16 SMs compute for longer than that gains.  Microseconds per iteration, checks included, against the exchange
// through L2: 20 x 26 0.67 : 1.60 (with one tile that needs no exchange 1.40), 40^2 0.64 : 1.61, 64^2 0.74 : 1.52, 84^2
// 1.00 : 1.46, 100^2 1.22 : 1.39, 108^2 1.35 : 1.39, 120^2 (992 points) 1.39 : 1.38, 128^2 1.79 : 1.38; 170 x 40 1.18 :
// 1.70, 250 x 50 (850 points) 1.61 : 1.51.  With a cluster barrier per iteration instead of counted stores: 20 x 26 0.90,
// 64^2 1.03, 84^2 1.22 (the barrier waits for every earlier write of a thread, and for all blocks instead of the
// neighbours).  Tiles of 32 points: a block's barrier takes less with fewer warps (20 x 26, kernel alone, with cluster
// barriers: 0.90 us with one block, 0.78 with two, 0.70 with four, 0.64 with eight, 0.61 with sixteen).
ResidentPlan cluster_plan(int64_t Nx, int64_t Ny, int device) {
    ResidentPlan best;
    const int64_t cols = Nx - 1, rows = Ny - 1, pts = cols * rows;
    const int most = cluster_limit(device);
    int tiles = 1;
    while (tiles < most && pts > (int64_t)tiles * 32) tiles *= 2;
    double best_cost = 0.0;
    for (; tiles >= 1 && !best.fits; tiles /= 2)   // (fewer only where a thin grid does not split so far)
        for (int ntx = 1; ntx <= tiles; ntx *= 2) {
            const int64_t W = ceil_div(cols, ntx), H = ceil_div(rows, tiles / ntx);
            ResidentPlan p;
            if (W < 2 || H < 2 || ceil_div(cols, W) != ntx || ceil_div(rows, H) != tiles / ntx || !threads_for(W, H, p))
                continue;
            const double cost = tile_cost(W, H, p);
            if ((W + 1) * rows_of((int)H, p.k) > CLUSTER_PTS || (best.fits && cost >= best_cost)) continue;
            p.cluster = true;
            set_tiles(p, cols, rows, W, H);
            best = p;
            best_cost = cost;
        }
    return best;
}

// The exchange through L2: which grids, and how many tiles.  Up to 512 x 4 points per SM (registers: 22 per point) the
// state fits, and is faster than the march wherever it does (3.2 against 5.8 us per iteration at 500^2, 1.4 against 4.3
// at 128^2).  One tile per 150 points: the exchange costs the same whatever the tiles' size, and smaller ones
// compute faster until they no longer do (128^2: 1.67 us, with 450 points 2.02, with 100 1.70); a small grid still
// leaves SMs to solves on other streams.
ResidentPlan resident_plan(int64_t Nx, int64_t Ny, int num_sms) {
    ResidentPlan best;
    const int64_t cols = Nx - 1, rows = Ny - 1, pts = cols * rows;
    double best_cost = 0.0;
    if (pts > (int64_t)num_sms * 512 * RES_MAX_K) return best;
    const int tiles = (int)std::min<int64_t>(num_sms, ceil_div(pts, 150));
    for (int ntx = 1; ntx <= tiles && ntx <= cols; ++ntx) {
        const int nty = (int)std::min<int64_t>(tiles / ntx, rows);
        const int64_t W = ceil_div(cols, ntx), H = ceil_div(rows, nty);
        ResidentPlan p;
        if (W < 2 || H < 2 || !threads_for(W, H, p)) continue;
        const double cost = tile_cost(W, H, p);
        if (best.fits && cost >= best_cost) continue;
        set_tiles(p, cols, rows, W, H);
        // (128 registers, the launch bound)
        p.share = (int)std::min<int64_t>(4, std::max(ceil_div(p.threads * 128, 65536 / 4), ceil_div(p.smem, 50 * 1024)));
        best = p;
        best_cost = cost;
    }
    return best;
}

namespace {
constexpr int ROOM_DEVICES = MAX_DEVICES;
std::mutex g_room_mutex;
int g_room_used[ROOM_DEVICES] = {};       // quarters of SMs held by solves that exchange through L2, by device
int g_room_clusters[ROOM_DEVICES] = {};   // solves that use a cluster
int g_room_solves[ROOM_DEVICES] = {};     // plain solves
int g_room_others[ROOM_DEVICES] = {};     // OtherWork
std::vector<const sf_ctx*> g_room_contexts;
// marker kernels without a context: until when, and the thread that launched them
std::atomic<int64_t> g_noalloc_until[ROOM_DEVICES];
std::atomic<size_t> g_noalloc_thread[ROOM_DEVICES];

size_t this_thread() { return std::hash<std::thread::id>()(std::this_thread::get_id()); }

int64_t now_ns() {
    return std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// (with the mutex) whether another context's marker kernels are under way
bool markers_at_work(const sf_ctx* ctx, int device) {
    const int64_t now = now_ns();
    if (g_noalloc_until[device].load(std::memory_order_relaxed) > now &&
        g_noalloc_thread[device].load(std::memory_order_relaxed) != this_thread())
        return true;
    for (const sf_ctx* c : g_room_contexts)
        if (c != ctx && c->device == device && c->markers_until.load(std::memory_order_relaxed) > now) return true;
    return false;
}
}  // namespace

void room_add_context(const sf_ctx* ctx) {
    std::lock_guard<std::mutex> lock(g_room_mutex);
    g_room_contexts.push_back(ctx);
}

void room_remove_context(const sf_ctx* ctx) {
    std::lock_guard<std::mutex> lock(g_room_mutex);
    g_room_contexts.erase(std::remove(g_room_contexts.begin(), g_room_contexts.end(), ctx), g_room_contexts.end());
}

// Taken to last 10 ms and 0.2 ns per marker (three deposits 0.11, rebin and advection 0.06) from the call on: beside
// whole-SM tiles they wait for the solve's next check first (up to 7 ms).
void markers_launched(sf_ctx* ctx, int device, int64_t nm) {
    if (device < 0 || device >= ROOM_DEVICES) return;
    if (!ctx) g_noalloc_thread[device].store(this_thread(), std::memory_order_relaxed);
    (ctx ? ctx->markers_until : g_noalloc_until[device]).store(now_ns() + 10000000 + nm / 5, std::memory_order_relaxed);
}

OtherWork::OtherWork(int device) : device_(device) {
    std::lock_guard<std::mutex> lock(g_room_mutex);
    if (device_ >= 0 && device_ < ROOM_DEVICES) ++g_room_others[device_];
}

OtherWork::~OtherWork() {
    std::lock_guard<std::mutex> lock(g_room_mutex);
    if (device_ >= 0 && device_ < ROOM_DEVICES) --g_room_others[device_];
}

bool ResidentRoom::known() const { return device_ >= 0 && device_ < ROOM_DEVICES; }

ResidentRoom::ResidentRoom(const sf_ctx* ctx, cudaStream_t s) : ctx_(ctx), device_(ctx->device), stream_(s) {
    std::lock_guard<std::mutex> lock(g_room_mutex);
    if (known()) ++g_room_solves[device_];
}

ResidentRoom::~ResidentRoom() {
    release();
    std::lock_guard<std::mutex> lock(g_room_mutex);
    if (known()) --g_room_solves[device_];
}

bool ResidentRoom::keeps(const ResidentPlan& plan) const {
    if (plan.cluster) return true;
    std::lock_guard<std::mutex> lock(g_room_mutex);
    return g_room_others[device_] == 0 && (plan.share < 4 || whole_sms());
}

bool ResidentRoom::whole_sms() const { return g_room_solves[device_] == 1 && !markers_at_work(ctx_, device_); }

bool ResidentRoom::acquire(const ResidentPlan& plan) {
    if (!plan.fits || !known() || held_ || cluster_) return false;
    const int need = plan.ntx * plan.nty * plan.share;
    std::lock_guard<std::mutex> lock(g_room_mutex);
    if (plan.cluster) {
        if (g_room_used[device_]) return false;
        ++g_room_clusters[device_];
        cluster_ = true;
        return true;
    }
    const int most = plan.share == 4 && whole_sms() ? 4 : 3;
    if (g_room_clusters[device_] || g_room_others[device_] || plan.share > most ||
        g_room_used[device_] + need > most * ctx_->num_sms)
        return false;
    g_room_used[device_] += need;
    held_ = need;
    return true;
}

void ResidentRoom::release() {
    if (!held_ && !cluster_) return;
    cudaStreamSynchronize(stream_);   // nothing of the solve runs any more
    std::lock_guard<std::mutex> lock(g_room_mutex);
    g_room_used[device_] -= held_;
    g_room_clusters[device_] -= cluster_;
    held_ = 0;
    cluster_ = false;
}

int resident_scratch(sf_ctx* ctx, const ResidentPlan& plan, cudaStream_t s) {
    if (plan.cluster) return SF_OK;
    const size_t bytes = (size_t)2 * plan.ntx * plan.nty * slots_of(plan.W, plan.H) * sizeof(ulonglong2);
    if (bytes <= ctx->halo.bytes) return SF_OK;
    int rc = ensure(ctx, ctx->halo, bytes);
    if (rc) return rc;
    SF_CUDA(cudaMemsetAsync(ctx->halo.ptr, 0, ctx->halo.bytes, s));
    ctx->halo_tag = 1;
    return SF_OK;
}

int resident_launch(sf_ctx* ctx, ResidentParams& p, const ResidentPlan& plan, cudaStream_t s) {
    const int tiles = plan.ntx * plan.nty;
    if (!plan.cluster) {
        // tags of earlier launches stay in the slots: new memory, and a wrap of the counter, start from zeroed slots
        if (ctx->halo_tag > 0xffffffffu - (uint32_t)p.iters - 1u) {
            SF_CUDA(cudaMemsetAsync(ctx->halo.ptr, 0, ctx->halo.bytes, s));
            ctx->halo_tag = 1;
        }
        p.comm = (ulonglong2*)ctx->halo.ptr;
        p.tag0 = ctx->halo_tag;
        ctx->halo_tag += (uint32_t)p.iters;
    }
    p.ntx = plan.ntx;
    p.nty = plan.nty;
    p.W = plan.W;
    p.H = plan.H;
    const int which = kernel_of(plan);
    static PerDevice ready[RES_KERNELS];
    const int rc = allow_smem(ready[which], ctx->device, (const void*)kKernels[which], RES_SMEM);
    if (rc) return rc;
    p.wait_ns = RES_WAIT_NS;
    int blocks = tiles;
    if (ctx->tiles_fail_ns) {   // sf_selftest_tile_wait
        p.wait_ns = (uint64_t)ctx->tiles_fail_ns;
        ctx->tiles_fail_ns = 0;
        if (plan.cluster)       // (a block is not sent to one that is not there)
            SF_CUDA(cudaMemsetAsync(p.err_flag, 1, sizeof(int), s));
        else
            --blocks;           // nothing fills the neighbours' slots
    }
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)plan.threads);
    cfg.dynamicSmemBytes = (size_t)plan.smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (plan.cluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)tiles;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kKernels[which], (const ResidentParams)p);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorInvalidClusterSize ||
        e == cudaErrorInvalidConfiguration) {
        (void)cudaGetLastError();
        return RESIDENT_LOST;
    }
    SF_CUDA(e);
    SF_LAUNCHED(ctx);
    return SF_OK;
}

}  // namespace sf
