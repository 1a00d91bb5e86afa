// sf_resident.cu -- many pseudo-transient iterations (StokesSolver_multixpu.jl:48-57) of a small grid in one launch.
//
// On a small grid an iteration's arithmetic takes less than launching a kernel for it.  Here the state stays on
// the chip for as many iterations as the reference's loop runs without an event (a residual check, a dt update):
//
//   * the grid is cut into at most one tile per SM; a thread owns the same points in every iteration and keeps their
//     P, rates and parameters in registers.  Vx, Vy and the stage-1 results of a tile (P, tau_xx, tau_yy, tau_xy) are in
//     shared memory.  An iteration is the two stages of k_pt_iter, a block barrier after each, and the exchange;
//   * the tiles exchange the velocities of their borders through L2: every value travels in a 16-byte slot as two
//     8-byte words {half, tag}, the tag being the iteration's number, so that a reader that sees its tag has the
//     value: one store and one load instead of data, fence and flag.  Slots are double-buffered by parity; a tile
//     cannot be two iterations ahead of one that it exchanges with, so a slot is never overwritten unread;
//   * the launch is cooperative (all tiles resident), and every wait has a wall-clock budget.
//
// A tile's halo column and row of P and tau are computed by both neighbours from the same values.  Every expression
// keeps the reference's order of operations (compiled without contraction): bit-identical to single iterations.
//
// What bounds it: latency.  At 128^2 (110 tiles of 150 points, 8 warps) an iteration takes 1.5 us, about half of it the
// exchange (a store to L2 and a load from it, two barriers) and half the two stages' dependent FP64 chains; at 511 x 385
// (1450 points per SM) 2.8 us, there mostly issue slots.  5.2 -> 1.65 us per iteration at 128^2 (k_pt_iter: one launch
// each), 8.3 -> 2.8 at 511 x 385, 4.5 -> 1.4 at 20 x 26, checks included.  Testing every point's flags and sending
// borders from the update itself took 905 instructions per warp and iteration at 511 x 385 and 4.2 us.
#include <algorithm>
#include <mutex>

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

// what a thread's point is: one whose Vx / Vy it updates (the others' are boundary entries, zero), one of the tile (not
// of its halo column or row), and the sides of the domain that it lies on
enum { PT_X = 1, PT_Y = 2, PT_OWN = 4, PT_I0 = 8, PT_I1 = 16, PT_J0 = 32, PT_J1 = 64,
       PT_BOUND = PT_I0 | PT_I1 | PT_J0 | PT_J1 };

// K points per thread
template <int K>
__global__ void __launch_bounds__(K == 1 ? 1024 : 512, 1) k_pt_resident(const __grid_constant__ ResidentParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int gave_up;
    const int W = p.W, H = p.H, pitch = W + 2;
    double* const sVx = reinterpret_cast<double*>(smem_raw);      // (H + 2) x (W + 2): entry (0, 0) is Vx(i0, j0)
    double* const sVy = sVx + (H + 2) * pitch;
    double* const sTxx = sVy + (H + 2) * pitch;                   // (H + 1) rows of the same pitch
    double* const sTyy = sTxx + (H + 1) * pitch;
    double* const sPn = sTyy + (H + 1) * pitch;
    double* const sTxy = sPn + (H + 1) * pitch;
    const int tid = threadIdx.x, NT = blockDim.x;
    const int bx = blockIdx.x % p.ntx, by = blockIdx.x / p.ntx;
    const int i0 = bx * W, j0 = by * H;
    const int Nx = p.Nx, Ny = p.Ny;
    const int64_t LD = p.LD;
    const double _dx = p._dx, _dy = p._dy;
    const bool has_l = bx > 0, has_r = bx + 1 < p.ntx, has_b = by > 0, has_t = by + 1 < p.nty;

    // ---- state and parameters onto the chip ----
    for (int n = tid; n < (H + 2) * pitch; n += NT) {
        const int b = n / pitch, a = n - b * pitch;
        const bool in = i0 + a <= Nx && j0 + b <= Ny;
        const int64_t o = i0 + a + (int64_t)(j0 + b) * LD;
        sVx[n] = in ? p.Vx_in[o] : 0.0;
        sVy[n] = in ? p.Vy_in[o] : 0.0;
    }
    double P[K], dvx[K], dvy[K], tp[K], mu2[K], mb[K], tx[K], ty[K], rho[K], gx[K], gy[K];
    int off[K];      // b * pitch + a of the thread's points (a <= W, b <= H: the tile and one more column and row)
    int kind[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int n = tid + k * NT;
        const int b = n / (W + 1), a = n - b * (W + 1);
        const int i = i0 + a, j = j0 + b;
        off[k] = b <= H ? b * pitch + a : 0;   // (points beyond the tile's compute on its first and store nothing)
        kind[k] = 0;
        P[k] = dvx[k] = dvy[k] = tp[k] = mu2[k] = mb[k] = tx[k] = ty[k] = rho[k] = gx[k] = gy[k] = 0.0;
        if (b > H) continue;
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
    const int hv = min(H, Ny - 1 - j0), wv = min(W, Nx - 1 - i0), comp1 = (H + 2) * pitch;
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
    int to0, from0, peer0;
    halo(tid, to0, from0, peer0);
    if (tid == 0) gave_up = 0;
    __syncthreads();

    for (int it = 0; it < p.iters; ++it) {
        // ---- stage 1: compute_P_tau! (:140-169) on the tile and one more column and row.  Evaluated at every point
        // (outside the domain on whatever is there; nothing that is kept depends on it) ----
        double sterm[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int o = off[k];
            const double vx00 = sVx[o], vx10 = sVx[o + pitch], vx11 = sVx[o + pitch + 1];
            const double vy00 = sVy[o], vy01 = sVy[o + 1], vy11 = sVy[o + pitch + 1];
            const double vx20 = sVx[o + 2 * pitch], vx21 = sVx[o + 2 * pitch + 1];
            const double dVx_dy = (vx10 - vx00) * _dy;
            const double dVy_dx = (vy01 - vy00) * _dx;
            const double txy = mb[k] * (dVx_dy + dVy_dx);
            const double dVx_dx = (vx11 - vx10) * _dx;
            const double dVy_dy = (vy11 - vy01) * _dy;
            const double div = dVx_dx + dVy_dy;
            P[k] = P[k] - tp[k] * div;
            const double third = 1.0 / 3.0 * div;
            const double txx = mu2[k] * (dVx_dx - third), tyy = mu2[k] * (dVy_dy - third);
            // the gravity term of compute_ResY (:189-202), from the old velocities
            const double av = 0.25 * (vx10 + vx11 + vx20 + vx21);
            sterm[k] = g_y * (rho[k] - dt * (av * gx[k] * 0.5 * _dx + vy11 * gy[k] * 0.5 * _dy));
            if (tid + k * NT < (W + 1) * (H + 1)) {
                sTxy[o] = txy;
                sPn[o] = P[k];
                sTxx[o] = txx;
                sTyy[o] = tyy;
            }
        }
        __syncthreads();
        // ---- stage 2: compute_dV!, compute_V! (:209-234), the boundary kernels (:53-56) ----
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int o = off[k];
            const double txy11 = sTxy[o + pitch + 1];
            const double Rx = (sTxx[o + 1] - sTxx[o]) * _dx + (txy11 - sTxy[o + 1]) * _dy - (sPn[o + 1] - P[k]) * _dx;
            const double Ry = (sTyy[o + pitch] - sTyy[o]) * _dy + (txy11 - sTxy[o + pitch]) * _dx -
                              (sPn[o + pitch] - P[k]) * _dy + sterm[k];
            dvx[k] = dampX * dvx[k] + Rx;
            dvy[k] = dampY * dvy[k] + Ry;
            // Vx(Nx-1) and Vy(Ny-1) are the zero entries of the boundary
            const double xn = (kind[k] & PT_X) ? sVx[o + pitch + 1] + tx[k] * dvx[k] : 0.0;
            const double yn = (kind[k] & PT_Y) ? sVy[o + pitch + 1] + ty[k] * dvy[k] : 0.0;
            if (kind[k] & PT_OWN) {
                sVx[o + pitch + 1] = xn;
                sVy[o + pitch + 1] = yn;
            }
            if (kind[k] & PT_BOUND) {
                if (kind[k] & PT_I0) {
                    sVx[o + pitch] = 0.0;
                    sVy[o + pitch] = yn;
                }
                if (kind[k] & PT_I1) sVy[o + pitch + 2] = yn;
                if (kind[k] & PT_J0) {
                    sVx[o + 1] = xn;
                    sVy[o + 1] = 0.0;
                }
                if (kind[k] & PT_J1) sVx[o + 2 * pitch + 1] = xn;
            }
        }
        __syncthreads();
        if (tiles == 1 || it + 1 == p.iters) continue;
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
                    if ((q & 63u) == 0u && global_timer_ns() - t0 > RES_WAIT_NS) {
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

    // ---- the state back, with the boundary entries ----
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (!(kind[k] & PT_OWN)) continue;
        const int o = off[k], b = o / pitch, a = o - b * pitch;
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
const ResKernel kKernels[RES_MAX_K + 1] = {nullptr, k_pt_resident<1>, k_pt_resident<2>, k_pt_resident<3>,
                                           k_pt_resident<4>};

// the last array is one row longer: stage 2 reads a row above its points, those of the halo row too
int smem_of(int W, int H) { return (2 * (H + 2) + 4 * (H + 1) + 1) * (W + 2) * 8; }

}  // namespace

// Which grids, and how many tiles.  Up to 512 x 4 points per SM (registers: 22 per point) the state fits, and is faster
// than the march wherever it does (3.5 against 5.8 us per iteration at 512^2, 1.65 against 4.3 at 128^2).  One tile up
// to 800 points: it needs no exchange (27^2: 1.66 us against 1.70 with five tiles, 33^2: 2.04 against 1.62, residual
// checks included).  Above, one per 150 points: the exchange costs the same whatever the tiles' size, and smaller ones
// compute faster until they no longer do (128^2: 1.67 us, with 450 points 2.02, with 100 1.70); a small grid still
// leaves SMs to solves on other streams.
ResidentPlan resident_plan(int64_t Nx, int64_t Ny, int num_sms) {
    ResidentPlan best;
    const int64_t cols = Nx - 1, rows = Ny - 1, pts = cols * rows;
    if (pts > (int64_t)num_sms * 512 * RES_MAX_K) return best;
    int tiles = 1;
    if (pts > 800) tiles = (int)std::min<int64_t>(num_sms, ceil_div(pts, 150));
    int64_t best_pts = 0;
    for (int ntx = 1; ntx <= tiles && ntx <= cols; ++ntx) {
        const int nty = (int)std::min<int64_t>(tiles / ntx, rows);
        const int64_t W = ceil_div(cols, ntx), H = ceil_div(rows, nty);
        const int64_t n = (W + 1) * (H + 1);
        if (W < 2 || H < 2 || (best.fits && n >= best_pts)) continue;
        const int64_t nx = ceil_div(cols, W), ny = ceil_div(rows, H);
        int k = 0, threads = 0;
        for (k = 1; k <= RES_MAX_K; ++k) {
            threads = (int)round_up(ceil_div(n, k), 32);
            if (threads <= (k == 1 ? 1024 : 512)) break;
        }
        if (k > RES_MAX_K) continue;
        best.fits = true;
        best.ntx = (int)nx;
        best.nty = (int)ny;
        best.W = (int)W;
        best.H = (int)H;
        best.k = k;
        best.threads = threads;
        best.smem = smem_of((int)W, (int)H);
        // registers: 64 per thread with one point (the launch bound), else up to 128
        const int regs = threads * (k == 1 ? 64 : 128);
        best.share = regs <= 65536 / 4 && best.smem <= 50 * 1024 ? 1
                     : regs <= 65536 / 2 && best.smem <= 100 * 1024 ? 2 : 4;
        best_pts = n;
    }
    return best;
}

namespace {
std::mutex g_room_mutex;
int g_room_used[64] = {};   // quarters of SMs held, by device
}

bool ResidentRoom::acquire(int device, int num_sms, const ResidentPlan& plan, cudaStream_t s) {
    if (!plan.fits || device < 0 || device >= 64) return false;
    const int need = plan.ntx * plan.nty * plan.share;
    std::lock_guard<std::mutex> lock(g_room_mutex);
    if (g_room_used[device] + need > 4 * num_sms) return false;
    g_room_used[device] += need;
    device_ = device;
    held_ = need;
    stream_ = s;
    return true;
}

void ResidentRoom::release() {
    if (device_ < 0) return;
    cudaStreamSynchronize(stream_);   // nothing of the solve runs any more
    std::lock_guard<std::mutex> lock(g_room_mutex);
    g_room_used[device_] -= held_;
    device_ = -1;
}

int resident_launch(sf_ctx* ctx, ResidentParams& p, const ResidentPlan& plan, cudaStream_t s) {
    const int tiles = plan.ntx * plan.nty;
    const size_t bytes = (size_t)2 * tiles * slots_of(plan.W, plan.H) * sizeof(ulonglong2);
    // tags of earlier launches stay in the slots: new memory, and a wrap of the counter, start from zeroed slots
    const bool fresh = bytes > ctx->halo.bytes, wrap = ctx->halo_tag > 0xffffffffu - (uint32_t)p.iters - 1u;
    int rc = ensure(ctx, ctx->halo, bytes);
    if (rc) return rc;
    if (fresh || wrap) {
        SF_CUDA(cudaMemsetAsync(ctx->halo.ptr, 0, ctx->halo.bytes, s));
        ctx->halo_tag = 1;
    }
    p.ntx = plan.ntx;
    p.nty = plan.nty;
    p.W = plan.W;
    p.H = plan.H;
    p.comm = (ulonglong2*)ctx->halo.ptr;
    p.tag0 = ctx->halo_tag;
    ctx->halo_tag += (uint32_t)p.iters;
    static bool ready[64][RES_MAX_K + 1] = {};
    if (!ready[ctx->device & 63][plan.k]) {
        SF_CUDA(cudaFuncSetAttribute((const void*)kKernels[plan.k], cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        ready[ctx->device & 63][plan.k] = true;
    }
    void* args[] = {&p};
    SF_CUDA(cudaLaunchCooperativeKernel((const void*)kKernels[plan.k], dim3((unsigned)tiles), dim3((unsigned)plan.threads),
                                        args, (size_t)plan.smem, s));
    SF_LAUNCHED(ctx);
    return SF_OK;
}

}  // namespace sf
