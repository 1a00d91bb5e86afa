// sf_core.cu -- context, errors, scratch, warning counters and
// marker initialisation (scripts/common.jl:40-110) for libstokesflow_b200.so.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>

#include "sf_internal.cuh"
#include "sf_tma.cuh"

namespace sf {

static thread_local std::string g_last_error;

void set_error(const std::string& msg) { g_last_error = msg; }

int fail(int status, const std::string& msg) {
    g_last_error = msg;
    return status;
}

int cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
    char buf[512];
    snprintf(buf, sizeof(buf), "%s failed: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
    g_last_error = buf;
    if (e == cudaErrorMemoryAllocation) return SF_ERR_OOM;
    if (e == cudaErrorNoDevice || e == cudaErrorInvalidDevice || e == cudaErrorInsufficientDriver)
        return SF_ERR_NO_DEVICE;
    return SF_ERR_CUDA;
}

int set_device(sf_ctx* ctx) {
    SF_CUDA(cudaSetDevice(ctx->device));
    return SF_OK;
}

// --------------------------------------------------------------------------
// peer access between the devices of ranks, and block copies between ranks
// --------------------------------------------------------------------------
namespace {
constexpr int MAX_DEV = 64;
std::mutex g_peer_mutex;
signed char g_peer[MAX_DEV][MAX_DEV] = {};   // 0: not asked yet, 1: dev reads / writes peer's memory, -1: cannot
}

int peer_access(int dev, int peer, bool* ok) {
    *ok = (dev == peer);
    if (dev == peer) return SF_OK;
    if (dev < 0 || peer < 0 || dev >= MAX_DEV || peer >= MAX_DEV) return fail(SF_ERR_NO_DEVICE, "peer_access: device index");
    std::lock_guard<std::mutex> lock(g_peer_mutex);
    if (g_peer[dev][peer] == 0) {
        int can = 0;
        SF_CUDA(cudaDeviceCanAccessPeer(&can, dev, peer));
        g_peer[dev][peer] = -1;
        if (can) {
            int cur = 0;
            SF_CUDA(cudaGetDevice(&cur));
            SF_CUDA(cudaSetDevice(dev));
            const cudaError_t e = cudaDeviceEnablePeerAccess(peer, 0);
            if (e == cudaSuccess || e == cudaErrorPeerAccessAlreadyEnabled) {
                (void)cudaGetLastError();
                g_peer[dev][peer] = 1;
            } else {
                (void)cudaGetLastError();   // not enabled: the copies go through the runtime
            }
            SF_CUDA(cudaSetDevice(cur));
        }
    }
    *ok = g_peer[dev][peer] == 1;
    return SF_OK;
}

__global__ void k_copy_block(double* __restrict__ dst, int64_t ld_dst, const double* __restrict__ src, int64_t ld_src,
                             int64_t w, int64_t h) {
    const int64_t n = w * h;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = k % w, j = k / w;
        dst[i + j * ld_dst] = src[i + j * ld_src];
    }
}

int copy_block(sf_ctx* ctx, cudaStream_t s, double* dst, int64_t ld_dst, const double* src, int64_t ld_src,
               int64_t w, int64_t h, int src_device) {
    if (w <= 0 || h <= 0) return SF_OK;
    bool direct = false;
    int rc = peer_access(ctx->device, src_device, &direct);
    if (rc) return rc;
    if (direct) {
        const int64_t n = w * h;
        const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), (int64_t)ctx->num_sms * 8));
        k_copy_block<<<g, 256, 0, s>>>(dst, ld_dst, src, ld_src, w, h);
        SF_LAUNCHED(ctx);
    } else {
        SF_CUDA(cudaMemcpy2DAsync(dst, (size_t)ld_dst * 8, src, (size_t)ld_src * 8, (size_t)w * 8, (size_t)h,
                                  cudaMemcpyDefault, s));
    }
    return SF_OK;
}

static size_t scratch_size(size_t bytes) { return (size_t)round_up((int64_t)bytes, 1 << 20); }

bool may_have(const Scratch& s, size_t bytes) {
    if (bytes <= s.bytes) return true;
    size_t free_bytes = 0, total = 0;
    if (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess) {
        (void)cudaGetLastError();
        return true;   // (the allocation will tell)
    }
    return scratch_size(bytes) <= free_bytes + s.bytes;
}

int ensure(sf_ctx* ctx, Scratch& s, size_t bytes) {
    if (bytes <= s.bytes) return SF_OK;
    (void)ctx;
    if (s.ptr) {
        SF_CUDA(cudaFree(s.ptr));
        s.ptr = nullptr;
        s.bytes = 0;
    }
    size_t want = scratch_size(bytes);
    cudaError_t e = cudaMalloc(&s.ptr, want);
    if (e != cudaSuccess) {
        s.ptr = nullptr;
        (void)cudaGetLastError();
        return cuda_fail(e, "cudaMalloc(scratch)", __FILE__, __LINE__);
    }
    s.bytes = want;
    return SF_OK;
}

// --------------------------------------------------------------------------
// marker initialisation, scripts/common.jl:40-110 (single rank)
// --------------------------------------------------------------------------
struct MarkerLayout {
    double xlimlo, xlimhi, ylimlo, ylimhi, dxm, dym;
    int64_t nmx, nmy;
};

// the layout of the rank at (cx, cy) of a dims_x x dims_y grid (common.jl:43-75): a side that is a physical
// boundary starts half a marker spacing in; a side shared with a neighbour leaves the markers the neighbour
// places (half a cell, adjusted for odd or even densities)
static MarkerLayout marker_layout_rank(int64_t md, double lx, double ly, double dx, double dy, int64_t nx, int64_t ny,
                                       int cx, int cy, int dimx, int dimy) {
    MarkerLayout L;
    L.dxm = dx / (double)md;
    L.dym = dy / (double)md;
    const bool xlo = cx == 0, xhi = cx == dimx - 1, ylo = cy == 0, yhi = cy == dimy - 1;   // :47-50
    const bool even = md % 2 == 0;
    const double x_less_hi = even ? L.dxm / 2 : L.dxm, y_less_hi = even ? L.dym / 2 : L.dym;   // :52-56
    const double x_less_lo = even ? L.dxm / 2 : 0.0, y_less_lo = even ? L.dym / 2 : 0.0;
    L.xlimlo = xlo ? L.dxm / 2 : dx / 2 + x_less_lo;                                          // :58-61
    L.xlimhi = xhi ? lx - L.dxm / 2 : lx - dx / 2 - x_less_hi;
    L.ylimlo = ylo ? L.dym / 2 : dy / 2 + y_less_lo;
    L.ylimhi = yhi ? ly - L.dym / 2 : ly - dy / 2 - y_less_hi;
    const int64_t lo_less = md / 2, hi_less = (md + 1) / 2;                                    // :63-64
    L.nmx = md * (nx - 1) - (xlo ? 0 : lo_less) - (xhi ? 0 : hi_less);                         // :66-67
    L.nmy = md * (ny - 1) - (ylo ? 0 : lo_less) - (yhi ? 0 : hi_less);
    return L;
}

static MarkerLayout marker_layout(int64_t md, double lx, double ly, double dx, double dy, int64_t nx, int64_t ny) {
    return marker_layout_rank(md, lx, ly, dx, dy, nx, ny, 0, 0, 1, 1);   // one rank: every side is physical
}

// Julia LinRange(a, b, n)[k] (1-based k): lerpi(k-1, n-1, a, b) = (1 - t)*a + t*b with t = (k-1)/(n-1), two
// products and a sum each rounded (this file is built without contraction).  That is the form the reference's
// golden values fit: the fma form of lerpi moves some markers by one ulp, enough to put a marker of
// test/test_StokesFlow2D.jl's case on the other side of the plume boundary
__host__ __device__ __forceinline__ double linrange_at(double a, double b, int64_t n, int64_t k) {
    if (n == 1) return a;
    double t = (double)(k - 1) / (double)(n - 1);
    return (1.0 - t) * a + t * b;
}

__host__ __device__ __forceinline__ void marker_position(const MarkerLayout& L, double jitter, uint64_t seed,
                                                         int64_t m, double* x, double* y) {
    int64_t ix = m / L.nmy + 1, iy = m % L.nmy + 1;  // x outer, y inner (common.jl:85-91)
    double xv = linrange_at(L.xlimlo, L.xlimhi, L.nmx, ix);
    double yv = linrange_at(L.ylimlo, L.ylimhi, L.nmy, iy);
    if (jitter != 0.0) {
        double ux = uniform01(seed, (uint64_t)(2 * m));
        double uy = uniform01(seed, (uint64_t)(2 * m + 1));
        // x .+= (u - 0.5) * jitter * dxm, two roundings per product (no contraction)
        xv = xv + (ux - 0.5) * jitter * L.dxm;
        yv = yv + (uy - 0.5) * jitter * L.dym;
    }
    *x = xv;
    *y = yv;
}

__global__ void k_init_markers(MarkerLayout L, double jitter, uint64_t seed, double* __restrict__ x,
                               double* __restrict__ y) {
    int64_t nm = L.nmx * L.nmy;
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < nm; m += (int64_t)gridDim.x * blockDim.x)
        marker_position(L, jitter, seed, m, &x[m], &y[m]);
}

// StokesFlow2D_multixpu.jl:387-404 density / viscosity closures
__host__ __device__ __forceinline__ double plume_eval(const sf_plume_model& M, double x, double y, double air,
                                                      double mat, double pl) {
    if (y < M.air_height) return air;
    double ddx = x - M.plume_x, ddy = y - M.plume_y;
    if (ddx * ddx + ddy * ddy < M.plume_r * M.plume_r) return pl;
    return mat;
}

__global__ void k_set_props(sf_plume_model M, const double* __restrict__ x, const double* __restrict__ y,
                            int64_t nm, double x0, double y0, double* __restrict__ rho, double* __restrict__ mu) {
    for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < nm; m += (int64_t)gridDim.x * blockDim.x) {
        double xx = x0 + x[m], yy = y0 + y[m];
        rho[m] = plume_eval(M, xx, yy, M.rho_air, M.rho_matrix, M.rho_plume);
        mu[m] = plume_eval(M, xx, yy, M.mu_air, M.mu_matrix, M.mu_plume);
    }
}

// The bounded wait of the persistent kernels (mbar_wait), on a shared-memory barrier that thread 0 completes
// (arrive != 0) or that nothing completes (arrive == 0): then every thread's wait gives up after budget_ns and
// the block reports it through *timed_out, exactly as the kernels report a tile copy that never landed.
__global__ void k_wait_selftest(int arrive, uint64_t budget_ns, int* __restrict__ timed_out) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (arrive && threadIdx.x == 0) mbar_arrive_expect_tx(&bar, 0);
    const bool ok = mbar_wait(&bar, 0, budget_ns);
    if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicExch(timed_out, 1);
}

}  // namespace sf

using namespace sf;

// ==========================================================================
// C ABI
// ==========================================================================
extern "C" {

int sf_version(void) { return (0 << 16) | (1 << 8) | 0; }

const char* sf_status_string(int status) {
    switch (status) {
        case SF_OK: return "ok";
        case SF_ERR_INVALID_ARG: return "invalid argument";
        case SF_ERR_CUDA: return "CUDA error";
        case SF_ERR_OOM: return "out of device memory";
        case SF_ERR_NO_DEVICE: return "no CUDA device";
        case SF_ERR_NONFINITE: return "non-finite residual";
        case SF_ERR_TOO_LARGE: return "size exceeds the supported maximum";
        case SF_ERR_BUSY: return "engine full; retry after instances finish";
        default: return "unknown status";
    }
}

const char* sf_last_error(void) { return g_last_error.c_str(); }

int sf_ctx_create(int device, sf_ctx** out) {
    if (!out) return fail(SF_ERR_INVALID_ARG, "sf_ctx_create: out is NULL");
    *out = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) {
        (void)cudaGetLastError();
        return fail(SF_ERR_NO_DEVICE, "sf_ctx_create: no CUDA device");
    }
    if (device < 0 || device >= n) return fail(SF_ERR_NO_DEVICE, "sf_ctx_create: device index out of range");
    sf_ctx* c = new sf_ctx();
    c->device = device;
    int rc = set_device(c);
    if (rc) { delete c; return rc; }
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) == cudaSuccess) c->num_sms = prop.multiProcessorCount;
    if (cudaMalloc(&c->d_counters, sizeof(unsigned long long) * CNT_N) != cudaSuccess ||
        cudaMalloc(&c->d_scalars, sizeof(double) * SC_N) != cudaSuccess ||
        cudaMalloc(&c->d_flags, sizeof(int) * FL_N) != cudaSuccess ||
        cudaMallocHost(&c->h_scalars, sizeof(double) * SC_N) != cudaSuccess ||
        cudaEventCreate(&c->ev_a) != cudaSuccess || cudaEventCreate(&c->ev_b) != cudaSuccess ||
        cudaEventCreate(&c->ev_c) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->ev_check[0], cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->ev_check[1], cudaEventDisableTiming) != cudaSuccess ||
        cudaStreamCreateWithFlags(&c->work, cudaStreamNonBlocking) != cudaSuccess) {
        cudaError_t le = cudaGetLastError();
        sf_ctx_destroy(c);
        return cuda_fail(le, "sf_ctx_create allocation", __FILE__, __LINE__);
    }
    cudaMemset(c->d_counters, 0, sizeof(unsigned long long) * CNT_N);
    cudaMemset(c->d_scalars, 0, sizeof(double) * SC_N);
    cudaMemset(c->d_flags, 0, sizeof(int) * FL_N);
    SF_CUDA(cudaDeviceSynchronize());
    room_add_context(c);
    *out = c;
    return SF_OK;
}

int sf_ctx_destroy(sf_ctx* c) {
    if (!c) return SF_OK;
    room_remove_context(c);
    cudaSetDevice(c->device);
    cudaDeviceSynchronize();
    mixed_engine_release(c);
    Scratch* all[] = {&c->keys,     &c->counts, &c->offsets,  &c->perm,  &c->records, &c->longs,
                      &c->scan_tmp, &c->fields, &c->partials, &c->mixed,  &c->exch, &c->halo};
    for (Scratch* s : all)
        if (s->ptr) cudaFree(s->ptr);
    if (c->d_counters) cudaFree(c->d_counters);
    if (c->d_scalars) cudaFree(c->d_scalars);
    if (c->d_flags) cudaFree(c->d_flags);
    if (c->work) cudaStreamDestroy(c->work);
    if (c->h_scalars) cudaFreeHost(c->h_scalars);
    cudaEvent_t evs[] = {c->ev_a, c->ev_b, c->ev_c, c->ev_check[0], c->ev_check[1]};
    for (cudaEvent_t ev : evs)
        if (ev) cudaEventDestroy(ev);
    delete c;
    return SF_OK;
}

int sf_ctx_scratch_bytes(sf_ctx* c, int64_t* bytes) {
    if (!c || !bytes) return fail(SF_ERR_INVALID_ARG, "sf_ctx_scratch_bytes: NULL argument");
    const Scratch* all[] = {&c->keys,     &c->counts, &c->offsets,  &c->perm,  &c->records, &c->longs,
                            &c->scan_tmp, &c->fields, &c->partials, &c->mixed,  &c->exch, &c->halo};
    int64_t b = 0;
    for (const Scratch* s : all) b += (int64_t)s->bytes;
    *bytes = b;
    return SF_OK;
}

int sf_ctx_launch_count(sf_ctx* c, int64_t* launches) {
    if (!c || !launches) return fail(SF_ERR_INVALID_ARG, "sf_ctx_launch_count: NULL argument");
    *launches = c->launches;
    return SF_OK;
}

int sf_get_warnings(sf_ctx* c, sf_warnings* out, int reset) {
    if (!c || !out) return fail(SF_ERR_INVALID_ARG, "sf_get_warnings: NULL argument");
    int rc = set_device(c);
    if (rc) return rc;
    unsigned long long h[CNT_N];
    SF_CUDA(cudaDeviceSynchronize());
    SF_CUDA(cudaMemcpy(h, c->d_counters, sizeof(h), cudaMemcpyDeviceToHost));
    out->bad_markers = (int64_t)h[CNT_BAD_MARKERS];
    out->empty_nodes = (int64_t)h[CNT_EMPTY_NODES];
    out->interp_failsafe = (int64_t)h[CNT_INTERP_FAILSAFE];
    out->markers_outside = (int64_t)h[CNT_OUTSIDE];
    if (reset) SF_CUDA(cudaMemset(c->d_counters, 0, sizeof(h)));
    return SF_OK;
}

int sf_selftest_bounded_wait(sf_ctx* c, int arrive, int64_t budget_ns, int32_t* timed_out) {
    if (!c || !timed_out) return fail(SF_ERR_INVALID_ARG, "sf_selftest_bounded_wait: NULL argument");
    if (budget_ns < 1 || budget_ns > 2000000000LL)
        return fail(SF_ERR_INVALID_ARG, "sf_selftest_bounded_wait: budget_ns must be in 1 .. 2e9");
    int rc = set_device(c);
    if (rc) return rc;
    int* d = c->d_flags + FL_SELFTEST;   // (the solvers' flags stay untouched)
    SF_CUDA(cudaMemsetAsync(d, 0, sizeof(int), c->work));
    k_wait_selftest<<<1, 128, 0, c->work>>>(arrive, (uint64_t)budget_ns, d);
    SF_LAUNCHED(c);
    SF_CUDA(cudaMemcpyAsync(timed_out, d, sizeof(int), cudaMemcpyDeviceToHost, c->work));
    SF_CUDA(cudaStreamSynchronize(c->work));
    return SF_OK;
}

int sf_selftest_tile_wait(sf_ctx* c, int64_t budget_ns) {
    if (!c) return fail(SF_ERR_INVALID_ARG, "sf_selftest_tile_wait: ctx is NULL");
    if (budget_ns < 1 || budget_ns > 2000000000LL)
        return fail(SF_ERR_INVALID_ARG, "sf_selftest_tile_wait: budget_ns must be in 1 .. 2e9");
    c->tiles_fail_ns = budget_ns;
    return SF_OK;
}

int sf_marker_count(int64_t md, int64_t nx, int64_t ny, int64_t* nmx, int64_t* nmy) {
    if (md < 1 || nx < 2 || ny < 2 || !nmx || !nmy) return fail(SF_ERR_INVALID_ARG, "sf_marker_count: bad arguments");
    *nmx = md * (nx - 1);
    *nmy = md * (ny - 1);
    return SF_OK;
}

double sf_uniform(uint64_t seed, uint64_t counter) { return uniform01(seed, counter); }

int sf_init_markers_host(int64_t md, double lx, double ly, double dx, double dy, int64_t nx, int64_t ny,
                         double jitter, uint64_t seed, double* x, double* y) {
    if (md < 1 || nx < 2 || ny < 2 || !x || !y) return fail(SF_ERR_INVALID_ARG, "sf_init_markers_host: bad arguments");
    MarkerLayout L = marker_layout(md, lx, ly, dx, dy, nx, ny);
    int64_t nm = L.nmx * L.nmy;
    for (int64_t m = 0; m < nm; ++m) marker_position(L, jitter, seed, m, &x[m], &y[m]);
    return SF_OK;
}

int sf_init_markers(sf_ctx* c, int64_t md, double lx, double ly, double dx, double dy, int64_t nx, int64_t ny,
                    double jitter, uint64_t seed, double* x, double* y, void* stream) {
    if (!c || md < 1 || nx < 2 || ny < 2 || !x || !y) return fail(SF_ERR_INVALID_ARG, "sf_init_markers: bad arguments");
    int rc = set_device(c);
    if (rc) return rc;
    MarkerLayout L = marker_layout(md, lx, ly, dx, dy, nx, ny);
    int64_t nm = L.nmx * L.nmy;
    if (nm == 0) return SF_OK;
    unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(nm, 256), (int64_t)c->num_sms * 16);
    k_init_markers<<<blocks, 256, 0, as_stream(stream)>>>(L, jitter, seed, x, y);
    SF_LAUNCHED(c);
    return SF_OK;
}

int sf_marker_count_rank(int64_t md, int64_t nx, int64_t ny, int32_t coord_x, int32_t coord_y, int32_t dims_x,
                         int32_t dims_y, int64_t* nmx, int64_t* nmy) {
    if (md < 1 || nx < 3 || ny < 3 || !nmx || !nmy || dims_x < 1 || dims_y < 1 || coord_x < 0 || coord_x >= dims_x ||
        coord_y < 0 || coord_y >= dims_y)
        return fail(SF_ERR_INVALID_ARG, "sf_marker_count_rank: bad arguments");
    MarkerLayout L = marker_layout_rank(md, 1.0, 1.0, 1.0, 1.0, nx, ny, coord_x, coord_y, dims_x, dims_y);
    *nmx = L.nmx;
    *nmy = L.nmy;
    return SF_OK;
}

int sf_init_markers_rank(sf_ctx* c, int64_t md, double lx, double ly, double dx, double dy, int64_t nx, int64_t ny,
                         int32_t coord_x, int32_t coord_y, int32_t dims_x, int32_t dims_y, double jitter,
                         uint64_t seed, double* x, double* y, void* stream) {
    if (!c || md < 1 || nx < 3 || ny < 3 || !x || !y || dims_x < 1 || dims_y < 1 || coord_x < 0 ||
        coord_x >= dims_x || coord_y < 0 || coord_y >= dims_y)
        return fail(SF_ERR_INVALID_ARG, "sf_init_markers_rank: bad arguments");
    int rc = set_device(c);
    if (rc) return rc;
    MarkerLayout L = marker_layout_rank(md, lx, ly, dx, dy, nx, ny, coord_x, coord_y, dims_x, dims_y);
    int64_t nm = L.nmx * L.nmy;
    if (nm <= 0) return SF_OK;
    unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(nm, 256), (int64_t)c->num_sms * 16);
    k_init_markers<<<blocks, 256, 0, as_stream(stream)>>>(L, jitter, seed, x, y);
    SF_LAUNCHED(c);
    return SF_OK;
}

int sf_set_marker_properties_host(const sf_plume_model* M, const double* x, const double* y, int64_t nm, double x0,
                                  double y0, double* rho, double* mu) {
    if (!M || nm < 0 || (nm > 0 && (!x || !y || !rho || !mu)))
        return fail(SF_ERR_INVALID_ARG, "sf_set_marker_properties_host: bad arguments");
    for (int64_t m = 0; m < nm; ++m) {
        double xx = x0 + x[m], yy = y0 + y[m];
        rho[m] = plume_eval(*M, xx, yy, M->rho_air, M->rho_matrix, M->rho_plume);
        mu[m] = plume_eval(*M, xx, yy, M->mu_air, M->mu_matrix, M->mu_plume);
    }
    return SF_OK;
}

int sf_set_marker_properties(sf_ctx* c, const sf_plume_model* M, const double* x, const double* y, int64_t nm,
                             double x0, double y0, double* rho, double* mu, void* stream) {
    if (!c || !M || nm < 0 || (nm > 0 && (!x || !y || !rho || !mu)))
        return fail(SF_ERR_INVALID_ARG, "sf_set_marker_properties: bad arguments");
    if (nm == 0) return SF_OK;
    int rc = set_device(c);
    if (rc) return rc;
    unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(nm, 256), (int64_t)c->num_sms * 16);
    k_set_props<<<blocks, 256, 0, as_stream(stream)>>>(*M, x, y, nm, x0, y0, rho, mu);
    SF_LAUNCHED(c);
    return SF_OK;
}

}  // extern "C"
