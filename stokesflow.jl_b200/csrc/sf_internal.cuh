// sf_internal.cuh -- shared internals of libstokesflow_b200.so: the context,
// status/error plumbing, grow-only scratch buffers and the small device
// helpers that every kernel file uses.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cmath>
#include <map>
#include <utility>
#include <string>

#include "stokesflow_b200.h"

namespace sf {

// --------------------------------------------------------------------------
// errors
// --------------------------------------------------------------------------
void set_error(const std::string& msg);
int fail(int status, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what, const char* file, int line);

#define SF_CUDA(call)                                                   \
    do {                                                                \
        cudaError_t e_ = (call);                                        \
        if (e_ != cudaSuccess) return ::sf::cuda_fail(e_, #call, __FILE__, __LINE__); \
    } while (0)

#define SF_CHECK_LAUNCH() SF_CUDA(cudaGetLastError())

// after every kernel launch: check it and count it on the context
#define SF_LAUNCHED(c)        \
    do {                      \
        SF_CHECK_LAUNCH();    \
        ++(c)->launches;      \
    } while (0)

#define SF_REQUIRE(cond, msg)                                           \
    do {                                                                \
        if (!(cond)) return ::sf::fail(SF_ERR_INVALID_ARG, msg);        \
    } while (0)

// --------------------------------------------------------------------------
// scratch: a grow-only device buffer owned by the context
// --------------------------------------------------------------------------
struct Scratch {
    void* ptr = nullptr;
    size_t bytes = 0;
};

// device-side warning counters, in the order of sf_warnings
enum { CNT_BAD_MARKERS = 0, CNT_EMPTY_NODES = 1, CNT_INTERP_FAILSAFE = 2, CNT_OUTSIDE = 3, CNT_N = 4 };

// device scalars used by the PT solve
// SC_DT: dt used by the stabilisation term; SC_DT_CHECK: dt of the residual
// check; SC_DT_OUT: dt returned by the solve; SC_MAXBITS (2 slots): max|Vx|,
// max|Vy| as ordered bit patterns during a reduction, zero between reductions;
// SC_TICKET: blocks of k_residuals that are done, zero between launches.
enum { SC_DT = 0, SC_DT_CHECK = 1, SC_ERR = 2, SC_SUM_RX = 3, SC_SUM_RY = 4, SC_SUM_DIV = 5,
       SC_MAX_VX = 6, SC_MAX_VY = 7, SC_SCALE = 8, SC_DT_OUT = 9,
       SC_ERR2 = 10 /* host: every other check's err */, SC_WAITS = 11 /* host: WAIT_* bits */, SC_MAXBITS = 12, SC_TICKET = 14, SC_N = 16 };

// d_flags: waits that gave up.  FL_COPY: for a tile copy; FL_SELFTEST; FL_TILES: of resident tiles for one another
enum { FL_COPY = 0, FL_SELFTEST = 1, FL_TILES = 2, FL_N = 4 };
enum { WAIT_COPY = 1, WAIT_TILES = 2 };   // the same as bits
__host__ __device__ __forceinline__ int wait_bits(const volatile int* flags) {
    return (flags[FL_COPY] ? WAIT_COPY : 0) | (flags[FL_TILES] ? WAIT_TILES : 0);
}

}  // namespace sf

struct sf_ctx {
    int device = 0;
    int num_sms = 148;
    // deposit / rebin scratch: cell keys and run ends, counts, offsets, the cell-ordered permutation, scan tiles, the
    // deposit's marker records and the lists of long cells
    sf::Scratch keys, counts, offsets, perm, scan_tmp, records, longs;
    // PT solve: padded internal fields, reduction partials; mixed/batched engine arena
    sf::Scratch fields, partials, mixed;
    // decomposed timestep: marker-exchange and overlap-sum staging
    sf::Scratch exch;
    // resident iterations: the tiles' halo slots, and the tag of the next iteration (1 at first: slots start zeroed)
    sf::Scratch halo;
    uint32_t halo_tag = 1;
    cudaStream_t work = nullptr;  // private non-blocking stream (graph capture needs a non-legacy stream)
    // device counters (unsigned long long[CNT_N]) and scalars (double[SC_N])
    unsigned long long* d_counters = nullptr;
    double* d_scalars = nullptr;
    double* h_scalars = nullptr;  // pinned mirror
    int* d_flags = nullptr;       // device error flags, int[FL_N]
    int64_t tiles_fail_ns = 0;    // self-test: the next resident launch fails, its waits giving up after this (0: no)
    cudaEvent_t ev_a = nullptr, ev_b = nullptr, ev_c = nullptr;
    cudaEvent_t ev_check[2] = {};  // the PT loop's residual checks
    int64_t launches = 0;         // kernels launched through this context
    // until when (steady clock, ns) marker kernels of this context are taken to run; other contexts' solves read it
    std::atomic<int64_t> markers_until{0};
    sf_engine* batch_engine = nullptr;  // the engine sf_solve_stokes_batch_mixed reuses across calls
    // sweep shapes the engines' autotuner measured best, by workload class (sf_mixed.cu)
    std::map<int, int> sweep_shapes;
};

namespace sf {

// Whether the device has the memory for `s` to hold `bytes`, what `s` holds now among it.
bool may_have(const Scratch& s, size_t bytes);
// Ensures `s` holds at least `bytes`; contents are not preserved.
int ensure(sf_ctx* ctx, Scratch& s, size_t bytes);
int set_device(sf_ctx* ctx);
// Whether device `dev` can read and write `peer`'s memory directly (NVLink / PCIe peer access), enabling it on
// first use; *ok is true for dev == peer.  Pairs without peer access copy through the runtime instead.
int peer_access(int dev, int peer, bool* ok);
// A w x h block of doubles (rows of w contiguous entries, leading dimensions ld_dst / ld_src) from src, which
// lives on src_device, to dst on ctx's device, queued on stream s of that device (current).  With peer access
// (or one device) a copy kernel on ctx's device reads src directly -- plain loads, no multicast; otherwise
// cudaMemcpy2DAsync does it.
int copy_block(sf_ctx* ctx, cudaStream_t s, double* dst, int64_t ld_dst, const double* src, int64_t ld_src,
               int64_t w, int64_t h, int src_device);
// frees the context's cached batch engine (sf_mixed.cu)
void mixed_engine_release(sf_ctx* ctx);

// true when no two of the n contexts (reached through get(i)) are the same: a rank's scratch is its own
template <typename Get>
bool distinct_contexts(int n, Get get) {
    for (int i = 0; i < n; ++i)
        for (int j = i + 1; j < n; ++j)
            if (get(i) == get(j)) return false;
    return true;
}
inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// launches `kern`; with `overlap`, under programmatic stream serialization: it may begin (launch, prologue)
// while the previous kernel on `s` drains, and must call griddep_wait() before it touches that kernel's
// results (sf_tma.cuh)
template <typename... Params, typename... Args>
cudaError_t launch_overlapped(bool overlap, void (*kern)(Params...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t s, Args&&... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// for the ledger of resident tiles (sf_resident.cuh): the contexts, and marker kernels over nm markers launched on a device
// (ctx NULL: without a context)
void room_add_context(const sf_ctx* ctx);
void room_remove_context(const sf_ctx* ctx);
void markers_launched(sf_ctx* ctx, int device, int64_t nm);

// What is done or looked up once per device; threads that come at the same time each do it, with the same outcome.
constexpr int MAX_DEVICES = 64;
struct PerDevice {
    std::atomic<int> value[MAX_DEVICES] = {};   // 0: not yet
    int get(int device) const { return device >= 0 && device < MAX_DEVICES ? value[device].load(std::memory_order_acquire) : 0; }
    void set(int device, int v) {
        if (device >= 0 && device < MAX_DEVICES) value[device].store(v, std::memory_order_release);
    }
};
// lets launches of `kern` on the current device, `device`, have `bytes` of dynamic shared memory
inline int allow_smem(PerDevice& done, int device, const void* kern, int bytes) {
    if (done.get(device)) return SF_OK;
    SF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    done.set(device, 1);
    return SF_OK;
}

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline int64_t round_up(int64_t a, int64_t b) { return ceil_div(a, b) * b; }

// --------------------------------------------------------------------------
// device helpers
// --------------------------------------------------------------------------

// scripts/common.jl:22-33 topleftIndexRelDist.  ix, iy are 1-based like the
// reference; q is floor((x - x_grid_min)/dx) kept in double so that NaN and
// huge values can be classified without undefined conversions.
struct TopLeft {
    double qx, qy;     // floor((x - xmin)/dx) = ix - 1
    double dxij, dyij;
};

__device__ __forceinline__ TopLeft topleft(double xmin, double ymin, double x, double y, double dx,
                                           double dy) {
    TopLeft t;
    t.qx = floor((x - xmin) / dx);
    t.qy = floor((y - ymin) / dy);
    double x_ix = xmin + t.qx * dx;   // x_grid_min + (ix - 1) * dx
    double y_iy = ymin + t.qy * dy;
    t.dxij = (x - x_ix) / dx;
    t.dyij = (y - y_iy) / dy;
    return t;
}

// a / b correctly rounded, from y = RN(1 / b): q = RN(a y) is within 1.5 ulp of a / b; one correction by its remainder
// brings it within 1 ulp, and then the remainder a - b q is exact and RN(q + r y) = RN(a / b) (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990: the theorem on a faithful quotient and a correctly
// rounded reciprocal).  Needs |a| of 2^-960 .. 2^960 (or 0) and b of 2^-60 .. 2^60, so that nothing is lost below the
// exponent range.  Five FP64 operations; the division is about twice that.
__device__ __forceinline__ double div_const(double a, double b, double y) {
    double q = a * y;
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

__device__ __forceinline__ bool div_const_takes_a(double a) {   // false for NaN and infinities
    const unsigned hi = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return hi - 0x08000000u < 0x70000000u || (hi | (unsigned)__double2loint(a)) == 0u;
}
inline bool div_const_takes(double b) { return b > 0x1p-60 && b < 0x1p60; }

// SplitMix64 finaliser; sf_uniform(seed, k) = top 53 bits of
// mix(mix(seed) ^ k*C) / 2^53.
__host__ __device__ __forceinline__ uint64_t splitmix64_mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__host__ __device__ __forceinline__ double uniform01(uint64_t seed, uint64_t counter) {
    uint64_t z = splitmix64_mix(splitmix64_mix(seed) ^ (counter * 0xD1B54A32D192ED03ull));
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// Julia max(x, 0) and min(x, l) for Float64: -0.0 < 0.0, NaN propagates.
__host__ __device__ __forceinline__ double jl_max0(double x) {
    if (x != x) return x;
    return (x < 0.0 || (x == 0.0 && std::signbit(x))) ? 0.0 : x;
}
__host__ __device__ __forceinline__ double jl_min(double x, double l) {
    if (x != x) return x;
    return (l < x) ? l : x;
}

}  // namespace sf
