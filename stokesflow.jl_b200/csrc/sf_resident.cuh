// sf_resident.cuh -- many pseudo-transient iterations of a small grid in one launch
// (sf_resident.cu): the kernel's parameters, its plan and its host-side launcher.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sf_internal.cuh"

namespace sf {

constexpr int RESIDENT_LOST = -1;           // (no sf_status) the tiles could not run: march
constexpr int RESIDENT_MIN_ITERS = 4;       // fewer are faster by the march
// iterations of one launch; of tiles that take a whole SM fewer, since kernels on other streams wait for its end (1.5 ms;
// a launch's load and store are 0.5% of that)
constexpr int RESIDENT_MAX_ITERS = 20000, RESIDENT_MAX_ITERS_WHOLE = 512;

struct ResidentParams {
    // the state that is read, the state that is written (other buffers) and the parameters, all in the padded layout
    const double *Vx_in, *Vy_in, *P_in, *dVx_in, *dVy_in;
    double *Vx_out, *Vy_out, *P_out, *dVx_out, *dVy_out;
    const double *rho, *mub, *mup2, *dtp, *dtx, *dty;   // mub = 2.0 mu_b 0.5, mup2 = 2 mu_p
    const double* dt_ptr;
    int Nx, Ny;
    int64_t LD;
    double _dx, _dy, g_y, dampX, dampY;
    int ntx, nty, W, H;          // tiles, and the points of one
    int iters;
    uint32_t tag0;               // iteration k (0-based) publishes with tag tag0 + k
    ulonglong2* comm;            // received halo entries, [parity][tile][slot]
    int* err_flag;               // set where a wait for another tile gave up; nothing is done where it is set already
    uint64_t wait_ns;            // (set by resident_launch)
    // of the last iteration, where wanted: tau and divV (NULL: not), and max|Vx|, max|Vy| as bit patterns, accumulated
    // onto what is there (NULL: not)
    double *txx, *tyy, *txy, *divV;
    unsigned long long* max_bits;
    const double* err;           // where given, nothing is done unless eps < *err < infinity
    double eps;
};

// whether the loop goes on after a check (StokesSolver_multixpu.jl:43, :75): for kernels launched behind the check
__device__ __forceinline__ bool goes_on(const double* err, double eps) { return *err > eps && !isinf(*err); }

struct ResidentPlan {
    bool fits = false;           // the grid is small enough
    bool cluster = false;        // the tiles are one thread-block cluster
    int ntx = 0, nty = 0, W = 0, H = 0, k = 0, threads = 0, smem = 0;
    int share = 0;               // quarters of an SM that a tile takes: 1 to 4
    int max_iters() const { return share == 4 ? RESIDENT_MAX_ITERS_WHOLE : RESIDENT_MAX_ITERS; }
};

// Room on a device for the tiles of a plan, held while a solve uses it.  The tiles of a launch wait for one another, so
// all must become resident whatever else runs: concurrent solves (other threads, streams and contexts) hold at most
// three quarters of every SM together.  Then a tile of one or two quarters always finds a place (an SM without one
// holds two quarters or three already, and not all SMs can); its launch ends; and what is left of three quarters finds its
// place in turn.  The last quarter stays free for kernels that are not resident: a solve that marches beside them waits
// for no launch of theirs.  A plan of whole SMs is for a solve that is alone on the device, and gives way when another
// one begins: a march of 64^2 would wait up to a launch of 511 x 385 at every step.
// A cluster is placed whole or not at all and needs no such room, but one that waits for a free group of SMs
// could stand before tiles that others wait for: clusters and tiles that exchange through L2 do not run together.
// A solve that gets no room marches instead (same results).  The ledger is this process's: tiles of other processes
// on the device (MPS) or a partition of it with fewer SMs are not in it.  There a launch may be refused, or a tile's wait
// for another may run out (RESIDENT_LOST): the solve begins again and marches.
class ResidentRoom {
   public:
    ResidentRoom(int device, int num_sms, cudaStream_t s);   // for the duration of a solve
    ~ResidentRoom();
    bool acquire(const ResidentPlan& plan);
    void release();
    bool alone() const;   // no other solve on the device

   private:
    bool known() const { return device_ >= 0 && device_ < 64; }
    int device_, num_sms_, held_ = 0;
    bool cluster_ = false;
    cudaStream_t stream_;
};

ResidentPlan cluster_plan(int64_t Nx, int64_t Ny, int device);
ResidentPlan resident_plan(int64_t Nx, int64_t Ny, int num_sms);
// the memory that a plan's tiles exchange through; before the launches
int resident_scratch(sf_ctx* ctx, const ResidentPlan& plan, cudaStream_t s);
// p.iters iterations; the tiles and the exchange's slots of p are set here.  RESIDENT_LOST: the device did not take them
int resident_launch(sf_ctx* ctx, ResidentParams& p, const ResidentPlan& plan, cudaStream_t s);

}  // namespace sf
