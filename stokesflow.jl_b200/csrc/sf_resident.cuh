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
// place in turn.  The last quarter stays free for solves that march beside them and wait for no launch of theirs.  A plan
// of whole SMs (222^2 - 257^2, 317^2 - 373^2, 387^2 - 529^2) is for a solve that is alone on the device: a march of 64^2
// would wait up to a launch of 511 x 385 at every step.
// Other work of this library comes first where it is known.  Beside an engine or batched solve under way, or a decomposed
// one, no tiles are placed that exchange through L2: their sweeps fill the device, and a quarter of every SM is too little
// (an engine's sweep takes 11.2 us beside 256^2 by single iterations, beside its tiles 67.7, beside its march 12.0; beside
// 450^2 12.7, 103 and 13.0; beside 300^2, which takes three quarters, 11.4, 22.9 and 12.3).  Beside marker kernels that
// another context has just launched no tiles of whole SMs are (three deposits of 128^2 beside 450^2: 331, 546 and 129 us; a
// rebin of 0.6 M markers 137, 453 and 104): other tiles gain more than such short kernels lose.  A solve gives its tiles up,
// or takes some, at a check.  A cluster has 16 SMs and leaves the others.  Kernels of other libraries are not known here;
// they wait for a launch's end (1.5 ms for whole SMs).
// A cluster is placed whole or not at all and needs no such room, but one that waits for a free group of SMs
// could stand before tiles that others wait for: clusters and tiles that exchange through L2 do not run together.
// A solve that gets no room marches instead (same results).  The ledger is this process's: tiles of other processes
// on the device (MPS) or a partition of it with fewer SMs are not in it.  There a launch may be refused, or a tile's wait
// for another may run out (RESIDENT_LOST): the solve begins again and marches.
class ResidentRoom {
   public:
    ResidentRoom(const sf_ctx* ctx, cudaStream_t s);   // for the duration of a solve
    ~ResidentRoom();
    bool acquire(const ResidentPlan& plan);
    void release();
    bool keeps(const ResidentPlan& plan) const;   // whether a solve that has room for the plan may go on using it

   private:
    bool known() const;
    bool whole_sms() const;   // (with the ledger's lock) no other solve, no marker kernels
    const sf_ctx* ctx_;
    int device_, held_ = 0;
    bool cluster_ = false;
    cudaStream_t stream_;
};

// Announces work on a device that is neither a plain solve nor marker kernels, for as long as it lives.
class OtherWork {
   public:
    explicit OtherWork(int device);
    ~OtherWork();
    OtherWork(const OtherWork&) = delete;
    OtherWork& operator=(const OtherWork&) = delete;

   private:
    int device_;
};

ResidentPlan cluster_plan(int64_t Nx, int64_t Ny, int device);
ResidentPlan resident_plan(int64_t Nx, int64_t Ny, int num_sms);
// the memory that a plan's tiles exchange through; before the launches
int resident_scratch(sf_ctx* ctx, const ResidentPlan& plan, cudaStream_t s);
// p.iters iterations; the tiles and the exchange's slots of p are set here.  RESIDENT_LOST: the device did not take them
int resident_launch(sf_ctx* ctx, ResidentParams& p, const ResidentPlan& plan, cudaStream_t s);

}  // namespace sf
