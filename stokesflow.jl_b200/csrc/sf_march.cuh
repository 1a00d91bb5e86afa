// sf_march.cuh -- several pseudo-transient iterations in one pass over memory
// (sf_march.cu): the kernel's parameters and its host-side launcher.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sf_internal.cuh"

namespace sf {

constexpr int MARCH_MAX_T = 3;   // iterations of one launch at most
constexpr int MARCH_CW = 64;     // columns of a strip with its halo
// the fields' slabs: the state's A buffers {Vx, Vy, P, dVx, dVy}, its B buffers, then {rho, mu_b, 2 mu_p, dtauP,
// dtauVx, dtauVy}; within each, the row of a slab that holds a field's row 0
constexpr int MARCH_Z_A = 0, MARCH_Z_B = 5, MARCH_Z_MAT = 10, MARCH_NZ = 16;
constexpr int MARCH_SKEW[MARCH_NZ] = {0, 0, 1, 2, 2, 0, 0, 1, 2, 2, 0, 1, 1, 1, 2, 2};

struct MarchMaps {
    CUtensorMap state, mat;      // boxes of MARCH_CW x 1 x 5 and MARCH_CW x 1 x 6 over the slabs
};

struct MarchParams {
    double* __restrict__ Vx_out;
    double* __restrict__ Vy_out;
    double* __restrict__ P_out;
    double* __restrict__ dVx_out;
    double* __restrict__ dVy_out;
    const double* __restrict__ dt_ptr;
    int z_in;                    // MARCH_Z_A or MARCH_Z_B: the buffers that are read
    int Nx, Ny;
    int64_t LD;
    double _dx, _dy, g_y, dampX, dampY;
    int ns, w, nseg, rows;       // strips, their columns, segments of a strip, their rows
    int* __restrict__ err_flag;
};

// Iterations per launch on an Nx x Ny grid.
int march_iterations(int64_t Nx, int64_t Ny);
// Splits an Nx x Ny grid into strips and segments for T iterations per launch (p.Nx, p.Ny set).
void march_plan(MarchParams& p, int T, int num_sms);
// T in 1 .. MARCH_MAX_T iterations
int march_launch(sf_ctx* ctx, const MarchMaps& maps, const MarchParams& p, int T, cudaStream_t s);

}  // namespace sf
