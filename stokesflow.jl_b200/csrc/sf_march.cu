// sf_march.cu -- T pseudo-transient iterations (StokesSolver_multixpu.jl:48-57) in one pass over memory.
//
// One iteration moves 104 bytes per point whatever it computes, so a kernel that does one iteration per launch
// cannot be faster than HBM allows.  Here a launch does T iterations:
//
//   * a warp owns a strip of columns (two per lane) and a segment of rows, and marches along y.  At row step r
//     level 1 computes the first iteration's velocities of row r-1 from the rows r-2 .. r of the old state;
//     level 2 takes them at once and computes the second iteration's row r-2, and so on; level T's row goes
//     to memory.  Whatever a level needs of its previous rows stays in registers, neighbours in x come by shuffle:
//     no stage arrays, no block barrier, no second evaluation of tau or P in y;
//   * warps do not exchange anything: a strip is computed with extra columns and a segment with T extra rows on
//     each side, whose results are dropped (their owners compute the same values);
//   * the rows of the eleven input fields come through a ring of shared-memory slots, two tensor copies per row
//     (the five state fields, the six parameter fields) that one lane issues NSS rows ahead, completion on an
//     mbarrier (bounded wait).  The fields' slabs are laid out skewed (sf_solve.cu), so that one box holds the rows
//     that a step reads.  Levels 2 .. T re-read the parameter rows from the ring;
//   * all five state fields are double-buffered, as a segment reads rows that its neighbours overwrite.
//
// The free-slip entries are set on the way from level to level as the reference's boundary kernels set them
// (:53-56), so every level sees the arrays the reference's iteration would.  Every expression keeps the
// reference's order of operations (and the file is compiled without contraction): bit-identical to T single
// iterations.
//
// What bounds it: at 2048^2 a launch of three iterations moves 549 MB (128 B per point and the halos) in 100 us, 5.4 TB/s,
// with the FP64 pipe some 60% busy; on smaller grids the halo rows of short segments.  85 -> 33.5 us per iteration at
// 2048^2, 241 -> 97 at 4001 x 3003, 24.6 -> 11.9 at 1024^2; in runs of seconds, which draw the 1000 W limit and settle at
// 1.69 GHz, 89.9 -> 37.5, 258 -> 105 and (1.86 GHz) 24.6 -> 12.4.  One warp per block, 234 registers, 8 blocks per SM (two warps
// per scheduler): two columns to a lane halve the shuffles, and 32 doubles in flight per lane hide the latencies that few
// warps would not (four per SM: 56 us at 2048^2; twelve with T = 2: 68; T = 4 spills: 63).  Every item runs the same code,
// the boundary entries as selects: with a leaner body for the items inside, the two bodies shared the instruction cache
// and the others finished late (37 us at 2048^2, 113 at 4001 x 3003); branches around the boundary entries cost as much.
// The first form of this kernel loaded each field's row by its own copy and divided by max(Nx, Ny): 50.6 us.
#include <algorithm>

#include "sf_march.cuh"
#include "sf_tma.cuh"

namespace sf {
namespace {

constexpr uint64_t MARCH_WAIT_NS = 2000000000ull;
constexpr int CW = MARCH_CW;                   // columns of a strip with its halo: two per lane
constexpr int ROW = CW * 8;
// a step's rows: Vx, Vy of row r, P of row r - 1, dVx, dVy of row r - 2 ...
constexpr int S_X = 0, S_Y = ROW, S_P = 2 * ROW, S_DX = 3 * ROW, S_DY = 4 * ROW, STATE_ROW = 5 * ROW;
// ... rho of row r, mu_b, 2 mu_p, dtauP of row r - 1, dtauVx, dtauVy of row r - 2
constexpr int M_RHO = 0, M_MUB = ROW, M_MUP2 = 2 * ROW, M_TP = 3 * ROW, M_TX = 4 * ROW, M_TY = 5 * ROW,
              MAT_ROW = 6 * ROW;
constexpr uint32_t ROW_TX = STATE_ROW + MAT_ROW;

// columns of a strip to the left of its own: the validity of a level's results shrinks by one column per level
// from both sides, and a lane stores velocity columns c and c + 1 from its left neighbour's and its own
constexpr int left_halo(int T) { return T == 1 ? 2 : 4; }

template <int T, int NSS>
struct Ring {
    // a state row is read at its own step only; a parameter row at its step and the T - 1 steps after it
    static constexpr int NSM = NSS + T - 1;
    static constexpr int BAR = NSS * STATE_ROW + NSM * MAT_ROW;
    static constexpr int BYTES = BAR + 8 * NSS;
};

__device__ __forceinline__ double from_right(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double from_left(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }

// what one iteration level keeps between two row steps; [h]: this lane's two columns c, c + 1.  Column c of the
// velocities is Vx(c + 1), Vy(c + 1) -- the entries that pressure column c's thread updates
struct Level {
    double X[2], Y[2], Yr;     // Vx, Vy of the row before, and Vy of the column to the right of the second one
    double S[2];               // Vx(c) + Vx(c + 1) of the row before
    double A[2], C[2];         // x differences of tau_xx and P of the pressure row before, times _dx
    double ty[2], Pn[2], Q[2]; // tau_yy, P and tau_xy of the row before
    double r1[2], r2[2], g[2]; // rho of the row before and the one before that; x difference of rho of the row before
};

__device__ __forceinline__ void lds2(const unsigned char* p, double* v) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    v[0] = t.x;
    v[1] = t.y;
}

// One row step of a level: X, Y, Xl (the column to the left of the first) and Yr arrive for row r; P0 is the old P
// of row r-1, dvx0 / dvy0 the damped rates of row r-2, m the parameter slot of step r.  Returns the new velocities
// of row r-1 and the rates of row r-2; L.Pn is the new P of row r-1.
__device__ __forceinline__ void march_step(Level& L, const MarchParams& k, double dt, const unsigned char* __restrict__ m,
                                           const double (&X)[2], const double (&Y)[2], double Xl, double Yr,
                                           const double (&P0)[2], const double (&dvx0)[2], const double (&dvy0)[2],
                                           double (&Xn)[2], double (&Yn)[2], double (&dvx)[2], double (&dvy)[2]) {
    double rh[4], mb[4], mu2[2], tp[2], tx[2], ty[2];
    lds2(m + M_RHO, rh);
    lds2(m + M_RHO + 16, rh + 2);
    lds2(m + M_MUB, mb);
    lds2(m + M_MUB + 16, mb + 2);
    lds2(m + M_MUP2, mu2);
    lds2(m + M_TP, tp);
    lds2(m + M_TX, tx);
    lds2(m + M_TY, ty);
    const double xl[2] = {Xl, X[0]};
    const double ypr[2] = {L.Y[1], L.Yr};
    double txx[2], tyy[2], Pn[2], Q[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        // compute_P_tau! (:140-169) at the pressure point of row r-1 and the shear node above it
        const double ex = (X[h] - xl[h]) * k._dx;
        const double ey = (Y[h] - L.Y[h]) * k._dy;
        const double div = ex + ey;
        Pn[h] = P0[h] - tp[h] * div;
        const double third = 1.0 / 3.0 * div;
        txx[h] = mu2[h] * (ex - third);
        tyy[h] = mu2[h] * (ey - third);
        const double sy = (X[h] - L.X[h]) * k._dy;
        const double sx = (ypr[h] - L.Y[h]) * k._dx;
        Q[h] = mb[h + 1] * (sy + sx);
    }
    const double txr = from_right(txx[0]), pr = from_right(Pn[0]), ql = from_left(Q[1]);
    const double txn[2] = {txx[1], txr}, pn[2] = {Pn[1], pr}, qn[2] = {ql, Q[0]};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        // compute_ResX (:176-182), compute_dV!, compute_V! at Vx row r-1
        const double Rx = L.A[h] + (Q[h] - L.Q[h]) * k._dy - L.C[h];
        dvx[h] = k.dampX * dvx0[h] + Rx;
        Xn[h] = L.X[h] + tx[h] * dvx[h];
        // compute_ResY (:189-202) at Vy row r-1
        const double av = 0.25 * (L.S[h] + xl[h] + X[h]);
        const double dyr = rh[h + 1] - L.r2[h];
        const double Ry = (tyy[h] - L.ty[h]) * k._dy + (Q[h] - qn[h]) * k._dx - (Pn[h] - L.Pn[h]) * k._dy +
                          k.g_y * (L.r1[h] - dt * (av * L.g[h] * 0.5 * k._dx + L.Y[h] * dyr * 0.5 * k._dy));
        dvy[h] = k.dampY * dvy0[h] + Ry;
        Yn[h] = L.Y[h] + ty[h] * dvy[h];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        L.X[h] = X[h];
        L.Y[h] = Y[h];
        L.S[h] = xl[h] + X[h];
        L.A[h] = (txn[h] - txx[h]) * k._dx;
        L.C[h] = (pn[h] - Pn[h]) * k._dx;
        L.ty[h] = tyy[h];
        L.Pn[h] = Pn[h];
        L.Q[h] = Q[h];
        L.r2[h] = L.r1[h];
        L.r1[h] = rh[h + 1];
        L.g[h] = rh[h + 2] - rh[h];
    }
    L.Yr = Yr;
}

// A strip's segment; edge: its columns or rows (halo included) see a side of the domain, so that its stores are not whole
// pairs of columns.
template <int T, int NSS>
__device__ __forceinline__ void march_segment(const MarchMaps& maps, const MarchParams& p, unsigned char* smem,
                                              int strip, int seg, const bool edge) {
    using R = Ring<T, NSS>;
    constexpr int NSM = R::NSM;
    unsigned char* const mats = smem + NSS * STATE_ROW;
    uint64_t* const bar = reinterpret_cast<uint64_t*>(smem + R::BAR);
    const int lane = threadIdx.x;
    const int Nx = p.Nx, Ny = p.Ny;
    // own pressure columns [ca, cb) of the Nx - 1, own velocity rows [ra, rb) of 1 .. Ny - 1
    const int ca = strip * p.w, cb = min(ca + p.w, Nx - 1);
    const int ra = 1 + seg * p.rows, rb = min(ra + p.rows, Ny);
    const int c0 = ca - left_halo(T);
    const int r0 = max(ra - T, 0);
    const int steps = (rb + T - r0 + 1) & ~1;   // rows r0 .. rb - 1 + T, one more for an even count

    // rows of step n; beyond the slabs the copies fill in zeros, and what they lead to is dropped
    int in_s = 0, in_m = 0, in_b = 0, in_n = 0;    // the slots that the next rows go to, and their step
    auto issue = [&]() {   // lane 0
        uint64_t* b = bar + in_b;
        mbar_arrive_expect_tx(b, ROW_TX);
        tma_load_3d(smem + in_s, &maps.state, b, c0, r0 + in_n, p.z_in);
        tma_load_3d(mats + in_m, &maps.mat, b, c0, r0 + in_n, MARCH_Z_MAT);
        ++in_n;
        in_s = (in_b + 1 == NSS) ? 0 : in_s + STATE_ROW;
        in_b = (in_b + 1 == NSS) ? 0 : in_b + 1;
        in_m = (in_m + MAT_ROW == NSM * MAT_ROW) ? 0 : in_m + MAT_ROW;
    };
    if (lane == 0)
        for (int n = 0; n < NSS && n < steps; ++n) issue();

    const double dt = *p.dt_ptr;
    Level L[T];
    double pdx[T][2], pdy[T][2];   // rates of level l's previous step: the next level's input one row later
    const unsigned char* mo[T];    // the parameter slot that level l reads
#pragma unroll
    for (int l = 0; l < T; ++l) {
        L[l] = Level{};
        mo[l] = mats + 16 * lane;
#pragma unroll
        for (int h = 0; h < 2; ++h) pdx[l][h] = pdy[l][h] = 0.0;
    }
    const int c = c0 + 2 * lane;                     // this lane's columns c, c + 1 (c is even)
    const bool own = c >= ca && c < cb;              // (inside the domain) both of them, or none
    int so = 0, sb = 0;                              // this step's state slot and barrier
    uint32_t phase = 0;
    // this row's output place: row r0 + n - T of the velocities
    int64_t out = (int64_t)(r0 - T) * p.LD + c;

    auto step = [&](int n) -> bool {
        if (!__all_sync(0xffffffffu, mbar_wait(bar + sb, phase, MARCH_WAIT_NS))) return false;
        const unsigned char* st = smem + so + 16 * lane;
        double X[2], Y[2], P0[2], dvx0[2], dvy0[2], Xl, Yr;
        {
            double t[4];
            lds2(st + S_X, t);
            lds2(st + S_X + 16, t + 2);
            Xl = t[0];
            X[0] = t[1];
            X[1] = t[2];
            lds2(st + S_Y, t);
            lds2(st + S_Y + 16, t + 2);
            Y[0] = t[1];
            Y[1] = t[2];
            Yr = t[3];
            lds2(st + S_P, P0);
            lds2(st + S_DX, dvx0);
            lds2(st + S_DY, dvy0);
        }
#pragma unroll
        for (int l = 0; l < T; ++l) {
            const int r = r0 + n - l;                          // this level's row
            const double Pold[2] = {L[l].Pn[0], L[l].Pn[1]};   // new P of row r - 2: the next level's input
            double Xn[2], Yn[2], dvx[2], dvy[2];
            march_step(L[l], p, dt, mo[l], X, Y, Xl, Yr, P0, dvx0, dvy0, Xn, Yn, dvx, dvy);
            {   // bc_x_zero! on Vx, bc_x_noflux! on Vy (selects, in strips inside too)
                const double y_right = from_right(Yn[0]), y_left = from_left(Yn[1]);
                if (c + 1 == -1) Yn[1] = y_right;
                if (c + 1 == Nx - 1) Yn[1] = Yn[0];
                if (c == Nx - 1) Yn[0] = y_left;
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (c + h == -1 || c + h == Nx - 2) Xn[h] = 0.0;
            }
            if (l + 1 < T) {
                // the velocities of row r - 1 enter level l + 1, whose row it is
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    X[h] = Xn[h];
                    Y[h] = Yn[h];
                    P0[h] = Pold[h];
                    dvx0[h] = pdx[l][h];
                    dvy0[h] = pdy[l][h];
                    pdx[l][h] = dvx[h];
                    pdy[l][h] = dvy[h];
                }
                {   // bc_y_noflux! on Vx, bc_y_zero! on Vy
                    Level& N = L[(l + 1 < T) ? l + 1 : l];
                    const int rn = r - 1;
                    if (rn == 1) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            N.X[h] = X[h];
                            N.Y[h] = 0.0;
                        }
                        N.Yr = 0.0;
                    }
                    if (rn == Ny - 1) Y[0] = Y[1] = 0.0;
                    if (rn == Ny) {
                        X[0] = N.X[0];
                        X[1] = N.X[1];
                    }
                }
                Xl = from_left(X[1]);
                Yr = from_right(Y[0]);
            } else if (!edge) {
                // the row r - 1 leaves, with P and the rates of pressure row r - 2; {c, c + 1} of Vx is an aligned pair
                const double x_left = from_left(Xn[1]), y_left = from_left(Yn[1]);
                if (own && r > ra && r <= rb) {
                    const int64_t q = out - p.LD;
                    *reinterpret_cast<double2*>(p.Vx_out + out) = make_double2(x_left, Xn[0]);
                    *reinterpret_cast<double2*>(p.Vy_out + out) = make_double2(y_left, Yn[0]);
                    *reinterpret_cast<double2*>(p.P_out + q) = make_double2(Pold[0], Pold[1]);
                    *reinterpret_cast<double2*>(p.dVx_out + q) = make_double2(dvx[0], dvx[1]);
                    *reinterpret_cast<double2*>(p.dVy_out + q) = make_double2(dvy[0], dvy[1]);
                }
            } else if (r > ra && r <= rb) {
                const int ro = r - 1;
                const bool last = cb == Nx - 1;
                const int64_t q = out - p.LD;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int col = c + h;
                    if (col >= ca && col < cb) {
                        p.P_out[q + h] = Pold[h];
                        if (col < Nx - 2) p.dVx_out[q + h] = dvx[h];   // the rates end one column (dVx) ...
                        if (ro < Ny - 1) p.dVy_out[q + h] = dvy[h];    // ... and one row (dVy) earlier
                    }
                    // velocity columns ca - 1 .. cb - 2 (the pairs of the vector stores), and to the far side
                    const bool vx_own = col >= ca - 1 && col <= (last ? Nx - 2 : cb - 2);
                    const bool vy_own = col >= ca - 1 && col <= (last ? Nx - 1 : cb - 2);
                    if (vx_own) p.Vx_out[out + h + 1] = Xn[h];
                    if (vy_own) p.Vy_out[out + h + 1] = (ro == Ny - 1) ? 0.0 : Yn[h];
                    // the ghost rows
                    if (ro == 1) {
                        if (vx_own) p.Vx_out[q + h + 1] = Xn[h];
                        if (vy_own) p.Vy_out[q + h + 1] = 0.0;
                    }
                    if (ro == Ny - 1 && vx_own) p.Vx_out[out + p.LD + h + 1] = Xn[h];
                }
            }
        }
        // every lane has read the slots that the next rows go to
        __syncwarp();
        if (lane == 0 && in_n < steps) issue();
#pragma unroll
        for (int l = T - 1; l > 0; --l) mo[l] = mo[l - 1];
        mo[0] = (mo[0] == mats + 16 * lane + (NSM - 1) * MAT_ROW) ? mats + 16 * lane : mo[0] + MAT_ROW;
        so = (sb + 1 == NSS) ? 0 : so + STATE_ROW;
        phase ^= (sb + 1 == NSS) ? 1u : 0u;
        sb = (sb + 1 == NSS) ? 0 : sb + 1;
        out += p.LD;
        return true;
    };
    // two steps a turn: the levels' previous-row values change registers instead of being moved
    for (int n = 0; n < steps; n += 2) {
        if (!step(n) || !step(n + 1)) {
            // a copy never completed: flag it, give the copies in flight a bounded chance to land, leave
            if (lane == 0) atomicExch(p.err_flag, 1);
            for (int q = 1; q < NSS; ++q) {
                if (++sb == NSS) {
                    sb = 0;
                    phase ^= 1u;
                }
                mbar_wait(bar + sb, phase, MARCH_WAIT_NS);
            }
            return;
        }
    }
}

template <int T, int NSS, int WPS>
__global__ void __launch_bounds__(32, WPS) k_pt_march(const __grid_constant__ MarchMaps maps,
                                                      const __grid_constant__ MarchParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int strip = blockIdx.x % p.ns, seg = blockIdx.x / p.ns;
    const int ca = strip * p.w, ra = 1 + seg * p.rows;
    if (threadIdx.x == 0) {
        uint64_t* bar = reinterpret_cast<uint64_t*>(smem + Ring<T, NSS>::BAR);
        for (int q = 0; q < NSS; ++q) mbar_init(bar + q, 1);
        fence_mbar_init();
    }
    __syncwarp();
    const bool edge = ca == 0 || ca + p.w + T >= p.Nx - 1 || ra - T <= 1 || ra + p.rows + T >= p.Ny - 1;
    march_segment<T, NSS>(maps, p, smem, strip, seg, edge);
}

template <int T, int NSS, int WPS>
int launch(sf_ctx* ctx, const MarchMaps& maps, const MarchParams& p, cudaStream_t s) {
    using R = Ring<T, NSS>;
    static PerDevice ready;
    const int rc = allow_smem(ready, ctx->device, (const void*)k_pt_march<T, NSS, WPS>, R::BYTES);
    if (rc) return rc;
    k_pt_march<T, NSS, WPS><<<(unsigned)(p.ns * p.nseg), 32, R::BYTES, s>>>(maps, p);
    SF_LAUNCHED(ctx);
    return SF_OK;
}

constexpr int WARPS_PER_SM = 8;

}  // namespace

// The rows above and below that a warp computes for a third iteration outweigh what it saves where segments are short but
// the launch is not all latency.  Microseconds per iteration with T = 2 : T = 3: 100^2 3.80 : 3.67, 150^2 3.77 : 3.64, 200^2
// 4.28 : 3.63, 225^2 4.28 : 3.65, 600 x 100 4.31 : 3.62; 250^2 4.26 : 4.33, 300^2 4.26 : 4.61, 350^2 5.29 : 5.63, 375^2 5.32 :
// 5.67, 900 x 150 5.33 : 5.67; 400^2 5.72 : 5.64, 425^2 5.81 : 5.64, 450^2 5.31 : 5.64, 475^2 5.77 : 5.64, 500^2 5.89 : 5.68, 600^2
// 6.72 : 6.39, 700^2 7.94 : 7.49, 800^2 9.68 : 9.32, 1024^2 13.95 : 12.21, 2048^2 54.4 : 37.3 (T = 1: 101.5).
// (Below 530^2 solves march only where no resident tiles are to be had.)
int march_iterations(int64_t Nx, int64_t Ny) {
    const int64_t points = Nx * Ny;
    return points >= 240 * 240 && points < 400 * 400 ? 2 : 3;
}

void march_plan(MarchParams& p, int T, int num_sms) {
    const int te = left_halo(T);
    const int cols = p.Nx - 1, rows = p.Ny - 1;
    if (te + cols <= CW - 2) {
        p.ns = 1;                      // the whole width with its ghost columns fits a strip
        p.w = (cols + 1) & ~1;
    } else {
        const int most = (CW - 1 - T - te) & ~1;
        p.ns = (cols + most - 1) / most;
        p.w = (cols + p.ns - 1) / p.ns;
        p.w += p.w & 1;
        p.ns = (cols + p.w - 1) / p.w;
    }
    const int slots = std::max(1, num_sms * WARPS_PER_SM / p.ns);
    p.rows = std::max((rows + slots - 1) / slots, 2);
    p.nseg = (rows + p.rows - 1) / p.rows;
}

int march_launch(sf_ctx* ctx, const MarchMaps& maps, const MarchParams& p, int T, cudaStream_t s) {
    switch (T) {
        case 1: return launch<1, 3, WARPS_PER_SM>(ctx, maps, p, s);
        case 2: return launch<2, 3, WARPS_PER_SM>(ctx, maps, p, s);
        default: return launch<3, 3, WARPS_PER_SM>(ctx, maps, p, s);
    }
}

}  // namespace sf
