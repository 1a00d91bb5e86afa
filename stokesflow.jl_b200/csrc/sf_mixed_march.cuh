// sf_mixed_march.cuh -- T FP32 sweeps of the mixed solve in one pass over memory (included by sf_mixed.cu, which defines
// the instance record Inst, its fields and its control word Ctl).
//
// The same march as the FP64 one (sf_march.cu): a warp owns a strip of columns, two per lane, and a segment of rows of
// one instance, keeps each sweep level's previous rows in registers and takes x neighbours by shuffle; rows arrive two
// at a time through a ring of bulk-tensor copies.  The expressions, their fused multiply-adds and divisions are k_pt32's,
// so a point gets the same bits here and there, however many sweeps a launch does.
//
// A warp recomputes rows and columns of its neighbours, whose rates must be the old ones: the rates need a second pair
// of buffers (Inst::rates_b), which the batched solve's arena has and an engine's arena, whose size is the caller's,
// has not.
//
// What bounds it: issue slots (57% active at 1024^2) and, on small sets, the halo rows of short segments and a launch's
// start.  One 1024^2 instance 17.5 -> 8.5 us per sweep (T = 3; one launch 25 us), 2048^2 59 -> 25.5, 16 instances of
// 128 .. 512 points per side 27.2 -> 15.6, 100^2 4.5 -> 2.8.  Some 500 warp instructions per row step of 64 columns and
// three sweeps, the same for every item (a leaner body for items inside the domain: 9.4 us at 1024^2).  With that leaner
// body: two warps per scheduler (8 per SM) 9.4 us, ten leave the schedulers uneven (11.4), twelve shorten the segments
// (11.0); four columns per lane need fewer instructions, but their code misses the instruction cache (2.6 of 5
// stall cycles; 11.3 - 14.6 us); T = 2 with 12 warps 11.8.  One sweep per launch is no faster than k_pt32.
#pragma once

namespace sf {
namespace mx {

constexpr int NC = 2;                    // columns of a lane
constexpr int ML = 4;                    // columns left of a strip's own: copies start on 16 bytes
constexpr int MPAIRS = 2;                // row pairs in flight

// a pair of rows of a strip in shared memory: [field][row][column].  State: Vx, Vy of rows r, r + 1, P of the row
// before each, the rates of the row before that; parameters: rho of rows r, r + 1; mu_b, mu_p and the divV residual of
// the row before each; the momentum residuals of the row before that
struct MRing {
    static constexpr int MC = 32 * NC;   // columns of a strip with its halo
    static constexpr int ROW = MC * 4, FIELD = 2 * ROW;
    static constexpr int X = 0, Y = FIELD, P = 2 * FIELD, VX = 3 * FIELD, VY = 4 * FIELD, STATE = 5 * FIELD;
    static constexpr int RHO = 0, MUB = FIELD, MUP = 2 * FIELD, RDIV = 3 * FIELD, RX = 4 * FIELD, RY = 5 * FIELD,
                         MAT = 6 * FIELD;
    static constexpr int MPS = MPAIRS + 1;   // a parameter row is read at its step and the T - 1 <= 2 after it
    static constexpr int BAR = MPAIRS * STATE + MPS * MAT;
    static constexpr int BYTES = BAR + 8 * MPAIRS;
    static constexpr uint32_t TX = STATE + MAT;
};

struct MItem { int inst, ca, ra, wr; };  // own columns from ca, own rows from ra; wr = columns | rows << 8

// what a sweep level keeps between two rows; [h]: this lane's columns c + h (velocity column c is Vx(c + 1))
struct MLevel {
    float X[NC], Y[NC], Yr, S[NC], A[NC], sy[NC], Q[NC], P[NC], r1[NC], r2[NC], g[NC], tx[NC], mu[NC];
    float mb[NC];                        // (stencil-maximum pseudo-step only)
};

struct MConst { float _dx, _dy, h_dx, h_dy, c_pt, cdx, cdy, g_dt, c1, c2; };

__device__ __forceinline__ float fr_right(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ float fr_left(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ void ldf2(const unsigned char* p, float* v) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x;
    v[1] = t.y;
}
__device__ __forceinline__ void stf2(float* p, const float* v) {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

// one row of a level, as march_step of sf_march.cu; m: this lane's place in the parameter row's slots
template <bool DMAX>
__device__ __forceinline__ void mstep(MLevel& L, const MConst& k, const unsigned char* __restrict__ m,
                                      const float (&X)[NC], const float (&Y)[NC], float Xl, float Yr,
                                      const float (&P0)[NC], const float (&rx0)[NC], const float (&ry0)[NC],
                                      float (&Xn)[NC], float (&Yn)[NC], float (&rxn)[NC], float (&ryn)[NC]) {
    using R = MRing;
    float rh[NC + 2], mb[NC + 1], mu[NC + 1], rd[NC], cx[NC], cy[NC];
    ldf2(m + R::RHO, rh);
    ldf2(m + R::RHO + 4 * NC, rh + NC);
    ldf2(m + R::MUB, mb);
    mb[NC] = *reinterpret_cast<const float*>(m + R::MUB + 4 * NC);
    ldf2(m + R::MUP, mu);
    mu[NC] = *reinterpret_cast<const float*>(m + R::MUP + 4 * NC);
    ldf2(m + R::RDIV, rd);
    ldf2(m + R::RX, cx);
    ldf2(m + R::RY, cy);
    float sxx[NC], syy[NC], pn[NC], Q[NC];
#pragma unroll
    for (int h = 0; h < NC; ++h) {
        const float xl = h ? X[h - 1] : Xl, ypr = h + 1 < NC ? L.Y[(h + 1) % NC] : L.Yr;
        const float ex = (X[h] - xl) * k._dx;
        const float ey = (Y[h] - L.Y[h]) * k._dy;
        const float d = ex + ey;
        const float full = d + rd[h];                        // divV of V_k + dV
        pn[h] = fmaf(-(k.c_pt * mu[h]), full, P0[h]);
        const float mu2 = 2.0f * mu[h];
        sxx[h] = fmaf(mu2, fmaf(-(1.0f / 3.0f), d, ex), -pn[h]);
        syy[h] = fmaf(mu2, fmaf(-(1.0f / 3.0f), d, ey), -pn[h]);
        const float a = (X[h] - L.X[h]) * k._dy;
        const float b = (ypr - L.Y[h]) * k._dx;
        Q[h] = mb[h + 1] * (a + b);
    }
    const float sr = fr_right(sxx[0]), ql = fr_left(Q[NC - 1]);
#pragma unroll
    for (int h = 0; h < NC; ++h) {
        const float xl = h ? X[h - 1] : Xl, qn = h ? Q[h - 1] : ql;
        const float Rx = fmaf(L.A[h], k._dx, fmaf(Q[h] - L.Q[h], k._dy, cx[h]));
        const float dv = fmaf(-k.cdx, rx0[h], rx0[h]) + Rx;
        rxn[h] = dv;
        const float tx = DMAX ? __fdividef(k.c1, fmaxf(L.tx[h], fmaxf(L.mb[h], mb[h + 1]))) : L.tx[h];
        Xn[h] = fmaf(tx, dv, L.X[h]);
        const float av = 0.25f * (L.S[h] + xl + X[h]);
        const float dyr = rh[h + 1] - L.r2[h];
        const float stab = fmaf(av * L.g[h], k.h_dx, (L.Y[h] * dyr) * k.h_dy);
        const float Ry = fmaf(syy[h] - L.sy[h], k._dy, fmaf(Q[h] - qn, k._dx, fmaf(-k.g_dt, stab, cy[h])));
        const float dw = fmaf(-k.cdy, ry0[h], ry0[h]) + Ry;
        ryn[h] = dw;
        const float ty = DMAX ? __fdividef(k.c1, fmaxf(fmaxf(L.mu[h], mu[h]), fmaxf(mb[h], mb[h + 1])))
                              : __fdividef(k.c2, L.mu[h] + mu[h]);
        Yn[h] = fmaf(ty, dw, L.Y[h]);
    }
#pragma unroll
    for (int h = 0; h < NC; ++h) {
        L.S[h] = (h ? X[h - 1] : Xl) + X[h];
        L.A[h] = (h + 1 < NC ? sxx[(h + 1) % NC] : sr) - sxx[h];
        L.X[h] = X[h];
        L.Y[h] = Y[h];
        L.sy[h] = syy[h];
        L.Q[h] = Q[h];
        L.P[h] = pn[h];
        L.r2[h] = L.r1[h];
        L.r1[h] = rh[h + 1];
        L.g[h] = rh[h + 2] - rh[h];
        // the pseudo-step of Vx between this row's pressure points, or (DMAX) the larger viscosity of the two
        L.tx[h] = DMAX ? fmaxf(mu[h], mu[h + 1]) : __fdividef(k.c2, mu[h] + mu[h + 1]);
        L.mu[h] = mu[h];
        if (DMAX) L.mb[h] = mb[h + 1];
    }
    L.Yr = Yr;
}

// position in the rings; carried from item to item (in_: lane 0's, of the next copies)
struct MPos { int b, m, in_b, in_m; uint32_t phase; };

// One item: T levels.  edge: its columns or rows (halo included) see a side of the domain; DMAX: the stencil-maximum
// pseudo-step.  false: a copy never came.
template <int T, bool DMAX>
__device__ __forceinline__ bool mitem(const CUtensorMap* __restrict__ maps, const Inst& I, const MItem& w, bool edge,
                                      int in, int rin, unsigned char* smem, MPos& pos) {
    using R = MRing;
    unsigned char* const mats = smem + MPAIRS * R::STATE;
    uint64_t* const bar = reinterpret_cast<uint64_t*>(smem + R::BAR);
    const int lane = threadIdx.x;
    const int Nx = I.Nx, Ny = I.Ny;
    const int ca = w.ca, cb = min(ca + (w.wr & 255), Nx - 1);
    const int ra = w.ra, rb = min(ra + (w.wr >> 8), Ny);
    const int c0 = ca - ML, r0 = max(ra - T, 0);
    const int pairs = (rb + T - r0 + 1) >> 1;
    const int64_t LD = I.LD32;

    int in_p = 0;
    const int zv = in ? G_VXB : G_VXA, zr = rin ? G_RVXB : G_RVX;
    auto issue = [&]() {   // lane 0; rows outside the fields come as zeros, and what they lead to is dropped
        uint64_t* b = bar + pos.in_b;
        const int r = r0 + 2 * in_p;
        unsigned char* st = smem + pos.in_b * R::STATE;
        unsigned char* mt = mats + pos.in_m * R::MAT;
        mbar_arrive_expect_tx(b, R::TX);
        tma_load_3d(st + R::X, maps + M_ROW2, b, c0, r, zv);
        tma_load_3d(st + R::P, maps + M_ROW1, b, c0, r - 1, zv + 2);
        tma_load_3d(st + R::VX, maps + M_ROW2, b, c0, r - 2, zr);
        tma_load_3d(mt + R::RHO, maps + M_ROW1, b, c0, r, G_RHO);
        tma_load_3d(mt + R::MUB, maps + M_ROW3, b, c0, r - 1, G_MUB);
        tma_load_3d(mt + R::RX, maps + M_ROW2, b, c0, r - 2, G_RX);
        ++in_p;
        pos.in_b ^= 1;
        pos.in_m = (pos.in_m + 1 == R::MPS) ? 0 : pos.in_m + 1;
    };
    static_assert(MPAIRS == 2, "two barriers in turn");
    if (lane == 0)
        for (int n = 0; n < MPAIRS && n < pairs; ++n) issue();

    MConst k;
    k._dx = I._dxf;
    k._dy = I._dyf;
    k.h_dx = 0.5f * I._dxf;
    k.h_dy = 0.5f * I._dyf;
    k.c_pt = I.c_ptscf;
    k.cdx = I.cdampXf;
    k.cdy = I.cdampYf;
    k.g_dt = I.g_dtf;
    k.c1 = I.c_vscf;
    k.c2 = 2.0f * I.c_vscf;

    float* const Vx_out = gf(I, in ? G_VXA : G_VXB);
    float* const Vy_out = gf(I, in ? G_VYA : G_VYB);
    float* const P_out = gf(I, in ? G_PA : G_PB);
    float* const Rvx = gf(I, rin ? G_RVX : G_RVXB);
    float* const Rvy = gf(I, rin ? G_RVY : G_RVYB);

    MLevel L[T];
    float prx[T][NC], pry[T][NC];
#pragma unroll
    for (int l = 0; l < T; ++l) {
        L[l] = MLevel{};
#pragma unroll
        for (int h = 0; h < NC; ++h) prx[l][h] = pry[l][h] = 0.f;
    }
    const int c = c0 + NC * lane;                    // a multiple of NC
    const bool own = c >= ca && c < cb;
    int64_t out = (int64_t)(r0 - T) * LD + c;
    const unsigned char* mt_prev = mats + 4 * NC * lane;   // the parameter rows of the pair before

    for (int p = 0; p < pairs; ++p) {
        if (!__all_sync(0xffffffffu, mbar_wait(bar + pos.b, pos.phase, WAIT_BUDGET_NS))) return false;
        const unsigned char* const st = smem + pos.b * R::STATE + 4 * NC * lane;
        const unsigned char* const mt = mats + pos.m * R::MAT + 4 * NC * lane;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float X[NC], Y[NC], P0[NC], rx0[NC], ry0[NC], Xl, Yr;
            {
                float t[NC + 2];
                ldf2(st + R::X + j * R::ROW, t);
                t[NC] = *reinterpret_cast<const float*>(st + R::X + j * R::ROW + 4 * NC);
                Xl = t[0];
#pragma unroll
                for (int h = 0; h < NC; ++h) X[h] = t[h + 1];
                ldf2(st + R::Y + j * R::ROW, t);
                ldf2(st + R::Y + j * R::ROW + 4 * NC, t + NC);
#pragma unroll
                for (int h = 0; h < NC; ++h) Y[h] = t[h + 1];
                Yr = t[NC + 1];
                ldf2(st + R::P + j * R::ROW, P0);
                ldf2(st + R::VX + j * R::ROW, rx0);
                ldf2(st + R::VY + j * R::ROW, ry0);
            }
#pragma unroll
            for (int l = 0; l < T; ++l) {
                const int r = r0 + 2 * p + j - l;
                // row l before row j of this pair: in this pair or the one before
                const unsigned char* m = (l <= j ? mt : mt_prev) + (((j - l) & 1) ? R::ROW : 0);
                float Pold[NC], Xn[NC], Yn[NC], rxn[NC], ryn[NC];
#pragma unroll
                for (int h = 0; h < NC; ++h) Pold[h] = L[l].P[h];
                mstep<DMAX>(L[l], k, m, X, Y, Xl, Yr, P0, rx0, ry0, Xn, Yn, rxn, ryn);
                {   // (as in sf_march.cu: every item, so that all take the same time)
                    const float y_right = fr_right(Yn[0]), y_left = fr_left(Yn[NC - 1]);
                    if (c + NC - 1 == -1) Yn[NC - 1] = y_right;
#pragma unroll
                    for (int h = NC - 1; h >= 0; --h) {
                        if (c + h == Nx - 1) Yn[h] = h ? Yn[(h + NC - 1) % NC] : y_left;
                        if (c + h == -1 || c + h == Nx - 2) Xn[h] = 0.f;
                    }
                }
                if (l + 1 < T) {
#pragma unroll
                    for (int h = 0; h < NC; ++h) {
                        X[h] = Xn[h];
                        Y[h] = Yn[h];
                        P0[h] = Pold[h];
                        rx0[h] = prx[l][h];
                        ry0[h] = pry[l][h];
                        prx[l][h] = rxn[h];
                        pry[l][h] = ryn[h];
                    }
                    {
                        MLevel& N = L[(l + 1 < T) ? l + 1 : l];
                        const int rn = r - 1;
                        if (rn == 1) {
#pragma unroll
                            for (int h = 0; h < NC; ++h) {
                                N.X[h] = X[h];
                                N.Y[h] = 0.f;
                            }
                            N.Yr = 0.f;
                        }
                        if (rn == Ny - 1) {
#pragma unroll
                            for (int h = 0; h < NC; ++h) Y[h] = 0.f;
                        }
                        if (rn == Ny) {
#pragma unroll
                            for (int h = 0; h < NC; ++h) X[h] = N.X[h];
                        }
                    }
                    Xl = fr_left(X[NC - 1]);
                    Yr = fr_right(Y[0]);
                } else if (!edge) {
                    float xs[NC], ys[NC];    // {Vx(c), ..}: the column to the left, then this lane's but its last
                    xs[0] = fr_left(Xn[NC - 1]);
                    ys[0] = fr_left(Yn[NC - 1]);
#pragma unroll
                    for (int h = 1; h < NC; ++h) {
                        xs[h] = Xn[h - 1];
                        ys[h] = Yn[h - 1];
                    }
                    if (own && r > ra && r <= rb) {
                        const int64_t q = out - LD;
                        stf2(Vx_out + out, xs);
                        stf2(Vy_out + out, ys);
                        stf2(P_out + q, Pold);
                        stf2(Rvx + q, rxn);
                        stf2(Rvy + q, ryn);
                    }
                } else if (r > ra && r <= rb) {
                    const int ro = r - 1;
                    const bool last = cb == Nx - 1;
                    const int64_t q = out - LD;
#pragma unroll
                    for (int h = 0; h < NC; ++h) {
                        const int col = c + h;
                        if (col >= ca && col < cb) {
                            P_out[q + h] = Pold[h];
                            if (col < Nx - 2) Rvx[q + h] = rxn[h];
                            if (ro < Ny - 1) Rvy[q + h] = ryn[h];
                        }
                        const bool vx_own = col >= ca - 1 && col <= (last ? Nx - 2 : cb - 2);
                        const bool vy_own = col >= ca - 1 && col <= (last ? Nx - 1 : cb - 2);
                        if (vx_own) Vx_out[out + h + 1] = Xn[h];
                        if (vy_own) Vy_out[out + h + 1] = (ro == Ny - 1) ? 0.f : Yn[h];
                        if (ro == 1) {
                            if (vx_own) Vx_out[q + h + 1] = Xn[h];
                            if (vy_own) Vy_out[q + h + 1] = 0.f;
                        }
                        if (ro == Ny - 1 && vx_own) Vx_out[out + LD + h + 1] = Xn[h];
                    }
                }
            }
            out += LD;
        }
        __syncwarp();   // every lane has read the slots that the next rows go to
        if (lane == 0 && in_p < pairs) issue();
        mt_prev = mt;
        pos.m = (pos.m + 1 == R::MPS) ? 0 : pos.m + 1;
        pos.phase ^= pos.b;
        pos.b ^= 1;
    }
    return true;
}

// Sweeps of launch `l` of a round for an instance whose budget is B: T a launch, and where a residual check follows the
// last one alone (the check reads the velocities before the last sweep from the other buffer).
__host__ __device__ __forceinline__ int march_sweeps(int l, int T, int B, bool check) {
    const int main = check ? B - 1 : B, launches = (main + T - 1) / T;
    if (l < launches) return main - l * T < T ? main - l * T : T;
    return check && l == launches ? 1 : 0;
}
__host__ __device__ __forceinline__ int march_launches(int T, int B, bool check) {
    return check ? (B - 1 + T - 1) / T + 1 : (B + T - 1) / T;
}

template <int T, int WPS>
__global__ void __launch_bounds__(32, WPS) k_march32(const CUtensorMap* __restrict__ maps, const Inst* __restrict__ insts,
                                                     const Ctl* __restrict__ ctl, const MItem* __restrict__ items,
                                                     const int* __restrict__ nitems_ptr, int launch_idx,
                                                     int* __restrict__ err_flag) {
    static_assert(T == 3, "what is left over: one or two sweeps");
    extern __shared__ __align__(128) unsigned char smem[];
    using R = MRing;
    uint64_t* const bar = reinterpret_cast<uint64_t*>(smem + R::BAR);
    MItem w = items[blockIdx.x];         // (the list has room for as many entries as the launch has blocks)
    const int nitems = *nitems_ptr;
    if (threadIdx.x == 0) {
        for (int q = 0; q < MPAIRS; ++q) mbar_init(bar + q, 1);
        fence_mbar_init();
    }
    __syncwarp();
    MPos pos = {0, 0, 0, 0, 0};
    int fenced = -1;
    bool first = true;
    for (int t = blockIdx.x; t < nitems; t += gridDim.x) {
        if (t != blockIdx.x) w = items[t];
        const Ctl cw = ctl[w.inst];
        const Inst& I = insts[w.inst];
        const int n = march_sweeps(launch_idx, T, cw.budget, (cw.flags & CTL_CHECK) != 0);
        if (n == 0) continue;
        const CUtensorMap* m = maps + (int64_t)w.inst * M_NUM_MARCH;
        if (fenced != w.inst) {
            if (threadIdx.x == 0)
                for (int q = M_ROW1; q <= M_ROW3; ++q) fence_tensormap_acquire(m + q);
            fenced = w.inst;
        }
        if (first) {   // the previous launch's fields are complete and visible from here on
            griddep_wait();
            griddep_launch_dependents();
            first = false;
        }
        const int in = (cw.parity ^ launch_idx) & 1, rin = (cw.rparity ^ launch_idx) & 1;
        const int cols = w.wr & 255, rows = w.wr >> 8;
        const bool edge = w.ca == 0 || w.ca + cols + T >= I.Nx - 1 || w.ra - T <= 1 || w.ra + rows + T >= I.Ny - 1;
        bool ok;
        if (I.dtau_max)
            ok = n == T ? mitem<T, true>(m, I, w, edge, in, rin, smem, pos)
                 : n == 2 ? mitem<2, true>(m, I, w, edge, in, rin, smem, pos)
                          : mitem<1, true>(m, I, w, edge, in, rin, smem, pos);
        else
            ok = n == T ? mitem<T, false>(m, I, w, edge, in, rin, smem, pos)
                 : n == 2 ? mitem<2, false>(m, I, w, edge, in, rin, smem, pos)
                          : mitem<1, false>(m, I, w, edge, in, rin, smem, pos);
        if (!ok) {
            // flag it, give the copies in flight a bounded chance to land, leave
            if (threadIdx.x == 0) atomicExch(err_flag, 1);
            pos.phase ^= pos.b;
            mbar_wait(bar + (pos.b ^ 1), pos.phase, WAIT_BUDGET_NS);
            return;
        }
    }
    if (first) griddep_wait();
}

}  // namespace mx
}  // namespace sf
