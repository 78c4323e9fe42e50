// Fixed-step N-band solves, many steps per launch (sm_100a).
//
// With a fixed step (RK4 / Fehlberg-5, SBEs.h:395-416, 596-624) the k-points
// of a solve are independent until the k-sum of the outputs, so a launch
// advances every k-point by up to S steps with its state on chip and writes
// one partial row of the outputs per warp and step; `wan_finish` sums the
// rows of each step and moves the solve's controller on.  One attempt launch
// and one control launch per step (wan_vg_attempt / wan_control) cost 30 + 12
// us on 14 520 k-points of the four-band KaneMele model, of which the
// arithmetic is under 2.
//
// wan_vg_steps: velocity gauge (SBEs.h:284-373, 787-805, 862-871) at N <= 3,
// one thread per k-point.  rho (the upper triangle) and H = diag(eps) + A.P
// live in registers, P in shared memory (one column per thread, so a warp's
// 16-byte loads are contiguous).
// wan_vg_rows: the same at N = 4 ... 8, one row of the matrices per lane.
// Both are FP64 in both methods, as wan_vg_attempt, which runs the adaptive
// Cash-Karp steps.
// wan_lw_steps: the length gauge of the analytic materials at N = 2, 3, 4.
//
// Measured (RK4, 367 steps, whole solve with its set-up): three bands 1.8 us a
// step at 14 520 k-points and 5.5 at 90 300 (rows: 3.7, 14.9); four bands rows
// 5.2 and 21 (one thread per k-point spills: 5.5, 21; with RK5 8.1 and 34
// against 9.7 and 39).
#include <cuda_runtime.h>

#include "sbe_wandev.cuh"
#include "sbe_wannier.h"

namespace sbe {

namespace {

constexpr int WS_T = 64;   // threads (k-points) per block

// Compile-time tableaux (SBEs.h:395-416).  ti(i): field-table column of
// stage i (NT distinct stage times); c: the fractions of those columns.
template <int RK> struct StepTab;
template <> struct StepTab<4> {
    static constexpr int S = 4, NT = 3;
    __host__ __device__ static constexpr double c(int t) { return t == 0 ? 0.0 : t == 1 ? 0.5 : 1.0; }
    __device__ static constexpr double a(int i, int j)
    {
        return (i == 1 && j == 0) ? 0.5 : (i == 2 && j == 1) ? 0.5 : (i == 3 && j == 2) ? 1.0 : 0.0;
    }
    __device__ static constexpr double b(int i) { return (i == 0 || i == 3) ? 1.0 / 6.0 : 2.0 / 6.0; }
    __device__ static constexpr int ti(int i) { return i == 0 ? 0 : (i == 3 ? 2 : 1); }
};
template <> struct StepTab<5> {
    static constexpr int S = 6, NT = 6;
    __host__ __device__ static constexpr double c(int t)
    {
        return t == 0 ? 0.0 : t == 1 ? 0.25 : t == 2 ? 3. / 8. : t == 3 ? 12. / 13. : t == 4 ? 1.0 : 0.5;
    }
    __device__ static constexpr double a(int i, int j)
    {
        return i == 1 ? (j == 0 ? 1.0 / 4.0 : 0.0)
             : i == 2 ? (j == 0 ? 3. / 32. : j == 1 ? 9. / 32. : 0.0)
             : i == 3 ? (j == 0 ? 1932. / 2197. : j == 1 ? -7200. / 2197. : j == 2 ? 7296. / 2197. : 0.0)
             : i == 4 ? (j == 0 ? 439. / 216. : j == 1 ? -8. : j == 2 ? 3680. / 513. : j == 3 ? -845. / 4104. : 0.0)
             : i == 5 ? (j == 0 ? -8. / 27. : j == 1 ? 2. : j == 2 ? -3544. / 2565 : j == 3 ? 1859. / 4104
                        : j == 4 ? -11. / 40. : 0.0)
             : 0.0;
    }
    __device__ static constexpr double b(int i)
    {
        return i == 0 ? 16. / 135. : i == 1 ? 0.0 : i == 2 ? 6656. / 12825. : i == 3 ? 28561. / 56430.
             : i == 4 ? -9. / 50. : 2. / 55.;
    }
    __device__ static constexpr int ti(int i) { return i; }
};

// Steps a launch of at most S takes from output step n: up to the end, and not
// past a step whose density snapshot is due (it is taken between launches).
__device__ __forceinline__ int launch_steps(const WanDev &P, int n, int S)
{
    int m = min(min(S, P.step_max), P.Nt - n);
    if (P.shot_every > 0) m = min(m, ((n + P.shot_every - 1) / P.shot_every) * P.shot_every + 1 - n);
    return m;
}

// Start of output step n and its length as the step controller forms them:
// steps end exactly on t_{n+1}.
__device__ __forceinline__ double step_start(const WanDev &P, int n)
{
    return n == 0 ? P.atmin : P.atmin + P.dt * n;
}
__device__ __forceinline__ double step_length(const WanDev &P, int n)
{
    return (P.atmin + P.dt * (n + 1)) - step_start(P, n);
}

// Sum of 16 values over a warp by halving exchanges: lanes 2i return value i
// (fixed pattern; 16 shuffles instead of 80).
__device__ __forceinline__ double warp_sum16(const double (&v)[16], int lane)
{
    double u[8], x[4], y[2];
    const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4, h1 = lane & 2;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        u[i] = (h4 ? v[i + 8] : v[i]) + __shfl_xor_sync(0xffffffffu, h4 ? v[i] : v[i + 8], 16);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        x[i] = (h3 ? u[i + 4] : u[i]) + __shfl_xor_sync(0xffffffffu, h3 ? u[i] : u[i + 4], 8);
#pragma unroll
    for (int i = 0; i < 2; ++i)
        y[i] = (h2 ? x[i + 2] : x[i]) + __shfl_xor_sync(0xffffffffu, h2 ? x[i] : x[i + 2], 4);
    double z = (h1 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, h1 ? y[0] : y[1], 2);
    return z + __shfl_xor_sync(0xffffffffu, z, 1);
}

// upper-triangle index of (m, n), m < n, among the off-diagonal elements
__host__ __device__ constexpr int oidx(int m, int n, int N) { return m * N - m * (m + 1) / 2 + (n - m - 1); }

}  // namespace

// A at the distinct stage times of every step: step_fld[n][NT][3]
__global__ void __launch_bounds__(128) wan_step_fields(const WanDev *__restrict__ Pp, int nt, int rk)
{
    const WanDev &P = *Pp;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.Nt * nt) return;
    const int n = i / nt, j = i % nt;
    const double tc = step_start(P, n), hs = step_length(P, n);
    const double c = rk == 4 ? StepTab<4>::c(j) : StepTab<5>::c(j);
    double A[3], E[3];
    laser_eval(P.laser, j == 0 ? tc : tc + c * hs, A, E);
    for (int d = 0; d < 3; ++d) P.step_fld[(size_t)i * 3 + d] = A[d];
}

// FP64-pipe bound where the grid fills the GPU, latency-bound (one warp per
// scheduler) below: at N = 3 an RK4 step is ~0.7e3 FP64 instructions per
// thread against 3 passes over P in shared memory (54 16-byte loads).
template <int N, int RK, int NA>
__global__ void __launch_bounds__(WS_T) wan_vg_steps(const WanDev *__restrict__ Pp,
                                                     const WanDev *const *__restrict__ descs,
                                                     const WanTileRef *__restrict__ tiles, int S)
{
    using TB = StepTab<RK>;
    constexpr int NN = N * N, NO = N * (N - 1) / 2;
    extern __shared__ __align__(16) double2 sP[];   // [NA][NN][WS_T] P, then [N][WS_T] (eps, f)
    const WanDev &P = tiles ? *descs[tiles[blockIdx.x].solve] : *Pp;
    const int tile0 = tiles ? tiles[blockIdx.x].tile : (int)blockIdx.x * (WS_T / WAN_WARPS);
    if (P.ctl->done) return;
    const int n0 = P.ctl->n, steps = launch_steps(P, n0, S);
    const int t = threadIdx.x, lane = t & 31;
    const int k = tile0 * WAN_WARPS + t;
    const bool live = k < P.nk;
    const int kc = live ? k : P.nk - 1;   // a thread past the grid shadows the last k-point
    double2 *const sE = sP + NA * NN * WS_T;
    for (int e = 0; e < NA * NN; ++e) sP[e * WS_T + t] = P.vg_P[(size_t)kc * (NA * NN) + e];
#pragma unroll
    for (int m = 0; m < N; ++m)
        sE[m * WS_T + t] = make_double2(P.vg_eps[(size_t)kc * N + m], P.vg_f[(size_t)kc * N + m]);
    const double wk = live ? P.weight[kc] : 0.0;
    const double g1 = P.g1, g2 = P.g2;
    double2 *rho = P.rho[0] + (size_t)kc * NN;
    double yd[N];
    double2 yo[NO];
#pragma unroll
    for (int m = 0; m < N; ++m) {
        yd[m] = rho[m * N + m].x;
#pragma unroll
        for (int n = m + 1; n < N; ++n) yo[oidx(m, n, N)] = rho[m * N + n];
    }
    const int ce = (P.nval * N + P.nval + 1) % NN;   // antelope.cpp:539-542
    const int nw = (P.nk + 31) / 32;
    double *part = P.step_part + (size_t)((tile0 * WAN_WARPS + t) >> 5) * WAN_NSLOT + (lane >> 1);
    const bool put = (lane & 1) == 0 && tile0 * WAN_WARPS + (t & ~31) < P.nk;

    for (int j = 0; j < steps; ++j) {
        const double *fl = P.step_fld + (size_t)(n0 + j) * TB::NT * 3;
        const double h = step_length(P, n0 + j);
        double2 H[NN];
        // one pass over P: H at the start of the step, and the currents there
        // (SBEs.h:694-760): Re sum_ij rho_ij P_a,ji, the diagonal -> intraband
        {
            double A[NA], v[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = 0.0;
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                A[a] = fl[a];
                double ie = 0.0, ia = 0.0;
#pragma unroll
                for (int e = 0; e < NN; ++e) {
                    const int m = e / N, n = e % N;
                    const double2 p = sP[(a * NN + e) * WS_T + t];
                    if (a == 0) H[e] = make_double2(m == n ? fma(A[a], p.x, sE[m * WS_T + t].x) : A[a] * p.x, A[a] * p.y);
                    else H[e] = make_double2(fma(A[a], p.x, H[e].x), fma(A[a], p.y, H[e].y));
                    // rho_nm P_mn
                    if (m == n) ia = fma(yd[m], p.x, ia);
                    else if (m < n) ie = fma(yo[oidx(m, n, N)].x, p.x, fma(yo[oidx(m, n, N)].y, p.y, ie));
                    else ie = fma(yo[oidx(n, m, N)].x, p.x, fma(-yo[oidx(n, m, N)].y, p.y, ie));
                }
                v[a < 2 ? a : WAN_SLOT_INTER_Z] = wk * ie;
                v[a < 2 ? 2 + a : WAN_SLOT_INTRA_Z] = wk * ia;
            }
#pragma unroll
            for (int m = 0; m < N; ++m) v[4 + m] = wk * yd[m];
#pragma unroll
            for (int e = 0; e < NN; ++e)
                if (e == ce) {
                    const int m = e / N, n = e % N;
                    v[4 + N] = wk * (m == n ? yd[m] : m < n ? yo[oidx(m, n, N)].x : yo[oidx(n, m, N)].x);
                    v[5 + N] = m == n ? 0.0 : wk * (m < n ? yo[oidx(m, n, N)].y : -yo[oidx(n, m, N)].y);
                }
            const double s = warp_sum16(v, lane);
            if (put) part[(size_t)j * nw * WAN_NSLOT] = s;
        }
        // the step
        double kd[TB::S][N], id[N];
        double2 ko[TB::S][NO], io[NO];
#pragma unroll
        for (int m = 0; m < N; ++m) id[m] = 0.0;
#pragma unroll
        for (int o = 0; o < NO; ++o) io[o] = make_double2(0.0, 0.0);
#pragma unroll
        for (int s = 0; s < TB::S; ++s) {
            double xd[N];
            double2 xo[NO];
#pragma unroll
            for (int m = 0; m < N; ++m) xd[m] = yd[m];
#pragma unroll
            for (int o = 0; o < NO; ++o) xo[o] = yo[o];
#pragma unroll
            for (int q = 0; q < s; ++q)
                if (TB::a(s, q) != 0.0) {
                    const double a = h * TB::a(s, q);
#pragma unroll
                    for (int m = 0; m < N; ++m) xd[m] = fma(a, kd[q][m], xd[m]);
#pragma unroll
                    for (int o = 0; o < NO; ++o)
                        xo[o] = make_double2(fma(a, ko[q][o].x, xo[o].x), fma(a, ko[q][o].y, xo[o].y));
                }
            if (s > 0 && TB::ti(s) != TB::ti(s - 1)) {
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                    const double Aa = fl[TB::ti(s) * 3 + a];
#pragma unroll
                    for (int e = 0; e < NN; ++e) {
                        const double2 p = sP[(a * NN + e) * WS_T + t];
                        if (a == 0)
                            H[e] = make_double2(e / N == e % N ? fma(Aa, p.x, sE[(e / N) * WS_T + t].x) : Aa * p.x, Aa * p.y);
                        else H[e] = make_double2(fma(Aa, p.x, H[e].x), fma(Aa, p.y, H[e].y));
                    }
                }
            }
            // -i((HY) - (HY)^dag) - Gamma o (Y - rho0)   (SBEs.h:808-819, 862-871)
#pragma unroll
            for (int m = 0; m < N; ++m) {
                double im = H[m * N + m].y * xd[m];   // Im (HY)_mm
#pragma unroll
                for (int l = 0; l < N; ++l) {
                    if (l == m) continue;
                    const double2 y = l < m ? xo[oidx(l, m, N)] : cconj(xo[oidx(m, l, N)]);
                    im = fma(H[m * N + l].x, y.y, fma(H[m * N + l].y, y.x, im));
                }
                kd[s][m] = 2.0 * im - g1 * (xd[m] - sE[m * WS_T + t].y);
#pragma unroll
                for (int n = m + 1; n < N; ++n) {
                    // c = (HY)_mn - conj (HY)_nm
                    const double2 w = xo[oidx(m, n, N)];
                    double2 c = make_double2(H[m * N + n].x * xd[n] - H[n * N + m].x * xd[m],
                                             H[m * N + n].y * xd[n] + H[n * N + m].y * xd[m]);
                    cfma(c, H[m * N + m], w);
                    // conj(H_nn conj(w)) = conj(H_nn) w
                    cfma(c, make_double2(-H[n * N + n].x, H[n * N + n].y), w);
#pragma unroll
                    for (int l = 0; l < N; ++l) {
                        if (l == m || l == n) continue;
                        const double2 yn = l < n ? xo[oidx(l, n, N)] : cconj(xo[oidx(n, l, N)]);   // Y_ln
                        const double2 ym = l < m ? xo[oidx(l, m, N)] : cconj(xo[oidx(m, l, N)]);   // Y_lm
                        cfma(c, H[m * N + l], yn);
                        // - conj(H_nl Y_lm)
                        const double2 hn = H[n * N + l];
                        c.x = fma(-hn.x, ym.x, fma(hn.y, ym.y, c.x));
                        c.y = fma(hn.x, ym.y, fma(hn.y, ym.x, c.y));
                    }
                    ko[s][oidx(m, n, N)] = make_double2(fma(-g2, w.x, c.y), fma(-g2, w.y, -c.x));
                }
            }
            if (TB::b(s) != 0.0) {
                const double b = h * TB::b(s);
#pragma unroll
                for (int m = 0; m < N; ++m) id[m] = fma(b, kd[s][m], id[m]);
#pragma unroll
                for (int o = 0; o < NO; ++o) io[o] = make_double2(fma(b, ko[s][o].x, io[o].x), fma(b, ko[s][o].y, io[o].y));
            }
        }
#pragma unroll
        for (int m = 0; m < N; ++m) yd[m] += id[m];
#pragma unroll
        for (int o = 0; o < NO; ++o) yo[o] = make_double2(yo[o].x + io[o].x, yo[o].y + io[o].y);
    }
    if (!live) return;
#pragma unroll
    for (int m = 0; m < N; ++m) {
        rho[m * N + m] = make_double2(yd[m], 0.0);
#pragma unroll
        for (int n = m + 1; n < N; ++n) {
            rho[m * N + n] = yo[oidx(m, n, N)];
            rho[n * N + m] = cconj(yo[oidx(m, n, N)]);
        }
    }
}

// ---------------------------------------------------- one row per lane
// Lanes per k-point and the shared-memory strides (in complex numbers) of a
// k-point's regions: Y, the packed upper triangle, read element by element at
// one address per group (odd stride: the groups of a warp hit distinct
// banks), and T, rows of LDT for the transpose (stride GT: the 8 lanes of a
// 16-byte phase hit distinct banks on row writes and on column reads).
template <int N> struct RowDim {
    static constexpr int G = N <= 4 ? 4 : 8, KW = 32 / G, NU = N * (N + 1) / 2;
    static constexpr int GY = NU | 1, LDT = N | 1;
    static constexpr int GT = G == 8 ? (N * LDT) | 1 : (N * LDT + 3) / 8 * 8 + 4;
};
constexpr int WR_T = 64;   // threads per block of the row kernel

// Velocity gauge at N = 4 ... 8: lane m of a k-point's group holds row m of
// rho, of P and of H in registers; H Y is formed one row per lane with Y read
// by element, and its conjugate transpose read back from shared memory.  Bound
// by shared memory (58 wavefronts per warp and stage at N = 4) and the FP64
// pipe (112 instructions) about equally, at 12 warps per SM.
template <int N, int RK>
__global__ void __launch_bounds__(WR_T, N <= 4 ? 6 : 4) wan_vg_rows(const WanDev *__restrict__ Pp,
                                                    const WanDev *const *__restrict__ descs,
                                                    const WanTileRef *__restrict__ tiles, int S)
{
    using TB = StepTab<RK>;
    using D = RowDim<N>;
    constexpr int NN = N * N, G = D::G, KW = D::KW;
    __shared__ double2 sY[WR_T / G * D::GY], sT[WR_T / G * D::GT];
    const WanDev &P = tiles ? *descs[tiles[blockIdx.x].solve] : *Pp;
    const int k0 = (tiles ? tiles[blockIdx.x].tile * WAN_WARPS : (int)blockIdx.x * (WR_T / G));
    if (P.ctl->done) return;
    const int n0 = P.ctl->n, steps = launch_steps(P, n0, S);
    const int lane = threadIdx.x & 31, grp = threadIdx.x / G, m = threadIdx.x % G;
    const int warp_k = k0 + (threadIdx.x >> 5) * KW;   // the warp's first k-point
    if (warp_k >= P.nk) return;                        // no block-wide barrier below
    const int k = k0 + grp;
    const bool live = k < P.nk;
    const int kc = live ? k : P.nk - 1;   // a group past the grid shadows the last k-point
    const int mr = m < N ? m : N - 1;     // idle lanes shadow the last row (and store nothing)
    const bool own = m < N;
    double2 *const Y = sY + grp * D::GY, *const T = sT + grp * D::GT;
    double2 p[2][N], y0[N];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int n = 0; n < N; ++n) p[a][n] = P.vg_P[((size_t)kc * 2 + a) * NN + mr * N + n];
    double2 *rho = P.rho[0] + (size_t)kc * NN;
#pragma unroll
    for (int n = 0; n < N; ++n) y0[n] = mr <= n ? rho[mr * N + n] : cconj(rho[n * N + mr]);
    const double eps = P.vg_eps[(size_t)kc * N + mr], f = P.vg_f[(size_t)kc * N + mr];
    const double wk = live && own ? P.weight[kc] : 0.0;
    const double g1 = P.g1, g2 = P.g2;
    const int ce = (P.nval * N + P.nval + 1) % NN, cr = ce / N, cc = ce % N;   // antelope.cpp:539-542
    double *const part = P.step_part + (size_t)(warp_k / KW) * WAN_NSLOT;
    const size_t pstride = (size_t)P.step_rows * WAN_NSLOT;

    for (int j = 0; j < steps; ++j) {
        const double *fl = P.step_fld + (size_t)(n0 + j) * TB::NT * 3;
        const double h = step_length(P, n0 + j);
        {   // currents at the start of the step (SBEs.h:694-760), occupations, coherence
            double v[4] = {0.0, 0.0, 0.0, 0.0}, oc = 0.0, co = 0.0;
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const bool dg = n == m;
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const double q = fma(y0[n].x, p[a][n].x, y0[n].y * p[a][n].y);   // Re rho_nm P_mn
                    v[a] += dg ? 0.0 : q;
                    v[2 + a] += dg ? q : 0.0;
                }
                if (dg) oc = y0[n].x;
                // element ce: its real part from row cr, its imaginary part (of
                // the conjugate) from row cc
                if (m == cr && n == cc) co = y0[n].x;
                else if (m == cc && n == cr) co = -y0[n].y;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] *= wk;
            oc *= wk;
            co *= wk;
            const bool h4 = lane & 16, h3 = lane & 8;
            double u0 = (h4 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h4 ? v[0] : v[2], 16);
            double u1 = (h4 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h4 ? v[1] : v[3], 16);
            double z = (h3 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, h3 ? u0 : u1, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
#pragma unroll
            for (int o = 16; o >= G; o >>= 1) {
                oc += __shfl_xor_sync(0xffffffffu, oc, o);
                co += __shfl_xor_sync(0xffffffffu, co, o);
            }
            double *row = part + (size_t)j * pstride;
            if ((lane & 7) == 0) row[lane >> 3] = z;
            if (lane < N) {
                row[4 + lane] = oc;
                if (lane == cr) row[4 + N] = co;
                if (lane == cc && cr != cc) row[5 + N] = co;
            }
        }
        double2 ks[TB::S][N], inc[N], H[N];
#pragma unroll
        for (int n = 0; n < N; ++n) inc[n] = make_double2(0.0, 0.0);
#pragma unroll
        for (int s = 0; s < TB::S; ++s) {
            double2 y[N];
#pragma unroll
            for (int n = 0; n < N; ++n) y[n] = y0[n];
#pragma unroll
            for (int q = 0; q < s; ++q)
                if (TB::a(s, q) != 0.0) {
                    const double a = h * TB::a(s, q);
#pragma unroll
                    for (int n = 0; n < N; ++n)
                        y[n] = make_double2(fma(a, ks[q][n].x, y[n].x), fma(a, ks[q][n].y, y[n].y));
                }
#pragma unroll
            for (int n = 0; n < N; ++n)
                if (own && n >= m) Y[m * N - m * (m - 1) / 2 + (n - m)] = y[n];
            if (s == 0 || TB::ti(s) != TB::ti(s - 1)) {   // row m of diag(eps) + A.P (SBEs.h:787-805)
                const double Ax = fl[TB::ti(s) * 3], Ay = fl[TB::ti(s) * 3 + 1];
#pragma unroll
                for (int n = 0; n < N; ++n)
                    H[n] = make_double2(fma(Ax, p[0][n].x, fma(Ay, p[1][n].x, n == m ? eps : 0.0)),
                                        fma(Ax, p[0][n].y, Ay * p[1][n].y));
            }
            __syncwarp();
            double2 c[N];
#pragma unroll
            for (int n = 0; n < N; ++n) c[n] = make_double2(0.0, 0.0);
#pragma unroll
            for (int l = 0; l < N; ++l)
#pragma unroll
                for (int n = l; n < N; ++n) {
                    const double2 v = Y[l * N - l * (l - 1) / 2 + (n - l)];   // Y_ln
                    cfma(c[n], H[l], v);
                    if (n != l) cfma(c[l], H[n], cconj(v));
                }
#pragma unroll
            for (int n = 0; n < N; ++n)
                if (own) T[m * D::LDT + n] = c[n];
            __syncwarp();
            // -i((HY) - (HY)^dag) - Gamma o (Y - rho0)   (SBEs.h:808-819, 862-871)
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const double2 d = T[n * D::LDT + mr];
                const double re = c[n].y + d.y, im = d.x - c[n].x;
                ks[s][n] = n == m ? make_double2(fma(-g1, y[n].x - f, re), 0.0)
                                  : make_double2(fma(-g2, y[n].x, re), fma(-g2, y[n].y, im));
                if (TB::b(s) != 0.0) {
                    const double b = h * TB::b(s);
                    inc[n] = make_double2(fma(b, ks[s][n].x, inc[n].x), fma(b, ks[s][n].y, inc[n].y));
                }
            }
        }
#pragma unroll
        for (int n = 0; n < N; ++n) y0[n] = make_double2(y0[n].x + inc[n].x, y0[n].y + inc[n].y);
    }
    if (live && own)
#pragma unroll
        for (int n = 0; n < N; ++n) rho[m * N + n] = y0[n];
}

// ============================================================= length gauge
// Models with their own current-operator tables (has_jtab: the analytic
// materials), plain FP64 method: rho in the Wannier basis, H0(k + A) from its
// Fourier tables, dephasing in the eigenbasis of H0 (SBEs.h:762-786, 831-861).
// A pair of lattice vectors (R, -R) is summed together: c sig + s tau with
// e^{iKR} = c + i s.

// Phase factors e^{iA(t)R} of a launch that starts at step n0: row j of
// step_cA, at the distinct stage times of step n0 + j.
__device__ void launch_phases(const WanDev &P, int n0, int j)
{
    const int n = n0 + j, nt = P.rk == 4 ? StepTab<4>::NT : StepTab<5>::NT;
    if (!P.step_cA || n >= P.Nt) return;
    double2 *out = P.step_cA + (size_t)j * nt * P.npair;
    for (int i = threadIdx.x; i < nt * P.npair; i += blockDim.x) {
        const int r = P.gpair[i % P.npair];
        const double *A = P.step_fld + ((size_t)n * nt + i / P.npair) * 3;
        double sn, cs;
        sincos(A[0] * P.V[2 * r] + A[1] * P.V[2 * r + 1], &sn, &cs);
        out[i] = make_double2(cs, sn);
    }
}

__global__ void __launch_bounds__(256) wan_step_phases(const WanDev *__restrict__ Pp)
{
    launch_phases(*Pp, Pp->ctl->n, blockIdx.x);
}

// Upper-triangle pair tables [np][2][NU] (sig, tau) of H (a < 0), or of the
// Hermitian part of J_a (Re Tr(rho J) sees no more), into shared memory
__device__ __forceinline__ void load_pairs(const WanDev &P, int N, int a, double2 *sh)
{
    const int NN = N * N, NU = N * (N + 1) / 2;
    const double2 *tb = static_cast<const double2 *>(a < 0 ? P.h : P.jt) + (a > 0 ? NN : 0);
    const int stride = a < 0 ? NN : 2 * NN;
    const double2 zero = make_double2(0.0, 0.0);
    for (int i = threadIdx.x; i < P.npair * NU; i += blockDim.x) {
        const int q = i / NU, r = P.gpair[q], r2 = P.gmate[q];
        int u = i % NU, m = 0;
        while (u >= N - m) { u -= N - m; ++m; }
        const int n = m + u;
        double2 x = tb[(size_t)r * stride + m * N + n], y = r2 < 0 ? zero : tb[(size_t)r2 * stride + m * N + n];
        if (a >= 0) {   // (T + T^dag) / 2: the adjoint of the entry at R belongs to -R
            const double2 xt = cconj(tb[(size_t)r * stride + n * N + m]);
            const double2 yt = r2 < 0 ? zero : cconj(tb[(size_t)r2 * stride + n * N + m]);
            x = make_double2(0.5 * (x.x + yt.x), 0.5 * (x.y + yt.y));
            y = make_double2(0.5 * (y.x + xt.x), 0.5 * (y.y + xt.y));
        }
        double2 *o = sh + q * 2 * NU + i % NU;
        o[0] = make_double2(x.x + y.x, x.y + y.y);
        o[NU] = make_double2(y.y - x.y, x.x - y.x);   // i (x - y)
    }
}

// Hermitian N x N matrix of one thread: real diagonal, upper off-diagonal
template <int N> struct Herm {
    static constexpr int NO = N * (N - 1) / 2;
    double d[N];
    double2 o[NO];
};
template <int N> __device__ __forceinline__ double2 el(const Herm<N> &A, int m, int n)   // m != n
{
    return m < n ? A.o[oidx(m, n, N)] : cconj(A.o[oidx(n, m, N)]);
}
template <int N> __device__ __forceinline__ double tr2(const Herm<N> &A, const Herm<N> &B)   // Tr(A B)
{
    double s = 0.0, t = 0.0, u = 0.0;   // separate chains: latency counts at one warp per scheduler
#pragma unroll
    for (int m = 0; m < N; ++m) s = fma(A.d[m], B.d[m], s);
#pragma unroll
    for (int i = 0; i < Herm<N>::NO; ++i) {
        t = fma(A.o[i].x, B.o[i].x, t);
        u = fma(A.o[i].y, B.o[i].y, u);
    }
    return fma(2.0, t + u, s);
}
template <int N> __device__ __forceinline__ void axpy(Herm<N> &A, double c, const Herm<N> &B)   // A += c B
{
#pragma unroll
    for (int m = 0; m < N; ++m) A.d[m] = fma(c, B.d[m], A.d[m]);
#pragma unroll
    for (int i = 0; i < Herm<N>::NO; ++i) A.o[i] = make_double2(fma(c, B.o[i].x, A.o[i].x), fma(c, B.o[i].y, A.o[i].y));
}
template <int N> __device__ __forceinline__ void clear(Herm<N> &A)
{
#pragma unroll
    for (int m = 0; m < N; ++m) A.d[m] = 0.0;
#pragma unroll
    for (int i = 0; i < Herm<N>::NO; ++i) A.o[i] = make_double2(0.0, 0.0);
}
template <int N> __device__ __forceinline__ void traceless(Herm<N> &A)
{
    double t = 0.0;
#pragma unroll
    for (int m = 0; m < N; ++m) t += A.d[m];
#pragma unroll
    for (int m = 0; m < N; ++m) A.d[m] = fma(t, -1.0 / N, A.d[m]);
}
// W = traceless part of A B for commuting A, B
template <int N> __device__ __forceinline__ void mul_traceless(Herm<N> &W, const Herm<N> &A, const Herm<N> &B)
{
#pragma unroll
    for (int m = 0; m < N; ++m) {
        double d = A.d[m] * B.d[m];
#pragma unroll
        for (int l = 0; l < N; ++l)
            if (l != m) {
                const double2 x = el<N>(A, m, l), y = el<N>(B, m, l);
                d = fma(x.x, y.x, fma(x.y, y.y, d));
            }
        W.d[m] = d;
#pragma unroll
        for (int n = m + 1; n < N; ++n) {
            const double2 x = A.o[oidx(m, n, N)], y = B.o[oidx(m, n, N)];
            double2 w = make_double2(fma(A.d[m], y.x, x.x * B.d[n]), fma(A.d[m], y.y, x.y * B.d[n]));
#pragma unroll
            for (int l = 0; l < N; ++l)
                if (l != m && l != n) cfma(w, el<N>(A, m, l), el<N>(B, l, n));
            W.o[oidx(m, n, N)] = w;
        }
    }
    traceless<N>(W);
}

// V^dag X V, rows p < q
template <int N> __device__ __forceinline__ void turn(Herm<N> &X, int p, int q, const Turn &t)
{
    t.own(X.d[p], X.o[oidx(p, q, N)], X.d[q]);
#pragma unroll
    for (int r = 0; r < N; ++r) {
        if (r == p || r == q) continue;
        double2 x = el<N>(X, r, p), y = el<N>(X, r, q);
        t.on(x, y, t.s);
        if (r < p) X.o[oidx(r, p, N)] = x;
        else X.o[oidx(p, r, N)] = cconj(x);
        if (r < q) X.o[oidx(r, q, N)] = y;
        else X.o[oidx(q, r, N)] = cconj(y);
    }
}
// D(Y) by eigenvectors, for k-points where bands crowd: Jacobi rotations of A until it is
// diagonal and of Y along with it, then Y's diagonal back through them.  Out of line.
template <int N> __device__ __noinline__ void eigen_diagonal(Herm<N> *D, const Herm<N> *A0, const Herm<N> *Y0)
{
    Turn rot[MAX_SWEEPS * Herm<N>::NO];
    Herm<N> A = *A0, Y = *Y0;
    int n = 0;
#pragma unroll 1
    for (int sweep = 0; sweep < MAX_SWEEPS; ++sweep) {
        double off = 0.0;
#pragma unroll
        for (int i = 0; i < Herm<N>::NO; ++i) off += A.o[i].x * A.o[i].x + A.o[i].y * A.o[i].y;
        if (!(off > 1e-36 * tr2<N>(A, A))) break;
#pragma unroll
        for (int p = 0; p < N - 1; ++p)
#pragma unroll
            for (int q = p + 1; q < N; ++q) {
                Turn t;
                double dl;
                t.find(A.d[p], A.d[q], A.o[oidx(p, q, N)], dl);
                turn<N>(Y, p, q, t);
                const double a = A.d[p] - dl, b = A.d[q] + dl;
                turn<N>(A, p, q, t);
                A.d[p] = a;
                A.d[q] = b;
                A.o[oidx(p, q, N)] = make_double2(0.0, 0.0);
                rot[n++] = t;
            }
    }
#pragma unroll
    for (int i = 0; i < Herm<N>::NO; ++i) Y.o[i] = make_double2(0.0, 0.0);
#pragma unroll 1
    while (n > 0) {   // the last rotation first
#pragma unroll
        for (int p = N - 2; p >= 0; --p)
#pragma unroll
            for (int q = N - 1; q > p; --q) {
                Turn t = rot[--n];
                t.s = make_double2(-t.s.x, -t.s.y);
                turn<N>(Y, p, q, t);
            }
    }
    *D = Y;
}

// D = the band-diagonal part of Y in the eigenbasis of A, U diag(U^dag Y U)
// U^dag, without the eigenbasis: for distinct eigenvalues it is the orthogonal
// projection (inner product Tr(XY)) of Y on the span of I, A, ..., A^{N-1},
// the matrices that commute with A.  The Lanczos recurrence from I (left
// multiplication by A is self-adjoint) gives an orthogonal basis of Hermitian
// matrices in N - 2 products, where a tracked eigenbasis takes B = U^dag A U,
// rotations until it is diagonal, and U diag U^dag.  Conditioned like the
// eigenvectors (rounding over the smallest gap) but for three close bands of
// N = 4 (bands_crowd), which go by eigenvectors.  N = 2 is the closed form (s.n) n
// of the Bloch vector.  A is made traceless.  Returns whether bands crowd; D is by
// eigenvectors then if EIG.
template <int N, bool EIG> __device__ __forceinline__ bool band_diagonal(Herm<N> &D, Herm<N> &A, const Herm<N> &Y)
{
    double ty = 0.0, th = 0.0;
#pragma unroll
    for (int m = 0; m < N; ++m) {
        ty += Y.d[m];
        th += A.d[m];
    }
    traceless<N>(A);
    const double a2 = tr2<N>(A, A), ia = a2 > 0.0 ? 1.0 / a2 : 0.0;
    clear<N>(D);
#pragma unroll
    for (int m = 0; m < N; ++m) D.d[m] = ty * (1.0 / N);
    axpy<N>(D, tr2<N>(A, Y) * ia, A);
    if constexpr (N > 2) {
        // a basis matrix that is rounding only (two bands meet) is left out
        Herm<N> W;
        mul_traceless<N>(W, A, A);
        axpy<N>(W, -tr2<N>(W, A) * ia, A);
        const double w2 = tr2<N>(W, W), iw = w2 > 1e-26 * a2 * a2 ? 1.0 / w2 : 0.0;
        axpy<N>(D, tr2<N>(W, Y) * iw, W);
        if constexpr (N > 3) {
            Herm<N> V;
            mul_traceless<N>(V, A, W);
            const double va = tr2<N>(V, A) * ia, vw = tr2<N>(V, W) * iw;
            axpy<N>(V, -va, A);
            axpy<N>(V, -vw, W);
            const double v2 = tr2<N>(V, V), iv = v2 > 1e-26 * a2 * w2 ? 1.0 / v2 : 0.0;
            axpy<N>(D, tr2<N>(V, Y) * iv, V);
            if (bands_crowd<N>(v2, v2 * iw, a2, fma(th * th, 1.0 / N, a2))) {
                if constexpr (EIG) {
                    Herm<N> d, a = A, y = Y;
                    eigen_diagonal<N>(&d, &a, &y);
                    D = d;
                }
                return true;
            }
        }
    }
    return false;
}

// H += a pair's term: table entry s [2][NU], phase e
template <int N> __device__ __forceinline__ void add_pair(Herm<N> &H, const double2 *s, double2 e)
{
    constexpr int NU = N * (N + 1) / 2;
#pragma unroll
    for (int m = 0; m < N; ++m)
#pragma unroll
        for (int n = m; n < N; ++n) {
            const int u = m * N - m * (m - 1) / 2 + n - m;
            const double2 sg = s[u], ta = s[NU + u];
            if (m == n) {
                H.d[m] = fma(e.x, sg.x, fma(e.y, ta.x, H.d[m]));
            } else {
                double2 &x = H.o[oidx(m, n, N)];
                x = make_double2(fma(e.x, sg.x, fma(e.y, ta.x, x.x)), fma(e.x, sg.y, fma(e.y, ta.y, x.y)));
            }
        }
}

// the tableaux of StepTab, for the run-time stage loop
__constant__ double c_step_a[2][6][6] = {
    {{0}, {0.5}, {0, 0.5}, {0, 0, 1.0}},
    {{0},
     {1.0 / 4.0},
     {3. / 32., 9. / 32.},
     {1932. / 2197., -7200. / 2197., 7296. / 2197.},
     {439. / 216., -8., 3680. / 513., -845. / 4104.},
     {-8. / 27., 2., -3544. / 2565, 1859. / 4104, -11. / 40.}}};
__constant__ double c_step_b[2][6] = {{1.0 / 6.0, 2.0 / 6.0, 2.0 / 6.0, 1.0 / 6.0},
                                      {16. / 135., 0.0, 6656. / 12825., 28561. / 56430., -9. / 50., 2. / 55.}};

constexpr int WL_T = 32;   // threads (k-points) per block
// shared memory: H and J tables, the step's phase factors, per thread e^{ikR},
// rho, its increment and the stage slopes
static int lw_bytes(int N, int rk, int npair)
{
    const int nt = rk == 4 ? StepTab<4>::NT : StepTab<5>::NT;
    return (3 * N * (N + 1) * npair + nt * npair + npair * WL_T) * 16 + (2 + (rk == 4 ? 1 : 5)) * N * N * WL_T * 8;
}

// N = 2, 3, 4, one thread per k-point.  H0, Y, D and the Lanczos basis are
// registers; rho, its increment and the stage slopes wait in shared memory, a
// column per thread.  The stage loop is a run-time loop, so that its body stays
// in the instruction cache.  One-warp blocks: small grids spread over every
// SM.  Latency-bound (a step is a serial chain of stages) until the grid gives
// every scheduler a few warps, FP64-pipe bound beyond.  Measured (whole solves
// of 367 steps with their set-up, us a step, 168 to 14 640 k-points alike): N =
// 2, 3, 4 RK4 2.5, 5.7, 9.5, RK5 4.1, 9.2, 15; one attempt and one control
// launch a step take 78 (N = 3, RK5, 2 400 k-points).
//
// lw_advance: false if bands crowded at a stage of a k-point; nothing but partial
// rows was written then.  EIG: those by eigenvectors (in a pass of their own: with
// the call in the first pass a step took 9.9 us, with the check alone 9.5, without 9.3).
template <int N, int RK, bool EIG>
__device__ __forceinline__ bool lw_advance(const WanDev &P, int k0, int S, unsigned char *smem)
{
    using TB = StepTab<RK>;
    using HN = Herm<N>;
    constexpr int NN = N * N, NU = N * (N + 1) / 2, NO = HN::NO, NK = RK == 4 ? 1 : 5;
    const int n0 = P.ctl->n, steps = launch_steps(P, n0, S), np = P.npair, ncA = TB::NT * np;
    const int t = threadIdx.x, lane = t & 31;
    const int k = k0 + t;
    const bool live = k < P.nk;
    const int kc = live ? k : P.nk - 1;   // a thread past the grid shadows the last k-point
    double2 *const htab = reinterpret_cast<double2 *>(smem), *const jtab = htab + 2 * NU * np;   // load_pairs; J_x, J_y
    double2 *const cA = jtab + 4 * NU * np, *const pk = cA + ncA;                                // pk: [np][WL_T]
    double *const sy = reinterpret_cast<double *>(pk + np * WL_T);   // [2 + NK][NN][WL_T]: rho, increment, slopes
    auto put = [&](int slot, const HN &A) {
#pragma unroll
        for (int m = 0; m < N; ++m) sy[(slot * NN + m) * WL_T + t] = A.d[m];
#pragma unroll
        for (int i = 0; i < NO; ++i) {
            sy[(slot * NN + N + 2 * i) * WL_T + t] = A.o[i].x;
            sy[(slot * NN + N + 2 * i + 1) * WL_T + t] = A.o[i].y;
        }
    };
    auto get = [&](int slot, HN &A) {
#pragma unroll
        for (int m = 0; m < N; ++m) A.d[m] = sy[(slot * NN + m) * WL_T + t];
#pragma unroll
        for (int i = 0; i < NO; ++i)
            A.o[i] = make_double2(sy[(slot * NN + N + 2 * i) * WL_T + t], sy[(slot * NN + N + 2 * i + 1) * WL_T + t]);
    };
    load_pairs(P, N, -1, htab);
    load_pairs(P, N, 0, jtab);
    load_pairs(P, N, 1, jtab + 2 * NU * np);
    double kv[3], wk;
    kpoint(P, kc, kv, wk);
    if (!live) wk = 0.0;
    for (int q = 0; q < np; ++q) {
        const int r = P.gpair[q];
        double sn, cs;
        sincos(kv[0] * P.V[2 * r] + kv[1] * P.V[2 * r + 1], &sn, &cs);
        pk[q * WL_T + t] = make_double2(cs, sn);
    }
    double2 *rho = P.rho[0] + (size_t)kc * NN;
    {
        HN Y;
#pragma unroll
        for (int m = 0; m < N; ++m) {
            Y.d[m] = rho[m * N + m].x;
#pragma unroll
            for (int n = m + 1; n < N; ++n) Y.o[oidx(m, n, N)] = rho[m * N + n];
        }
        put(0, Y);
    }
    const double g1 = P.g1, g2 = P.g2, gd = g1 - g2;
    const int ce = (P.nval * N + P.nval + 1) % NN;   // antelope.cpp:539-542
    const int nw = P.step_rows;
    double *part = P.step_part + (size_t)((k0 + t) >> 5) * WAN_NSLOT + (lane >> 1);
    const bool wr = (lane & 1) == 0;
    // the step's phase factors go to shared memory; the next step's first 64
    // are on their way in registers meanwhile
    const double2 *cg = P.step_cA;
    bool crowded = false;
    double2 pre[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) pre[x] = t + x * WL_T < ncA ? cg[t + x * WL_T] : make_double2(0.0, 0.0);

    for (int j = 0; j < steps; ++j, cg += ncA) {
        __syncwarp();
#pragma unroll
        for (int x = 0; x < 2; ++x)
            if (t + x * WL_T < ncA) cA[t + x * WL_T] = pre[x];
        for (int i = t + 2 * WL_T; i < ncA; i += WL_T) cA[i] = cg[i];
        __syncwarp();
        if (j + 1 < steps)
#pragma unroll
            for (int x = 0; x < 2; ++x)
                if (t + x * WL_T < ncA) pre[x] = cg[ncA + t + x * WL_T];
        const double h = step_length(P, n0 + j);
        HN H;
#pragma unroll 1
        for (int s = 0; s < TB::S; ++s) {
            const int ti = RK == 4 ? (s + 1) / 2 : s;
            double z[4];   // current sums of the step's start
            HN Y, K;
            get(0, Y);
            for (int q = RK == 4 ? max(0, s - 1) : 0; q < s; ++q) {
                const double a = h * c_step_a[RK - 4][s][q];
                get(2 + (RK == 4 ? 0 : q), K);
                axpy<N>(Y, a, K);
            }
            HN X[2];
            if (s == 0) {   // with the currents' operators (Hermitian parts)
                clear<N>(H);
                clear<N>(X[0]);
                clear<N>(X[1]);
#pragma unroll 1
                for (int q = 0; q < np; ++q) {
                    const double2 e = cmul(pk[q * WL_T + t], cA[q]);
                    add_pair<N>(H, htab + q * 2 * NU, e);
                    add_pair<N>(X[0], jtab + q * 2 * NU, e);
                    add_pair<N>(X[1], jtab + (np + q) * 2 * NU, e);
                }
            } else if (!(RK == 4 && s == 2)) {   // RK4's midpoint stages share H0
                clear<N>(H);
#pragma unroll 2
                for (int q = 0; q < np; ++q) add_pair<N>(H, htab + q * 2 * NU, cmul(pk[q * WL_T + t], cA[ti * np + q]));
            }
            {
                HN A = H;
                crowded |= band_diagonal<N, EIG>(K, A, Y);   // K = D(Y)
            }
            if (s == 0) {   // currents at k + A(t_n) (SBEs.h:694-760): intraband Re Tr(D J), the rest interband
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    z[2 + a] = tr2<N>(K, X[a]);
                    z[a] = tr2<N>(Y, X[a]) - z[2 + a];
                }
                double v[16];
#pragma unroll
                for (int q = 0; q < 16; ++q) v[q] = q < 4 ? wk * z[q] : 0.0;
#pragma unroll
                for (int m = 0; m < N; ++m) v[4 + m] = wk * Y.d[m];
#pragma unroll
                for (int e = 0; e < NN; ++e)
                    if (e == ce) {
                        const int m = e / N, n = e % N;
                        const double2 y = m == n ? make_double2(Y.d[m], 0.0) : el<N>(Y, m, n);
                        v[4 + N] = wk * y.x;
                        v[5 + N] = wk * y.y;
                    }
                const double sum = warp_sum16(v, lane);
                if (wr) part[(size_t)j * nw * WAN_NSLOT] = sum;
            }
            // -i((HY) - (HY)^dag) - (g2 Y + (g1 - g2) D)   (SBEs.h:808-861)
            const double b = h * c_step_b[RK - 4][s];
#pragma unroll
            for (int m = 0; m < N; ++m) {
                double im = 0.0;   // Im (HY)_mm
#pragma unroll
                for (int l = 0; l < N; ++l) {
                    if (l == m) continue;
                    const double2 x = el<N>(H, m, l), y = el<N>(Y, l, m);
                    im = fma(x.x, y.y, fma(x.y, y.x, im));
                }
                K.d[m] = fma(-gd, K.d[m], fma(-g2, Y.d[m], 2.0 * im));
            }
#pragma unroll
            for (int m = 0; m < N; ++m)
#pragma unroll
                for (int n = m + 1; n < N; ++n) {
                    const int o = oidx(m, n, N);
                    const double2 w = Y.o[o], x = H.o[o];
                    // c = (HY)_mn - conj (HY)_nm
                    const double hd = H.d[m] - H.d[n], yd = Y.d[n] - Y.d[m];
                    double2 c = make_double2(fma(hd, w.x, x.x * yd), fma(hd, w.y, x.y * yd));
#pragma unroll
                    for (int l = 0; l < N; ++l) {
                        if (l == m || l == n) continue;
                        cfma(c, el<N>(H, m, l), el<N>(Y, l, n));
                        const double2 p = el<N>(Y, m, l), q = el<N>(H, l, n);   // - Y_ml H_ln
                        c.x = fma(-p.x, q.x, fma(p.y, q.y, c.x));
                        c.y = fma(-p.x, q.y, fma(-p.y, q.x, c.y));
                    }
                    K.o[o] = make_double2(fma(-gd, K.o[o].x, fma(-g2, w.x, c.y)), fma(-gd, K.o[o].y, fma(-g2, w.y, -c.x)));
                }
            if (RK == 4 || s < NK) put(2 + (RK == 4 ? 0 : s), K);
            if (s > 0) get(1, Y);
            else clear<N>(Y);
            axpy<N>(Y, b, K);   // the increment
            if (s + 1 < TB::S) {
                put(1, Y);
            } else {
                get(0, K);
                axpy<N>(K, 1.0, Y);
                put(0, K);
            }
        }
    }
    if (N > 3 && !EIG && __any_sync(0xffffffffu, live && crowded)) return false;
    if (!live) return true;
    HN Y;
    get(0, Y);
#pragma unroll
    for (int m = 0; m < N; ++m) {
        rho[m * N + m] = make_double2(Y.d[m], 0.0);
#pragma unroll
        for (int n = m + 1; n < N; ++n) {
            rho[m * N + n] = Y.o[oidx(m, n, N)];
            rho[n * N + m] = cconj(Y.o[oidx(m, n, N)]);
        }
    }
    return true;
}
template <int N, int RK> __device__ __noinline__ void lw_advance_eig(const WanDev &P, int k0, int S, unsigned char *smem)
{
    lw_advance<N, RK, true>(P, k0, S, smem);
}

template <int N, int RK>
__global__ void __launch_bounds__(WL_T) wan_lw_steps(const WanDev *__restrict__ Pp,
                                                     const WanDev *const *__restrict__ descs,
                                                     const WanTileRef *__restrict__ tiles, int S)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const WanDev &P = tiles ? *descs[tiles[blockIdx.x].solve] : *Pp;
    const int k0 = tiles ? tiles[blockIdx.x].tile * WAN_WARPS : (int)blockIdx.x * WL_T;
    if (P.ctl->done) return;
    if (!lw_advance<N, RK, false>(P, k0, S, smem)) {
        if constexpr (N > 3) lw_advance_eig<N, RK>(P, k0, S, smem);
    }
}

// Block (j, solve): the sums of the launch's step j over the solve's partial
// rows (fixed order).  The solve's last block to finish moves its controller
// past the launch's steps; every block has read it by then.
__global__ void __launch_bounds__(256) wan_finish(const WanDev *__restrict__ Pp, const WanDev *const *__restrict__ descs,
                                                  int S)
{
    __shared__ double red[16][WAN_NSLOT];
    const WanDev &P = descs ? *descs[blockIdx.y] : *Pp;
    WanCtl *ctl = P.ctl;
    const int j = blockIdx.x, t = threadIdx.x;
    if (ctl->done) {
        if (j == 0 && t == 0) ctl->shot = -1;   // a snapshot is taken once
        return;
    }
    const int n0 = ctl->n, steps = launch_steps(P, n0, S);
    if (j < steps) {
        const int slot = t % WAN_NSLOT, g = t / WAN_NSLOT, nw = P.step_rows;
        const double *p = P.step_part + (size_t)j * nw * WAN_NSLOT + slot;
        double s0 = 0.0, s1 = 0.0;
        int i = g;
        for (; i + 16 < nw; i += 32) {
            s0 += p[(size_t)i * WAN_NSLOT];
            s1 += p[(size_t)(i + 16) * WAN_NSLOT];
        }
        if (i < nw) s0 += p[(size_t)i * WAN_NSLOT];
        red[g][slot] = s0 + s1;
        __syncthreads();
        if (t < WAN_NSLOT) {
            double s = 0.0;
            for (int q = 0; q < 16; ++q) s += red[q][t];
            P.jout[(size_t)(n0 + j) * WAN_NSLOT + t] = s;
        }
    }
    for (int x = j; x < WAN_STEPS; x += gridDim.x) launch_phases(P, n0 + steps, x);   // of the next launch, whatever its S
    __syncthreads();
    if (t == 0) {
        __threadfence();
        if (atomicAdd(P.step_ticket, 1u) == gridDim.x - 1) {
            *P.step_ticket = 0u;
            ctl->shot = -1;
            ctl->n = n0 + steps;
            // a step whose end the sum t + dt misses by rounding counts one
            // more (empty) step, as the step controller counts it
            long long cnt = steps;
            for (int n = n0; n < n0 + steps; ++n)
                cnt += !(step_start(P, n) + P.dt >= P.atmin + P.dt * (n + 1) - 1e-12 * P.dt);
            ctl->steps += cnt;
            ctl->attempts += cnt;
            ctl->tc = step_start(P, n0 + steps);
            ctl->need_current = 1;
            if (P.shot_every > 0 && (n0 + steps - 1) % P.shot_every == 0) ctl->shot = n0 + steps - 1;
            if (n0 + steps >= P.Nt) ctl->done = 1;
        }
    }
}

// ============================================================= launchers
// Velocity gauge: one thread per k-point while a k-point's matrices fit a
// thread's registers without spilling (N <= 3), else one row per lane; both
// sides measured at the head of this file.  Length gauge: the plain method on
// models with current-operator tables, N <= 4.  The mixed method keeps the
// FP32 Fourier sums and the tolerances of wan_attempt; more bands and dipole
// tables stay with it and with wan_attempt_g, and so do solves with bands that
// meet at a grid point (to 1e-7 of their spread): what the dephasing does
// inside such a pair depends on its basis, which only a tracked eigenbasis
// carries along; and small grids where three bands crowd (wan_crowded_slow).
enum StepMode : int { VG_THREAD = 1, VG_ROWS = 2, LW_THREAD = 3 };
static int row_lanes(int N) { return N <= 4 ? 4 : 8; }
// dynamic shared memory of a block
static int steps_bytes(int mode, int N, int na, int rk, int npair)
{
    if (mode == VG_THREAD) return (na * N * N + N) * WS_T * 16;
    return mode == LW_THREAD ? lw_bytes(N, rk, npair) : 0;
}
constexpr int STEPS_MAX_BYTES = 96 * 1024;   // at least two blocks per SM
int wan_steps(const WanDev &w)
{
    if (w.lean || (w.rk != 4 && w.rk != 5) || w.N < 2 || w.N > WAN_MAXN) return 0;
    if (w.vg) return w.N <= 3 ? VG_THREAD : VG_ROWS;
    if (w.mixed || !w.has_jtab || w.has_dip || w.cont || w.N > 4 || w.degenerate) return 0;
    return steps_bytes(LW_THREAD, w.N, 2, w.rk, w.nR) <= STEPS_MAX_BYTES ? LW_THREAD : 0;
}
// A k-point where bands crowd makes its block take its pass again, with eigenvectors.
// Measured with such points, us a step or attempt, against the tracked kernels:
// wan_lw_steps (N = 4, RK4) 50 / 40 on 168 points, 52 / 77 on 3 720, 55 / 199 on
// 14 640; wan_attempt_p (Cash-Karp) at 64, 10 000 and 60 000 points, all of them or
// one in 30 crowded, N = 4: 208, 243, 812 all and 206, 292 some / 97, 207, 818; N = 5:
// 450, 582, 3015 and 507, 768 / 164, 769, 4261; N = 6: 500, 595, 3268 and 595, 1221 /
// 146, 390, 1433.
bool wan_crowded_slow(const WanDev &w, unsigned long long points)
{
    if (points == 0) return false;
    if (wan_steps(w)) return w.nk < 2048;
    return w.N < 6 ? w.nk < 10000 : w.nk < 60000 || points * 32 > (unsigned long long)w.nk;
}
static int block_threads(int mode) { return mode == VG_ROWS ? WR_T : mode == LW_THREAD ? WL_T : WS_T; }
int wan_steps_rows(const WanDev &w)
{
    const int kw = wan_steps(w) == VG_ROWS ? 32 / row_lanes(w.N) : 32;
    return (w.nk + kw - 1) / kw;
}
int wan_steps_fields(int rk) { return rk == 4 ? StepTab<4>::NT : StepTab<5>::NT; }
int wan_steps_unit(int mode, int N)
{
    return block_threads(mode) / (mode == VG_ROWS ? row_lanes(N) : 1) / WAN_WARPS;
}

using StepKernel = void (*)(const WanDev *, const WanDev *const *, const WanTileRef *, int);
template <int RK> static StepKernel steps_kernel(int mode, int N, int na)
{
    if (mode == VG_THREAD) {
        if (N == 2) return na == 3 ? wan_vg_steps<2, RK, 3> : wan_vg_steps<2, RK, 2>;   // 3: the continuum model
        return N == 3 ? wan_vg_steps<3, RK, 2> : nullptr;
    }
    if (mode == LW_THREAD)
        return N == 2 ? wan_lw_steps<2, RK> : N == 3 ? wan_lw_steps<3, RK> : N == 4 ? wan_lw_steps<4, RK> : nullptr;
    switch (N) {
    case 4: return wan_vg_rows<4, RK>;
    case 5: return wan_vg_rows<5, RK>;
    case 6: return wan_vg_rows<6, RK>;
    case 7: return wan_vg_rows<7, RK>;
    case 8: return wan_vg_rows<8, RK>;
    default: return nullptr;
    }
}

cudaError_t launch_wan_steps(const WanStepClass &c, const WanDev *dw, const WanDev *const *descs,
                             const WanTileRef *tiles, int nblocks, int S, cudaStream_t st)
{
    const StepKernel f = c.rk == 4 ? steps_kernel<4>(c.mode, c.N, c.na)
                                   : c.rk == 5 ? steps_kernel<5>(c.mode, c.N, c.na) : nullptr;
    if (!f) return cudaErrorInvalidValue;
    const int sm = steps_bytes(c.mode, c.N, c.na, c.rk, c.npair);
    if (sm > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, STEPS_MAX_BYTES);
        if (e != cudaSuccess) return e;
    }
    f<<<nblocks, block_threads(c.mode), sm, st>>>(dw, descs, tiles, S);
    return cudaGetLastError();
}
WanStepClass wan_step_class(const WanDev &w)
{
    WanStepClass c;
    c.mode = wan_steps(w);
    c.N = w.N;
    c.na = w.cont ? 3 : 2;
    c.rk = w.rk;
    c.npair = c.mode == LW_THREAD ? w.npair : 0;
    return c;
}

cudaError_t launch_wan_finish(const WanDev *dw, const WanDev *const *descs, int nsolves, int S, cudaStream_t st)
{
    wan_finish<<<dim3(S, nsolves), 256, 0, st>>>(dw, descs, S);
    return cudaGetLastError();
}

cudaError_t launch_wan_step_fields(const WanDev &w, const WanDev *dw, cudaStream_t st)
{
    const int nt = wan_steps_fields(w.rk);
    wan_step_fields<<<(w.Nt * nt + 127) / 128, 128, 0, st>>>(dw, nt, w.rk);
    if (w.step_cA) wan_step_phases<<<WAN_STEPS, 256, 0, st>>>(dw);
    return cudaGetLastError();
}

}  // namespace sbe
