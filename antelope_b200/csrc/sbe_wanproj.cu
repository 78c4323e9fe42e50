// Projection attempt kernel of the N-band length gauge (sm_100a): explicit
// tables with the -dH/dk + i[D, H] current operator (SyntheticWannier), one
// attempted step of every k-point per launch.
//
// The same step as wan_attempt -- SBEs::GenDifferentialDM (SBEs.h:762-872)
// with the Wannier model form (Materials/Wannier90.h:297-387) and the currents
// of SBEs::GenInterIntraCurrent (SBEs.h:694-760) -- with two changes of
// algorithm.
//
//  - No eigenbasis.  The dephasing and the intraband current need only the
//    band-diagonal part D(Y) = U diag(U^dag Y U) U^dag of rho, which for distinct
//    bands is the orthogonal projection (inner product Tr(XY)) of Y on the
//    matrices that commute with H0.  The Lanczos recurrence P_{j+1} = H0 P_j -
//    a_j P_j - b_j P_{j-1} from I gives an orthogonal basis of them in N - 2
//    products; tracking the eigenbasis took 1.9 rotation steps a stage of four
//    products each, and half of the kernel's time.  Conditioned like the
//    eigenvectors: over a 100 x 100 grid of N = 6 models D(Y) is within 1.5e-14
//    of the eigensolver's, its own rounding over the smallest gap.
//  - Fourier sums in two levels.  A row of the grid has k = k_row + f b, so the
//    vectors R with equal b.R share their phase along the row: with G_g =
//    sum of h_R e^{i(k_row + A).R} over such a group, H0(k + A) = sum_g G_g
//    e^{i f g} has 7 terms instead of 37 on the N = 6 model's vectors.  wan_next
//    forms the G (and those of E.D) of every row and stage between attempts.
//    FP64 method only: the mixed method keeps its FP32 sums over the pairs.
//
// Layout: G lanes per k-point (8 for N > 4), one warp per block; lane l owns
// the upper elements u = l + G j of the state, and lane m < N forms row m of
// the products, the other factor read by element at one address per group.
#include <cuda_runtime.h>

#include <algorithm>

#include "sbe_wandev.cuh"
#include "sbe_wannier.h"

namespace sbe {

namespace {

constexpr unsigned ALL = 0xffffffffu;
constexpr int SPREAD = 148;   // SMs of a B200

// Tableaux (SBEs.h:395-416; Cash-Karp 4(5), ACM TOMS 16 (1990) 201) for the
// run-time stage loop: RK4, Fehlberg-5, Cash-Karp; e = b - b*
struct PTab {
    int S;
    double c[6], a[6][6], b[6], e[6];
};
__constant__ PTab c_tab[3] = {
    {4, {0, 0.5, 0.5, 1.0}, {{0}, {0.5}, {0, 0.5}, {0, 0, 1.0}}, {1.0 / 6.0, 2.0 / 6.0, 2.0 / 6.0, 1.0 / 6.0}, {0}},
    {6,
     {0, 0.25, 3. / 8., 12. / 13., 1.0, 0.5},
     {{0},
      {1.0 / 4.0},
      {3. / 32., 9. / 32.},
      {1932. / 2197., -7200. / 2197., 7296. / 2197.},
      {439. / 216., -8., 3680. / 513., -845. / 4104.},
      {-8. / 27., 2., -3544. / 2565, 1859. / 4104, -11. / 40.}},
     {16. / 135., 0.0, 6656. / 12825., 28561. / 56430., -9. / 50., 2. / 55.},
     {0}},
    {6,
     {0, 1. / 5., 3. / 10., 3. / 5., 1., 7. / 8.},
     {{0},
      {1. / 5.},
      {3. / 40., 9. / 40.},
      {3. / 10., -9. / 10., 6. / 5.},
      {-11. / 54., 5. / 2., -70. / 27., 35. / 27.},
      {1631. / 55296., 175. / 512., 575. / 13824., 44275. / 110592., 253. / 4096.}},
     {37. / 378., 0, 250. / 621., 125. / 594., 0, 512. / 1771.},
     {37. / 378. - 2825. / 27648., 0., 250. / 621. - 18575. / 48384., 125. / 594. - 13525. / 55296., 0. - 277. / 14336.,
      512. / 1771. - 1. / 4.}}};
__device__ __forceinline__ int tab_of(int rk) { return rk == 4 ? 0 : rk == 5 ? 1 : 2; }

template <int N> struct PD {
    static constexpr int G = N <= 4 ? 4 : 8, KW = 32 / G, NN = N * N, NU = N * (N + 1) / 2;
    static constexpr int NO = (NU + G - 1) / G;   // owned upper elements per lane
    static constexpr int LDT = N | 1;
    // a k-point's shared memory in complex numbers: Y, H0, H0 + E.D packed, T rows
    // (odd stride: the groups of a warp read one element each from distinct banks)
    static constexpr int Y = 0, H0 = NU, HT = 2 * NU, T = 3 * NU, END = (T + N * LDT) | 1;
};
__host__ __device__ constexpr int up(int m, int n, int N) { return m * N - m * (m - 1) / 2 + (n - m); }

template <int N> __device__ __forceinline__ double2 herm(const double2 *P, int a, int b)
{
    return a <= b ? P[up(a, b, N)] : cconj(P[up(b, a, N)]);
}
// Re sum_n a_n conj(b_n): three chains
template <int N> __device__ __forceinline__ double row_dot(const double2 (&a)[N], const double2 (&b)[N])
{
    double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int n = 0; n < N; ++n) {
        s[(2 * n) % 3] = fma(a[n].x, b[n].x, s[(2 * n) % 3]);
        s[(2 * n + 1) % 3] = fma(a[n].y, b[n].y, s[(2 * n + 1) % 3]);
    }
    return (s[0] + s[1]) + s[2];
}
template <int G> __device__ __forceinline__ double gsum(double v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(ALL, v, o);
    return v;
}

// c = row a times the Hermitian matrix M (packed upper triangle, each element
// read once at one address per group)
template <int N> __device__ __forceinline__ void row_herm(double2 (&c)[N], const double2 (&a)[N], const double2 *M)
{
#pragma unroll
    for (int n = 0; n < N; ++n) c[n] = make_double2(0.0, 0.0);
#pragma unroll
    for (int l = 0; l < N; ++l)
#pragma unroll
        for (int n = l; n < N; ++n) {
            const double2 x = M[up(l, n, N)];
            cfma(c[n], a[l], x);
            if (n != l) cfma(c[l], a[n], cconj(x));
        }
}

}  // namespace

// Shared memory of a block: slopes, the groups' matrices, the phases along the row
template <int N> static int proj_bytes(int ngrp)
{
    using D = PD<N>;
    return (5 * D::NO * 32 + D::KW * D::END + D::KW * ngrp) * 16;
}

template <int N>
__global__ void __launch_bounds__(32, N <= 4 ? 16 : 12)
    wan_attempt_p(const WanDev *__restrict__ Pp, const WanDev *const *__restrict__ descs,
                  const WanTileRef *__restrict__ tiles)
{
    using D = PD<N>;
    constexpr int G = D::G, KW = D::KW, NU = D::NU, NO = D::NO, NN = D::NN;
    extern __shared__ __align__(16) double2 sm[];
    const WanDev &P = tiles ? *descs[tiles[blockIdx.x].solve] : *Pp;
    // KW k-points; consecutive units (they share the tables of a row) to the
    // blocks of one SM, which get every SPREAD-th block of the grid
    int unit;
    if (tiles) {
        unit = tiles[blockIdx.x].tile * WAN_WARPS / KW;
    } else {
        const int nu = (P.nk + KW - 1) / KW, i = (int)blockIdx.x % SPREAD;
        unit = (int)((long long)i * nu / SPREAD) + (int)blockIdx.x / SPREAD;
        if (unit >= (int)((long long)(i + 1) * nu / SPREAD)) return;
    }
    const WanCtl &ctl = *P.ctl;
    if (ctl.done) return;
    const int lane = threadIdx.x, grp = lane / G, m = lane % G;
    const int k = unit * KW + grp;
    const bool live = k < P.nk, own = m < N;
    const int kc = live ? k : P.nk - 1;   // a group past the grid shadows the last k-point
    const int mr = own ? m : N - 1;
    double2 *const ks = sm;                                      // [5][NO][32] slopes, a column per lane
    double2 *const v = ks + 5 * NO * 32 + grp * D::END;
    const int ng = P.gr_n, nent = 2 * ng - 1;                    // group pairs (g = 0 first), table entries
    double2 *const ph = ks + 5 * NO * 32 + KW * D::END + grp * ng;
    const double h = ctl.hs;
    const int buf = ctl.buf;
    const bool cur = ctl.need_current;
    const PTab &tb = c_tab[tab_of(P.rk)];
    const int S = tb.S;
    double kv[3], wk;
    kpoint(P, kc, kv, wk);
    // the row of this k-point and its phases along it
    const int nf = P.gr_nf, kg = P.k_offset + kc, row = kg / nf - P.gr_row0;
    const double f1 = nf == 1 ? 0.0 : double(kg % nf) / (nf - 1) - 0.5;
    for (int q = m; q < ng; q += G) {
        double sn, cs;
        sincos(f1 * P.gr_a[q], &sn, &cs);
        ph[q] = make_double2(cs, sn);
    }
    // owned upper elements: (row, column) packed in bytes
    int om[NO], on[NO];
    double2 r64[NO];
    const double2 *rho = P.rho[buf] + (size_t)kc * NN;
#pragma unroll
    for (int j = 0; j < NO; ++j) {
        int u = min(m + G * j, NU - 1), a = 0;
        while (u >= N - a) { u -= N - a; ++a; }
        om[j] = a;
        on[j] = a + u;
        r64[j] = __ldcg(rho + om[j] * N + on[j]);
        if (om[j] == on[j]) r64[j].y = 0.0;
    }
    const bool dip = P.has_dip;
    const int NQ = dip ? 2 : 1;
    const double g1 = P.g1, g2 = P.g2, gd = g1 - g2;
    const bool deph = g1 != 0.0 || g2 != 0.0;
    double emax = 0.0;
    double2 kl[NO];   // the last stage's slope
    const size_t ent = (size_t)nent * NO * NQ * G;   // table entries of a (row, stage)
    const double2 *tab = P.gr_tab + (size_t)row * S * ent + m;
    __syncwarp();

#pragma unroll 1
    for (int s = 0; s < S; ++s, tab += ent) {
        // stage input Y = rho + h sum_j a_sj k_j
#pragma unroll
        for (int j = 0; j < NO; ++j) {
            double2 y = r64[j];
            for (int i = 0; i < s; ++i) {
                const double a = h * tb.a[s][i];
                const double2 q = ks[(i * NO + j) * 32 + lane];
                y = make_double2(fma(a, q.x, y.x), fma(a, q.y, y.y));
            }
            if (m + G * j < NU) v[D::Y + m + G * j] = y;
        }
        // H0 and E.D at the owned elements; the next stage's table lines (128
        // bytes each) are fetched towards L1 meanwhile
        if (s + 1 < S)
            for (int i = lane * 8; i < (int)ent; i += 256)
                asm volatile("prefetch.global.L1 [%0];" ::"l"(tab - m + ent + i));
        double2 a0[NO], a1[NO];
#pragma unroll
        for (int j = 0; j < NO; ++j) {
            a0[j] = __ldg(tab + (size_t)j * NQ * G);
            a1[j] = dip ? __ldg(tab + (size_t)(j * NQ + 1) * G) : make_double2(0.0, 0.0);
        }
#pragma unroll 1
        for (int q = 1; q < ng; ++q) {
            const double2 e = ph[q];
            const double2 *t0 = tab + (size_t)(2 * q - 1) * NO * NQ * G, *t1 = t0 + (size_t)NO * NQ * G;
#pragma unroll
            for (int j = 0; j < NO; ++j) {
                const double2 sg = __ldg(t0 + j * NQ * G), ta = __ldg(t1 + j * NQ * G);
                a0[j] = make_double2(fma(e.x, sg.x, fma(e.y, ta.x, a0[j].x)), fma(e.x, sg.y, fma(e.y, ta.y, a0[j].y)));
                if (dip) {
                    const double2 sd = __ldg(t0 + (j * NQ + 1) * G), td = __ldg(t1 + (j * NQ + 1) * G);
                    a1[j] = make_double2(fma(e.x, sd.x, fma(e.y, td.x, a1[j].x)), fma(e.x, sd.y, fma(e.y, td.y, a1[j].y)));
                }
            }
        }
#pragma unroll
        for (int j = 0; j < NO; ++j) {
            if (m + G * j >= NU) continue;
            if (om[j] == on[j]) a0[j].y = a1[j].y = 0.0;
            v[D::H0 + m + G * j] = a0[j];
            v[D::HT + m + G * j] = make_double2(a0[j].x + a1[j].x, a0[j].y + a1[j].y);
        }
        __syncwarp();
        const bool with_cur = cur && s == 0;
        double tot[2] = {0.0, 0.0};
        // S_a waits in the columns of slopes that do not exist yet
        double2 *const sv = ks + NO * 32 + lane;   // [a][j] at (a NO + j) 32
        if (with_cur) {
            // total current Re Tr(Y J_a), J_a = -i S_a + i [D_a, H0] (S_a = sum R_a h_R
            // e^{iKR}): over the owned upper elements, with C = H0 Y - (H0 Y)^dag, the
            // diagonal Y_mm Im(S_mm) - Im(C_mm) Re(D_mm), off it -2 Im(Y_mn conj(S_mn))
            // - 2 Im(C_mn conj(D_mn))
            const int NC = dip ? 4 : 2;   // S_x, S_y (, D_x, D_y)
            const double2 *tc = P.gr_cur + (size_t)row * nent * NO * NC * G + m;
            double2 dd[2][NO], sx[2][NO];
#pragma unroll
            for (int j = 0; j < NO; ++j)
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    sx[a][j] = __ldg(tc + (size_t)(j * NC + a) * G);
                    dd[a][j] = dip ? __ldg(tc + (size_t)(j * NC + 2 + a) * G) : make_double2(0.0, 0.0);
                }
#pragma unroll 1
            for (int q = 1; q < ng; ++q) {
                const double2 e = ph[q];
                const double2 *t0 = tc + (size_t)(2 * q - 1) * NO * NC * G, *t1 = t0 + (size_t)NO * NC * G;
#pragma unroll
                for (int j = 0; j < NO; ++j)
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        const double2 x = __ldg(t0 + (j * NC + a) * G), y = __ldg(t1 + (j * NC + a) * G);
                        double2 &z = sx[a][j];
                        z = make_double2(fma(e.x, x.x, fma(e.y, y.x, z.x)), fma(e.x, x.y, fma(e.y, y.y, z.y)));
                        if (dip) {
                            const double2 x2 = __ldg(t0 + (j * NC + 2 + a) * G), y2 = __ldg(t1 + (j * NC + 2 + a) * G);
                            double2 &z2 = dd[a][j];
                            z2 = make_double2(fma(e.x, x2.x, fma(e.y, y2.x, z2.x)), fma(e.x, x2.y, fma(e.y, y2.y, z2.y)));
                        }
                    }
            }
            if (dip) {
                double2 hr[N], c[N];
#pragma unroll
                for (int l = 0; l < N; ++l) hr[l] = herm<N>(v + D::H0, mr, l);
                row_herm<N>(c, hr, v + D::Y);
                if (own)
#pragma unroll
                    for (int n = 0; n < N; ++n) v[D::T + m * D::LDT + n] = c[n];
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < NO; ++j) {
                if (m + G * j >= NU) continue;
                double2 c = make_double2(0.0, 0.0);
                if (dip) {
                    const double2 c1 = v[D::T + om[j] * D::LDT + on[j]], c2 = v[D::T + on[j] * D::LDT + om[j]];
                    c = make_double2(c1.x - c2.x, c1.y + c2.y);
                }
                const double2 y = v[D::Y + m + G * j];
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const double2 x = sx[a][j], d = dd[a][j];
                    sv[(a * NO + j) * 32] = x;
                    if (om[j] == on[j]) tot[a] += y.x * x.y - c.y * d.x;
                    else tot[a] -= 2.0 * (y.y * x.x - y.x * x.y) + 2.0 * (c.y * d.x - c.x * d.y);
                }
            }
            __syncwarp();
        }
        {   // row m of (H0 + E.D) Y
            double2 hr[N], c[N];
#pragma unroll
            for (int l = 0; l < N; ++l) hr[l] = herm<N>(v + D::HT, mr, l);
            row_herm<N>(c, hr, v + D::Y);
            if (own)
#pragma unroll
                for (int n = 0; n < N; ++n) v[D::T + m * D::LDT + n] = c[n];
        }
        __syncwarp();   // HT is free for the projection below
        if (deph || with_cur) {
            double2 p[N], q[N], y[N], d[N];   // rows of P_j, P_{j-1}, Y and D(Y)
            double t0 = 0.0, ty = 0.0;
#pragma unroll
            for (int n = 0; n < N; ++n) {
                p[n] = own ? herm<N>(v + D::H0, mr, n) : make_double2(0.0, 0.0);
                y[n] = own ? herm<N>(v + D::Y, mr, n) : make_double2(0.0, 0.0);
                q[n] = make_double2(0.0, 0.0);
                if (n == m) { t0 = p[n].x; ty = y[n].x; }
            }
            t0 = gsum<G>(t0) * (1.0 / N);
            ty = gsum<G>(ty) * (1.0 / N);
#pragma unroll
            for (int n = 0; n < N; ++n) {
                if (n == m) p[n].x -= t0;
                d[n] = make_double2(n == m ? ty : 0.0, 0.0);
            }
            double p2 = gsum<G>(row_dot<N>(p, p));
            const double py = gsum<G>(row_dot<N>(p, y));
            const double a2 = p2;
            double ip = p2 > 0.0 ? 1.0 / p2 : 0.0, b = 0.0;
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const double x = py * ip;
                d[n] = make_double2(fma(x, p[n].x, d[n].x), fma(x, p[n].y, d[n].y));
            }
#pragma unroll
            for (int j = 2; j < N; ++j) {
                double2 w[N];
                row_herm<N>(w, p, v + D::H0);
                const double a = gsum<G>(row_dot<N>(w, p)) * ip;
#pragma unroll
                for (int n = 0; n < N; ++n) {
                    w[n].x = fma(-a, p[n].x, fma(-b, q[n].x, w[n].x));
                    w[n].y = fma(-a, p[n].y, fma(-b, q[n].y, w[n].y));
                    if (j == 2 && n == m) w[n].x -= p2 * (1.0 / N);   // Tr(H0 P_1) / N
                    q[n] = p[n];
                }
                const double w2 = gsum<G>(row_dot<N>(w, w)), wy = gsum<G>(row_dot<N>(w, y));
                // a basis matrix that is rounding only (two bands meet) is left out
                const bool ok = w2 > 1e-26 * a2 * p2;
                b = w2 * ip;
                ip = ok ? 1.0 / w2 : 0.0;
                p2 = w2;
                const double x = wy * ip;
#pragma unroll
                for (int n = 0; n < N; ++n) {
                    p[n] = w[n];
                    d[n] = make_double2(fma(x, p[n].x, d[n].x), fma(x, p[n].y, d[n].y));
                }
                if (!ok)
#pragma unroll
                    for (int n = 0; n < N; ++n) p[n] = make_double2(0.0, 0.0);
            }
            if (own)
#pragma unroll
                for (int n = 0; n < N; ++n)
                    if (n >= m) v[D::HT + up(m, n, N)] = d[n];
        }
        __syncwarp();
        if (with_cur) {
            // intraband current Re Tr(D(Y) J_a) = Re Tr(D(Y) (-i S_a)): D(Y) commutes with H0
            double ii[2] = {0.0, 0.0};
            double *out = P.cur_part + (size_t)unit * WAN_NSLOT;
#pragma unroll
            for (int j = 0; j < NO; ++j) {
                if (m + G * j >= NU) continue;
                const double2 y = v[D::HT + m + G * j];
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const double2 x = sv[(a * NO + j) * 32];
                    if (om[j] == on[j]) ii[a] += y.x * x.y;
                    else ii[a] -= 2.0 * (y.y * x.x - y.x * x.y);
                }
            }
            const double w = live ? wk : 0.0;
            double z[4] = {w * (tot[0] - ii[0]), w * (tot[1] - ii[1]), w * ii[0], w * ii[1]};
            const bool h4 = lane & 16, h3 = lane & 8;
            double u0 = (h4 ? z[2] : z[0]) + __shfl_xor_sync(ALL, h4 ? z[0] : z[2], 16);
            double u1 = (h4 ? z[3] : z[1]) + __shfl_xor_sync(ALL, h4 ? z[1] : z[3], 16);
            double x = (h3 ? u1 : u0) + __shfl_xor_sync(ALL, h3 ? u0 : u1, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(ALL, x, o);
            if ((lane & 7) == 0) out[lane >> 3] = x;
            // occupations, and the element of the coherence file (antelope.cpp:539-542)
            const int ce = (P.nval * N + P.nval + 1) % NN;
            double oc = own ? w * v[D::Y + up(mr, mr, N)].x : 0.0;
            const double2 yc = herm<N>(v + D::Y, ce / N, ce % N);
            double co = m == 0 ? w * yc.x : m == 1 ? w * yc.y : 0.0;
#pragma unroll
            for (int o = 16; o >= G; o >>= 1) {
                oc += __shfl_xor_sync(ALL, oc, o);
                co += __shfl_xor_sync(ALL, co, o);
            }
            if (lane < N) out[4 + lane] = oc;
            if (lane < 2) out[4 + N + lane] = co;
        }
        // -i((HY) - (HY)^dag) - (g2 Y + (g1 - g2) D(Y)) at the owned elements (SBEs.h:808-861)
#pragma unroll
        for (int j = 0; j < NO; ++j) {
            const int u = min(m + G * j, NU - 1);
            const double2 c = v[D::T + om[j] * D::LDT + on[j]], c2 = v[D::T + on[j] * D::LDT + om[j]];
            double2 kn = make_double2(c.y + c2.y, c2.x - c.x);
            if (deph) {
                const double2 d = v[D::HT + u], y = v[D::Y + u];
                kn.x -= g2 * y.x + gd * d.x;
                kn.y -= g2 * y.y + gd * d.y;
            }
            if (om[j] == on[j]) kn.y = 0.0;
            if (s + 1 < S) ks[(s * NO + j) * 32 + lane] = kn;
            else kl[j] = kn;
        }
        __syncwarp();
    }
    // trial state and error estimate
    double2 *rout = P.rho[1 - buf] + (size_t)kc * NN;
#pragma unroll
    for (int j = 0; j < NO; ++j) {
        if (m + G * j >= NU || !live) continue;
        double2 inc = make_double2(0.0, 0.0), er = inc;
        for (int s = 0; s < S; ++s) {
            const double2 q = s + 1 < S ? ks[(s * NO + j) * 32 + lane] : kl[j];
            const double b = h * tb.b[s], e = h * tb.e[s];
            inc = make_double2(fma(b, q.x, inc.x), fma(b, q.y, inc.y));
            er = make_double2(fma(e, q.x, er.x), fma(e, q.y, er.y));
        }
        const double2 x = make_double2(r64[j].x + inc.x, r64[j].y + inc.y);
        __stcg(rout + om[j] * N + on[j], x);
        if (om[j] != on[j]) __stcg(rout + on[j] * N + om[j], cconj(x));
        emax = fmax(emax, sqrt(er.x * er.x + er.y * er.y));
    }
    if (P.rk == 45) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) emax = fmax(emax, __shfl_xor_sync(ALL, emax, o));
        // non-negative doubles order as their bits; a NaN's are above all
        if (lane == 0) atomicMax(P.gr_err, (unsigned long long)__double_as_longlong(fabs(emax)));
    }
}

// Between attempts: the sums of the attempt's outputs (fixed order), the step
// controller's decision -- every block takes it from the same numbers -- and
// the row tables of the next attempt, one (row, stage) item per block and
// turn.  The last block to finish moves the controller on; every block has
// read it by then.  `first`: tables of the first attempt only.
template <int N>
__global__ void __launch_bounds__(128) wan_next(const WanDev *__restrict__ Pp, const WanDev *const *__restrict__ descs,
                                                bool first)
{
    using D = PD<N>;
    constexpr int G = D::G, NU = D::NU, NO = D::NO, NN = D::NN;
    __shared__ __align__(16) unsigned char sp[sizeof(WanDev)];
    __shared__ WanCtl c;
    __shared__ double AE[6][6], red[128];
    __shared__ double2 pr[WAN_MAXR], ph[WAN_MAXR];
    __shared__ int idx[WAN_MAXR];
    __shared__ double V[2 * WAN_MAXR];
    // the descriptor, the controller and the vectors come in one round trip each:
    // the launch is a chain of latencies
    const WanDev *Pg = descs ? descs[blockIdx.y] : Pp;
    const int t = threadIdx.x;
    static_assert(sizeof(WanDev) % 8 == 0, "copied in 8-byte words");
    for (int i = t; i < (int)(sizeof(WanDev) / 8); i += blockDim.x)
        reinterpret_cast<unsigned long long *>(sp)[i] = reinterpret_cast<const unsigned long long *>(Pg)[i];
    __syncthreads();
    const WanDev &P = *reinterpret_cast<const WanDev *>(sp);
    if (t < (int)(sizeof(WanCtl) / 8))
        reinterpret_cast<unsigned long long *>(&c)[t] = reinterpret_cast<const unsigned long long *>(P.ctl)[t];
    const double emax = first ? 0.0 : __longlong_as_double((long long)*P.gr_err);
    for (int i = t; i < 2 * P.nR; i += blockDim.x) V[i] = P.V[i];
    if (t < P.nR) idx[t] = P.gr_idx[t];
    __syncthreads();
    if (c.done) {
        if (blockIdx.x == 0 && t == 0) P.ctl->shot = -1;   // a snapshot is taken once
        return;
    }
    const PTab &tb = c_tab[tab_of(P.rk)];
    const int S = tb.S;
    // phases of every vector at a row's k (f = 0)
    auto row_phases = [&](int item) {
        const int row = item / S, N0 = P.gr_fast ? P.Ngrid[0] : 1;
        const double f0 = N0 == 1 ? 0.0 : double(P.gr_row0 + row) / (N0 - 1) - 0.5;
        for (int r = t; r < P.nR; r += blockDim.x) {
            const double kx = P.origin[0] + f0 * P.axes[0], ky = P.origin[1] + f0 * P.axes[1];
            double sn, cs;
            sincos(kx * V[2 * r] + ky * V[2 * r + 1], &sn, &cs);
            pr[r] = make_double2(cs, sn);
        }
    };
    const int need_current = c.need_current, n = c.n;
    __syncthreads();
    // the decision, by the last thread, while the others start on the row
    if (!first && t == (int)blockDim.x - 1) control_decide(P, &c, emax);
    row_phases(blockIdx.x);
    if (!first && need_current) {
        const int nu = (P.nk + D::KW - 1) / D::KW;
        for (int slot = blockIdx.x; slot < 6 + N; slot += gridDim.x) {
            const double *p = P.cur_part + slot;
            double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
            int i = t;
            for (; i + 384 < nu; i += 512) {
                s0 += p[(size_t)i * WAN_NSLOT];
                s1 += p[(size_t)(i + 128) * WAN_NSLOT];
                s2 += p[(size_t)(i + 256) * WAN_NSLOT];
                s3 += p[(size_t)(i + 384) * WAN_NSLOT];
            }
            for (; i < nu; i += 128) s0 += p[(size_t)i * WAN_NSLOT];
            red[t] = (s0 + s1) + (s2 + s3);
            __syncthreads();
            for (int o = 64; o > 0; o >>= 1) {
                if (t < o) red[t] += red[t + o];
                __syncthreads();
            }
            if (t == 0) P.jout[(size_t)n * WAN_NSLOT + slot] = red[0];
            __syncthreads();
        }
    }
    __syncthreads();
    if (!c.done) {
        const int ng = P.gr_n, nent = 2 * ng - 1;
        const bool dip = P.has_dip;
        const int NQ = dip ? 2 : 1, NC = dip ? 4 : 2;
        if (t < S) laser_eval(P.laser, t == 0 ? c.tc : c.tc + tb.c[t] * c.hs, &AE[t][0], &AE[t][3]);
        const double2 *h = static_cast<const double2 *>(P.h), *d = static_cast<const double2 *>(P.d);
        for (int item = blockIdx.x; item < P.gr_rows * S; item += gridDim.x) {
            const int row = item / S, s = item % S;
            __syncthreads();
            if (item != (int)blockIdx.x) row_phases(item);
            // times the stage's e^{iA.R}
            for (int r = t; r < P.nR; r += blockDim.x) {
                double sn, cs;
                sincos(AE[s][0] * V[2 * r] + AE[s][1] * V[2 * r + 1], &sn, &cs);
                ph[r] = cmul(pr[r], make_double2(cs, sn));
            }
            __syncthreads();
            const bool cur = s == 0 && c.need_current;
            const double ex = AE[s][3], ey = AE[s][4];
            double2 *out = P.gr_tab + (size_t)item * nent * NO * NQ * G;
            double2 *oc = P.gr_cur + (size_t)row * nent * NO * NC * G;
            for (int w = t; w < ng * NU; w += blockDim.x) {
                const int q = w / NU, u = w % NU;
                int mu = u, a = 0;
                while (mu >= N - a) { mu -= N - a; ++a; }
                const int e = a * N + a + mu;
                double2 x[2][6];   // h, E.D, S_x, S_y, D_x, D_y of the group at +g and -g
#pragma unroll
                for (int z = 0; z < 2; ++z) {
#pragma unroll
                    for (int y = 0; y < 6; ++y) x[z][y] = make_double2(0.0, 0.0);
                    const int i1 = P.gr_off[2 * q + z + 1];
#pragma unroll 4
                    for (int i = P.gr_off[2 * q + z]; i < i1; ++i) {
                        const int r = idx[i];
                        const double2 hp = cmul(h[(size_t)r * NN + e], ph[r]);
                        x[z][0] = make_double2(x[z][0].x + hp.x, x[z][0].y + hp.y);
                        if (dip) {
                            cfma(x[z][4], d[((size_t)r * 2) * NN + e], ph[r]);
                            cfma(x[z][5], d[((size_t)r * 2 + 1) * NN + e], ph[r]);
                        }
                        if (cur) {
                            const double vx = V[2 * r], vy = V[2 * r + 1];
                            x[z][2] = make_double2(fma(vx, hp.x, x[z][2].x), fma(vx, hp.y, x[z][2].y));
                            x[z][3] = make_double2(fma(vy, hp.x, x[z][3].x), fma(vy, hp.y, x[z][3].y));
                        }
                    }
                    x[z][1] = make_double2(fma(ey, x[z][5].x, ex * x[z][4].x), fma(ey, x[z][5].y, ex * x[z][4].y));
                }
                const int j = u / G, l = u % G;
                // sig = G_g + G_-g, tau = i (G_g - G_-g); the group g = 0 is sig alone
                auto store = [&](double2 *o, int nq, int y, const double2 &xp, const double2 &xm) {
                    if (q == 0) {
                        o[(size_t)(j * nq + y) * G + l] = xp;
                    } else {
                        o[((size_t)((2 * q - 1) * NO + j) * nq + y) * G + l] = make_double2(xp.x + xm.x, xp.y + xm.y);
                        o[((size_t)(2 * q * NO + j) * nq + y) * G + l] = make_double2(xm.y - xp.y, xp.x - xm.x);
                    }
                };
                store(out, NQ, 0, x[0][0], x[1][0]);
                if (dip) store(out, NQ, 1, x[0][1], x[1][1]);
                if (cur) {
                    store(oc, NC, 0, x[0][2], x[1][2]);
                    store(oc, NC, 1, x[0][3], x[1][3]);
                    if (dip) {
                        store(oc, NC, 2, x[0][4], x[1][4]);
                        store(oc, NC, 3, x[0][5], x[1][5]);
                    }
                }
            }
        }
    }
    if (first) return;
    __syncthreads();
    if (t == 0) {
        __threadfence();
        if (atomicAdd(P.step_ticket, 1u) == gridDim.x - 1) {
            *P.step_ticket = 0u;
            *P.gr_err = 0ull;
            *P.ctl = c;
        }
    }
}

// ============================================================= launchers
bool wan_proj_applies(const WanDev &w)
{
    return !w.mixed && !w.vg && !w.cont && !w.has_jtab && !w.degenerate && w.N >= 3 && w.N <= 6 && w.nR >= 1 &&
           w.Ngrid[2] == 1;
}
bool wan_proj(const WanDev &w) { return w.gr_tab != nullptr && wan_proj_applies(w); }

// Entries of the row tables per row (gr_tab has one set per stage)
int wan_proj_entries(int N, int ngrp, int nq)
{
    const int G = N <= 4 ? 4 : 8;
    return (2 * ngrp - 1) * ((N * (N + 1) / 2 + G - 1) / G) * nq * G;
}
int wan_proj_unit(int N) { return N <= 4 ? 2 : 1; }   // tiles per block

template <int N>
static cudaError_t proj_attempt(const WanDev *dw, const WanDev *const *descs, const WanTileRef *tiles, int nblocks,
                                int ngrp, cudaStream_t st)
{
    const int grid = tiles ? nblocks : (nblocks + SPREAD - 1) / SPREAD * SPREAD;
    wan_attempt_p<N><<<grid, 32, proj_bytes<N>(ngrp), st>>>(dw, descs, tiles);
    return cudaGetLastError();
}
cudaError_t launch_wan_attempt_p(int N, int ngrp, const WanDev *dw, const WanDev *const *descs, const WanTileRef *tiles,
                                 int nblocks, cudaStream_t st)
{
    if (nblocks <= 0) return cudaSuccess;
    switch (N) {
    case 3: return proj_attempt<3>(dw, descs, tiles, nblocks, ngrp, st);
    case 4: return proj_attempt<4>(dw, descs, tiles, nblocks, ngrp, st);
    case 5: return proj_attempt<5>(dw, descs, tiles, nblocks, ngrp, st);
    case 6: return proj_attempt<6>(dw, descs, tiles, nblocks, ngrp, st);
    default: return cudaErrorInvalidValue;
    }
}
cudaError_t launch_wan_next(int N, const WanDev *dw, const WanDev *const *descs, int nsolves, int nitems, bool first,
                            cudaStream_t st)
{
    const dim3 grid(std::min(nitems, 1184), nsolves);   // 8 blocks of 128 threads per SM
    switch (N) {
    case 3: wan_next<3><<<grid, 128, 0, st>>>(dw, descs, first); break;
    case 4: wan_next<4><<<grid, 128, 0, st>>>(dw, descs, first); break;
    case 5: wan_next<5><<<grid, 128, 0, st>>>(dw, descs, first); break;
    case 6: wan_next<6><<<grid, 128, 0, st>>>(dw, descs, first); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace sbe
