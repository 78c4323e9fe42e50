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
//    eigenvectors -- over a 100 x 100 grid of N = 6 models D(Y) is within 1.5e-14
//    of the eigensolver's, its own rounding over the smallest gap -- except where
//    three or more bands crowd (bands_crowd); those k-points go by eigenvectors.
//  - Fourier sums in two levels.  A row of the grid has k = k_row + f b, so the
//    vectors R with equal b.R share their phase along the row: with G_g =
//    sum of h_R e^{i(k_row + A).R} over such a group, H0(k + A) = sum_g G_g
//    e^{i f g} has 7 terms instead of 37 on the N = 6 model's vectors.  wan_next
//    forms the G (and those of E.D) of every row and stage between attempts.
//    FP64 method only: the mixed method keeps its FP32 sums over the pairs.
//
// Layout: one warp per block; N/2 lanes per k-point for even N, two rows of its
// matrices each, and N lanes for odd N, one row each (PD below): 10 k-points per
// warp at N = 6.  All lanes work, only the kept half of each Hermitian product is
// formed, and an element read from shared memory serves two rows.  That read was
// the limit of one row per lane in groups of 8 (a 16-byte element at one address
// per group costs 4 wavefronts, whatever the number of groups; 4 k-points per
// warp, 6 of 8 lanes at work): Cash-Karp attempts of N = 6, 4, 3 on 200 x 300
// points took 681, 251 and 144 us, now 380, 141 and 111; on 100 x 100 162, 82 and
// 52, now 88, 52 and 46; on 8 x 8 68, 61 and 41, now 65, 42 and 38.  What does not
// fit the 255 registers of N = 6 stays in shared memory (the slope while the
// projection adds to it) or is read again (the state): 11 and 6 % more with both
// kept, their spills missing an L1 that the blocks' shared memory leaves 28 KB.
// Bound: latencies at two warps a scheduler; FP64 issue a quarter to a third of
// the time.
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

// A k-point's G lanes share its Hermitian matrices by circulant diagonals: lane m
// owns row m (and m + N/2 when N is even) of the elements (r, r + d mod N), d <=
// N/2 -- of the diagonal d = N/2 of an even N the rows r < N/2 only.  Every lane
// then has the same elements relative to its row, and equal work.
template <int N> struct PD {
    static constexpr bool EVEN = N % 2 == 0;
    static constexpr int M = N / 2, G = EVEN ? M : N, KW = 32 / G, LW = KW * G, NN = N * N;
    static constexpr int DO = EVEN ? N - 1 : M;   // owned elements off the diagonal
    static constexpr int NE = DO + 1;             // entries of an owned set; the last: its diagonal elements
    static constexpr int NM = (M + 1) * N;        // slots [d][r] of a matrix (d = N/2 of an even N twice)
    // a k-point's two matrices in complex numbers: Y, then H0; H0 + E.D (T, P); the
    // stride puts the lanes of a warp's groups on distinct banks
    static constexpr int Y = 0, HT = NM;
    static constexpr int END = 2 * NM + (N == 5 ? 5 : N == 3 ? 1 : N == 6 ? 3 : 2);
    static constexpr int TN = (N - 1 - M) * N;    // slots of the product's unowned elements
    __host__ __device__ static constexpr int slot(int d, int r) { return d * N + r; }
};

// o += a x (conj(x) if CJ), of numbers known real (ar, xr) and of the parts of
// o that are wanted; all four known when the loops are unrolled
__device__ __forceinline__ void mac(double2 &o, const double2 &a, bool ar, const double2 &x, bool xr, bool cj, bool re, bool im)
{
    if (re) {
        o.x = fma(a.x, x.x, o.x);
        if (!ar && !xr) o.x = fma(cj ? a.y : -a.y, x.y, o.x);
    }
    if (im) {
        if (!xr) o.y = fma(cj ? -a.x : a.x, x.y, o.y);
        if (!ar) o.y = fma(a.y, x.x, o.y);
    }
}
// Tr(XY) of a lane's owned elements: three chains
template <int N> __device__ __forceinline__ double dot(const double2 (&a)[PD<N>::NE], const double2 (&b)[PD<N>::NE])
{
    constexpr int DO = PD<N>::DO;
    double s = 0.0, t = 0.0;
#pragma unroll
    for (int j = 0; j < DO; ++j) {
        s = fma(a[j].x, b[j].x, s);
        t = fma(a[j].y, b[j].y, t);
    }
    double u = a[DO].x * b[DO].x;
    if (PD<N>::EVEN) u = fma(a[DO].y, b[DO].y, u);
    return fma(2.0, s + t, u);
}
// sum over a group's lanes, in lane order (the same bits in every lane)
template <int G> __device__ __forceinline__ double gsum(double v, int base)
{
    double s = __shfl_sync(ALL, v, base);
#pragma unroll
    for (int i = 1; i < G; ++i) s += __shfl_sync(ALL, v, base + i);
    return s;
}
// an owned set to its slots
template <int N> __device__ __forceinline__ void put(double2 *P, const double2 (&x)[PD<N>::NE], int m)
{
    using D = PD<N>;
#pragma unroll
    for (int d = 1; d <= D::M; ++d) P[D::slot(d, m)] = x[d - 1];
    P[m].x = x[D::DO].x;
    if (D::EVEN) {
        P[D::slot(D::M, m + D::M)] = cconj(x[D::M - 1]);
#pragma unroll
        for (int d = 1; d < D::M; ++d) P[D::slot(d, m + D::M)] = x[D::M + d - 1];
        P[m + D::M].x = x[D::DO].y;
    }
}
// element (l, c) relative to the lane's row: ro[i] = (m + i) mod N
template <int N> __device__ __forceinline__ double2 elem(const double2 *P, const int (&ro)[N], int l, int c)
{
    using D = PD<N>;
    const int d = (c - l + N) % N;
    if (d == 0) return make_double2(P[ro[l]].x, 0.0);
    if (d <= D::M) return P[D::slot(d, ro[l])];
    return cconj(P[D::slot(N - d, ro[c])]);
}
// the lane's rows of a matrix, columns relative to row m
template <int N> struct Rows {
    double2 a[N], b[N];   // row m, row m + N/2
    __device__ __forceinline__ void load(const double2 *P, const int (&ro)[N])
    {
#pragma unroll
        for (int c = 0; c < N; ++c) {
            a[c] = elem<N>(P, ro, 0, c);
            if (PD<N>::EVEN) b[c] = elem<N>(P, ro, PD<N>::M, c);
        }
    }
};
// w = (H P) at the owned elements (H, P commute: the product is Hermitian); each
// element of P is read once
template <int N>
__device__ __forceinline__ void product(double2 (&w)[PD<N>::NE], const Rows<N> &H, const double2 *P, const int (&ro)[N])
{
    using D = PD<N>;
    constexpr int M = D::M;
    double2 oa[N], ob[N];
#pragma unroll
    for (int c = 0; c < N; ++c) oa[c] = ob[c] = make_double2(0.0, 0.0);
    // columns a lane keeps: of row m 0 .. N/2, of row m + N/2 the N/2 from its own
    auto add = [&](int l, int c, const double2 &x, bool cj) {   // the term of column c with H's element l
        if (c <= M) mac(oa[c], H.a[l], l == 0, x, l == c, cj, true, c != 0);
        const int d = (c - M + N) % N;
        if (D::EVEN && d < M) mac(ob[c], H.b[l], l == M, x, l == c, cj, true, d != 0);
    };
#pragma unroll
    for (int l = 0; l < N; ++l)
#pragma unroll
        for (int c = l; c < N; ++c) {
            const double2 x = elem<N>(P, ro, l, c);
            add(l, c, x, false);
            if (l != c) add(c, l, x, true);
        }
#pragma unroll
    for (int d = 1; d <= M; ++d) w[d - 1] = oa[d];
    w[D::DO] = make_double2(oa[0].x, 0.0);
    if (D::EVEN) {
#pragma unroll
        for (int d = 1; d < M; ++d) w[M + d - 1] = ob[(M + d) % N];
        w[D::DO].y = ob[M].x;
    }
}
// c = (H Y) - (H Y)^dag at the owned elements, its imaginary diagonal in the last
// entry; T: room for the elements that other lanes need (may be H's own slots)
template <int N>
__device__ __forceinline__ void commutator(double2 (&w)[PD<N>::NE], const double2 *Hs, const double2 *Y, double2 *T,
                                           const int (&ro)[N])
{
    using D = PD<N>;
    constexpr int M = D::M;
    Rows<N> H;
    H.load(Hs, ro);
    double2 oa[N], ob[N];
#pragma unroll
    for (int c = 0; c < N; ++c) oa[c] = ob[c] = make_double2(0.0, 0.0);
    auto add = [&](int l, int c, const double2 &x, bool cj) {
        mac(oa[c], H.a[l], l == 0, x, l == c, cj, c != 0, true);
        if (D::EVEN) mac(ob[c], H.b[l], l == M, x, l == c, cj, c != M, true);
    };
#pragma unroll
    for (int l = 0; l < N; ++l)
#pragma unroll
        for (int c = l; c < N; ++c) {
            const double2 x = elem<N>(Y, ro, l, c);
            add(l, c, x, false);
            if (l != c) add(c, l, x, true);
        }
    __syncwarp();
#pragma unroll
    for (int d = M + 1; d < N; ++d) {
        T[(d - M - 1) * N + ro[0]] = oa[d];
        if (D::EVEN) T[(d - M - 1) * N + ro[M]] = ob[(M + d) % N];
    }
    __syncwarp();
    auto diff = [](const double2 &x, const double2 &y) { return make_double2(x.x - y.x, x.y + y.y); };
#pragma unroll
    for (int d = 1; d <= M; ++d)
        w[d - 1] = diff(oa[d], D::EVEN && d == M ? ob[0] : T[(N - d - M - 1) * N + ro[d]]);
    w[D::DO] = make_double2(2.0 * oa[0].y, 0.0);
    if (D::EVEN) {
#pragma unroll
        for (int d = 1; d < M; ++d) w[M + d - 1] = diff(ob[(M + d) % N], T[(N - d - M - 1) * N + ro[(M + d) % N]]);
        w[D::DO].y = 2.0 * ob[M].y;
    }
    __syncwarp();
}
// Re Tr(X (-i S)) of the owned elements, S anti-Hermitian with its imaginary
// diagonal in the last entry
template <int N>
__device__ __forceinline__ double tr_s(const double2 (&x)[PD<N>::NE], const double2 (&s)[PD<N>::NE])
{
    constexpr int DO = PD<N>::DO;
    double t = 0.0;
#pragma unroll
    for (int j = 0; j < DO; ++j) t += x[j].y * s[j].x - x[j].x * s[j].y;
    double u = x[DO].x * s[DO].x;
    if (PD<N>::EVEN) u += x[DO].y * s[DO].y;
    return u - 2.0 * t;
}


// D(Y) by eigenvectors, for the k-points where bands crowd, the groups of the warp at
// once: Jacobi rotations of A until it is diagonal and of Y along with it, then Y's
// diagonal back through them.  In a round a lane has one of the N/2 disjoint pairs
// and keeps its rotation; the blocks between two pairs (and, of odd N, between a pair
// and the row left over) are dealt out to the group's lanes.  Two matrices of room,
// no eigenvectors kept.
template <int N> struct Slots {   // elements of a Hermitian matrix in its slots, each kept once
    using D = PD<N>;
    double2 *P;
    __device__ __forceinline__ double2 *at(int r, int c, bool &cj) const
    {
        const int d = c >= r ? c - r : c - r + N;
        cj = d > D::M || (D::EVEN && d == D::M && r >= D::M);
        return P + (cj ? D::slot(N - d, c) : D::slot(d, r));
    }
    __device__ __forceinline__ double2 get(int r, int c) const
    {
        bool cj;
        const double2 x = *at(r, c, cj);
        return cj ? cconj(x) : x;
    }
    __device__ __forceinline__ void set(int r, int c, const double2 &x) const
    {
        bool cj;
        double2 *p = at(r, c, cj);
        *p = cj ? cconj(x) : x;
    }
};
// The row at place x of round rd (pair i: places 2 i and 2 i + 1), round robin
template <int N> __device__ __forceinline__ int round_row(int rd, int x)
{
    constexpr int n = N % 2 ? N : N - 1;
    if (N % 2 == 0 && x == 1) return N - 1;
    const int j = (x >> 1) + N % 2, y = x == N - 1 && N % 2 ? rd : rd + (x & 1 ? n - j : j);
    return y >= n ? y - n : y;
}
// A round's rotations on the blocks off the pairs of X (and of X2)
template <int N, int NM>
__device__ __forceinline__ void turn_blocks(const Slots<N> (&X)[NM], int rd, const Turn &own, int m, int base, bool work)
{
    constexpr int NP = N / 2, NB = NP * (NP - 1) / 2, NT = NB + N % 2 * NP, G = PD<N>::G;
#pragma unroll 1
    for (int x0 = 0; x0 < NM * NT; x0 += G) {
        const int x = min(x0 + m, NM * NT - 1), e = x % NT;
        const int i = e < NB ? (NP == 3 && e == 2) : e - NB, j = e < NB ? (NP == 3 ? min(e + 1, 2) : 1) : NP;
        Turn ti, tj;
        ti.c = __shfl_sync(ALL, own.c, base + i);
        ti.s = make_double2(__shfl_sync(ALL, own.s.x, base + i), __shfl_sync(ALL, own.s.y, base + i));
        tj.c = __shfl_sync(ALL, own.c, base + min(j, NP - 1));
        tj.s = make_double2(__shfl_sync(ALL, own.s.x, base + min(j, NP - 1)), __shfl_sync(ALL, own.s.y, base + min(j, NP - 1)));
        if (!work || x0 + m >= NM * NT) continue;
        const Slots<N> Z = NM == 1 || x < NT ? X[0] : X[NM - 1];
        const int p = round_row<N>(rd, 2 * i), q = round_row<N>(rd, 2 * i + 1), r = round_row<N>(rd, 2 * j);
        double2 pr = Z.get(p, r), qr = Z.get(q, r);
        if (j < NP) {
            const int u = round_row<N>(rd, 2 * j + 1);
            double2 pu = Z.get(p, u), qu = Z.get(q, u);
            tj.on(pr, pu, tj.s);
            tj.on(qr, qu, tj.s);
            ti.on(pu, qu, cconj(ti.s));
            Z.set(p, u, pu);
            Z.set(q, u, qu);
        }
        ti.on(pr, qr, cconj(ti.s));
        Z.set(p, r, pr);
        Z.set(q, r, qr);
    }
}
// at: the group's matrices in shared memory, A in the second slots and Y in the
// first; D(Y) is left in the second.  Groups without `work` only pass through.
template <int N> __device__ __noinline__ void eigen_diagonal(int at, int m, int base, bool work)
{
    using D = PD<N>;
    constexpr int NP = N / 2, NR = N % 2 ? N : N - 1, G = D::G;
    extern __shared__ __align__(16) double2 sm[];
    double2 *const v = sm + at;
    const Slots<N> AY[2] = {{v + D::HT}, {v + D::Y}}, A[1] = {{v + D::HT}};
    Turn rot[MAX_SWEEPS * NR];
    const bool mine = work && m < NP;
    const int place = 2 * min(m, NP - 1);
    int n = 0;
#pragma unroll 1
    for (int sweep = 0; sweep < MAX_SWEEPS; ++sweep) {
        double off = 0.0, all = 0.0;
#pragma unroll 1
        for (int e = m; e < N * N; e += G) {
            const double2 z = A[0].get(e / N, e % N);
            const bool diag = e / N == e % N;
            const double q = diag ? z.x * z.x : fma(z.x, z.x, z.y * z.y);
            all += q;
            off += diag ? 0.0 : q;
        }
        off = gsum<G>(off, base);
        all = gsum<G>(all, base);
        if (!__any_sync(ALL, work && off > 1e-36 * all)) break;
#pragma unroll 1
        for (int rd = 0; rd < NR; ++rd, ++n) {
            const int p = round_row<N>(rd, place), q = round_row<N>(rd, place + 1);
            Turn t;
            t.c = 1.0;
            t.s = make_double2(0.0, 0.0);
            if (mine) {
                double dl, a = v[D::Y + p].x, b = v[D::Y + q].x;
                double2 z = AY[1].get(p, q);
                t.find(v[D::HT + p].x, v[D::HT + q].x, A[0].get(p, q), dl);
                v[D::HT + p].x -= dl;
                v[D::HT + q].x += dl;
                A[0].set(p, q, make_double2(0.0, 0.0));
                t.own(a, z, b);
                v[D::Y + p].x = a;
                v[D::Y + q].x = b;
                AY[1].set(p, q, z);
            }
            rot[n] = t;
            turn_blocks<N, 2>(AY, rd, t, m, base, work);
            __syncwarp();
        }
    }
    if (work)
        for (int e = m; e < D::NM; e += G) v[D::HT + e] = make_double2(e < N ? v[D::Y + e].x : 0.0, 0.0);
    __syncwarp();
#pragma unroll 1
    while (n > 0) {   // D = V D' V^dag, the last rotation first
        const int rd = --n % NR, p = round_row<N>(rd, place), q = round_row<N>(rd, place + 1);
        Turn t = rot[n];
        t.s = make_double2(-t.s.x, -t.s.y);
        if (mine) {
            double a = v[D::HT + p].x, b = v[D::HT + q].x;
            double2 z = A[0].get(p, q);
            t.own(a, z, b);
            v[D::HT + p].x = a;
            v[D::HT + q].x = b;
            A[0].set(p, q, z);
        }
        turn_blocks<N, 1>(A, rd, t, m, base, work);
        __syncwarp();
    }
}

}  // namespace

// Shared memory of a block: slopes, the groups' matrices, the phases along the row
template <int N> static int proj_bytes(int ngrp, int S)
{
    using D = PD<N>;
    return (S * D::NE * 32 + D::KW * D::END + D::KW * ngrp) * 16;
}

// One attempted step of a unit of KW k-points; false: bands crowd at a stage of one
// of them, and nothing but current sums was written.  EIG: those k-points by
// eigenvectors, in a pass of its own (with the call in the first pass N = 6 took 390
// us an attempt of 200 x 300 points, with the check alone 380, without 367).
template <int N, bool EIG>
__device__ __forceinline__ bool attempt(const WanDev &P, int unit)
{
    extern __shared__ __align__(16) double2 sm[];
    using D = PD<N>;
    constexpr int G = D::G, KW = D::KW, LW = D::LW, NE = D::NE, DO = D::DO, M = D::M, NN = D::NN;
    const WanCtl &ctl = *P.ctl;
    // lanes past the last group shadow its first lanes: same values, to the same
    // addresses where the group shares them
    const int lane = threadIdx.x, grp = min(lane / G, KW - 1), m = lane < LW ? lane % G : lane - LW;
    const int base = grp * G;
    const int k = unit * KW + grp;
    const bool live = k < P.nk && lane < LW;
    const int kc = min(k, P.nk - 1);   // a group past the grid shadows the last k-point
    const int S = c_tab[tab_of(P.rk)].S;
    double2 *const ks = sm + lane;                               // [S][NE][32] slopes, a column per lane
    double2 *const v = sm + S * NE * 32 + grp * D::END;
    constexpr int CR = 2 * D::NM;                                // past the matrices: |H0|^2; have bands crowded?
    if (N > 3 && m == 0) v[CR].y = 0.0;
    const int ng = P.gr_n, nent = 2 * ng - 1;                    // group pairs (g = 0 first), table entries
    double2 *const ph = sm + S * NE * 32 + KW * D::END + grp * ng;
    const double h = ctl.hs;
    const int buf = ctl.buf;
    const bool cur = ctl.need_current;
    const PTab &tb = c_tab[tab_of(P.rk)];
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
    int ro[N];   // rows and columns relative to the lane's row
#pragma unroll
    for (int i = 0; i < N; ++i) ro[i] = m + i < N ? m + i : m + i - N;
    // the owned element j < DO: row m (m + N/2) and its column
    auto erow = [&](int j) { return j < M ? ro[0] : ro[M % N]; };
    auto ecol = [&](int j) { return j < M ? ro[j + 1] : ro[(j + 1) % N]; };
    // the state's owned elements; at N = 6 read again at each stage: they do not
    // fit the registers beside the projection's matrices
    constexpr bool KEEP = N < 6;
    const double2 *rho = P.rho[buf] + (size_t)kc * NN;
    auto state = [&](double2 (&r)[NE]) {
#pragma unroll
        for (int j = 0; j < DO; ++j) {
            const int a = erow(j), b = ecol(j);
            r[j] = __ldcg(rho + min(a, b) * N + max(a, b));
            if (a > b) r[j].y = -r[j].y;
        }
        r[DO].x = __ldcg(&rho[m * (N + 1)].x);
        r[DO].y = D::EVEN ? __ldcg(&rho[(m + M) * (N + 1)].x) : 0.0;
    };
    double2 r64[NE];
    if (KEEP) state(r64);
    const bool dip = P.has_dip;
    const int NQ = dip ? 2 : 1;
    const double g1 = P.g1, g2 = P.g2, gd = g1 - g2;
    const bool deph = g1 != 0.0 || g2 != 0.0;
    const size_t ent = (size_t)nent * NE * NQ * G;   // table entries of a (row, stage)
    const double2 *tab = P.gr_tab + (size_t)row * S * ent + m;
    __syncwarp();

#pragma unroll 1
    for (int s = 0; s < S; ++s, tab += ent) {
        // H0 and E.D at the owned elements
        double2 y[NE], a0[NE], a1[NE];
        if (!KEEP) state(y);
        {
#pragma unroll
            for (int j = 0; j < NE; ++j) {
                a0[j] = __ldg(tab + (size_t)j * NQ * G);
                a1[j] = dip ? __ldg(tab + (size_t)(j * NQ + 1) * G) : make_double2(0.0, 0.0);
            }
#pragma unroll 1
            for (int q = 1; q < ng; ++q) {
                const double2 e = ph[q];
                const double2 *t0 = tab + (size_t)(2 * q - 1) * NE * NQ * G, *t1 = t0 + (size_t)NE * NQ * G;
#pragma unroll
                for (int j = 0; j < NE; ++j) {
                    const double2 sg = __ldg(t0 + j * NQ * G), ta = __ldg(t1 + j * NQ * G);
                    a0[j] = make_double2(fma(e.x, sg.x, fma(e.y, ta.x, a0[j].x)), fma(e.x, sg.y, fma(e.y, ta.y, a0[j].y)));
                    if (dip) {
                        const double2 sd = __ldg(t0 + (j * NQ + 1) * G), td = __ldg(t1 + (j * NQ + 1) * G);
                        a1[j] = make_double2(fma(e.x, sd.x, fma(e.y, td.x, a1[j].x)), fma(e.x, sd.y, fma(e.y, td.y, a1[j].y)));
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < NE; ++j) a1[j] = make_double2(a0[j].x + a1[j].x, a0[j].y + a1[j].y);
        }
        // stage input Y = rho + h sum_j a_sj k_j
        if (KEEP)
#pragma unroll
            for (int j = 0; j < NE; ++j) y[j] = r64[j];
#pragma unroll 1
        for (int i = 0; i < s; ++i) {
            const double a = h * tb.a[s][i];
#pragma unroll
            for (int j = 0; j < NE; ++j) {
                const double2 q = ks[(i * NE + j) * 32];
                y[j] = make_double2(fma(a, q.x, y[j].x), fma(a, q.y, y[j].y));
            }
        }
        const bool with_cur = cur && s == 0;
        put<N>(v + D::Y, y, m);
        if (!with_cur) put<N>(v + D::HT, a1, m);
        else put<N>(v + D::HT, a0, m);
        __syncwarp();
        double tot[2] = {0.0, 0.0};
        if (with_cur) {
            // total current Re Tr(Y J_a), J_a = -i S_a + i [D_a, H0] (S_a = sum R_a h_R
            // e^{iKR}): over the owned elements, with C = H0 Y - (H0 Y)^dag, the
            // diagonal Y_mm Im(S_mm) - Im(C_mm) Re(D_mm), off it -2 Im(Y_mn conj(S_mn))
            // - 2 Im(C_mn conj(D_mn)).  S_a, T and H0 + E.D wait in the columns of
            // slopes that do not exist yet.
            const int NC = dip ? 4 : 2;   // S_x, S_y (, D_x, D_y)
            const double2 *tc = P.gr_cur + (size_t)row * nent * NE * NC * G + m;
            double2 c[NE];
#pragma unroll
            for (int j = 0; j < NE; ++j) ks[(3 * NE + j) * 32] = a1[j];
            if (dip) commutator<N>(c, v + D::HT, v + D::Y, sm + grp * D::TN, ro);
#pragma unroll 1
            for (int a = 0; a < 2; ++a) {
                double2 x[NE], d[NE];
#pragma unroll
                for (int j = 0; j < NE; ++j) {
                    x[j] = __ldg(tc + (size_t)(j * NC + a) * G);
                    d[j] = dip ? __ldg(tc + (size_t)(j * NC + 2 + a) * G) : make_double2(0.0, 0.0);
                }
#pragma unroll 1
                for (int q = 1; q < ng; ++q) {
                    const double2 e = ph[q];
                    const double2 *t0 = tc + (size_t)(2 * q - 1) * NE * NC * G, *t1 = t0 + (size_t)NE * NC * G;
#pragma unroll
                    for (int j = 0; j < NE; ++j) {
                        const double2 x1 = __ldg(t0 + (j * NC + a) * G), y1 = __ldg(t1 + (j * NC + a) * G);
                        x[j] = make_double2(fma(e.x, x1.x, fma(e.y, y1.x, x[j].x)), fma(e.x, x1.y, fma(e.y, y1.y, x[j].y)));
                        if (dip) {
                            const double2 x2 = __ldg(t0 + (j * NC + 2 + a) * G), y2 = __ldg(t1 + (j * NC + 2 + a) * G);
                            d[j] = make_double2(fma(e.x, x2.x, fma(e.y, y2.x, d[j].x)), fma(e.x, x2.y, fma(e.y, y2.y, d[j].y)));
                        }
                    }
                }
                double t = tr_s<N>(y, x);
                if (dip) {
                    double u = 0.0;
#pragma unroll
                    for (int j = 0; j < DO; ++j) u += c[j].y * d[j].x - c[j].x * d[j].y;
                    t -= 2.0 * u + c[DO].x * d[DO].x;
                    if (D::EVEN) t -= c[DO].y * d[DO].y;
                }
#pragma unroll
                for (int j = 0; j < NE; ++j) ks[((a + 1) * NE + j) * 32] = x[j];
                if (a == 0) tot[0] = t;
                else tot[1] = t;
            }
            double *out = P.cur_part + (size_t)unit * WAN_NSLOT;
            const double w = live ? wk : 0.0;
            // lane l < N: occupation l; the next two: the element of the coherence
            // file (antelope.cpp:539-542)
            const int ce = (P.nval * N + P.nval + 1) % NN, ca = ce / N, cb = ce % N, cd = (cb - ca + N) % N;
            const bool up = cd <= M;
            const double *src = reinterpret_cast<const double *>(sm + S * NE * 32 + D::Y);
            if (lane < N) src += 2 * lane;
            else src += 2 * (up ? D::slot(cd, ca) : D::slot(N - cd, cb)) + (lane == N + 1);
            double oc = 0.0;
#pragma unroll 2
            for (int g = 0; g < KW; ++g) {
                const double wg = __shfl_sync(ALL, w, g * G);
                if (lane < N + 2) oc = fma(wg, src[2 * g * D::END], oc);
            }
            if (lane == N + 1) oc = cd == 0 ? 0.0 : up ? oc : -oc;
            if (lane < N + 2) out[4 + lane] = oc;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < NE; ++j) a1[j] = ks[(3 * NE + j) * 32];
            put<N>(v + D::HT, a1, m);
            __syncwarp();
        }
        // the slope -i [H0 + E.D, Y] - g2 Y, to which the projection adds
        double2 *const kn = ks + s * NE * 32;
        double2 c[NE];
        {
            commutator<N>(c, v + D::HT, v + D::Y, v + D::HT, ro);
#pragma unroll
            for (int j = 0; j < NE; ++j)
                c[j] = j < DO ? make_double2(fma(-g2, y[j].x, c[j].y), fma(-g2, y[j].y, -c[j].x))
                              : make_double2(fma(-g2, y[j].x, c[j].x), fma(-g2, y[j].y, c[j].y));
            if (!KEEP || !(deph || with_cur))
#pragma unroll
                for (int j = 0; j < NE; ++j) kn[j * 32] = c[j];
        }
        if (deph || with_cur) {
            double2 *const Ps = v + D::HT;
            double2 p[NE], q[NE], d[NE];   // P_j, P_{j-1} and D(Y)
#pragma unroll
            for (int j = 0; j < NE; ++j) p[j] = a0[j];
            if (!D::EVEN) p[DO].y = 0.0;
            const double t0 = gsum<G>(p[DO].x + p[DO].y, base) * (1.0 / N);
            const double ty = gsum<G>(D::EVEN ? y[DO].x + y[DO].y : y[DO].x, base) * (1.0 / N);
            p[DO].x -= t0;
            if (D::EVEN) p[DO].y -= t0;
            put<N>(v + D::Y, p, m);   // A: H0 without its trace (Y is done with)
            double p2 = gsum<G>(dot<N>(p, p), base);
            const double py = gsum<G>(dot<N>(p, y), base);
            const double a2 = p2;
            double ip = p2 > 0.0 ? 1.0 / p2 : 0.0, b = 0.0;
            if (N > 3 && m == 0) v[CR].x = fma(N * t0, t0, a2);   // |H0|^2
#pragma unroll
            for (int j = 0; j < NE; ++j) {
                const double x = py * ip;
                d[j] = make_double2(x * p[j].x, x * p[j].y);
                q[j] = make_double2(0.0, 0.0);
            }
            d[DO].x += ty;
            if (D::EVEN) d[DO].y += ty;
            __syncwarp();
            Rows<N> H;
            H.load(v + D::Y, ro);
#pragma unroll 1
            for (int i = 2; i < N; ++i) {
                double2 w[NE];
                product<N>(w, H, i == 2 ? v + D::Y : Ps, ro);
                const double a = gsum<G>(dot<N>(w, p), base) * ip;
#pragma unroll
                for (int j = 0; j < NE; ++j) {
                    w[j].x = fma(-a, p[j].x, fma(-b, q[j].x, w[j].x));
                    w[j].y = fma(-a, p[j].y, fma(-b, q[j].y, w[j].y));
                    q[j] = p[j];
                }
                if (i == 2) {   // Tr(A P_1) / N
                    w[DO].x -= p2 * (1.0 / N);
                    if (D::EVEN) w[DO].y -= p2 * (1.0 / N);
                }
                const double w2 = gsum<G>(dot<N>(w, w), base), wy = gsum<G>(dot<N>(w, y), base);
                // a basis matrix that is rounding only (two bands meet) is left out
                const bool ok = w2 > 1e-26 * a2 * p2;
                b = w2 * ip;
                ip = ok ? 1.0 / w2 : 0.0;
                p2 = w2;
                const double x = wy * ip;
#pragma unroll
                for (int j = 0; j < NE; ++j) {
                    d[j] = make_double2(fma(x, w[j].x, d[j].x), fma(x, w[j].y, d[j].y));
                    p[j] = ok ? w[j] : make_double2(0.0, 0.0);
                }
                if (i + 1 < N) put<N>(Ps, p, m);
                __syncwarp();
            }
            if (N > 3 && !EIG && m == 0 && bands_crowd<N>(p2, b, a2, v[CR].x)) v[CR].y = 1.0;
            if constexpr (EIG) {
                const bool bad = bands_crowd<N>(p2, b, a2, v[CR].x);
                if (__any_sync(ALL, live && bad)) {
                    for (int e = m; e < D::NM; e += G)
                        if (lane < LW) Ps[e] = v[D::Y + e];
                    __syncwarp();
                    put<N>(v + D::Y, y, m);
                    __syncwarp();
                    eigen_diagonal<N>((int)(v - sm), m, base, live && bad);
                    if (bad) {
                        const Slots<N> Dy{Ps};
#pragma unroll
                        for (int j = 0; j < DO; ++j) d[j] = Dy.get(erow(j), ecol(j));
                        d[DO] = make_double2(Ps[m].x, D::EVEN ? Ps[m + M].x : 0.0);
                    }
                    __syncwarp();
                }
            }
#pragma unroll
            for (int j = 0; j < NE; ++j) {
                const double2 x = KEEP ? c[j] : kn[j * 32];
                kn[j * 32] = make_double2(fma(-gd, d[j].x, x.x), fma(-gd, d[j].y, x.y));
            }
            if (with_cur) {
                // intraband current Re Tr(D(Y) J_a) = Re Tr(D(Y) (-i S_a)): D(Y) commutes with H0
                double ii[2];
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    double2 x[NE];
#pragma unroll
                    for (int j = 0; j < NE; ++j) x[j] = ks[((a + 1) * NE + j) * 32];
                    ii[a] = tr_s<N>(d, x);
                }
                double *out = P.cur_part + (size_t)unit * WAN_NSLOT;
                const double w = live ? wk : 0.0;
                double z[4] = {w * (tot[0] - ii[0]), w * (tot[1] - ii[1]), w * ii[0], w * ii[1]};
                const bool h4 = lane & 16, h3 = lane & 8;
                double u0 = (h4 ? z[2] : z[0]) + __shfl_xor_sync(ALL, h4 ? z[0] : z[2], 16);
                double u1 = (h4 ? z[3] : z[1]) + __shfl_xor_sync(ALL, h4 ? z[1] : z[3], 16);
                double x = (h3 ? u1 : u0) + __shfl_xor_sync(ALL, h3 ? u0 : u1, 8);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(ALL, x, o);
                if ((lane & 7) == 0) out[lane >> 3] = x;
            }
        }
    }
    if (N > 3 && !EIG) {
        __syncwarp();
        if (__any_sync(ALL, live && v[CR].y != 0.0)) return false;
    }
    // trial state and error estimate
    double emax = 0.0;
    double2 *rout = P.rho[1 - buf] + (size_t)kc * NN;
    double2 er[NE];
#pragma unroll
    for (int j = 0; j < NE; ++j) er[j] = make_double2(0.0, 0.0);
    double2 inc[NE];
    if (!KEEP) state(r64);
#pragma unroll
    for (int j = 0; j < NE; ++j) inc[j] = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int s = 0; s < S; ++s) {
        const double b = h * tb.b[s], e = h * tb.e[s];
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            const double2 q = ks[(s * NE + j) * 32];
            inc[j] = make_double2(fma(b, q.x, inc[j].x), fma(b, q.y, inc[j].y));
            er[j] = make_double2(fma(e, q.x, er[j].x), fma(e, q.y, er[j].y));
        }
    }
    if (live) {
#pragma unroll
        for (int j = 0; j < DO; ++j) {
            const double2 x = make_double2(r64[j].x + inc[j].x, r64[j].y + inc[j].y);
            const int a = erow(j), b = ecol(j);
            __stcg(rout + a * N + b, x);
            __stcg(rout + b * N + a, cconj(x));
            emax = fmax(emax, sqrt(er[j].x * er[j].x + er[j].y * er[j].y));
        }
        __stcg(rout + m * (N + 1), make_double2(r64[DO].x + inc[DO].x, 0.0));
        emax = fmax(emax, fabs(er[DO].x));
        if (D::EVEN) {
            __stcg(rout + (m + M) * (N + 1), make_double2(r64[DO].y + inc[DO].y, 0.0));
            emax = fmax(emax, fabs(er[DO].y));
        }
    }
    if (P.rk == 45) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) emax = fmax(emax, __shfl_xor_sync(ALL, emax, o));
        // non-negative doubles order as their bits (fmax has dropped a NaN, as in wan_attempt)
        if (lane == 0) atomicMax(P.gr_err, (unsigned long long)__double_as_longlong(emax));
    }
    return true;
}
// A block's unit of KW k-points (-1: none): consecutive units (they share the tables of a
// row) go to the blocks of one SM, which get every SPREAD-th block of the grid
template <int N> __device__ __forceinline__ int block_unit(const WanDev &P, const WanTileRef *tiles)
{
    if (tiles) return tiles[blockIdx.x].tile;
    const int nu = (P.nk + PD<N>::KW - 1) / PD<N>::KW, i = (int)blockIdx.x % SPREAD;
    const int unit = (int)((long long)i * nu / SPREAD) + (int)blockIdx.x / SPREAD;
    return unit < (int)((long long)(i + 1) * nu / SPREAD) ? unit : -1;
}
template <int N>
__device__ __noinline__ void attempt_eig(const WanDev *Pp, const WanDev *const *descs, const WanTileRef *tiles)
{
    const WanDev &P = tiles ? *descs[tiles[blockIdx.x].solve] : *Pp;
    attempt<N, true>(P, block_unit<N>(P, tiles));
}

template <int N>
__global__ void __launch_bounds__(32, N == 6 || N == 4 ? 8 : N == 5 ? 12 : 16)
    wan_attempt_p(const WanDev *__restrict__ Pp, const WanDev *const *__restrict__ descs,
                  const WanTileRef *__restrict__ tiles)
{
    const WanDev &P = tiles ? *descs[tiles[blockIdx.x].solve] : *Pp;
    const int unit = block_unit<N>(P, tiles);
    if (unit < 0 || P.ctl->done) return;
    if (!attempt<N, false>(P, unit)) {
        if constexpr (N > 3) attempt_eig<N>(Pp, descs, tiles);
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
    constexpr int G = D::G, NE = D::NE, DO = D::DO, M = D::M, NN = D::NN, NU = N * (N + 1) / 2;
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
            double2 *out = P.gr_tab + (size_t)item * nent * NE * NQ * G;
            double2 *oc = P.gr_cur + (size_t)row * nent * NE * NC * G;
            for (int w = t; w < ng * NU; w += blockDim.x) {
                // owned element j of lane l; the diagonal ones last, two to an entry
                const int q = w / NU, u = w % NU, j = u / G, l = u % G;
                const int r0 = j < DO ? (j < M ? l : l + M) : l + (j - DO) * M;
                const int c0 = j < DO ? (r0 + 1 + (j < M ? j : j - M)) % N : r0;
                const bool low = r0 > c0;   // from the upper triangle by symmetry
                const int e = low ? c0 * N + r0 : r0 * N + c0;
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
                // sig = G_g + G_-g, tau = i (G_g - G_-g); the group g = 0 is sig alone.
                // Of the diagonal the real part (h, D Hermitian), of S the imaginary one.
                auto store = [&](double2 *o, int nq, int y, double2 sg, double2 ta, bool anti) {
                    const size_t step = (size_t)NE * nq * G;
                    o += (size_t)max(2 * q - 1, 0) * step + (size_t)(min(j, DO) * nq + y) * G + l;
                    if (j < DO) {
                        if (low) {
                            sg = anti ? make_double2(-sg.x, sg.y) : cconj(sg);
                            ta = anti ? make_double2(-ta.x, ta.y) : cconj(ta);
                        }
                        o[0] = sg;
                        if (q > 0) o[step] = ta;
                    } else {
                        double *z = reinterpret_cast<double *>(o) + (j - DO);
                        z[0] = anti ? sg.y : sg.x;
                        if (q > 0) z[2 * step] = anti ? ta.y : ta.x;
                        if (!D::EVEN) {
                            z[1] = 0.0;
                            if (q > 0) z[2 * step + 1] = 0.0;
                        }
                    }
                };
                auto pair = [&](double2 *o, int nq, int y, const double2 &xp, const double2 &xm, bool anti) {
                    store(o, nq, y, q == 0 ? xp : make_double2(xp.x + xm.x, xp.y + xm.y), make_double2(xm.y - xp.y, xp.x - xm.x),
                          anti);
                };
                pair(out, NQ, 0, x[0][0], x[1][0], false);
                if (dip) pair(out, NQ, 1, x[0][1], x[1][1], false);
                if (cur) {
                    pair(oc, NC, 0, x[0][2], x[1][2], true);
                    pair(oc, NC, 1, x[0][3], x[1][3], true);
                    if (dip) {
                        pair(oc, NC, 2, x[0][4], x[1][4], false);
                        pair(oc, NC, 3, x[0][5], x[1][5], false);
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
    return !w.lean && !w.mixed && !w.vg && !w.cont && !w.has_jtab && !w.degenerate && w.N >= 3 && w.N <= 6 && w.nR >= 1 &&
           w.Ngrid[2] == 1;
}
bool wan_proj(const WanDev &w) { return w.gr_tab != nullptr && wan_proj_applies(w); }

// Entries of the row tables per row (gr_tab has one set per stage)
int wan_proj_entries(int N, int ngrp, int nq)
{
    const int even = N % 2 == 0, G = even ? N / 2 : N, NE = even ? N : (N + 1) / 2;   // PD
    return (2 * ngrp - 1) * NE * nq * G;
}
int wan_proj_unit(int N) { return 32 / (N % 2 == 0 ? N / 2 : N); }

template <int N>
static cudaError_t proj_attempt(const WanDev *dw, const WanDev *const *descs, const WanTileRef *tiles, int nblocks,
                                int ngrp, int S, cudaStream_t st)
{
    const int grid = tiles ? nblocks : (nblocks + SPREAD - 1) / SPREAD * SPREAD;
    wan_attempt_p<N><<<grid, 32, proj_bytes<N>(ngrp, S), st>>>(dw, descs, tiles);
    return cudaGetLastError();
}
cudaError_t launch_wan_attempt_p(int N, int ngrp, int S, const WanDev *dw, const WanDev *const *descs, const WanTileRef *tiles,
                                 int nblocks, cudaStream_t st)
{
    if (nblocks <= 0) return cudaSuccess;
    switch (N) {
    case 3: return proj_attempt<3>(dw, descs, tiles, nblocks, ngrp, S, st);
    case 4: return proj_attempt<4>(dw, descs, tiles, nblocks, ngrp, S, st);
    case 5: return proj_attempt<5>(dw, descs, tiles, nblocks, ngrp, S, st);
    case 6: return proj_attempt<6>(dw, descs, tiles, nblocks, ngrp, S, st);
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
