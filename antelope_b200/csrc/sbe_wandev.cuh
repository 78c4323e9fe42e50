// Device helpers of the N-band kernels: complex arithmetic, the laser, the
// Runge-Kutta tableaux and the k-grid.  Included by the N-band translation
// units inside namespace sbe.
#pragma once

#include "sbe_wannier.h"

namespace sbe {
namespace {

template <class Real> struct Cx;
template <> struct Cx<double> { using T = double2; };
template <> struct Cx<float> { using T = float2; };

template <class T> __device__ __forceinline__ T cx(double re, double im)
{
    T r;
    r.x = (decltype(r.x))re;
    r.y = (decltype(r.y))im;
    return r;
}
template <class T> __device__ __forceinline__ T cmul(T a, T b)
{
    T r;
    r.x = fma(a.x, b.x, -(a.y * b.y));
    r.y = fma(a.x, b.y, a.y * b.x);
    return r;
}
template <class T> __device__ __forceinline__ T cmulc(T a, T b)  // conj(a) * b
{
    T r;
    r.x = fma(a.x, b.x, a.y * b.y);
    r.y = fma(a.x, b.y, -(a.y * b.x));
    return r;
}
template <class T> __device__ __forceinline__ void cfma(T &acc, T a, T b)  // acc += a b
{
    acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
    acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}
template <class T> __device__ __forceinline__ void cfmac(T &acc, T a, T b)  // acc += conj(a) b
{
    acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
    acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
}
template <class T> __device__ __forceinline__ T cconj(T a)
{
    a.y = -a.y;
    return a;
}

// ---- laser on the device (laser.h:150-322), FP64
__device__ double envelope(const PulseDev &q, double t, bool d)
{
    const double ef = q.envfactor;
    double to;
    switch (q.env) {
        case 2:  // cos4
            if (fabs(t) > q.twidth) return 0;
            if (d) return -4. * ef * sin(t * ef) * pow(cos(t * ef), 3.);
            return pow(cos(t * ef), 4.);
        case 4:  // sin2 (extension)
            if (fabs(t) > q.twidth) return 0;
            if (d) return -2. * ef * sin(t * ef) * cos(t * ef);
            return cos(t * ef) * cos(t * ef);
        case 3:  // cos4_clipped
            if (fabs(t) > q.twidth) return 0;
            if (t > q.twidth_clipped) to = t - q.twidth_clipped;
            else if (t > -q.twidth_clipped) return d ? 0. : 1.;
            else to = t + q.twidth_clipped;
            if (d) return -4. * ef * sin(to * ef) * pow(cos(to * ef), 3.);
            return pow(cos(to * ef), 4.);
        case 0:  // gauss
            if (d) return 2 * t * ef * exp(ef * t * t);
            return exp(ef * t * t);
        default:  // gauss_clipped
            if (t > q.twidth_clipped) to = t - q.twidth_clipped;
            else if (t > -q.twidth_clipped) return d ? 0. : 1.;
            else to = t + q.twidth_clipped;
            if (d) return 2 * to * ef * exp(ef * to * to);
            return exp(ef * to * to);
    }
}

__device__ void laser_eval(const LaserDev &L, double t, double *A, double *E)
{
    double a[3] = {0, 0, 0}, e[3] = {0, 0, 0};
    for (int i = 0; i < L.npulses; ++i) {
        const PulseDev &q = L.p[i];
        const double kt = t - q.t0;
        double s, c;
        sincos(kt * q.w0 - q.cep, &s, &c);
        const double f = envelope(q, kt, false), fp = envelope(q, kt, true);
        const double ax = -q.A0x * s * f, ay = q.A0y * c * f;
        const double ex = q.E0x * c * f - q.A0x * s * fp;
        const double ey = q.E0y * s * f + q.A0y * c * fp;
        for (int dd = 0; dd < 3; ++dd) {
            a[dd] += ax * q.xdir[dd] + ay * q.ydir[dd];
            e[dd] += ex * q.xdir[dd] + ey * q.ydir[dd];
        }
    }
    for (int dd = 0; dd < 3; ++dd) {
        A[dd] = a[dd] - L.init_A[dd];
        E[dd] = e[dd] - L.init_E[dd];
    }
}

// ---- tableaux (SBEs.h:395-416; Cash-Karp 4(5) for the adaptive steps)
struct WTab {
    int S;
    double c[6], a[6][6], b[6], e[6];  // e = b - b* (error weights)
};
__device__ void tableau(int rk, WTab &T)
{
    for (int i = 0; i < 6; ++i) {
        T.c[i] = T.b[i] = T.e[i] = 0;
        for (int j = 0; j < 6; ++j) T.a[i][j] = 0;
    }
    if (rk == 4) {
        T.S = 4;
        T.c[1] = 0.5; T.c[2] = 0.5; T.c[3] = 1.0;
        T.a[1][0] = 0.5; T.a[2][1] = 0.5; T.a[3][2] = 1.0;
        T.b[0] = 1.0 / 6.0; T.b[1] = 2.0 / 6.0; T.b[2] = 2.0 / 6.0; T.b[3] = 1.0 / 6.0;
    } else if (rk == 5) {
        T.S = 6;
        T.c[1] = 0.25; T.c[2] = 3. / 8.; T.c[3] = 12. / 13.; T.c[4] = 1.0; T.c[5] = 0.5;
        T.a[1][0] = 1.0 / 4.0;
        T.a[2][0] = 3. / 32.; T.a[2][1] = 9. / 32.;
        T.a[3][0] = 1932. / 2197.; T.a[3][1] = -7200. / 2197.; T.a[3][2] = 7296. / 2197.;
        T.a[4][0] = 439. / 216.; T.a[4][1] = -8.; T.a[4][2] = 3680. / 513.; T.a[4][3] = -845. / 4104.;
        T.a[5][0] = -8. / 27.; T.a[5][1] = 2.; T.a[5][2] = -3544. / 2565; T.a[5][3] = 1859. / 4104;
        T.a[5][4] = -11. / 40.;
        T.b[0] = 16. / 135.; T.b[2] = 6656. / 12825.; T.b[3] = 28561. / 56430.; T.b[4] = -9. / 50.;
        T.b[5] = 2. / 55.;
    } else {  // Cash-Karp (J. R. Cash, A. H. Karp, ACM TOMS 16 (1990) 201)
        T.S = 6;
        T.c[1] = 1. / 5.; T.c[2] = 3. / 10.; T.c[3] = 3. / 5.; T.c[4] = 1.; T.c[5] = 7. / 8.;
        T.a[1][0] = 1. / 5.;
        T.a[2][0] = 3. / 40.; T.a[2][1] = 9. / 40.;
        T.a[3][0] = 3. / 10.; T.a[3][1] = -9. / 10.; T.a[3][2] = 6. / 5.;
        T.a[4][0] = -11. / 54.; T.a[4][1] = 5. / 2.; T.a[4][2] = -70. / 27.; T.a[4][3] = 35. / 27.;
        T.a[5][0] = 1631. / 55296.; T.a[5][1] = 175. / 512.; T.a[5][2] = 575. / 13824.;
        T.a[5][3] = 44275. / 110592.; T.a[5][4] = 253. / 4096.;
        T.b[0] = 37. / 378.; T.b[2] = 250. / 621.; T.b[3] = 125. / 594.; T.b[5] = 512. / 1771.;
        const double bs[6] = {2825. / 27648., 0., 18575. / 48384., 13525. / 55296., 277. / 14336., 1. / 4.};
        for (int i = 0; i < 6; ++i) T.e[i] = T.b[i] - bs[i];
    }
}

// k-grid point (momaxis.h:147-186, 349-383) and its trapezoid weight
__device__ void kpoint(const WanDev &P, int kl, double kv[3], double &wt)
{
    const int N0 = P.Ngrid[0], N1 = P.Ngrid[1], N2 = P.Ngrid[2];
    const int k = P.k_offset + kl;  // local index -> flat grid index
    const int ii[3] = {k / (N1 * N2), (k / N2) % N1, k % N2};
    const int NNg[3] = {N0, N1, N2};
    double f[3];
    wt = 1.0;
    for (int dd = 0; dd < 3; ++dd) {
        f[dd] = (NNg[dd] == 1) ? 0.0 : double(ii[dd]) / (NNg[dd] - 1) - 0.5;
        if (NNg[dd] != 1 && (ii[dd] == 0 || ii[dd] == NNg[dd] - 1)) wt /= 2;
    }
    for (int dd = 0; dd < 3; ++dd)
        kv[dd] = P.origin[dd] + f[0] * P.axes[0 * 3 + dd] + f[1] * P.axes[1 * 3 + dd] + f[2] * P.axes[2 * 3 + dd];
}

// Where the Lanczos projections of wan_attempt_p and wan_lw_steps lose the
// eigenvectors' accuracy: do bands crowd?  A basis matrix amplifies the rounding
// of the one before by r_j^-1/2, r_j = |P_j|^2 / (|A|^2 |P_{j-1}|^2) (A: H0 without
// its trace), so D(Y) is good to some eps / sqrt(prod r_j), where eigenvectors are to
// eps / gap.  A close pair makes one small factor and costs nothing beyond eps / gap;
// a cluster of m bands of relative width d costs eps / d^(m-1).  The projection stands
// where the product is not small, or is mostly the last r_j's doing (of N = 4: or the
// other's).  The product telescopes to |P_{N-1}|^2 / |A|^(2N-2); hh = |H0|^2 in place of
// one |A|^2 is H0's own rounding.  p2, b: |P_{N-1}|^2 and its ratio to the one
// before.  Not for N = 3: three close bands are the whole spectrum there.
//
// The limits, from 160 000 random spectra with clusters in random frames (|Y| = 1):
// errors left are below 4e-13, or below 20 eps / gap at N = 4 and 8 at N = 5, 6; a
// factor of 8 (N = 6) to 57 (N = 4) below the smallest product on 240 000 k-points of
// 40 random six-, five- and four-band tables, which none of this should slow down.
template <int N> __device__ __forceinline__ bool bands_crowd(double p2, double b, double a2, double hh)
{
    constexpr double least = N == 4 ? 1e-7 : N == 5 ? 1e-8 : 1e-9, others = N == 6 ? 1e-4 : 1e-3;
    double s = hh;
#pragma unroll
    for (int j = 3; j < N; ++j) s *= a2;
    return N > 3 && p2 < least * s * a2 && p2 < others * s * b && (N != 4 || b < others * a2);
}
// The same from band energies
template <int N> __device__ bool bands_crowd(const double *e)
{
    double a[N], p[N], q[N], t0 = 0.0, a2 = 0.0, b = 0.0;
    for (int n = 0; n < N; ++n) t0 += e[n] / N;
    for (int n = 0; n < N; ++n) {
        p[n] = a[n] = e[n] - t0;
        q[n] = 0.0;
        a2 += a[n] * a[n];
    }
    double p2 = a2;
    for (int j = 2; j < N && p2 > 0.0; ++j) {
        double s = 0.0, w2 = 0.0;
        for (int n = 0; n < N; ++n) s += a[n] * p[n] * p[n];
        for (int n = 0; n < N; ++n) {
            const double w = (a[n] - s / p2) * p[n] - b * q[n] - (j == 2 ? p2 / N : 0.0);
            q[n] = p[n];
            p[n] = w;
            w2 += w * w;
        }
        b = w2 / p2;
        p2 = w2;
    }
    return !(p2 > 0.0) || bands_crowd<N>(p2, b, a2, a2 + N * t0 * t0);
}

// Jacobi rotation of the 2 x 2 block (a, z; conj z, b): V = (c, s; -conj s, c) makes
// V^dag (...) V diagonal, a - dl and b + dl
struct Turn {
    double c;
    double2 s;
    __device__ __forceinline__ void find(double a, double b, double2 z, double &dl)
    {
        const double m2 = fma(z.x, z.x, z.y * z.y), d = b - a;
        c = 1.0;
        s = make_double2(0.0, 0.0);
        dl = 0.0;
        if (m2 > 0.0) {
            const double rh = rsqrt(fma(d, d, 4.0 * m2));   // of twice the angle: cos |d| rh, sin 2 |z| rh
            const double c2 = fma(0.5 * fabs(d), rh, 0.5), rc = rsqrt(c2), g = copysign(rh * rc, d);
            c = c2 * rc;
            s = make_double2(z.x * g, z.y * g);
            dl = m2 * g * rc;
        }
    }
    // (x, y) -> (x, y) V of a row of a matrix; V^dag (x, y) of a column takes conj(s)
    __device__ __forceinline__ void on(double2 &x, double2 &y, double2 s) const
    {
        const double2 u = x;
        x = make_double2(fma(-s.x, y.x, fma(-s.y, y.y, c * u.x)), fma(-s.x, y.y, fma(s.y, y.x, c * u.y)));
        y = make_double2(fma(s.x, u.x, fma(-s.y, u.y, c * y.x)), fma(s.x, u.y, fma(s.y, u.x, c * y.y)));
    }
    // V^dag B V of the pair's own block (a, z; conj z, b)
    __device__ __forceinline__ void own(double &a, double2 &z, double &b) const
    {
        double2 p = make_double2(a, 0.0), q = z, r = cconj(z), t = make_double2(b, 0.0);
        on(p, q, s);
        on(r, t, s);
        on(p, r, cconj(s));
        on(q, t, cconj(s));
        a = p.x;
        z = q;
        b = t.x;
    }
};
constexpr int MAX_SWEEPS = 12;

// Accept or reject an attempt of error emax and set up the next one.  The
// step-size rule is the oracle's (oracle/sbe_oracle.c, run_adaptive).
__device__ void control_decide(const WanDev &P, WanCtl *ctl, double emax)
{
    ctl->attempts++;
    ctl->need_current = 0;
    ctl->shot = -1;
    ctl->emax = emax;
    const double dt = P.dt, tend = P.atmin + dt * (ctl->n + 1);
    bool accept = true;
    if (P.rk == 45) {
        if (emax <= P.tol) {
            double fac = emax > 0 ? 0.9 * pow(P.tol / emax, 0.2) : 5.0;
            if (fac > 5.0) fac = 5.0;
            if (!ctl->last || fac < 1.0) ctl->h = ctl->hs * (fac < 0.2 ? 0.2 : fac);
            if (ctl->h > dt) ctl->h = dt;
        } else {
            accept = false;
            double fac = 0.9 * pow(P.tol / emax, 0.25);
            ctl->h = ctl->hs * (fac < 0.1 ? 0.1 : fac);
            ctl->rejects++;
            if (!(ctl->h > 1e-12 * dt)) {
                ctl->error = 1;
                ctl->done = 1;
                return;
            }
        }
    }
    if (accept) {
        ctl->buf ^= 1;
        ctl->steps++;
        if (ctl->last) {
            ctl->tc = tend;
            // the state is now past interval n: its snapshot (after step n,
            // antelope.cpp:342) is due when n is a multiple of the interval
            if (P.shot_every > 0 && ctl->n % P.shot_every == 0) ctl->shot = ctl->n;
            ctl->n++;
            if (ctl->n >= P.Nt) {
                ctl->done = 1;
                return;
            }
            ctl->need_current = 1;
        } else {
            ctl->tc = ctl->tc + ctl->hs;
        }
    }
    // next attempt
    const double tend2 = P.atmin + dt * (ctl->n + 1);
    ctl->hs = ctl->h;
    ctl->last = 0;
    if (ctl->tc + ctl->hs >= tend2 - 1e-12 * dt) {
        ctl->hs = tend2 - ctl->tc;
        ctl->last = 1;
    }
}

}  // namespace
}  // namespace sbe
