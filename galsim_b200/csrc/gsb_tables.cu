// FP64 on-device construction of the FT tables and the leaf sizing (stepk / maxk).
//
//   ogata_*      Ogata (2005) nodes and weights for h = 2^-5 .. 2^-20, plus the first 10^6
//                zeros of J0, built once per device (gsb_init).
//   hankel_*     the reference's adaptive Hankel transform (src/math/Hankel.cpp:179-249),
//                one warp per transform, terms summed 32 at a time with a warp prefix sum.
//   ogata_log_*  the quadrature's levels resampled onto a uniform grid in ln x, so that a table
//                of transforms on a uniform ln k grid is a correlation (sersic_table_kernel).
//   sersic_*     SersicInfo (src/SBSersic.cpp:301-667): HLR and missing-flux radii by
//                Brent, the ln k table of the Hankel transform, its high-k fit and maxk,
//                and the natural cubic spline (src/Table.cpp:634-686).
//   kolmogorov_* KolmogorovInfo stepk (src/SBKolmogorov.cpp:338-420).
//   prepare_*    per-leaf derived constants and stepk / maxk.
#include <algorithm>
#include <mutex>
#include <vector>

#include "gsb_internal.cuh"
#include "gsb_interp.cuh"

namespace gsb {

namespace {

constexpr int kLevMin = 5;
constexpr int kMaxRounds = 128;      // rounds of ln k nodes per truncated table build (status flags)
// ln k nodes per truncated table and round: a table's nodes past its stopping point are integrated
// only up to the end of the round in which its scan stops
constexpr int kTableRound = 64;
constexpr int kLevMax = 20;
constexpr long long kNroot = 1000000;

// 2^(j/256), j = 0..255, correctly rounded (computed on the host in extended precision by
// ogata_init): the table of exp_tab256_core.
__device__ double g_exp2_256[256];

// The same method with a 256-entry table 2^(j/256) (`tab`, correctly rounded, filled by the
// caller): |r| <= ln2/512, so the degree-4 Taylor polynomial of e^r suffices (truncation
// < 4e-17 relative), two fused multiply-adds fewer than exp_tab_core.  Evaluated through
// gsb_exp_fp64_ex alone.
__device__ __forceinline__ double exp_tab256_core(double x, const double* tab)
{
    const double kShift = 6755399441055744.0;               // 1.5 * 2^52
    const double s = __dadd_rn(__dmul_rn(x, 369.3299304675746), kShift);   // 256 / ln2
    const int n = __double2loint(s);
    const double t = s - kShift;
    double r = fma(-t, 0.0027076061740622863, x);            // ln2/256, leading double
    r = fma(-t, 9.058776616587108e-20, r);                   // ln2/256, remainder
    const int j = n & 255;
    const int m = n >> 8;
    double p = fma(r, 1. / 24., 1. / 6.);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.);
    p = fma(p, r, 1.);
    const double v = tab[j] * p;
    return __hiloint2double(__double2hiint(v) + (m << 20), __double2loint(v));
}

__global__ void ogata_root_kernel(double2* root, long long nroot)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= nroot) return;
    const double z = bessel_j0_zero(i + 1);
    root[i] = make_double2(z, y0(z) / j1(z));
}

// Node i of level h: (log x, w) with x = pi/h psi(h xi) and the Ogata weight w.
__device__ inline double2 ogata_node(const double2* root, double h, long long i)
{
    const double2 r = root[i];
    const double t = h * r.x / kPi;
    const double x = kPi / h * ogata_psi(t);
    const double w = r.y * kPi * x * j0(x) * ogata_dpsi(t);
    return make_double2(log(x), w);
}

__global__ void ogata_level_kernel(double2* xw, const double2* root, double h, long long n)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    xw[i] = ogata_node(root, h, i);
}

__device__ inline double warp_total(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Running-sum estimate refresh: every chunk for the first kEagerChunks chunks (short sums stop
// there), then every kLazyChunks chunks.
constexpr int kEagerChunks = 2;
constexpr int kLazyChunks = 16;

// Sum_i w_i f(x_i / k) / k^2 for h = 2^-lev with the reference's stopping rule: stop at the
// first term whose magnitude is below 1e-15 |running sum| (Hankel.cpp:117-141).  The integrand
// is called with log(x_i / k) = log x_i - log k (nodes store log x), which spares a division
// and a logarithm per term.  Each lane keeps the sum of its own terms; the warp total is formed
// only every few chunks, and the stopping test uses that total.  The stop can therefore move by
// terms below 1e-15 of the sum, which changes the result only at that level.
template <class F>
__device__ double warp_ogata_sum(const OgataTables& og, const F& f, double k, int lev)
{
    const int lane = threadIdx.x & 31;
    const double h = ldexp(1.0, -lev);
    const long long nmax = (long long)fmin(kPi / h, 1e6);
    const bool tab = lev >= og.lev_min && lev <= og.lev_max;
    const double2* xw = tab ? og.xw + og.off[lev - og.lev_min] : nullptr;
    const double logk = log(k);
    double acc = 0., thresh = 0.;
    int chunk = 0;
    for (long long base = 0; base < nmax; base += 32, ++chunk) {
        const long long i = base + lane;
        const bool valid = i < nmax;
        double step = 0.;
        if (valid) {
            const double2 n = tab ? xw[i] : ogata_node(og.root, h, i);
            step = n.y * f(n.x - logk);
        }
        const unsigned mask = __ballot_sync(0xffffffffu, valid && fabs(step) < thresh);
        if (mask) {
            const int last = __ffs(mask) - 1;
            return warp_total(acc + (lane <= last ? step : 0.)) / (k * k);
        }
        acc += step;
        if (chunk < kEagerChunks || (chunk % kLazyChunks) == kLazyChunks - 1)
            thresh = 1e-15 * fabs(warp_total(acc));
    }
    return warp_total(acc) / (k * k);
}

// AdaptiveHankelIntegrator::integrate (Hankel.cpp:179-219).  `status` is set to 1 when
// the halving ran past 2^-60 without meeting the tolerance.
template <class F>
__device__ double warp_hankel(const OgataTables& og, const F& f, double k, double relerr,
                              double abserr, int* status)
{
    int lev = 5;
    double h0 = 1. / 32.;
    while (h0 > 100. * k && lev < 60) { h0 *= 0.5; ++lev; }
    double ans0 = warp_ogata_sum(og, f, k, lev);
    double ans1 = warp_ogata_sum(og, f, k, lev + 1);
    double err = fabs(ans1 - ans0);
    while ((err > relerr * ans1 && (err > abserr || fabs(ans1) > 2. * fabs(ans0))) || ans1 == 0.) {
        ++lev;
        if (lev > 60) { if (status) *status = 1; break; }
        ans0 = ans1;
        ans1 = warp_ogata_sum(og, f, k, lev + 1);
        err = fabs(ans1 - ans0);
    }
    return ans1;
}

// The quadrature levels on a uniform grid in ln x.  A level-l sum for a radial profile whose
// transform is wanted on a uniform ln k grid,
//     S_l(k) = sum_i w_i f(x_i / k) = sum_i w_i G(ln x_i - ln k),     G(y) = f(e^y),
// samples a smooth G at the scattered ln x_i.  With G band-limited well below pi / h, its value
// between the points of a grid of spacing h is the windowed-sinc sum
//     G(u h) = sum_q phi(u - q) G(q h),   phi(t) = sinc(t) exp(beta (sqrt(1 - (2 t / W)^2) - 1)),
// (the "exponential of semicircle" window of Barnett, Magland and af Klinteberg, SIAM J. Sci. Comput. 41, 2019)
// so the nodes can be spread onto the grid once and for all, A_l[q] = sum_i w_i phi(ln x_i / h - q),
// and S_l(k) = sum_q A_l[q] G(q h - ln k): one array of G per profile serves every ln k on the
// grid and every level, and a term costs one multiply-add instead of an exponential.  The A_l
// depend on the spacing alone.  Against the scattered sums (Sersic n from 0.3 to 6.2, every
// level): 1e-15 of the flux at n <= 0.5, 5e-12 where the level's own cancellation is largest.
constexpr int kLogW = 48;                 // window width in grid points
constexpr double kLogBeta = 34.;
constexpr double kLogMaxStep = 0.0333;    // largest grid spacing (the spectrum of G at n = 0.3 is
                                          // 1e-19 at pi / h; larger n decays faster)
constexpr int kLogLev0 = kLevMin;
constexpr int kLogLevels = 57;            // levels 5 .. 61: all the halving can reach

struct OgataLog {
    double h;
    const double* a;
    int have;                             // levels that are spread (kLogLev0 on)
    int qmin[kLogLevels], len[kLogLevels], off[kLogLevels];
};

// A_l[q]: the nodes within W / 2 grid points of q (the node list is ascending in ln x), a block per grid point
// and slice of its nodes, the slices added up by ogata_log_sum_kernel.  (Half of a level's nodes lie within
// the last 20 grid points: a block per grid point alone took 1.6 ms a level of a million nodes.)
constexpr int kLogSlices = 16;
__global__ void __launch_bounds__(256) ogata_log_kernel(const double2* __restrict__ xw, int n, double h, int qmin,
                                                        double* __restrict__ slices)
{
    const int q = qmin + int(blockIdx.x);
    auto lower = [&](double u) {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (xw[mid].x / h < u) lo = mid + 1; else hi = mid;
        }
        return lo;
    };
    __shared__ int range[2];
    if (threadIdx.x < 2) range[threadIdx.x] = lower(q + (threadIdx.x == 0 ? -0.5 : 0.5) * kLogW);
    __syncthreads();
    const int i0 = range[0], i1 = range[1];
    double sum = 0.;
    for (int i = i0 + int(blockIdx.y) * 256 + threadIdx.x; i < i1; i += 256 * kLogSlices) {
        const double t = xw[i].x / h - q;
        const double v = 2. * t / kLogW;
        const double s = fabs(t) < 1e-9 ? 1. : sinpi(t) / (kPi * t);
        sum += xw[i].y * s * exp(kLogBeta * (sqrt(fmax(1. - v * v, 0.)) - 1.));
    }
    sum = warp_total(sum);
    __shared__ double part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) sum += part[w];
        slices[blockIdx.x * kLogSlices + blockIdx.y] = sum;
    }
}

__global__ void ogata_log_sum_kernel(const double* __restrict__ slices, int len, double* __restrict__ a)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= len) return;
    double sum = 0.;
    for (int c = 0; c < kLogSlices; ++c) sum += slices[q * kLogSlices + c];
    a[q] = sum;
}

// The Sersic profile and its n-derivative along the table's moving grid (GSB_TABLES_DN) at
// y = ln(x / k):  f = exp(-u), u = e^(y/n);  the sum T(k) = sum_j w_j f(x_j / k) has dT/dn along
// k = k(n) with d ln k / dn = c equal to sum_j w_j [df/dn - c r df/dr](x_j / k), and
// df/dn = f u ln r / n^2, r df/dr = -f u / n.
__device__ __forceinline__ double2 sersic_sample(double y, double invn, double dnc)
{
    const double v = y * invn;
    const double u = exp(fmin(v, 7.));
    const double f = exp(-u);
    return make_double2(f, f * u * invn * (v + dnc));
}

// acc[c][r] += sum_q A[q] g[q mul - p (m + r)] (and the same with gd for DN) over q = qlo .. qhi, in the class c = (q - qlo)
// mod kLogSums: several sums, so that the chain of one node's multiply-adds is not the time, counted from the
// level's first point (qlo is a multiple of kLogSums from it), so that a node's value does not depend on how many
// nodes a thread takes.  g points at the sample of d = 0, and samples from top on are 0.  With p = mul = 1 (P1) the array is
// padded with them and the R nodes of a thread share each sample through a window in registers: one
// shared-memory read (lane stride R doubles, R odd: no bank conflicts) and one broadcast read feed R
// multiply-adds.
constexpr int kLogSums = 2;
template <int R, bool DN, bool P1>
__device__ __forceinline__ void correlate(const double* __restrict__ A, int qlo, int qhi, const double* g,
                                          const double* gd, int m, int p, int mul, int top, double (&acc)[kLogSums][R],
                                          double (&dacc)[kLogSums][R])
{
    double w[R], wd[R];
    if (P1) {
#pragma unroll
        for (int r = 1; r < R; ++r) {
            w[r] = g[qlo - m - r];
            if (DN) wd[r] = gd[qlo - m - r];
        }
    }
    auto step = [&](int c, int q) {
        const double a = A[q];
        if (P1) {
            w[0] = g[q - m];
            if (DN) wd[0] = gd[q - m];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                acc[c][r] = fma(a, w[r], acc[c][r]);
                if (DN) dacc[c][r] = fma(a, wd[r], dacc[c][r]);
            }
#pragma unroll
            for (int r = R - 1; r > 0; --r) {
                w[r] = w[r - 1];
                if (DN) wd[r] = wd[r - 1];
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int d = min(q * mul - p * (m + r), top);
                acc[c][r] = fma(a, g[d], acc[c][r]);
                if (DN) dacc[c][r] = fma(a, gd[d], dacc[c][r]);
            }
        }
    };
    int q = qlo;
#pragma unroll (R == 1 ? 4 : 3)
    for (; q + kLogSums - 1 <= qhi; q += kLogSums) {
#pragma unroll
        for (int c = 0; c < kLogSums; ++c) step(c, q + c);
    }
#pragma unroll
    for (int c = 0; c < kLogSums - 1; ++c)
        if (q + c <= qhi) step(c, q + c);
}

// Truncated Hankel transform (math::hankel_trunc, src/math/Hankel.cpp:249-255) of a radial
// profile f, as SersicInfo::buildFT (src/SBSersic.cpp:453-457) and SBMoffat::setupFT
// (src/SBMoffat.cpp:587-592) call it:
//   I(k) = int_0^t r f(r) J0(k r) dr,   f = exp(-r^(1/n)) (Sersic), (1 + r^2)^-beta (Moffat).
// The reference integrates adaptively (Gauss-Kronrod-Patterson to relerr 1e-6); here the
// integral is taken to near FP64 precision by 16-point Gauss-Legendre on panels between
// consecutive zeros of J0(k r) (the first interval graded toward r = 0 in 48 halvings, where
// the Sersic r^(1/n) has its cusp), so the two agree to the reference's integration error.
// One warp per node: lanes 0-15 and 16-31 take two panels at a time, one Legendre node each.
__device__ inline void gauss_legendre16(int q, double* x, double* w)
{
    // node q of P_16 by Newton's method from the Tricomi estimate, weight 2 / ((1 - x^2) P'^2)
    double z = cos(kPi * (q + 0.75) / 16.5), dp = 1.;
    for (int it = 0; it < 10; ++it) {
        double p0 = 1., p1 = z;
        for (int m = 2; m <= 16; ++m) {
            const double p2 = ((2. * m - 1.) * z * p1 - (m - 1.) * p0) / m;
            p0 = p1;
            p1 = p2;
        }
        dp = 16. * (z * p1 - p0) / (z * z - 1.);
        z -= p1 / dp;
    }
    *x = z;
    *w = 2. / ((1. - z * z) * dp * dp);
}

struct SersicRadial {
    double invn;
    __device__ double operator()(double r) const { return exp(-pow(r, invn)); }
};
struct MoffatRadial {
    double beta;
    __device__ double operator()(double r) const { return pow(1. + r * r, -beta); }
};

template <class F>
__device__ double warp_hankel_trunc(const OgataTables& og, const F& f, double k, double t, int* status)
{
    const int lane = threadIdx.x & 31, half = lane >> 4;
    double xq, wq;
    gauss_legendre16(lane & 15, &xq, &wq);
    const double rfirst = fmin(og.root[0].x / k, t);
    constexpr int M = 48;
    double acc = 0.;
    for (long long jp = 0;; jp += 2) {
        // panel jp (lanes 0-15) and jp + 1 (lanes 16-31)
        const long long j = jp + half;
        double a, b;
        bool live;
        if (j < M) {
            a = ldexp(rfirst, int(j - M));
            b = ldexp(rfirst, int(j + 1 - M));
            live = true;
        } else {
            const long long m = j - M;                      // panel between zeros m and m + 1 (1-based)
            if (m + 1 >= og.nroot) { if (status) *status = 1; live = false; a = b = t; }
            else {
                a = m == 0 ? rfirst : og.root[m - 1].x / k;
                b = fmin(og.root[m].x / k, t);
                live = a < t;
            }
        }
        if (!__any_sync(0xffffffffu, live)) break;
        if (live) {
            const double h = 0.5 * (b - a), r = a + h * (1. + xq);
            acc += wq * h * r * f(r) * j0(k * r);
        }
    }
    return warp_total(acc);
}

struct KolmKValue {
    __device__ double operator()(double logk) const { return exp_tab(-exp_tab(logk * (5. / 3.))); }
};

// (1 - P(2n, z)) Gamma(2n) - target   (SersicMissingFlux, SBSersic.cpp:541-556)
struct SersicMissingFlux {
    double twon, gam, target;
    __device__ double operator()(double z) const { return (1. - gamma_p(twon, z)) * gam - target; }
};

// CalculateB (SBSersic.cpp:627-658)
__device__ RootResult sersic_b(double n, double gamma2n, double flux_fraction)
{
    const double invn = 1. / n, invnsq = invn * invn;
    const double b1 = 2. * n - 1. / 3.;
    const double b2 = b1 + (8. / 405.) * invn + (46. / 25515.) * invnsq +
                      (131. / 1148175.) * invn * invnsq;
    SersicMissingFlux f{2. * n, gamma2n, (1. - 0.5 * flux_fraction) * gamma2n};
    return solve_bracket_lower_limit(f, b1, b2, 0.);
}

// calculateMissingFluxRadius (SBSersic.cpp:558-625); result in units of r0.
__device__ RootResult sersic_missing_flux_radius(double n, double gamma2n, double b,
                                                 double missing_frac)
{
    const double missing_flux = missing_frac * gamma2n;
    double z1 = -log(missing_flux);
    double z;
    if (n == 0.5) {
        z = z1;
    } else {
        z = 4. * (n + 1.);
        const double twonm1 = 2. * n - 1.;
        double z2 = z1 + twonm1 * log(z) + twonm1 / z + twonm1 * (2. * n - 3.) / (2. * z * z);
        if (z2 > z1 && z2 - z1 < 0.01) z2 = z1 + 0.01;
        else if (z2 < z1 && z2 - z1 > -0.01) z2 = z1 - 0.01;
        if (z1 < 0.) z1 = b;
        SersicMissingFlux f{2. * n, gamma2n, missing_flux};
        RootResult r = solve_bracket_upper(f, z1, z2);
        if (!r.ok) return {0., false};
        z = r.x;
    }
    return {pow(z, n), true};
}

// Truncated Sersic sizes (sersic.py:218-247 with SersicTruncatedScale / SersicIntegratedFlux,
// src/SBSersic.cpp:332-336, 688-775): per profile (n, size, trunc, flags) with flags bit 0 = size
// is a half-light radius, bit 1 = flux_untruncated:
//   r0 = size                                 (scale radius given)
//   r0 = hlr / b_untruncated(n)^n             (hlr given, flux_untruncated)
//   r0 = hlr * CalculateTruncatedScale(n, b, trunc / hlr)   (hlr of the truncated profile)
// and the flux fraction gamma_p(2n, (trunc / r0)^(1/n)) inside trunc.
struct SersicTruncatedHLR {
    double twon, x, gam;
    __device__ double operator()(double b) const
    { return (2. * gamma_p(twon, b) - gamma_p(twon, x * b)) * gam; }
};

__global__ void sersic_truncation_kernel(const double* in, int count, double* out, int* status)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const double n = in[4 * i], size = in[4 * i + 1], trunc = in[4 * i + 2];
    const int flags = int(in[4 * i + 3]);
    const double gamma2n = tgamma(2. * n);
    double r0 = size;
    if (flags & 1) {
        const RootResult rb = sersic_b(n, gamma2n, 1.);
        if (!rb.ok) { atomicOr(status, 1); return; }
        if (flags & 2) {
            r0 = size / pow(rb.x, n);
        } else {
            // b solves gamma_p(2n, b) = gamma_p(2n, x b) / 2, x = (trunc / hlr)^(1/n), bracketed
            // by the asymptotic guess (or b / 2) and the untruncated b (SBSersic.cpp:688-768)
            const double x = pow(trunc / size, 1. / n);
            double b1 = (log(0.5) + (2. * n - 1.) * log(x)) / (x - 1.);
            if (b1 < 1e-3 * rb.x) b1 = 0.5 * rb.x;
            const RootResult rt = solve_bracket_lower_limit(SersicTruncatedHLR{2. * n, x, gamma2n}, b1, rb.x, 0.);
            if (!rt.ok) { atomicOr(status, 1); return; }
            r0 = size / pow(rt.x, n);
        }
    }
    out[2 * i] = r0;
    out[2 * i + 1] = gamma_p(2. * n, pow(trunc / r0, 1. / n));
}

// Per-table constants.  A block holds 32 tables and three warps, one per independent part (the
// low-k series and grid, the half-light radius, the missing-flux radius):
// each part is a chain of dependent FP64 divisions, so taking them side by side rather than in
// one thread sets the kernel's time (a few hundred tables: 65-100 us in one thread each).
__global__ void __launch_bounds__(96) sersic_setup_kernel(const double* n_arr, const double* trunc_arr, int count,
                                                           gsb_gsparams gsp, double* header, int stride,
                                                           double* dheader)
{
    __shared__ int bad_b[32], bad_r[32];
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int s = blockIdx.x * 32 + lane;
    const bool live = s < count;
    double* H = header + (size_t)(live ? s : 0) * kSersicHeader;
    const double n = live ? n_arr[s] : 1.;
    const double trunc = live && trunc_arr ? trunc_arr[s] : 0.;      // in units of r0
    const double gamma2n = tgamma(2. * n);
    // truncated profiles (SBSersic.cpp:332-352, 393-424): the flux fraction inside trunc and the
    // moments of the truncated profile
    const double z = trunc > 0. ? pow(trunc, 1. / n) : 0.;
    const double ff = trunc > 0. ? gamma_p(2. * n, z) : 1.;
    if (live && part == 0) {
        double gamma4n = tgamma(4. * n);
        double gamma6n = tgamma(6. * n);
        double gamma8n = tgamma(8. * n);
        if (trunc > 0.) {
            gamma4n *= gamma_p(4. * n, z);
            gamma6n *= gamma_p(6. * n, z);
            gamma8n *= gamma_p(8. * n, z);
        }
        // buildFT low-k series (SBSersic.cpp:386-424)
        const double kderiv2 = -gamma4n / (4. * gamma2n) / ff;
        const double kderiv4 = gamma6n / (64. * gamma2n) / ff;
        const double kderiv6 = gamma8n / (2304. * gamma2n) / ff;
        const double kmin = pow(gsp.kvalue_accuracy / kderiv6, 1. / 6.);
        const double dlogk = gsp.table_spacing * sqrt(sqrt(gsp.kvalue_accuracy / 10.));
        int ncand = 0;
        const double logk_end = log(500.);
        for (double logk = log(kmin) - 0.001; logk < logk_end && ncand < stride; logk += dlogk)
            ++ncand;
        H[kSH_N] = n;
        H[kSH_NUSED] = 0;
        H[kSH_FRONT] = log(kmin) - 0.001;
        H[kSH_DA] = dlogk;
        H[kSH_KSQMIN] = kmin * kmin;
        H[kSH_KSQMAX] = 0.;
        H[kSH_KD2] = kderiv2;
        H[kSH_KD4] = kderiv4;
        H[kSH_HIGHA] = 0.;
        H[kSH_HIGHB] = 0.;
        H[kSH_MAXK] = kmin;
        H[kSH_DLOGK] = dlogk;
        H[kSH_NCAND] = ncand;
        H[kSH_TRUNC] = trunc;
        H[kSH_FLUXFRAC] = ff;
        if (dheader) {
            // d/dn of the low-k coefficients (ratios of Gamma functions)
            double* D = dheader + (size_t)s * kSersicDHeader;
            const double psi2 = digamma(2. * n);
            D[kSD_DKD2] = kderiv2 * (4. * digamma(4. * n) - 2. * psi2);
            D[kSD_DKD4] = kderiv4 * (6. * digamma(6. * n) - 2. * psi2);
            D[kSD_DHIGHA] = 0.;
            D[kSD_DHIGHB] = 0.;
            // front = ln k_min - 0.001 with k_min = (kvalue_accuracy / kderiv6)^(1/6)
            D[kSD_DFRONT] = -(8. * digamma(8. * n) - 2. * psi2) / 6.;
        }
    } else if (part == 1) {
        const RootResult rb = sersic_b(n, gamma2n, ff);
        bad_b[lane] = !rb.ok;
        if (live) {
            const double b = rb.x;
            H[kSH_RE] = pow(b, n);
            if (dheader) {
                // d ln(r_e / r0) / dn, r_e = b^n: db/dn from P(2n, b) = 1/2 by implicit differentiation
                const double dPdb = exp(-b + (2. * n - 1.) * log(b) - lgamma(2. * n));
                const double dbdn = -2. * gamma_p_da(2. * n, b) / dPdb;
                dheader[(size_t)s * kSersicDHeader + kSD_DLNRE] = log(b) + n * dbdn / b;
            }
        }
    } else if (part == 2) {
        // stepK (SBSersic.cpp:304-318): the untruncated missing-flux radius (its lower bracket falls
        // back to the profile's own b, :589-592), capped at trunc
        double b = 0.;
        if (-log(gsp.folding_threshold * gamma2n) < 0.) b = sersic_b(n, gamma2n, ff).x;
        const RootResult rr = sersic_missing_flux_radius(n, gamma2n, b, gsp.folding_threshold);
        bad_r[lane] = !rr.ok;
        double R = rr.x;
        if (trunc > 0. && trunc < R) R = trunc;
        R = fmax(R, gsp.stepk_minimum_hlr);
        if (live) H[kSH_STEPK] = kPi / R;
    }
    __syncthreads();
    if (live && part == 0) H[kSH_STATUS] = bad_r[lane] ? 3 : bad_b[lane] ? 2 : 0;
}

// Running state of a truncated table's stopping scan (buildFT, SBSersic.cpp:436-509): the 10-point
// high-k least-squares fit, advanced one round of nodes at a time so that few nodes past the
// stopping point are integrated.
struct SersicScan {
    double sf, skf, sk, sk2;
    double fit[10];
    int fit_size, fit_head, n_correct, nused, done;
};

__global__ void sersic_scan_init_kernel(const double* header, int count, SersicScan* scan)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= count) return;
    SersicScan& S = scan[s];
    const double* H = header + (size_t)s * kSersicHeader;
    S.sf = S.skf = S.sk = S.sk2 = 0.;
    S.fit_size = S.fit_head = S.n_correct = S.nused = 0;
    S.done = H[kSH_TRUNC] <= 0. || int(H[kSH_NCAND]) < 2 ? 1 : 0;
}

// One warp per node of this round for the truncated tables (trunc > 0): the truncated Hankel transform / hankel_norm, hankel_norm = flux fraction n Gamma(2n).
__global__ void __launch_bounds__(256) sersic_trunc_nodes_kernel(const double* header, int count, int i0,
                                    int nround, const __grid_constant__ OgataTables og, const SersicScan* scan,
                                    double* vals, int stride, const int* prev_live, int* status_out)
{
    if (prev_live && *prev_live == 0) return;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long s = warp / nround;
    const int i = i0 + int(warp % nround);
    if (s >= count) return;
    const double* H = header + s * kSersicHeader;
    if (H[kSH_TRUNC] <= 0. || scan[s].done) return;
    if (i >= int(H[kSH_NCAND])) return;
    const double n = H[kSH_N];
    const double k = exp(H[kSH_FRONT] + i * H[kSH_DLOGK]);
    const double hankel_norm = H[kSH_FLUXFRAC] * n * tgamma(2. * n);
    int st = 0;
    const double v = warp_hankel_trunc(og, SersicRadial{1. / n}, k, H[kSH_TRUNC], &st) / hankel_norm;
    if ((threadIdx.x & 31) == 0) {
        vals[s * stride + i] = v;
        if (st) atomicOr(status_out, 1);
    }
}

// The stopping scan of the truncated tables, whose nodes are integrated in rounds (the others stop
// inside sersic_table_kernel).  live_out is set when a table still needs nodes after this round; a
// zero prev_live (the previous round's flag) means every table has stopped and the launch returns
// at once.
__global__ void sersic_scan_kernel(const double* header, int count, int stride, int i0, int nround,
                                   gsb_gsparams gsp, const double* vals, SersicScan* scan,
                                   const int* prev_live, int* live_out)
{
    if (prev_live && *prev_live == 0) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= count) return;
    if (scan[s].done) return;
    SersicScan S = scan[s];
    const double* H = header + (size_t)s * kSersicHeader;
    const double* v = vals + (size_t)s * stride;
    const int ncand = int(H[kSH_NCAND]);
    const double front = H[kSH_FRONT], dlogk = H[kSH_DLOGK];
    const int n_fit = 10;
    const int iend = min(i0 + nround, ncand);
    for (int i = i0; i < iend; ++i) {
        const double logk = front + i * dlogk;
        const double k = exp(logk), ksq = k * k;
        const double val = v[i];
        const double f0 = val * ksq;
        if (fabs(val) > gsp.maxk_threshold) { S.n_correct = 0; }
        else {
            const double den = n_fit * S.sk2 - S.sk * S.sk;
            const double a = (S.sf * S.sk2 - S.sk * S.skf) / den;
            const double b = (n_fit * S.skf - S.sk * S.sf) / den;
            const double f0_pred = a + b / k;
            if (fabs(f0 - f0_pred) / ksq < gsp.kvalue_accuracy) ++S.n_correct;
            else S.n_correct = 0;
            // (one node more than the stop itself: sersic_table_kernel forms its window sums
            // afresh, and a stop that its rounding moved would read the next node)
            if (S.n_correct >= 6) { S.done = 1; S.nused = iend; scan[s] = S; return; }
        }
        const double inv_k = 1. / k;
        if (S.fit_size == n_fit) {
            const double k_back = exp(logk - n_fit * dlogk);
            const double f_back = S.fit[S.fit_head];
            const double inv_k_back = 1. / k_back;
            S.sf += f0 - f_back;
            S.skf += f0 * inv_k - f_back * inv_k_back;
            S.sk += inv_k - inv_k_back;
            S.sk2 += inv_k * inv_k - inv_k_back * inv_k_back;
            S.fit[S.fit_head] = f0;
            S.fit_head = (S.fit_head + 1) % n_fit;
        } else {
            S.sf += f0;
            S.skf += f0 * inv_k;
            S.sk += inv_k;
            S.sk2 += inv_k * inv_k;
            S.fit[S.fit_size++] = f0;
        }
    }
    if (iend >= ncand) S.done = 1;
    S.nused = iend;
    scan[s] = S;
    if (!S.done && live_out) *live_out = 1;
}

// Natural cubic spline second derivatives z of nodes (x, y) (Thomas algorithm; c is scratch).
// TSpline setup, src/Table.cpp:634-686.
__device__ void natural_spline(const double* x, const double* y, double* z, double* c, int N)
{
    for (int i = 0; i < N; ++i) z[i] = 0.;
    if (N == 3) {
        z[1] = 3. * ((y[2] - y[1]) / (x[2] - x[1]) - (y[1] - y[0]) / (x[1] - x[0])) / (x[2] - x[0]);
    } else if (N > 3) {
        for (int i = 1; i <= N - 2; ++i)
            z[i] = 6. * ((y[i + 1] - y[i]) / (x[i + 1] - x[i]) - (y[i] - y[i - 1]) / (x[i] - x[i - 1]));
        double bb = 2. * (x[2] - x[0]);
        for (int i = 1; i <= N - 2; ++i) {
            z[i] /= bb;
            if (i == N - 2) break;
            const double aa = x[i + 1] - x[i];
            const double cc = aa / bb;
            c[i - 1] = cc;
            bb = 2. * (x[i + 2] - x[i]);
            bb -= aa * cc;
            z[i + 1] -= aa * z[i];
        }
        for (int i = N - 3; i > 0; --i) z[i] -= c[i - 1] * z[i + 1];
    }
}

// One Sersic table per block: the transforms at the ln k nodes (the reference's adaptive halving,
// AdaptiveHankelIntegrator::integrate, Hankel.cpp:179-219, on the resampled levels), buildFT's
// stopping rule, high-k fit and maxk (SBSersic.cpp:436-537) and the natural spline (Table.cpp:634-686).
//
// The samples of G (and of its n-derivative) over the whole grid the table can reach are formed
// once in shared memory; a warp then takes 32 R consecutive nodes, R a thread, through the levels
// in step: a node starts at its own level (h0 = 1/32 halved while h0 > 100 k), keeps its last two
// sums and drops out at the first level where the reference's test passes.  After each chunk of
// THREADS x R nodes every thread tests its own nodes for the stop, so nodes past the stop cost at
// most the rest of a chunk.  The spline's tridiagonal system on the uniform grid,
// z_(i-1) + 4 z_i + z_(i+1) = d_i, is solved by its Green's function (-lambda)^|e| / (2 sqrt 3),
// lambda = 2 - sqrt 3 (2e-18 at |e| = 31), with d continued odd about both ends.
//
// Bound by the latency of the multiply-add chains and the shared-memory reads that feed them (R = 3:
// one read per three).  4096 tables, n in 0.5 .. 4: 1.05 ms, where integrating each node pair by
// its scattered sums (three exponentials a pair of terms) in rounds with a scan and a spline
// kernel after them took 10.3 ms; 113 tables 0.16 ms (0.31 with one
// sum a node and the level values read from L2), 1.4 before.
// R = 1 with 512 threads serves builds of a few tables per SM (kSmallBuild), where a block's
// latency counts and SMs are idle.
//
// Dynamic shared memory: [G samples | (DN) derivative samples | values | (DN) derivative values | flags |
// staged level values], gcap + pad doubles a sample array and stride doubles a value array; the
// spline's right-hand side takes the place of the samples.
template <int R, int THREADS, bool DN, bool P1>
__global__ void __launch_bounds__(THREADS, THREADS > 64 ? 1 : 8) sersic_table_kernel(
    double* header, int count, int stride, gsb_gsparams gsp, const __grid_constant__ OgataLog lg, int p, int mul,
    int gcap, int pad, int stage, const SersicScan* scan, const double* tvals, double4* nodes, double4* dnodes, double* dheader,
    int* status_out)
{
    extern __shared__ double tsm[];
    __shared__ int s_stop, s_above, s_below;
    const int lane = threadIdx.x & 31;
    // slots hold ascending n; the costly large-n tables are taken first so that they do not form
    // the tail of the launch
    const int s = count - 1 - int(blockIdx.x);
    double* H = header + (size_t)s * kSersicHeader;
    double* g = tsm;
    double* gd = g + gcap + pad;
    double* V = DN ? gd + gcap + pad : gd;
    double* DV = V + stride;
    const bool trunc = H[kSH_TRUNC] > 0.;
    int ncand = int(H[kSH_NCAND]);
    if (ncand < 2) {
        if (threadIdx.x == 0) { H[kSH_STATUS] = 5; H[kSH_NUSED] = 0; }
        return;
    }
    const double n = H[kSH_N], invn = 1. / n;
    const double front = H[kSH_FRONT], dlogk = H[kSH_DLOGK];
    const double norm = n * tgamma(2. * n);
    const double abserr = gsp.integration_abserr * norm;
    const double dnc = DN ? dheader[(size_t)s * kSersicDHeader + kSD_DFRONT] : 0.;
    // samples d = d0 .. dmax at y = d hs - front; beyond dmax f = exp(-u) is 0 (u > 745)
    const double hs = lg.h / mul;
    const int dmax = int(floor((front + 6.6134 * n) / hs));
    const int d0 = dmax - gcap + 1;
    if (trunc) {
        ncand = min(ncand, scan[s].nused);
        for (int i = threadIdx.x; i < ncand; i += THREADS) V[i] = tvals[(size_t)s * stride + i];
    } else {
        for (int j = threadIdx.x; j < gcap + pad; j += THREADS) {
            const double2 v = j < gcap ? sersic_sample((d0 + j) * hs - front, invn, dnc) : make_double2(0., 0.);
            g[j] = v.x;
            if (DN) gd[j] = v.y;
        }
    }
    if (threadIdx.x == 0) { s_stop = ncand; s_above = s_below = -1; }
    __syncthreads();

    const int n_fit = 10;
    // The fit's four sums (f0, f0 / k, 1 / k, 1 / k^2 over the 10 nodes before node i) are running
    // sums, as in the reference: they carry the rounding of the first nodes' 1 / k, which at
    // large n is what the fit consists of, so the order of the additions is kept.  Their steps are
    // formed by all threads, then four lanes run through the chunk.
    constexpr int CHUNK = THREADS * R;
    __shared__ double sums[4][CHUNK];
    __shared__ double s_end[4], s_fit[2];
    double carry = 0.;                       // lanes 0-3 of warp 0: the sum before the next chunk
    auto fit = [&](double sf, double skf, double sk, double sk2, double& a, double& b) {
        const double den = n_fit * sk2 - sk * sk;
        a = (sf * sk2 - sk * skf) / den;
        b = (n_fit * skf - sk * sf) / den;
    };

    unsigned char* ok = reinterpret_cast<unsigned char*>(DN ? DV + stride : V + stride);
    // the first `stage` level values, for the small builds: a block alone on its SM would wait for each
    // line of them from L2
    double* staged = reinterpret_cast<double*>(ok + ((stride + 15) & ~7));
    for (int i = threadIdx.x; i < stage; i += THREADS) staged[i] = lg.a[i];
    __syncthreads();
    for (int c0 = 0; c0 < ncand; c0 += THREADS * R) {
        const int c1 = min(ncand, c0 + THREADS * R);
        const int w0 = c0 + int(threadIdx.x >> 5) * 32 * R;      // this warp's nodes w0 .. w0 + 32 R - 1
        if (!trunc && w0 < c1) {
            const int m = w0 + lane * R;
            double prev[R], cur[R], dcur[R], ksq[R];
            int lev[R];
            unsigned run = 0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const double k = exp(front + (m + r) * dlogk);
                ksq[r] = k * k;
                prev[r] = cur[r] = dcur[r] = 0.;
                int l = kLogLev0;
                for (double h0 = 1. / 32.; h0 > 100. * k && l < 60; h0 *= 0.5) ++l;
                lev[r] = l;
                if (m + r < c1) run |= 1u << r;
            }
            int l = lev[R - 1];                                   // k ascends: the warp's lowest level
            l = __reduce_min_sync(0xffffffffu, run ? l : 99);
            const int mlast = min(c1 - 1, w0 + 32 * R - 1);
            while (__any_sync(0xffffffffu, run != 0u)) {
                // the reference halves until its level counter passes 60: the last sum is at 61
                if (l >= kLogLev0 + lg.have) {
                    if (lane == 0) atomicOr(status_out, lg.have == kLogLevels ? 1 : 2);   // (2: spread more)
                    break;
                }
                const int j = l - kLogLev0;
                const int qmin = lg.qmin[j];
                const double* A = (lg.off[j] + lg.len[j] <= stage ? staged : lg.a) + lg.off[j] - qmin;
                // the nodes still at work in this warp bound the samples that count
                int mhi = 0;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if ((run >> r & 1u) && l >= lev[r]) mhi = m + r;
                mhi = __reduce_max_sync(0xffffffffu, mhi);
                const int dhi = p * mhi + dmax, dlo = d0 + p * mlast + (R - 1) * p;
                const int qhi = min(qmin + lg.len[j] - 1, dhi >= 0 ? dhi / mul : -((mul - 1 - dhi) / mul));
                // samples below d0 (levels far beyond the usual) are formed on the fly
                const int qlo = max(qmin, dlo >= 0 ? (dlo + mul - 1) / mul : -(-dlo / mul));
                double acc[kLogSums][R], dacc[kLogSums][R];
#pragma unroll
                for (int c = 0; c < kLogSums; ++c)
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[c][r] = dacc[c][r] = 0.;
                int q = qmin;
                for (; q < min(qlo, qhi + 1); q += kLogSums) {
#pragma unroll
                    for (int c = 0; c < kLogSums; ++c) {
                        if (q + c > qhi) continue;
                        const double a = A[q + c];
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const double2 v = sersic_sample(((q + c) * mul - p * (m + r)) * hs - front, invn, dnc);
                            acc[c][r] = fma(a, v.x, acc[c][r]);
                            if (DN) dacc[c][r] = fma(a, v.y, dacc[c][r]);
                        }
                    }
                }
                // (lanes past mlast read other samples of the array, or its zero padding)
                if (q <= qhi)
                    correlate<R, DN, P1>(A, q, qhi, g - d0, gd - d0, min(m, mlast), p, mul, dmax + 1, acc, dacc);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (!(run >> r & 1u) || l < lev[r]) continue;
                    prev[r] = cur[r];
                    cur[r] = (acc[0][r] + acc[1][r]) / ksq[r];
                    if (DN) dcur[r] = (dacc[0][r] + dacc[1][r]) / ksq[r];
                    if (l == lev[r]) continue;
                    const double err = fabs(cur[r] - prev[r]);
                    const bool more = (err > gsp.integration_relerr * cur[r] &&
                                       (err > abserr || fabs(cur[r]) > 2. * fabs(prev[r]))) || cur[r] == 0.;
                    if (!more) run &= ~(1u << r);
                }
                ++l;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (m + r >= c1) continue;
                const double v = cur[r] / norm;
                V[m + r] = v;
                // node value y = v k^2 = T(k) / norm with norm = n Gamma(2n) and k = k_i(n):
                // dy/dn = (dT/dn) / norm - y (1/n + 2 psi(2n)), dT/dn from the second correlation.
                if (DN) DV[m + r] = (dcur[r] / norm - v * (1. / n + 2. * digamma(2. * n))) * ksq[r];
            }
        }
        __syncthreads();
        for (int i = c0 + threadIdx.x; i < c1; i += THREADS) {
            const double logk = front + i * dlogk;
            const double k = exp(logk), ksq = k * k, f0 = V[i] * ksq, inv_k = 1. / k;
            const int j = i - c0;
            if (i >= n_fit) {
                const double k_back = exp(logk - n_fit * dlogk);
                const double kb = exp(front + (i - n_fit) * dlogk);
                const double f_back = V[i - n_fit] * (kb * kb);
                const double inv_k_back = 1. / k_back;
                sums[0][j] = f0 - f_back;
                sums[1][j] = f0 * inv_k - f_back * inv_k_back;
                sums[2][j] = inv_k - inv_k_back;
                sums[3][j] = inv_k * inv_k - inv_k_back * inv_k_back;
            } else {
                sums[0][j] = f0;
                sums[1][j] = f0;             // times 1 / k and 1 / k^2 below, fused with the addition
                sums[2][j] = inv_k;
                sums[3][j] = inv_k;
            }
        }
        __syncthreads();
        if (threadIdx.x < 4) {
            double* sm = sums[threadIdx.x];
            int j = 0;
            for (; j < c1 - c0 && c0 + j < n_fit; ++j) {
                const double v = sm[j], inv_k = 1. / exp(front + (c0 + j) * dlogk);
                const double next = threadIdx.x == 1 ? fma(v, inv_k, carry) : threadIdx.x == 3 ? fma(v, v, carry) : carry + v;
                sm[j] = carry;
                carry = next;
            }
#pragma unroll 8
            for (; j < c1 - c0; ++j) {
                const double v = sm[j];
                sm[j] = carry;
                carry += v;
            }
        }
        __syncthreads();
        // the stop: the fifth in a row of the nodes below maxk_threshold that the fit predicts
        for (int i = c0 + threadIdx.x; i < c1; i += THREADS) {
            const int j = i - c0;
            const double k = exp(front + i * dlogk), ksq = k * k;
            bool good = false;
            if (!(fabs(V[i]) > gsp.maxk_threshold)) {
                double a, b;
                fit(sums[0][j], sums[1][j], sums[2][j], sums[3][j], a, b);
                good = fabs(V[i] * ksq - (a + b / k)) / ksq < gsp.kvalue_accuracy;
            }
            ok[i] = good;
        }
        __syncthreads();
        for (int i = max(c0, 4) + int(threadIdx.x); i < c1; i += THREADS)
            if (ok[i] && ok[i - 1] && ok[i - 2] && ok[i - 3] && ok[i - 4]) atomicMin(&s_stop, i);
        __syncthreads();
        // the last node whose fit was taken (the stop, if any), and the last above the threshold
        const int end = min(c1, s_stop + 1);
        for (int i = c0 + threadIdx.x; i < end; i += THREADS)
            atomicMax(fabs(V[i]) > gsp.maxk_threshold ? &s_above : &s_below, i);
        __syncthreads();
        if (threadIdx.x == 0 && s_below >= c0) {
            const int j = s_below - c0;
            fit(sums[0][j], sums[1][j], sums[2][j], sums[3][j], s_fit[0], s_fit[1]);
        }
        if (s_stop < ncand) break;
    }
    if (threadIdx.x < 4) s_end[threadIdx.x] = carry;
    const bool stopped = s_stop < ncand;
    const int N = stopped ? s_stop + 1 : ncand;
    // the spline's right-hand side, in the samples' place
    double* D = tsm;
    const double ih2 = 6. / (dlogk * dlogk);
    auto f0 = [&](int i) { const double k = exp(front + i * dlogk); return V[i] * (k * k); };
    for (int i = threadIdx.x; i < N; i += THREADS) {
        const bool in = i > 0 && i < N - 1;
        D[i] = in ? ih2 * ((f0(i + 1) - f0(i)) - (f0(i) - f0(i - 1))) : 0.;
    }
    __syncthreads();
    const double back = front + (N - 1) * dlogk;
    if (threadIdx.x == 0) {
        double a, b, maxk, ksq_max;
        if (s_below >= 0) {
            a = s_fit[0];
            b = s_fit[1];
            maxk = (s_above >= 0 ? exp(front + s_above * dlogk) : sqrt(H[kSH_KSQMIN])) * exp(dlogk);
        } else {
            fit(s_end[0], s_end[1], s_end[2], s_end[3], a, b);
            maxk = sqrt(a / gsp.maxk_threshold);
            for (int it = 0; it < 3; ++it) maxk = sqrt((a - b / maxk) / gsp.maxk_threshold);
        }
        if (stopped) {
            const double k = exp(back);
            ksq_max = k * k;
        } else {
            ksq_max = exp(2. * back);
        }
        H[kSH_NUSED] = N;
        H[kSH_DA] = (back - front) / (N - 1);
        H[kSH_KSQMAX] = ksq_max;
        H[kSH_HIGHA] = a;
        H[kSH_HIGHB] = b;
        H[kSH_MAXK] = maxk;
    }
    // z_i = sum_e G(e) d_(i + e), d odd about nodes 0 and N - 1 (period 2 (N - 1))
    auto green = [&](const double* d, int i) {
        const int L = N - 1;
        const double lam = -0.26794919243112270647;        // sqrt 3 - 2
        if (N < 3) return 0.;
        auto at = [&](int j) {
            j %= 2 * L;
            if (j < 0) j += 2 * L;
            return j <= L ? d[j] : -d[2 * L - j];
        };
        double w = 1., sum = d[i];
        if (i >= 31 && i + 31 <= L) {
            for (int e = 1; e <= 31; ++e) { w *= lam; sum = fma(w, d[i - e] + d[i + e], sum); }
        } else {
            for (int e = 1; e <= 31; ++e) { w *= lam; sum = fma(w, at(i - e) + at(i + e), sum); }
        }
        return sum * 0.28867513459481288225;               // 1 / (2 sqrt 3)
    };
    double4* nd = nodes + (size_t)s * stride;
    // .w: k^2 at the node, for the evaluators' spline offset 0.5 ln(k_i^2 / k^2)
    for (int i = threadIdx.x; i < N; i += THREADS) {
        const double x = front + i * dlogk;
        nd[i] = make_double4(x - front, f0(i), (i == 0 || i == N - 1) ? 0. : green(D, i), exp(2. * x));
    }
    if (DN) {
        // The spline is linear in its node values, so d/dn of the interpolant is the spline of
        // the node derivatives on the same grid.  Likewise the high-k fit is linear in the f0
        // values of its window: the 10 nodes before the stopping node, or the last 10 nodes
        // when the scan ran to the end of the candidate grid.
        double4* dn = dnodes + (size_t)s * stride;
        __syncthreads();
        for (int i = threadIdx.x; i < N; i += THREADS)
            D[i] = i > 0 && i < N - 1 ? ih2 * ((DV[i + 1] - DV[i]) - (DV[i] - DV[i - 1])) : 0.;
        __syncthreads();
        for (int i = threadIdx.x; i < N; i += THREADS)
            dn[i] = make_double4(front + i * dlogk - front, DV[i], (i == 0 || i == N - 1) ? 0. : green(D, i), 0.);
        if (threadIdx.x == 0) {
            // The fit's 1/k_i move too: d(1/k_i)/dn = -c / k_i with c = dfront/dn.
            double* Dh = dheader + (size_t)s * kSersicDHeader;
            const double c = dnc;
            const int wend = stopped ? N - 1 : N;
            const int wbeg = wend - n_fit > 0 ? wend - n_fit : 0;
            double sk = 0., sk2 = 0., sf = 0., skf = 0., dsf = 0., dskf = 0.;
            for (int i = wbeg; i < wend; ++i) {
                const double inv_k = exp(-(front + i * dlogk));
                const double f = f0(i), df = DV[i];
                sk += inv_k;
                sk2 += inv_k * inv_k;
                sf += f;
                skf += f * inv_k;
                dsf += df;
                dskf += (df - c * f) * inv_k;
            }
            const double dsk = -c * sk, dsk2 = -2. * c * sk2;
            const double den = n_fit * sk2 - sk * sk, dden = n_fit * dsk2 - 2. * sk * dsk;
            const double na = sf * sk2 - sk * skf, dna = dsf * sk2 + sf * dsk2 - dsk * skf - sk * dskf;
            const double nb = n_fit * skf - sk * sf, dnb = n_fit * dskf - dsk * sf - sk * dsf;
            Dh[kSD_DHIGHA] = (dna * den - na * dden) / (den * den);
            Dh[kSD_DHIGHB] = (dnb * den - nb * dden) / (den * den);
        }
    }
}

// Truncated Moffat FT tables (SBMoffat::setupFT, src/SBMoffat.cpp:565-625).  Per slot
// (beta, t = trunc / rD): the values
//     v(k) = 2 (beta - 1) / F  int_0^t r (1 + r^2)^-beta J0(k r) dr,  F = 1 - (1 + t^2)^(1 - beta)
// on the reference's grid k = 0, dk, 2 dk, ... (its running sum, k < 50), one warp per node for
// all candidate nodes at once; then, per slot, the reference's stopping rule (5 nodes in a row
// with |v| <= kvalue_accuracy end the table), maxk (the last node with |v| > maxk_threshold,
// refined linearly toward the next node) and the natural cubic spline in k^2.
__global__ void moffat_setup_kernel(int count, double* header)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= count) return;
    double* H = header + (size_t)s * kMoffatHeader;
    H[kMH_FLUXFACTOR] = 1. - pow(1. + H[kMH_TRUNC] * H[kMH_TRUNC], 1. - H[kMH_BETA]);
}

__global__ void __launch_bounds__(256) moffat_nodes_kernel(const double* header, int count, const double* kgrid,
                                                           int ncand, const __grid_constant__ OgataTables og,
                                                           double* vals, int* status_out)
{
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long s = warp / ncand;
    const int i = int(warp % ncand);
    if (s >= count) return;
    const double* H = header + s * kMoffatHeader;
    const double b = H[kMH_BETA];
    const double prefactor = 2. * (b - 1.) / H[kMH_FLUXFACTOR];
    int st = 0;
    const double v = prefactor * warp_hankel_trunc(og, MoffatRadial{b}, kgrid[i], H[kMH_TRUNC], &st);
    if ((threadIdx.x & 31) == 0) {
        vals[s * ncand + i] = v;
        if (st) atomicOr(status_out, 1);
    }
}

// One warp per slot; dynamic shared memory 4 * ncand doubles.
__global__ void __launch_bounds__(32) moffat_finalize_kernel(double* header, int count, const double* kgrid,
                                                             int ncand, gsb_gsparams gsp, const double* vals,
                                                             double4* nodes)
{
    extern __shared__ double msm[];
    const int s = blockIdx.x;
    const int lane = threadIdx.x;
    if (s >= count) return;
    double* xs = msm;
    double* ys = xs + ncand;
    double* zs = ys + ncand;
    double* cs = zs + ncand;
    const double* v = vals + (size_t)s * ncand;
    for (int i = lane; i < ncand; i += 32) {
        xs[i] = kgrid[i] * kgrid[i];
        ys[i] = v[i];
    }
    __syncwarp();
    __shared__ int n_used;
    if (lane == 0) {
        double* H = header + (size_t)s * kMoffatHeader;
        // the reference's loop over k: maxk bookkeeping and the stopping rule
        int im = 0, nbelow = 0, N = ncand;
        for (int i = 0; i < ncand; ++i) {
            const double a = fabs(ys[i]);
            if (a > gsp.maxk_threshold) im = i;
            nbelow = a > gsp.kvalue_accuracy ? 0 : nbelow + 1;
            if (nbelow == 5) { N = i + 1; break; }
        }
        double maxk = kgrid[im];
        // the refinement between k1 = maxk and k2 = maxk + dk (both tabulated nodes when k2 < 50,
        // where the spline returns the node values)
        const double k2 = maxk + H[kMH_DK];
        if (k2 < 50. && im + 1 < N) {
            const double f1 = fabs(ys[im]), f2 = fabs(ys[im + 1]);
            maxk = (maxk * (f2 - gsp.maxk_threshold) + k2 * (gsp.maxk_threshold - f1)) / (f2 - f1);
        }
        if (N >= 2) natural_spline(xs, ys, zs, cs, N);
        H[kMH_NUSED] = N;
        H[kMH_KSQMAX] = xs[N - 1];
        H[kMH_MAXK] = maxk;
        if (N < 2) H[kMH_STATUS] = 5;
        n_used = N;
    }
    __syncwarp();
    const int N = n_used;
    double4* nd = nodes + (size_t)s * ncand;
    for (int i = lane; i < N; i += 32) nd[i] = make_double4(xs[i], ys[i], zs[i], 0.);
}

// Scale radius of truncated Moffat profiles from the half-light radius
// (MoffatCalculateScaleRadiusFromHLR, src/SBMoffat.cpp:103-160): Brent on
//     2 f(re) - f(rm) = 0,   f(R) = 1 - (1 + R^2 / rd^2)^(1 - beta),
// bracketed upward from the untruncated radius r1 and 2 r1.
struct MoffatScaleRadiusFunc {
    double re, rm, beta;
    __device__ double operator()(double rd) const
    {
        const double fre = 1. - pow(1. + (re * re) / (rd * rd), 1. - beta);
        const double frm = 1. - pow(1. + (rm * rm) / (rd * rd), 1. - beta);
        return 2. * fre - frm;
    }
};

__global__ void moffat_scale_radius_kernel(const double* in, int count, double* out, int* status)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const double beta = in[3 * i], re = in[3 * i + 1], rm = in[3 * i + 2];
    const double r1 = re / sqrt(pow(0.5, 1. / (1. - beta)) - 1.);
    // beta <= 1 has no finite untruncated radius to start from: the reference's bracketing
    // fails there too
    if (!(r1 > 0.) || !isfinite(r1)) { atomicOr(status, 1); out[i] = 0.; return; }
    if (rm == 0.) { out[i] = r1; return; }
    const RootResult r = solve_bracket_upper(MoffatScaleRadiusFunc{re, rm, beta}, r1, 2. * r1);
    if (!r.ok) { atomicOr(status, 1); out[i] = 0.; return; }
    out[i] = r.x;
}

// KolmogorovInfo: x-space radial profile by Hankel transform of exp(-k^{5/3}) at
// r = exp(-3 + i dlogr); only the last tabulated point matters for stepk.
__global__ void kolmogorov_nodes_kernel(int ncand, double dlogr, gsb_gsparams gsp, const __grid_constant__ OgataTables og,
                                        double* vals, int* status_out)
{
    const int i = int((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
    if (i >= ncand) return;
    const double r = exp(-3. + i * dlogr);
    KolmKValue f;
    int st = 0;
    const double v = warp_hankel(og, f, r, gsp.integration_relerr, gsp.integration_abserr, &st) /
                     (2. * kPi);
    if ((threadIdx.x & 31) == 0) {
        vals[i] = v;
        if (st) atomicOr(status_out, 1);
    }
}

__global__ void kolmogorov_finalize_kernel(int ncand, double dlogr, gsb_gsparams gsp,
                                           const double* vals, double* out, double4* nodes, double* scratch)
{
    // the reference's loop: entries (r, f(r)) from r = e^-3 until f r^2 / 1.67 < thresh (that
    // entry included), after the analytic f(0) = XVAL_ZERO (SBKolmogorov.cpp:352-384)
    const double thresh = gsp.shoot_accuracy / (2. * kPi);
    double r1 = 0., F1 = 0.;
    int nused = 0;
    for (int i = 0; i < ncand; ++i) {
        const double r = exp(-3. + i * dlogr);
        r1 = r; F1 = vals[i];
        nused = i + 1;
        if (vals[i] * r * r / 1.67 < thresh) break;
    }
    const double n = 11. / 3.;
    double R = pow(2. * kPi * F1 * pow(r1, n) / ((n - 2.) * gsp.folding_threshold), 1. / (n - 2.));
    const double hlr = 2.992939911888651 * 0.5548101137;
    R = fmax(R, gsp.stepk_minimum_hlr * hlr);
    out[0] = kPi / R;
    // the radial table's natural spline in r (Table::spline, src/Table.cpp:634-686), for the
    // real-space drawing of Kolmogorov leaves
    const int N = nused + 1;
    double* xs = scratch;
    double* ys = xs + N;
    double* zs = ys + N;
    double* cs = zs + N;
    xs[0] = 0.;
    ys[0] = 0.0876786563672346;     // XVAL_ZERO = (3/5) Gamma(6/5) / (2 pi)
    for (int i = 0; i < nused; ++i) { xs[i + 1] = exp(-3. + i * dlogr); ys[i + 1] = vals[i]; }
    natural_spline(xs, ys, zs, cs, N);
    for (int i = 0; i < N; ++i) nodes[i] = make_double4(xs[i], ys[i], zs[i], 0.);
    out[1] = N;
}

// kV2 for the Moffat maxk solve (MoffatMaxKSolver, SBMoffat.cpp:481-520), normalised to 1
// at k = 0, as a function of ksq.
template <bool WARP>
struct MoffatKV2 {
    int mode;
    double nu, lognorm, thresh;
    __device__ double operator()(double ksq) const
    {
        const double k = sqrt(ksq);
        double v;
        if (mode == 1) v = exp(-k);
        else if (mode == 2) v = exp(-k) * (1. + k);
        else if (mode == 3) v = exp(-k) * (3. + (3. + k) * k) / 3.;
        else v = moffat_kv_fp64<WARP>(nu, lognorm, k);
        return v - thresh;
    }
};

struct MoffatRefs {
    const double* header;
    const double4* node;
    int count, stride;
};

struct ImageRefs {
    const ImageSlot* slots;
    const double* info;
    const double2* k64;
    const float2* k32;
    int count;
};

// WARP: a warp per leaf, all lanes in step (few leaves, where the chain of one thread is the time);
// else a thread per leaf.
template <bool WARP>
__global__ void prepare_leaves_kernel(const __grid_constant__ gsb_template tpl, int n_stamps, gsb_gsparams gsp,
                                      gsb_leaf* leaves, const double* sersic_header, MoffatRefs moffat,
                                      double kolm_stepk, ImageRefs images, double* info, int* status_out)
{
    const long long idx = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / (WARP ? 32 : 1);
    if (idx >= (long long)n_stamps * tpl.n_leaves) return;
    const int l = int(idx % tpl.n_leaves);
    gsb_leaf& L = leaves[idx];
    const int type = tpl.leaf_type[l];
    double stepk = 0., maxk = 0.;
    for (int i = 0; i < 8; ++i) L.d[i] = 0.;
    switch (type) {
      case GSB_GAUSSIAN: {
        // gaussian.py:148-155 and SBGaussian.cpp:63-73
        const double sigma = L.p[0];
        L.d[0] = sigma;
        L.d[1] = -2. * log(gsp.kvalue_accuracy);
        L.d[2] = pow(gsp.kvalue_accuracy * 48., 1. / 3.);
        maxk = sqrt(-2. * log(gsp.maxk_threshold)) / sigma;
        const double R = fmax(sqrt(-2. * log(gsp.folding_threshold)),
                              gsp.stepk_minimum_hlr * 1.1774100225154747);
        stepk = kPi / (R * sigma);
        break;
      }
      case GSB_EXPONENTIAL: {
        // exponential.py:131-136, SBExponential.cpp:65-79 and ExponentialInfo :513-543
        const double r0 = L.p[0];
        const double ksq_max = pow(gsp.kvalue_accuracy, -1. / 1.5) - 1.;
        L.d[0] = r0;
        L.d[1] = ksq_max;
        L.d[2] = sqrt(ksq_max);
        maxk = pow(gsp.maxk_threshold, -1. / 3.) / r0;
        const double logx = log(gsp.folding_threshold);
        double R = -logx;
        for (int i = 0; i < 3; ++i) R = log(1. + R) - logx;
        R = fmax(R, gsp.stepk_minimum_hlr * 1.6783469900166605);
        stepk = kPi / R / r0;
        break;
      }
      case GSB_SERSIC: {
        // SBSersic.cpp:71-90 (r0 from hlr via SersicHLR, sersic.py:224-227), :301-324
        const double* H = sersic_header + (size_t)L.table * kSersicHeader;
        const double r0 = (L.flags & GSB_LEAF_SIZE_IS_HLR) ? L.p[1] / H[kSH_RE] : L.p[1];
        L.d[0] = r0;
        maxk = H[kSH_MAXK] / r0;
        stepk = H[kSH_STEPK] / r0;
        if (H[kSH_STATUS] != 0.) atomicOr(status_out, 2);
        break;
      }
      case GSB_MOFFAT: {
        // SBMoffat.cpp:163-244 (kV selection), :481-549 (maxK, stepK)
        const double beta = L.p[0], rD = L.p[1], trunc = L.p[2];
        double maxRrD, flux_factor = 1.;
        L.d[0] = rD;
        L.d[1] = L.flux;
        if (trunc > 0.) {
            // the FT from the slot's spline in k^2 (kV_trunc, SBMoffat.cpp:339-345); the slot
            // must have been built for this (beta, trunc / rD)
            const int slot = L.table;
            if (slot < 0 || slot >= moffat.count) { atomicOr(status_out, 64); break; }
            const double* H = moffat.header + (size_t)slot * kMoffatHeader;
            if (fabs(H[kMH_BETA] - beta) > 1e-12 * fabs(beta) ||
                fabs(H[kMH_TRUNC] - trunc / rD) > 1e-12 * (trunc / rD)) { atomicOr(status_out, 128); break; }
            if (H[kMH_STATUS] != 0.) atomicOr(status_out, 256);
            maxRrD = trunc / rD;
            flux_factor = H[kMH_FLUXFACTOR];
            L.d[2] = 4;
            L.d[3] = H[kMH_DK];
            L.d[4] = H[kMH_KSQMAX];
            L.d[5] = H[kMH_NUSED];
            L.d[6] = __longlong_as_double((long long)(moffat.node + (size_t)slot * moffat.stride));
            maxk = H[kMH_MAXK] / rD;
        } else {
            const double kacc = gsp.kvalue_accuracy;
            int mode = 0;
            double nu = beta - 1.;
            if (fabs(beta - 1.5) < kacc) { mode = 1; }
            else if (fabs(beta - 2.) < kacc) { nu = 1.; }
            else if (fabs(beta - 2.5) < kacc) { mode = 2; }
            else if (fabs(beta - 3.) < kacc) { nu = 2.; }
            else if (fabs(beta - 3.5) < kacc) { mode = 3; }
            else if (fabs(beta - 4.) < kacc) { nu = 3.; }
            L.d[2] = mode;
            L.d[3] = nu;
            const double lognorm = (1. - nu) * log(2.) - lgamma(nu);
            L.d[4] = lognorm;
            MoffatKV2<WARP> f{mode, nu, lognorm, gsp.maxk_threshold};
            RootResult r = solve_bracket_upper(f, 0., 100.);
            if (!r.ok) atomicOr(status_out, 4);
            maxk = sqrt(r.x) / rD;
            maxRrD = sqrt(pow(gsp.xvalue_accuracy, 1. / (1. - beta)) - 1.);
        }
        const double maxR = maxRrD * rD;
        if (beta <= 1.1) {
            stepk = kPi / maxR;
        } else {
            double R = pow(gsp.folding_threshold, 0.5 / (1. - beta)) * rD;
            if (R > maxR) R = maxR;
            // getHalfLightRadius (SBMoffat.cpp:247-258), of the truncated profile when truncated
            const double hlr = rD * sqrt(pow(1. - 0.5 * flux_factor, 1. / (1. - beta)) - 1.);
            R = fmax(R, gsp.stepk_minimum_hlr * hlr);
            stepk = kPi / R;
        }
        break;
      }
      case GSB_KOLMOGOROV: {
        // kolmogorov.py:163-226 (k0), :281-287; SBKolmogorov.cpp:117-121
        const double k0 = 2.992939911888651 / L.p[0];
        L.d[0] = 1. / k0;
        maxk = pow(-log(gsp.kvalue_accuracy), 0.6) * k0;
        stepk = kolm_stepk * k0;
        break;
      }
      case GSB_AIRY: {
        // airy.py:217-222, SBAiry.cpp:66-81, 332-356, 432-445
        const double lod = L.p[0], obs = L.p[1];
        const double D = 1. / lod;
        L.d[0] = 1. / (D * kPi);
        L.d[1] = L.flux / (kPi * (1. - obs * obs));
        L.d[2] = obs;
        L.d[3] = obs * obs;
        maxk = 2. * kPi / lod;
        double R = (obs == 0.) ? 1. / (gsp.folding_threshold * 0.5 * kPi * kPi)
                               : 1. / (gsp.folding_threshold * 0.5 * kPi * kPi * (1. - obs));
        R = fmax(R, gsp.stepk_minimum_hlr * 0.5348321477);
        stepk = kPi / R * D;
        break;
      }
      case GSB_BOX: {
        // box.py:100-106, SBBox.cpp:74-77
        const double w = L.p[0], hgt = L.p[1];
        L.d[0] = w / (2. * kPi);
        L.d[1] = hgt / (2. * kPi);
        maxk = 2. / (gsp.maxk_threshold * fmin(w, hgt));
        stepk = kPi / fmax(w, hgt);
        break;
      }
      case GSB_INTERPOLATED: {
        // SBInterpolatedImage.cpp:97-152: kscale = (N/2) / pi maps k to the k-image's sample
        // index, maxk1 = urange / uscale cuts where the x interpolant's transform is
        // negligible.  stepk holds the flux radius R and maxk the scanned maxk (image units),
        // which the host turns into the profile's world stepk / maxk.
        const int slot = L.table;
        const int xc = int(L.p[0]), kc = int(L.p[1]);
        if (slot < 0 || slot >= images.count) { atomicOr(status_out, 16); break; }
        if (xc < GSB_INTERP_DELTA || xc > GSB_INTERP_SINC || kc < GSB_INTERP_NEAREST ||
            kc > GSB_INTERP_LANCZOS) { atomicOr(status_out, 32); break; }
        // a Lanczos k interpolant: p[2] holds its coefficient block {n, conserve_dc, K_1..5};
        // n <= 3 (at most 7 taps per axis)
        const double* kt = reinterpret_cast<const double*>(__double_as_longlong(L.p[2]));
        if (kc == GSB_INTERP_LANCZOS && (kt == nullptr || kt[0] < 1. || kt[0] > 3.)) {
            atomicOr(status_out, 512);
            break;
        }
        const ImageSlot& I = images.slots[slot];
        if (xc != I.desc.x_interp) { atomicOr(status_out, 1024); break; }
        const int N = I.desc.N;
        L.d[0] = (N / 2) / kPi;
        // a Lanczos x interpolant's urange is its table's uMax (Lanczos::urange)
        L.d[1] = (xc == GSB_INTERP_LANCZOS ? I.desc.x_table[3] : interp_urange(xc, gsp.kvalue_accuracy)) /
                 (1. / (2. * kPi));
        L.d[5] = __longlong_as_double((long long)I.desc.x_table);
        L.d[2] = xc + 16 * kc;
        L.d[3] = __longlong_as_double(kc == GSB_INTERP_LANCZOS ? (long long)kt : 0LL);
        L.d[4] = N;
        L.d[6] = __longlong_as_double((long long)(images.k64 + I.k_offset));
        L.d[7] = __longlong_as_double((long long)(images.k32 + I.k_offset));
        stepk = images.info[2 * slot];
        maxk = images.info[2 * slot + 1];
        break;
      }
      default:
        atomicOr(status_out, 8);
    }
    info[2 * idx] = stepk;
    info[2 * idx + 1] = maxk;
}

}  // namespace

namespace {
__global__ void exp_tab_kernel(const double* x, double* y, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = exp_tab(x[i]);
}

__global__ void exp_tab256_kernel(const double* x, double* y, int n)
{
    __shared__ double etab[256];
    etab[threadIdx.x] = g_exp2_256[threadIdx.x];
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = x[i] < -708. ? 0. : exp_tab256_core(x[i], etab);
}
}  // namespace

int exp_fp64(const double* d_x, double* d_y, int n, int table_size, cudaStream_t stream)
{
    if (n <= 0) return GSB_OK;
    if (table_size == 256)
        exp_tab256_kernel<<<(n + 255) / 256, 256, 0, stream>>>(d_x, d_y, n);
    else
        exp_tab_kernel<<<(n + 255) / 256, 256, 0, stream>>>(d_x, d_y, n);
    GSB_CUDA_CHECK(cudaGetLastError());
    return GSB_OK;
}

int ogata_init(DeviceState* st)
{
    {
        double tab[256];
        for (int j = 0; j < 256; ++j) tab[j] = (double)exp2l((long double)j / 256.L);
        GSB_CUDA_CHECK(cudaMemcpyToSymbol(g_exp2_256, tab, sizeof(tab)));
    }
    GSB_CUDA_CHECK(cudaMalloc(&st->d_status, sizeof(int)));
    GSB_CUDA_CHECK(cudaMalloc(&st->d_root, sizeof(double2) * kNroot));
    ogata_root_kernel<<<(unsigned)((kNroot + 255) / 256), 256>>>(st->d_root, kNroot);
    GSB_CUDA_CHECK(cudaGetLastError());
    long long total = 0;
    OgataTables og{};
    og.lev_min = kLevMin;
    og.lev_max = kLevMax;
    for (int lev = kLevMin; lev <= kLevMax; ++lev) {
        const double h = ldexp(1.0, -lev);
        const long long n = (long long)std::min(M_PI / h, 1e6);
        og.off[lev - kLevMin] = total;
        og.cnt[lev - kLevMin] = n;
        total += n;
    }
    GSB_CUDA_CHECK(cudaMalloc(&st->d_xw, sizeof(double2) * total));
    for (int lev = kLevMin; lev <= kLevMax; ++lev) {
        const long long n = og.cnt[lev - kLevMin];
        ogata_level_kernel<<<(unsigned)((n + 255) / 256), 256>>>(
            st->d_xw + og.off[lev - kLevMin], st->d_root, ldexp(1.0, -lev), n);
        GSB_CUDA_CHECK(cudaGetLastError());
    }
    GSB_CUDA_CHECK(cudaDeviceSynchronize());
    og.xw = st->d_xw;
    og.root = st->d_root;
    og.nroot = kNroot;
    st->og = og;
    return GSB_OK;
}

// Upper bound on the Sersic table length for these n values and GSParams.
static int sersic_stride(const double* h_n, int count, const gsb_gsparams* gsp)
{
    double nmax = 0.;
    for (int i = 0; i < count; ++i) nmax = std::max(nmax, h_n[i]);
    const double kderiv6 = std::exp(std::lgamma(8. * nmax) - std::lgamma(2. * nmax)) / 2304.;
    const double kmin = std::pow(gsp->kvalue_accuracy / kderiv6, 1. / 6.);
    const double dlogk = gsp->table_spacing * std::sqrt(std::sqrt(gsp->kvalue_accuracy / 10.));
    const double span = std::log(500.) - (std::log(kmin) - 0.001);
    return int(span / dlogk) + 4;
}

// The resampled quadrature levels of each device and spacing, kept while they are among the last
// few spacings used (a spacing is a GSParams setting: a program has one or two; 0.4 MB each).  Levels are
// spread as far as a build needs them: those up to level 15 (n <= 2) take 0.4 ms, up to 20 (n <= 4) 2.5, all 57,
// most of a million nodes each, 60.
namespace {
struct LogEntry {
    double* a = nullptr;
    OgataLog lg{};
    unsigned long long used = 0;
};
constexpr int kLogEntries = 4;
LogEntry g_log[64][kLogEntries];
unsigned long long g_log_clock = 0;
std::mutex g_log_mutex;
}  // namespace

// The first `need` levels for grid spacing h (g_log_mutex held).
static int ogata_log_levels(DeviceState* st, double h, int need, cudaStream_t stream, OgataLog* out)
{
    int dev = 0;
    cudaGetDevice(&dev);
    LogEntry* slots = g_log[dev & 63];
    LogEntry* e = slots;
    bool found = false;
    for (int i = 0; i < kLogEntries && !found; ++i) {
        found = slots[i].a && slots[i].lg.h == h;
        if (found || slots[i].used < e->used) e = &slots[i];
    }
    need = std::min(std::max(need, 1), kLogLevels);
    if (found && e->lg.have >= need) {
        e->used = ++g_log_clock;
        *out = e->lg;
        return GSB_OK;
    }
    OgataLog lg{};
    lg.h = h;
    int total = 0, cnt[kLogLevels], longest = 0;
    auto psi = [](double t) { return t * std::tanh(0.5 * M_PI * std::sinh(t)); };
    for (int j = 0; j < kLogLevels; ++j) {
        const double hl = std::ldexp(1.0, -(kLogLev0 + j));
        cnt[j] = int(std::min(M_PI / hl, double(kNroot)));
        // the first and last node: J0's first zero, and its cnt-th to McMahon's leading term
        const double t0 = hl * 2.404825557695773 / M_PI, t1 = hl * (cnt[j] - 0.25);
        const double x0 = M_PI / hl * psi(t0), x1 = M_PI / hl * psi(t1);
        lg.qmin[j] = int(std::floor(std::log(x0) / h)) - kLogW / 2 - 1;
        lg.len[j] = int(std::ceil(std::log(x1) / h)) + kLogW / 2 + 1 - lg.qmin[j] + 1;
        lg.off[j] = total;
        total += lg.len[j];
        longest = std::max(longest, lg.len[j]);
    }
    // a new spacing takes the place of the one used longest ago; more levels of a known one are added to
    // its array (builds in flight read the levels they were given)
    if (!found) {
        cudaFree(e->a);
        e->a = nullptr;
        e->lg = OgataLog{};
        GSB_CUDA_CHECK(cudaMalloc(&e->a, sizeof(double) * (total + (size_t)kLogSlices * longest)));
    }
    const int have = e->lg.have;
    double2* d_tmp = nullptr;
    double* d_slices = e->a + total;                      // (this function's alone: the mutex is held to its end)
    cudaError_t ce = cudaSuccess;
    if (kLogLev0 + need - 1 > kLevMax) ce = cudaMalloc(&d_tmp, sizeof(double2) * kNroot);
    for (int j = have; j < need && ce == cudaSuccess; ++j) {
        const int lev = kLogLev0 + j;
        const double2* xw = d_tmp;
        if (lev <= kLevMax) xw = st->d_xw + st->og.off[lev - kLevMin];
        else ogata_level_kernel<<<(cnt[j] + 255) / 256, 256, 0, stream>>>(d_tmp, st->d_root, std::ldexp(1.0, -lev), cnt[j]);
        ogata_log_kernel<<<dim3(lg.len[j], kLogSlices), 256, 0, stream>>>(xw, cnt[j], h, lg.qmin[j], d_slices);
        ogata_log_sum_kernel<<<(lg.len[j] + 127) / 128, 128, 0, stream>>>(d_slices, lg.len[j], e->a + lg.off[j]);
        ce = cudaGetLastError();
    }
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(stream);
    if (d_tmp) cudaFree(d_tmp);
    if (ce != cudaSuccess) {
        cudaGetLastError();
        if (!found) {
            cudaFree(e->a);
            e->a = nullptr;
        }
        return set_error(GSB_ERR_CUDA, std::string("resampled quadrature levels: ") + cudaGetErrorString(ce));
    }
    lg.a = e->a;
    lg.have = need;
    e->lg = lg;
    e->used = ++g_log_clock;
    *out = lg;
    return GSB_OK;
}

// Builds of at most this many tables per SM take one 512-thread block of single nodes a table: 400
// tables 295 us against 448 with the three-node blocks, 580 tables 403 against 465; it grows by
// 0.6 us a table from there, and the others reach 466 us at 1024.
constexpr int kSmallBuild = 4;

template <int R, int THREADS>
static int launch_sersic_tables(gsb_tables* t, int count, int stride, double nmax, const gsb_gsparams* gsp,
                                const OgataLog& lg, int p, int mul, const SersicScan* scan, double4* dnode, double* dheader,
                                int* d_status, cudaStream_t stream)
{
    // the samples a table of index nmax reaches from its level-12 sums down to its last node; smaller
    // n reach less far up
    const double kderiv6 = std::exp(std::lgamma(8. * nmax) - std::lgamma(2. * nmax)) / 2304.;
    const double front = std::log(gsp->kvalue_accuracy / kderiv6) / 6.;
    const int reach = std::max(0, int((front + 6.6134 * nmax) / lg.h * mul)) + 1 - std::min(0, lg.qmin[12 - kLogLev0]) * mul;
    const bool window = p == 1 && mul == 1;
    const int pad = window ? 33 * R : 1;
    const bool dn = dheader != nullptr;
    // per table: the samples (or the spline's right-hand side), the values, one flag byte a node
    const size_t fixed = (size_t)stride * (dn ? 2 : 1) * sizeof(double) + ((stride + 15) & ~7);
    const size_t room = 226 * 1024 - sizeof(double) * 4 * THREADS * R;
    const size_t per = sizeof(double) * (dn ? 2 : 1);
    // as many samples as the tables need, at least the right-hand side's room (samples that do not
    // fit are formed on the fly)
    size_t gcap = ((size_t)reach + (size_t)p * stride + 63) / 64 * 64;
    const size_t least = std::max<size_t>(64, dn ? stride / 2 + 1 : stride);
    if (fixed + per * (least + pad) > room) return set_error(GSB_ERR_UNSUPPORTED, "Sersic table too long");
    gcap = std::max(std::min(gcap, (room - fixed) / per - pad), least);
    // one-node builds: the levels 5 .. 20 next to them where they fit
    int stage = 0;
    for (int j = 0; R == 1 && j < 16; ++j)
        if (fixed + per * (gcap + pad) + sizeof(double) * (lg.off[j] + lg.len[j]) <= room) stage = lg.off[j] + lg.len[j];
    const size_t sm = fixed + per * (gcap + pad) + sizeof(double) * stage;
    auto go = [&](auto kernel) -> int {
        if (sm + sizeof(double) * 4 * THREADS * R > 47 * 1024)
            GSB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
        kernel<<<count, THREADS, sm, stream>>>(t->d_header, count, stride, *gsp, lg, p, mul, int(gcap), pad, stage, scan, t->d_val,
                                               t->d_node, dnode, dheader, d_status);
        GSB_CUDA_CHECK(cudaGetLastError());
        return GSB_OK;
    };
    if (window) return dn ? go(sersic_table_kernel<R, THREADS, true, true>) : go(sersic_table_kernel<R, THREADS, false, true>);
    return dn ? go(sersic_table_kernel<R, THREADS, true, false>) : go(sersic_table_kernel<R, THREADS, false, false>);
}

int sersic_tables_build(gsb_tables* t, const double* h_n, const double* h_trunc, int count,
                        const gsb_gsparams* gsp, bool with_dn, cudaStream_t stream)
{
    DeviceState* st = device_state();
    if (!st->ready) return set_error(GSB_ERR_INVALID, "gsb_init has not been called");
    for (int i = 0; i < count; ++i) {
        if (!(h_n[i] >= 0.3 && h_n[i] <= 6.2))
            return set_error(GSB_ERR_INVALID, "Sersic index out of range [0.3, 6.2]");
        if (h_trunc && !(h_trunc[i] >= 0.))
            return set_error(GSB_ERR_INVALID, "Sersic truncation radius must be >= 0");
    }
    if (count <= 0) { t->count = 0; return GSB_OK; }
    bool has_trunc = false;
    for (int i = 0; h_trunc && i < count; ++i) has_trunc |= h_trunc[i] > 0.;
    if (has_trunc && with_dn)
        return set_error(GSB_ERR_UNSUPPORTED, "n-derivative tables of truncated Sersic profiles are not built");
    const int stride = sersic_stride(h_n, count, gsp);
    if ((size_t)count > t->cap_slots || (size_t)count * stride > t->cap_nodes) {
        cudaFree(t->d_header); cudaFree(t->d_node); cudaFree(t->d_val); cudaFree(t->d_scan);
        cudaFree(t->d_n); cudaFree(t->d_status);
        t->d_header = nullptr; t->d_node = nullptr; t->d_val = nullptr; t->d_scan = nullptr;
        t->d_n = nullptr; t->d_status = nullptr;
        t->cap_slots = std::max<size_t>(count, t->cap_slots);
        t->cap_nodes = std::max<size_t>((size_t)count * stride, t->cap_nodes);
        GSB_CUDA_CHECK(cudaMalloc(&t->d_header, sizeof(double) * kSersicHeader * t->cap_slots));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_node, sizeof(double4) * t->cap_nodes));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_val, sizeof(double) * t->cap_nodes));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_scan, sizeof(SersicScan) * t->cap_slots));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_n, sizeof(double) * t->cap_slots));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_status, sizeof(int) * (1 + kMaxRounds)));
    }
    if (with_dn && ((size_t)count > t->cap_dn_slots || (size_t)count * stride > t->cap_dn_nodes)) {
        cudaFree(t->d_dheader); cudaFree(t->d_dnode);
        t->d_dheader = nullptr; t->d_dnode = nullptr;
        t->cap_dn_slots = std::max<size_t>(count, t->cap_dn_slots);
        t->cap_dn_nodes = std::max<size_t>((size_t)count * stride, t->cap_dn_nodes);
        GSB_CUDA_CHECK(cudaMalloc(&t->d_dheader, sizeof(double) * kSersicDHeader * t->cap_dn_slots));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_dnode, sizeof(double4) * t->cap_dn_nodes));
    }
    t->has_dn = with_dn;
    double* dheader = with_dn ? t->d_dheader : nullptr;
    double4* dnode = with_dn ? t->d_dnode : nullptr;
    t->count = count;
    t->stride = stride;
    double* d_n = t->d_n;
    int* d_status = t->d_status;
    GSB_CUDA_CHECK(cudaMemcpyAsync(d_n, h_n, sizeof(double) * count, cudaMemcpyHostToDevice, stream));
    double* d_trunc = nullptr;
    if (has_trunc) {
        if ((size_t)count > t->cap_trunc) {
            cudaFree(t->d_trunc);
            t->d_trunc = nullptr;
            t->cap_trunc = count;
            GSB_CUDA_CHECK(cudaMalloc(&t->d_trunc, sizeof(double) * t->cap_trunc));
        }
        d_trunc = t->d_trunc;
        GSB_CUDA_CHECK(cudaMemcpyAsync(d_trunc, h_trunc, sizeof(double) * count, cudaMemcpyHostToDevice, stream));
    }
    if ((stride + kTableRound - 1) / kTableRound > kMaxRounds) return set_error(GSB_ERR_UNSUPPORTED, "Sersic table too long");
    OgataLog lg;
    const double dlogk = gsp->table_spacing * std::sqrt(std::sqrt(gsp->kvalue_accuracy / 10.));
    // the resampled levels' spacing: the nodes' own, a p-th of it where that is too wide, or the largest multiple
    // (mul) that is not: a sum has as many terms as the levels' range in ln x has steps (2000 tables at
    // kvalue_accuracy 1e-9, spacing 0.003: 226 ms on the nodes' own spacing, 22 on ten times that)
    const int p = std::max(1, int(std::ceil(dlogk / kLogMaxStep)));
    const int mul = std::max(1, int(kLogMaxStep / dlogk));
    // held until the launch that reads the resampled levels is queued: an eviction frees only
    // after the device has finished it
    std::unique_lock<std::mutex> lock(g_log_mutex, std::defer_lock);
    double nmax = 0.;
    for (int i = 0; i < count; ++i) nmax = std::max(nmax, h_n[i]);
    // levels: at the default accuracies the last one that a table's nodes ask for is 13, 15, 18, 20, 22 and 26 at
    // n = 1.5, 2, 3, 4, 5 and 6.2; and two from the one that its lowest node starts at.  A node that asks for
    // more has the build run again with three more.
    int need = 2;
    {
        const double kderiv6 = std::exp(std::lgamma(8. * nmax) - std::lgamma(2. * nmax)) / 2304.;
        const double k = std::exp(std::log(gsp->kvalue_accuracy / kderiv6) / 6. - 0.001);
        for (double h0 = 1. / 32.; h0 > 100. * k && need < kLogLevels; h0 *= 0.5) ++need;
        need = std::max(need, int(10.5 + 2.55 * nmax) - kLogLev0 + 1);
    }
    // truncated tables: rounds of kTableRound ln k nodes, each followed by the stopping scan
    const int rounds = has_trunc ? (stride + kTableRound - 1) / kTableRound : 0;
    if (rounds > kMaxRounds) return set_error(GSB_ERR_UNSUPPORTED, "Sersic table too long");
    int h_status = 0;
    for (;; need = std::max(need, lg.have) + 3) {
        lock.lock();
        {
            const int rc = ogata_log_levels(st, dlogk / p * mul, need, stream, &lg);
            if (rc) return rc;
        }
        // d_status[0]: convergence status; d_status[1 + r]: some table still needs nodes after round r
        GSB_CUDA_CHECK(cudaMemsetAsync(d_status, 0, sizeof(int) * (1 + rounds), stream));
        sersic_setup_kernel<<<(count + 31) / 32, 96, 0, stream>>>(d_n, d_trunc, count, *gsp, t->d_header, stride, dheader);
        GSB_CUDA_CHECK(cudaGetLastError());
        SersicScan* scan = static_cast<SersicScan*>(t->d_scan);
        if (has_trunc) {
            sersic_scan_init_kernel<<<(count + 127) / 128, 128, 0, stream>>>(t->d_header, count, scan);
            GSB_CUDA_CHECK(cudaGetLastError());
            for (int r = 0; r < rounds; ++r) {
                const int* prev_live = r > 0 ? d_status + r : nullptr;
                const long long tw = (long long)count * kTableRound;
                sersic_trunc_nodes_kernel<<<(unsigned)((tw * 32 + 255) / 256), 256, 0, stream>>>(
                    t->d_header, count, r * kTableRound, kTableRound, st->og, scan, t->d_val, stride, prev_live, d_status);
                GSB_CUDA_CHECK(cudaGetLastError());
                sersic_scan_kernel<<<(count + 63) / 64, 64, 0, stream>>>(t->d_header, count, stride, r * kTableRound,
                                                                         kTableRound, *gsp, t->d_val, scan, prev_live,
                                                                         d_status + 1 + r);
                GSB_CUDA_CHECK(cudaGetLastError());
            }
        }
        {
            const int rc = count <= kSmallBuild * st->sm_count
                               ? launch_sersic_tables<1, 512>(t, count, stride, nmax, gsp, lg, p, mul, scan, dnode, dheader, d_status, stream)
                               : launch_sersic_tables<3, 64>(t, count, stride, nmax, gsp, lg, p, mul, scan, dnode, dheader, d_status, stream);
            if (rc) return rc;
        }
        lock.unlock();
        GSB_CUDA_CHECK(cudaMemcpyAsync(&h_status, d_status, sizeof(int), cudaMemcpyDeviceToHost, stream));
        GSB_CUDA_CHECK(cudaStreamSynchronize(stream));
        if (!(h_status & 2)) break;
    }
    if (h_status) return set_error(GSB_ERR_NUMERIC, "Sersic Hankel transform did not converge");
    return GSB_OK;
}

int sersic_truncation(int count, const double* h_in, double* h_out, cudaStream_t stream)
{
    if (count <= 0) return GSB_OK;
    double *d_in = nullptr, *d_out = nullptr;
    int* d_status = nullptr;
    GSB_CUDA_CHECK(cudaMallocAsync(&d_in, sizeof(double) * 4 * count, stream));
    GSB_CUDA_CHECK(cudaMallocAsync(&d_out, sizeof(double) * 2 * count, stream));
    GSB_CUDA_CHECK(cudaMallocAsync(&d_status, sizeof(int), stream));
    GSB_CUDA_CHECK(cudaMemsetAsync(d_status, 0, sizeof(int), stream));
    GSB_CUDA_CHECK(cudaMemcpyAsync(d_in, h_in, sizeof(double) * 4 * count, cudaMemcpyHostToDevice, stream));
    sersic_truncation_kernel<<<(count + 127) / 128, 128, 0, stream>>>(d_in, count, d_out, d_status);
    GSB_CUDA_CHECK(cudaGetLastError());
    int h_status = 0;
    GSB_CUDA_CHECK(cudaMemcpyAsync(h_out, d_out, sizeof(double) * 2 * count, cudaMemcpyDeviceToHost, stream));
    GSB_CUDA_CHECK(cudaMemcpyAsync(&h_status, d_status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    GSB_CUDA_CHECK(cudaStreamSynchronize(stream));
    cudaFreeAsync(d_in, stream);
    cudaFreeAsync(d_out, stream);
    cudaFreeAsync(d_status, stream);
    if (h_status) return set_error(GSB_ERR_NUMERIC, "truncated Sersic scale radius root find did not converge");
    return GSB_OK;
}

// The reference's k grid of SBMoffat::setupFT: k = 0, dk, 2 dk, ... as a running sum, k < 50.
static std::vector<double> moffat_kgrid(const gsb_gsparams* gsp)
{
    const double dk = gsp->table_spacing * std::sqrt(std::sqrt(gsp->kvalue_accuracy / 10.));
    std::vector<double> k;
    for (double x = 0.; x < 50.; x += dk) k.push_back(x);
    return k;
}

int moffat_tables_build(gsb_tables* t, const double* h_beta, const double* h_trunc, int count,
                        const gsb_gsparams* gsp, cudaStream_t stream)
{
    DeviceState* st = device_state();
    if (!st->ready) return set_error(GSB_ERR_INVALID, "gsb_init has not been called");
    for (int i = 0; i < count; ++i) {
        if (!(h_trunc[i] > 0.) || !std::isfinite(h_trunc[i]))
            return set_error(GSB_ERR_INVALID, "Moffat table needs trunc / scale_radius > 0");
        if (!(h_beta[i] > 0.) || h_beta[i] == 1. || !std::isfinite(h_beta[i]))
            return set_error(GSB_ERR_INVALID, "truncated Moffat beta must be > 0 and != 1 (at beta = 1 the "
                                              "flux normalisation 2 (beta - 1) / (1 - (1 + t^2)^(1 - beta)) is 0/0)");
    }
    if (count <= 0) { t->moffat_count = 0; return GSB_OK; }
    if (!(gsp->kvalue_accuracy > 0.) || !(gsp->table_spacing > 0.))
        return set_error(GSB_ERR_INVALID, "kvalue_accuracy and table_spacing must be > 0");
    const std::vector<double> kg = moffat_kgrid(gsp);
    const int ncand = int(kg.size());
    const size_t fsm = sizeof(double) * 4 * (size_t)ncand;
    if (fsm > 227 * 1024)
        return set_error(GSB_ERR_UNSUPPORTED, "truncated Moffat table too long for this kvalue_accuracy / "
                                              "table_spacing (more than 7264 nodes)");
    if ((size_t)count > t->cap_mslots || (size_t)count * ncand > t->cap_mnodes || (size_t)ncand > t->cap_mk) {
        cudaFree(t->d_mheader); cudaFree(t->d_mnode); cudaFree(t->d_mval); cudaFree(t->d_mk); cudaFree(t->d_mstatus);
        t->d_mheader = nullptr; t->d_mnode = nullptr; t->d_mval = nullptr; t->d_mk = nullptr; t->d_mstatus = nullptr;
        t->cap_mslots = std::max<size_t>(count, t->cap_mslots);
        t->cap_mnodes = std::max<size_t>((size_t)count * ncand, t->cap_mnodes);
        t->cap_mk = std::max<size_t>(ncand, t->cap_mk);
        GSB_CUDA_CHECK(cudaMalloc(&t->d_mheader, sizeof(double) * kMoffatHeader * t->cap_mslots));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_mnode, sizeof(double4) * t->cap_mnodes));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_mval, sizeof(double) * t->cap_mnodes));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_mk, sizeof(double) * t->cap_mk));
        GSB_CUDA_CHECK(cudaMalloc(&t->d_mstatus, sizeof(int)));
    }
    t->moffat_count = count;
    t->moffat_stride = ncand;
    // slot headers: (beta, trunc / rD, dk) from the host, the rest written on the device
    std::vector<double> hh((size_t)kMoffatHeader * count, 0.);
    for (int i = 0; i < count; ++i) {
        hh[(size_t)i * kMoffatHeader + kMH_BETA] = h_beta[i];
        hh[(size_t)i * kMoffatHeader + kMH_TRUNC] = h_trunc[i];
        hh[(size_t)i * kMoffatHeader + kMH_DK] = ncand > 1 ? kg[1] : 0.;
    }
    GSB_CUDA_CHECK(cudaMemcpyAsync(t->d_mheader, hh.data(), sizeof(double) * hh.size(), cudaMemcpyHostToDevice,
                                   stream));
    GSB_CUDA_CHECK(cudaMemcpyAsync(t->d_mk, kg.data(), sizeof(double) * ncand, cudaMemcpyHostToDevice, stream));
    GSB_CUDA_CHECK(cudaMemsetAsync(t->d_mstatus, 0, sizeof(int), stream));
    moffat_setup_kernel<<<(count + 127) / 128, 128, 0, stream>>>(count, t->d_mheader);
    GSB_CUDA_CHECK(cudaGetLastError());
    const int threads = 256;
    const long long nwarps = (long long)count * ncand;
    moffat_nodes_kernel<<<(unsigned)((nwarps * 32 + threads - 1) / threads), threads, 0, stream>>>(
        t->d_mheader, count, t->d_mk, ncand, st->og, t->d_mval, t->d_mstatus);
    GSB_CUDA_CHECK(cudaGetLastError());
    if (fsm > 48 * 1024)
        GSB_CUDA_CHECK(cudaFuncSetAttribute(moffat_finalize_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            int(fsm)));
    moffat_finalize_kernel<<<count, 32, fsm, stream>>>(t->d_mheader, count, t->d_mk, ncand, *gsp, t->d_mval,
                                                       t->d_mnode);
    GSB_CUDA_CHECK(cudaGetLastError());
    int h_status = 0;
    GSB_CUDA_CHECK(cudaMemcpyAsync(&h_status, t->d_mstatus, sizeof(int), cudaMemcpyDeviceToHost, stream));
    GSB_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (h_status) return set_error(GSB_ERR_NUMERIC, "truncated Moffat Hankel transform ran out of J0 zeros");
    return GSB_OK;
}

int moffat_scale_radius(int count, const double* h_in, double* h_out, cudaStream_t stream)
{
    if (count <= 0) return GSB_OK;
    double *d_in = nullptr, *d_out = nullptr;
    int* d_status = nullptr;
    GSB_CUDA_CHECK(cudaMallocAsync(&d_in, sizeof(double) * 3 * count, stream));
    GSB_CUDA_CHECK(cudaMallocAsync(&d_out, sizeof(double) * count, stream));
    GSB_CUDA_CHECK(cudaMallocAsync(&d_status, sizeof(int), stream));
    GSB_CUDA_CHECK(cudaMemsetAsync(d_status, 0, sizeof(int), stream));
    GSB_CUDA_CHECK(cudaMemcpyAsync(d_in, h_in, sizeof(double) * 3 * count, cudaMemcpyHostToDevice, stream));
    moffat_scale_radius_kernel<<<(count + 127) / 128, 128, 0, stream>>>(d_in, count, d_out, d_status);
    GSB_CUDA_CHECK(cudaGetLastError());
    int h_status = 0;
    GSB_CUDA_CHECK(cudaMemcpyAsync(h_out, d_out, sizeof(double) * count, cudaMemcpyDeviceToHost, stream));
    GSB_CUDA_CHECK(cudaMemcpyAsync(&h_status, d_status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    GSB_CUDA_CHECK(cudaStreamSynchronize(stream));
    cudaFreeAsync(d_in, stream);
    cudaFreeAsync(d_out, stream);
    cudaFreeAsync(d_status, stream);
    if (h_status) return set_error(GSB_ERR_NUMERIC, "Solve error: Moffat scale radius root find did not converge");
    return GSB_OK;
}

// The Kolmogorov radial spline of each device (its GSParams are those of the stepk cached in
// the device state).
namespace {
struct KolmRadial {
    double4* nodes = nullptr;
    int n = 0, cap = 0;
};
KolmRadial g_kolm_radial[64];
}  // namespace

static int kolmogorov_build(const gsb_gsparams* gsp, cudaStream_t stream)
{
    DeviceState* st = device_state();
    int dev = 0;
    cudaGetDevice(&dev);
    KolmRadial& kr = g_kolm_radial[dev & 63];
    const double key[13] = {double(gsp->minimum_fft_size), double(gsp->maximum_fft_size),
                            gsp->folding_threshold, gsp->stepk_minimum_hlr, gsp->maxk_threshold,
                            gsp->kvalue_accuracy, gsp->xvalue_accuracy, gsp->table_spacing,
                            gsp->realspace_relerr, gsp->realspace_abserr, gsp->integration_relerr,
                            gsp->integration_abserr, gsp->shoot_accuracy};
    if (st->kolm_valid && std::equal(key, key + 13, st->kolm_key)) return GSB_OK;
    const double dlogr = gsp->table_spacing * std::sqrt(std::sqrt(gsp->xvalue_accuracy / 10.));
    int ncand = 0;
    for (double logr = -3.; logr < std::log(1.e4); logr += dlogr) ++ncand;
    if (ncand + 1 > kr.cap) {
        cudaFree(kr.nodes);
        kr.nodes = nullptr;
        kr.cap = 0;
        GSB_CUDA_CHECK(cudaMalloc(&kr.nodes, sizeof(double4) * (ncand + 1)));
        kr.cap = ncand + 1;
    }
    double* d_vals = nullptr;
    int* d_status = nullptr;
    double* d_out = nullptr;
    double* d_scratch = nullptr;
    GSB_CUDA_CHECK(cudaMallocAsync(&d_vals, sizeof(double) * ncand, stream));
    GSB_CUDA_CHECK(cudaMallocAsync(&d_status, sizeof(int), stream));
    GSB_CUDA_CHECK(cudaMallocAsync(&d_out, sizeof(double) * 2, stream));
    GSB_CUDA_CHECK(cudaMallocAsync(&d_scratch, sizeof(double) * 4 * (ncand + 1), stream));
    GSB_CUDA_CHECK(cudaMemsetAsync(d_status, 0, sizeof(int), stream));
    kolmogorov_nodes_kernel<<<(ncand * 32 + 255) / 256, 256, 0, stream>>>(ncand, dlogr, *gsp, st->og,
                                                                          d_vals, d_status);
    GSB_CUDA_CHECK(cudaGetLastError());
    kolmogorov_finalize_kernel<<<1, 1, 0, stream>>>(ncand, dlogr, *gsp, d_vals, d_out, kr.nodes, d_scratch);
    GSB_CUDA_CHECK(cudaGetLastError());
    double h_out[2] = {0., 0.};
    int h_status = 0;
    GSB_CUDA_CHECK(cudaMemcpyAsync(h_out, d_out, sizeof(double) * 2, cudaMemcpyDeviceToHost, stream));
    GSB_CUDA_CHECK(cudaMemcpyAsync(&h_status, d_status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    GSB_CUDA_CHECK(cudaFreeAsync(d_vals, stream));
    GSB_CUDA_CHECK(cudaFreeAsync(d_status, stream));
    GSB_CUDA_CHECK(cudaFreeAsync(d_out, stream));
    GSB_CUDA_CHECK(cudaFreeAsync(d_scratch, stream));
    GSB_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (h_status) return set_error(GSB_ERR_NUMERIC, "Kolmogorov Hankel transform did not converge");
    std::copy(key, key + 13, st->kolm_key);
    st->kolm_stepk = h_out[0];
    kr.n = int(h_out[1]);
    st->kolm_valid = true;
    return GSB_OK;
}

int kolmogorov_stepk(const gsb_gsparams* gsp, cudaStream_t stream, double* out)
{
    const int rc = kolmogorov_build(gsp, stream);
    if (rc) return rc;
    *out = device_state()->kolm_stepk;
    return GSB_OK;
}

// The radial spline nodes (r, f, y2, 0) of KolmogorovInfo for these GSParams (gsb_real.cu).
int kolmogorov_radial(const gsb_gsparams* gsp, cudaStream_t stream, const double4** nodes, int* n)
{
    const int rc = kolmogorov_build(gsp, stream);
    if (rc) return rc;
    int dev = 0;
    cudaGetDevice(&dev);
    *nodes = g_kolm_radial[dev & 63].nodes;
    *n = g_kolm_radial[dev & 63].n;
    return GSB_OK;
}

int prepare_leaves(const gsb_template* tpl, int n_stamps, const gsb_gsparams* gsp, gsb_leaf* d_leaves,
                   const gsb_tables* t, double* d_info, cudaStream_t stream)
{
    DeviceState* st = device_state();
    if (!st->ready) return set_error(GSB_ERR_INVALID, "gsb_init has not been called");
    bool need_kolm = false, need_sersic = false, need_images = false;
    for (int l = 0; l < tpl->n_leaves; ++l) {
        if (tpl->leaf_type[l] == GSB_KOLMOGOROV) need_kolm = true;
        if (tpl->leaf_type[l] == GSB_SERSIC) need_sersic = true;
        if (tpl->leaf_type[l] == GSB_INTERPOLATED) need_images = true;
    }
    if (need_sersic && (!t || t->count == 0))
        return set_error(GSB_ERR_INVALID, "Sersic leaves need built FT tables");
    if (need_images && (!t || t->n_images == 0))
        return set_error(GSB_ERR_INVALID, "InterpolatedImage leaves need built image slots");
    ImageRefs images{};
    if (t) images = ImageRefs{t->d_images, t->d_image_info, t->d_k64, t->d_k32, t->n_images};
    MoffatRefs moffat{};
    if (t) moffat = MoffatRefs{t->d_mheader, t->d_mnode, t->moffat_count, t->moffat_stride};
    double kolm = 0.;
    if (need_kolm) {
        const int rc = kolmogorov_stepk(gsp, stream, &kolm);
        if (rc) return rc;
    }
    int* d_status = st->d_status;
    GSB_CUDA_CHECK(cudaMemsetAsync(d_status, 0, sizeof(int), stream));
    const long long n = (long long)n_stamps * tpl->n_leaves;
    if (n > 0) {
        // a warp per leaf while that does not fill the GPU
        if (n <= 16LL * st->sm_count)
            prepare_leaves_kernel<true><<<(unsigned)((n * 32 + 127) / 128), 128, 0, stream>>>(
                *tpl, n_stamps, *gsp, d_leaves, t ? t->d_header : nullptr, moffat, kolm, images, d_info, d_status);
        else
            prepare_leaves_kernel<false><<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(
                *tpl, n_stamps, *gsp, d_leaves, t ? t->d_header : nullptr, moffat, kolm, images, d_info, d_status);
        GSB_CUDA_CHECK(cudaGetLastError());
    }
    int h_status = 0;
    GSB_CUDA_CHECK(cudaMemcpyAsync(&h_status, d_status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    GSB_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (h_status & 8) return set_error(GSB_ERR_INVALID, "unknown leaf type");
    if (h_status & 16) return set_error(GSB_ERR_INVALID, "InterpolatedImage leaf names no built image slot");
    if (h_status & 32) return set_error(GSB_ERR_UNSUPPORTED, "interpolant not built (x: Delta, Nearest, "
                                                             "Linear, Cubic, Quintic, Lanczos; k: the same "
                                                             "but Delta)");
    if (h_status & 512) return set_error(GSB_ERR_INVALID, "a Lanczos k interpolant needs its coefficient "
                                                          "block in p[2] (n <= 3)");
    if (h_status & 1024) return set_error(GSB_ERR_INVALID, "InterpolatedImage leaf's x interpolant differs "
                                                           "from its image slot's");
    if (h_status & 2) return set_error(GSB_ERR_NUMERIC, "Sersic radius root finding failed");
    if (h_status & 4) return set_error(GSB_ERR_NUMERIC, "Moffat maxk root finding failed");
    if (h_status & 64) return set_error(GSB_ERR_INVALID, "truncated Moffat leaf names no built Moffat table slot");
    if (h_status & 128) return set_error(GSB_ERR_INVALID, "truncated Moffat leaf's table slot was built for "
                                                          "another (beta, trunc / scale_radius)");
    if (h_status & 256) return set_error(GSB_ERR_NUMERIC, "truncated Moffat table is empty");
    return GSB_OK;
}

}  // namespace gsb
