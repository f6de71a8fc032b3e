// ksp_device.cuh -- device-side numerics of the linear-response neutrino integrator.
//
// Background cosmology (Omega_nu(a) from Fermi-Dirac tables, H(a)), natural cubic
// splines, the Fermi-Dirac kernel J(x), and a warp-cooperative QAG integrator that
// makes the same adaptive decisions as QUADPACK's QAG with the 61-point Gauss-Kronrod
// rule (the integrator the reference calls through GSL, delta_tot_table.c:404,597).
// Each function names the reference file:line whose arithmetic it follows.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <float.h>
#include "gk61_table.h"

#define KSP_HD __host__ __device__ __forceinline__

namespace ksp {

// kspace_neutrino_const.h:9-19, gadget_defines.h:8, omega_nu_single.c:10-14,85
constexpr int kNuSpecies = 3;
constexpr int kNRhoTab = 200;
constexpr int kQagLimit = 200;  // GSL_VAL
constexpr double kLightCgs = 2.99792458e10;
constexpr double kBolEvK = 8.61734e-5;
constexpr double kHubble = 3.24077929e-18;
constexpr double kHbar = 6.582119e-16;
constexpr double kStefanBoltzmann = 5.670373e-5;
constexpr double kGravity = 6.67408e-8;
constexpr double kNuSw = 100.0;
constexpr double kFloatAcc = 1e-6;
constexpr double kPi = 3.14159265358979323846;
constexpr double kZeta3 = 1.202056903159594;

// Status bits written by kernels (host maps them to reference error codes).
enum : unsigned {
    kStGsl = 1u << 0,        // QAG failed / interpolation out of range  -> 2001
    kStDnuNaN = 1u << 1,     // delta_nu is NaN                          -> 2004
    kStGridNaN = 1u << 2,    // correction factor is NaN                 -> 5
    kStKmax = 1u << 3,       // k beyond transfer table                  -> 2
    kStKWarn = 1u << 4,      // k < keff_0 / 2 (reference prints to stderr, continues)
    kStTimeout = 1u << 5,    // a bounded wait expired
};
// the errors after which the reference terminates before it corrects the grid: the
// correction pass leaves the grid as it is when one of them is set
constexpr unsigned kStAbort = kStGsl | kStDnuNaN | kStGridNaN | kStKmax | kStTimeout;

// omega_nu_single.h:27-34: tabulated rho_nu(a) of one species (natural cubic spline in log a)
struct RhoTable {
    int has_table;
    double mnu;
    double loga[kNRhoTab], rhonu[kNRhoTab], c[kNRhoTab];
    // filled with c (k_rho_splines): the node-independent spline terms of each segment
    // (as cspline_seg forms them), 1 / knot spacing and 1 / mnu, for fsl_integrand
    double sb[kNRhoTab], sd[kNRhoTab];
    double inv_dx, imnu;
};

// omega_nu_single.h:100-113 (_omega_nu, _hybrid_nu) plus the parameters of the host's
// hubble_function (delta_tot_table_test.c:33-45; curvature as gadget-2/0003 patch:38).
struct Background {
    double rhocrit, kBtnu, tcmb0, conv, omegag0;
    double irhocrit, ihubble;  // 1 / rhocrit, 1 / hubble
    int deg[kNuSpecies];
    double mnu[kNuSpecies];
    double mnu_J[kNuSpecies];  // mass inside J's argument (get_delta_nu's mnu, delta_tot_table.c:507)
    int hyb_enabled;
    double nufrac_low[kNuSpecies], nu_crit_time, vcrit;
    double Omega_nonu_H, OmegaLambda, OmegaK, hubble;
    int radiation;
    RhoTable tab[kNuSpecies];
    // A host H(a) of another form, tabulated: log H as a natural cubic spline in log a on
    // htab_n uniform knots from htab_lo with spacing htab_h, 4 coefficients per segment
    // (device copy for kernels, host copy for host-side evaluation); htab_n = 0: the
    // analytic form above.
    const double* htab_d;
    const double* htab_h;
    int htab_n;
    double htab_lo, htab_dx;
};

// ------------------------------------------------------------------ splines
#ifdef __CUDACC__
// Integers in the order of the doubles: an FP64 comparison takes the FP64 pipe's 16 cycles.
__device__ __forceinline__ long long order_key(double v) {
    const long long b = __double_as_longlong(v);
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
#endif
// Segment i with x[i] <= v < x[i+1] (v == x[n-1] -> n-2), as GSL's bsearch.
KSP_HD int seg_bsearch(const double* x, int n, double v) {
    int lo = 0, hi = n - 1;
#ifdef __CUDA_ARCH__
    const long long k = order_key(v);
#endif
    while (hi > lo + 1) {
        const int mid = (lo + hi) >> 1;
#ifdef __CUDA_ARCH__
        if (order_key(x[mid]) > k) hi = mid; else lo = mid;
#else
        if (x[mid] > v) hi = mid; else lo = mid;
#endif
    }
    return lo;
}

// Natural cubic spline (c = S''/2 at the knots) evaluated on segment i.
KSP_HD double cspline_seg(const double* x, const double* y, const double* c, int i, double v) {
    const double h = x[i + 1] - x[i], dx = v - x[i];
    const double b = (y[i + 1] - y[i]) / h - h * (c[i + 1] + 2.0 * c[i]) / 3.0;
    const double d = (c[i + 1] - c[i]) / (3.0 * h);
    return y[i] + dx * (b + dx * (c[i] + dx * d));
}

// ------------------------------------------------------------------ background
// omega_nu_single.c:100-114 (rho_nu conversion factor)
KSP_HD double rho_nu_conversion() {
    double convert = 4 * kPi * 2;
    const double chbar = 1. / (2 * kPi * kLightCgs * kHbar);
    convert *= (chbar * chbar * chbar);
    convert *= (1.60217646e-12 / kLightCgs / kLightCgs);
    return convert;
}

// omega_nu_single.c:156-160
KSP_HD double non_rel_rho_nu(double a, double kT, double amnu, double kTamnu2, double conv) {
    return amnu * (kT * kT * kT) / (a * a * a * a) *
           (1.5 * kZeta3 + kTamnu2 * 45. / 4. * 1.0369277551433704 +
            2835. / 32. * kTamnu2 * kTamnu2 * 1.0083492773819229 +
            80325 / 32. * kTamnu2 * kTamnu2 * kTamnu2 * 1.0020083928260826) * conv;
}

// omega_nu_single.c:164-167
KSP_HD double rel_rho_nu(double a, double kT, double conv) {
    const double t = kPi * kT / a, t2 = t * t;
    return 7 * (t2 * t2) / 120. * conv;
}

// omega_nu_single.c:171-202
// loga_in: log(a) when the caller has it (NaN: computed here)
KSP_HD double rho_nu(const RhoTable& T, double a, double kT, double conv, double loga_in = NAN) {
    const double amnu = a * T.mnu;
    const double kTamnu2 = (kT * kT / amnu / amnu);
    if (kNuSw * kNuSw * kTamnu2 < 1) return non_rel_rho_nu(a, kT, amnu, kTamnu2, conv);
    if (amnu < 1e-6 * kT) return rel_rho_nu(a, kT, conv);
    const double loga = loga_in == loga_in ? loga_in : log(a);
    if (!T.has_table || loga < T.loga[0]) {
        if (amnu < 1e-4 * kT) return rel_rho_nu(a, kT, conv);
        return non_rel_rho_nu(a, kT, amnu, kTamnu2, conv);
    }
    // uniform knots: guess the segment, then settle it against the stored knots
    const double inv = (kNRhoTab - 1) / (T.loga[kNRhoTab - 1] - T.loga[0]);
    int i = (int)((loga - T.loga[0]) * inv);
    i = i < 0 ? 0 : (i > kNRhoTab - 2 ? kNRhoTab - 2 : i);
    while (i > 0 && loga < T.loga[i]) i--;
    while (i < kNRhoTab - 2 && loga >= T.loga[i + 1]) i++;
    return cspline_seg(T.loga, T.rhonu, T.c, i, loga);
}

// omega_nu_single.c:246-257
KSP_HD double particle_nu_fraction(const Background& B, double a, int i) {
    if (!B.hyb_enabled) return 0;
    if (a > B.nu_crit_time) return B.nufrac_low[i];
    return 0;
}

// omega_nu_single.c:55-65
KSP_HD double omega_nu(const Background& B, double a, double loga = NAN) {
    double rhonu = 0;
    for (int mi = 0; mi < kNuSpecies; mi++)
        if (B.deg[mi] > 0) rhonu += B.deg[mi] * rho_nu(B.tab[mi], a, B.kBtnu, B.conv, loga);
    return rhonu / B.rhocrit;
}

// omega_nu_single.c:69-74
KSP_HD double omega_nu_nopart(const Background& B, double a) {
    return omega_nu(B, a) - omega_nu(B, 1) * particle_nu_fraction(B, a, 0) / (a * a * a);
}

// omega_nu_single.c:262-279
KSP_HD double omega_nu_single(const Background& B, double a, int i) {
    if (B.deg[i] == 0) {
        for (int j = i; j >= 0; j--)
            if (B.deg[j]) { i = j; break; }
    }
    const double om = rho_nu(B.tab[i], a, B.kBtnu, B.conv) / B.rhocrit;
    double part = rho_nu(B.tab[i], 1, B.kBtnu, B.conv) / B.rhocrit;
    part *= particle_nu_fraction(B, a, i) / (a * a * a);
    return om - part;
}

// log H at log a from the tabulated spline (the end segments continue past the table)
KSP_HD double hubble_tab_log(const Background& B, double la) {
#ifdef __CUDA_ARCH__
    const double* t = B.htab_d;
#else
    const double* t = B.htab_h;
#endif
    int i = (int)floor((la - B.htab_lo) / B.htab_dx);
    i = i < 0 ? 0 : (i > B.htab_n - 2 ? B.htab_n - 2 : i);
    const double dx = la - (B.htab_lo + i * B.htab_dx);
    const double* c = t + 4 * i;
    return c[0] + dx * (c[1] + dx * (c[2] + dx * c[3]));
}

// delta_tot_table_test.c:33-45 (+ curvature, gadget-2/0003 patch:38); Omega_g as
// omega_nu_single.c:77-81.
KSP_HD double hubble(const Background& B, double a, double loga = NAN) {
    if (B.htab_n > 0) return exp(hubble_tab_log(B, loga == loga ? loga : log(a)));
    const double a3 = a * a * a;
    double om = B.Omega_nonu_H / a3 + B.OmegaLambda;
    if (B.OmegaK != 0.0) om += B.OmegaK / (a * a);
    om += omega_nu(B, a, loga);
    if (B.radiation) om += B.omegag0 / (a3 * a);
    return B.hubble * sqrt(om);
}

#ifdef __CUDACC__
// rho_nu for fsl_integrand: the same branches as rho_nu, of kT / (a m), with 1/a given and the
// table spline in per-segment polynomial form (RhoTable::sb, sd).
__device__ __forceinline__ double rho_nu_ia(const RhoTable& T, double ia, double loga, double kT, double conv) {
    const double kTamnu = kT * ia * T.imnu;
    bool nonrel = kNuSw * kTamnu < 1;
    bool rel = !nonrel && kTamnu > 1e6;
    if (!nonrel && !rel && (!T.has_table || loga < T.loga[0])) {
        rel = kTamnu > 1e4;
        nonrel = !rel;
    }
    if (nonrel) {
        const double t = kTamnu * kTamnu;
        return T.mnu * (kT * kT * kT) * (ia * ia * ia) *
               (1.5 * kZeta3 + t * (45. / 4. * 1.0369277551433704 +
                                    t * (2835. / 32. * 1.0083492773819229 + t * (80325 / 32. * 1.0020083928260826)))) *
               conv;
    }
    if (rel) {
        const double t = kPi * kT * ia, t2 = t * t;
        return 7 * (t2 * t2) / 120. * conv;
    }
    // a rounding across a knot is harmless: the segments' polynomials meet there
    int i = (int)((loga - T.loga[0]) * T.inv_dx);
    i = i < 0 ? 0 : (i > kNRhoTab - 2 ? kNRhoTab - 2 : i);
    const double dx = loga - T.loga[i];
    return T.rhonu[i] + dx * (T.sb[i] + dx * (T.c[i] + dx * T.sd[i]));
}

// 1 / H at a = 1 / ia with H as hubble() forms it.
__device__ __forceinline__ double inv_hubble_ia(const Background& B, double x, double ia) {
    const double ia2 = ia * ia, ia3 = ia2 * ia;
    double om = B.Omega_nonu_H * ia3 + B.OmegaLambda;
    if (B.OmegaK != 0.0) om += B.OmegaK * ia2;
    double rhonu = 0;
    for (int mi = 0; mi < kNuSpecies; mi++)
        if (B.deg[mi] > 0) rhonu += B.deg[mi] * rho_nu_ia(B.tab[mi], ia, x, B.kBtnu, B.conv);
    om += rhonu * B.irhocrit;
    if (B.radiation) om += B.omegag0 * (ia3 * ia);
    return rsqrt(om) * B.ihubble;
}
// The fslength integrand 1/(a^2 H(a)) at a = e^x (delta_tot_table.c:378-383): one exp, one
// reciprocal square root and no division, ~60 FP64 operations (with 1/a and 1/H divided out, 90).
__device__ __forceinline__ double fsl_integrand(const Background& B, double x) {
    if (B.htab_n > 0) return exp(-2.0 * x - hubble_tab_log(B, x));
    const double ia = exp(-x);
    return ia * ia * inv_hubble_ia(B, x, ia);
}
#endif

// delta_tot_table.c:613-617
KSP_HD double get_delta_tot(double dnu, double dcdm, double OmegaNua3, double Omeganonu, double Omeganu1,
                            double partnu) {
    const double fcdm = 1 - OmegaNua3 / (Omeganonu + Omeganu1);
    return fcdm * (dcdm + dnu * OmegaNua3 / (Omeganonu + Omeganu1 * partnu));
}

// ------------------------------------------------------------------ J(x)
// delta_tot_table.c:417-428
KSP_HD double specialJ_fit(double x) {
    if (x <= 0.) return 1.;
    const double x2 = x * x, x4 = x2 * x2, x8 = x4 * x4;
    return (1. + 0.0168 * x2 + 0.0407 * x4) / (1. + 2.1734 * x2 + 1.6787 * exp(4.1811 * log(x)) + 0.1467 * x8);
}

// sin(y)/y: Taylor series 1 - y^2/6 + y^4/120 - y^6/5040 + y^8/362880 near 0.
KSP_HD double sinc_j0(double y) {
    if (fabs(y) < 0.05) {
        const double t = y * y;
        return 1.0 - t / 6.0 * (1.0 - t / 20.0 * (1.0 - t / 42.0 * (1.0 - t / 72.0)));
    }
    return sin(y) / y;
}

// delta_tot_table.c:431-463 with qc > 0: sum over n = 1..19 of -(-1)^n e^{-n qc} /
// (n^2 + x^2)^2 times
//   (n^2 + n^3 qc + x^2 (n qc - 1)) qc sinc(qc x) + (2 n + n^2 qc + qc x^2) cos(qc x).
// The sine and the cosine do not depend on n: A and B are their factors' sums.  The weights
// e^{-n qc} are powers of e1 = e^{-qc}; four terms share a division.
KSP_HD void specialJ_sums(double x2, double qc, double e1, double* A_out, double* B_out) {
    double en = 1.0, A = 0.0, B = 0.0;
    for (int n0 = 1; n0 < 20; n0 += 4) {
        double d[4], w[4], a[4], c[4];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (int j = 0; j < 4; j++) {
            const double n = n0 + j;
            en *= e1;
            w[j] = n0 + j < 20 ? ((j & 1) ? -en : en) : 0.0;  // n0 is odd
            const double t = n * n + x2;
            d[j] = t * t;
            a[j] = n * n * (1.0 + n * qc) + x2 * (n * qc - 1.0);
            c[j] = n * (2.0 + n * qc) + qc * x2;
        }
        const double d01 = d[0] * d[1], d23 = d[2] * d[3], inv = 1.0 / (d01 * d23);
        const double w0 = w[0] * d[1] * d23, w1 = w[1] * d[0] * d23, w2 = w[2] * d01 * d[3], w3 = w[3] * d01 * d[2];
        A += inv * (w0 * a[0] + w1 * a[1] + w2 * a[2] + w3 * a[3]);
        B += inv * (w0 * c[0] + w1 * c[1] + w2 * c[2] + w3 * c[3]);
    }
    *A_out = A;
    *B_out = B;
}
KSP_HD double specialJ_series(double x, double qc, double nufrac_low) {
    double A, B;
    specialJ_sums(x * x, qc, exp(-qc), &A, &B);
    return (A * qc * sinc_j0(qc * x) + B * cos(qc * x)) / (1.5 * kZeta3 * (1 - nufrac_low));
}

// delta_tot_table.c:442-463
KSP_HD double specialJ(double x, double qc, double nufrac_low) {
    return qc > 0 ? specialJ_series(x, qc, nufrac_low) : specialJ_fit(x);
}

// Index of the largest error among e[0..n) (lowest index on ties), on every lane of
// the warp.  Errors are >= 0, so their IEEE bit patterns order as the numbers do: the
// comparisons run on the integer pipe (a NaN, never chosen by the floating-point
// comparison, gets key -1; with nothing else in the list it is entry 0, as in QUADPACK's
// search, whose first candidate that is).
__device__ __forceinline__ long long err_key(double e) {
    const long long b = __double_as_longlong(e);
    return (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL ? -1LL : b;
}
__device__ __forceinline__ int warp_argmax_err(const double* e, int n) {
    const int lane = threadIdx.x & 31;
    long long best = -1;
    int bk = lane;
    for (int i = lane; i < n; i += 32) {
        const long long v = err_key(e[i]);
        if (v > best) { best = v; bk = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long ob = __shfl_down_sync(0xffffffffu, best, o);
        const int ok = __shfl_down_sync(0xffffffffu, bk, o);
        if (ob > best || (ob == best && ok < bk)) { best = ob; bk = ok; }
    }
    return __shfl_sync(0xffffffffu, bk, 0);
}

// ------------------------------------------------------------------ QAG (GK61)
#ifdef __CUDACC__
// The expanded 61-node table, the nodes of the embedded Gauss rule (odd i of the rule's table)
// first: slots 0-14 -x_1, -x_3, ..., 15-29 +x_1, ..., 30-44 -x_0, -x_2, ..., 45-59 +x_0, ..., 60 the
// centre.  A lane's second node (slots 32 on) then has no part in the Gauss sum.
struct Gk61Nodes {
    double x[61], wk[61], wg[32];
};

// the rule in memory: as arrays of the functions that index them they were copied to every
// thread's stack first (744 bytes, half a microsecond of each integral kernel's start)
static __device__ const double kGkXK[31] = KSP_GK61_XK_INIT;
static __device__ const double kGkWK[31] = KSP_GK61_WK_INIT;
static __device__ const double kGkWG[31] = KSP_GK61_WG_INIT;
__device__ __forceinline__ int gk61_index(int j) {  // i of slot j's +-x_i
    return j < 30 ? 2 * (j < 15 ? j : j - 15) + 1 : 2 * (j < 45 ? j - 30 : j - 45);  // 60: i = 30
}
__device__ __forceinline__ double gk61_x(int j) {  // abscissa of slot j
    const double x = __ldg(kGkXK + gk61_index(j));
    return j == 60 ? 0.0 : (j < 15 || (j >= 30 && j < 45) ? -x : x);
}
// slot of the s-th node in ascending x
__device__ __forceinline__ int gk61_ascending(int s) {
    const int i = s <= 30 ? s : 60 - s, up = s > 30 ? 1 : 0;
    return s == 30 ? 60 : ((i & 1) ? (i >> 1) + 15 * up : 30 + (i >> 1) + 15 * up);
}
__device__ __forceinline__ void gk61_fill(Gk61Nodes& n, int tid, int nthreads) {
    for (int j = tid; j < 61; j += nthreads) {
        const int i = gk61_index(j);
        n.x[j] = gk61_x(j);
        n.wk[j] = __ldg(kGkWK + i);
        if (j < 32) n.wg[j] = j < 30 ? __ldg(kGkWG + i) : 0.0;
    }
}

__device__ __forceinline__ double warp_sum_to0(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double bcast0(double v) { return __shfl_sync(0xffffffffu, v, 0); }

// QUADPACK error estimate: err = resasc * min(1, (200 |err|/resasc)^1.5), floored at
// 50 eps resabs (Piessens et al. 1983, qk rules).  With x = 200 |err| below resasc the estimate
// is x sqrt(x / resasc), formed as x^2 / sqrt(x resasc): one reciprocal square root in place of
// pow, or of a division and a square root, whose dependent FP64 chains are on the QAG's
// critical path.
// Values that are not negative are compared by their bits, on the integer pipe: an FP64
// comparison takes the FP64 pipe's 16 cycles.
__device__ __forceinline__ long long bits_of(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ double rescale_error(double err, double resabs, double resasc) {
    err = fabs(err);
    if (bits_of(resasc) != 0 && bits_of(err) != 0) {
        const double x = 200.0 * err, p = x * resasc;
        const int hp = __double2hiint(p);
        if (hp >= 0x05d00000 && hp < 0x7ff00000) {  // 2^-930 <= p, finite: neither is a NaN
            err = bits_of(x) >= bits_of(resasc) ? resasc : x * (x * rsqrt(p));
        } else if (x >= resasc) {
            err = resasc;
        } else {
            const double t = x / resasc;
            err = resasc * (t * sqrt(t));
        }
    }
    if (bits_of(resabs) > bits_of(DBL_MIN / (50.0 * DBL_EPSILON))) {
        const double fl = 50.0 * DBL_EPSILON * resabs;
        if (bits_of(fl) > bits_of(err)) err = fl;  // (a NaN among them: err was one)
    }
    return err;
}

struct GkOut { double result, abserr, resabs, resasc; };

// The GK61 sums of one or two intervals from the node values of a warp (fv[2 t + m]: node
// lane + 32 m of interval t, 0 past the 61st), and the rule's outputs, identical on every
// lane.  The FP64 pipe takes 16 cycles a warp instruction whatever its lanes do, so the count
// is what matters: the sums of both intervals are reduced together by a butterfly that
// halves the set of values each lane carries at every step, and where no value is negative
// (a density history's sign does not change: nearly always) |f| sums to what f does: the
// Kronrod and Gauss sums take 6 additions per lane, resasc's two 5.
__device__ __forceinline__ void gk61_lane_sums(const Gk61Nodes& N, const double* fv, int nint, const double* h,
                                               GkOut* out) {
    const int lane = threadIdx.x & 31;
    const bool two = lane < 29;  // the lane has a second node
    const double k0 = N.wk[lane], k1 = two ? N.wk[32 + lane] : 0.0;
    const double g0 = N.wg[lane];
    const int b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    double rk[2], rg[2];
#pragma unroll
    for (int t = 0; t < 2; t++) {
        rk[t] = fma(k1, fv[2 * t + 1], k0 * fv[2 * t]);
        rg[t] = g0 * fv[2 * t];
    }
    const int signs = __double2hiint(fv[0]) | __double2hiint(fv[1]) | __double2hiint(fv[2]) | __double2hiint(fv[3]);
    const bool negative = __any_sync(0xffffffffu, signs < 0);
    // interval 0 goes to the lanes below 16, 1 to the others; there Kronrod below bit 3, Gauss above
    const double ka = (b4 ? rk[1] : rk[0]) + __shfl_xor_sync(0xffffffffu, b4 ? rk[0] : rk[1], 16);
    const double ga = (b4 ? rg[1] : rg[0]) + __shfl_xor_sync(0xffffffffu, b4 ? rg[0] : rg[1], 16);
    double y = (b3 ? ga : ka) + __shfl_xor_sync(0xffffffffu, b3 ? ka : ga, 8);
    double ra = 0.0;
    if (negative) {  // warp-uniform
        double r[2];
#pragma unroll
        for (int t = 0; t < 2; t++) r[t] = fma(k1, fabs(fv[2 * t + 1]), k0 * fabs(fv[2 * t]));
        ra = (b4 ? r[1] : r[0]) + __shfl_xor_sync(0xffffffffu, b4 ? r[0] : r[1], 16);
        ra += __shfl_xor_sync(0xffffffffu, ra, 8);
        // one more value each: |f| on the lanes with bit 2
        const double give = b2 ? y : ra, keep = b2 ? ra : y;
        y = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    } else {
        y += __shfl_xor_sync(0xffffffffu, y, 4);
    }
    y += __shfl_xor_sync(0xffffffffu, y, 2);
    y += __shfl_xor_sync(0xffffffffu, y, 1);
    const double rk0 = __shfl_sync(0xffffffffu, y, 0), rk1 = __shfl_sync(0xffffffffu, y, 16);
    // distances from the mean, half the Kronrod sum
    const double s0 = fma(k1, fabs(fma(-0.5, rk0, fv[1])), k0 * fabs(fma(-0.5, rk0, fv[0])));
    const double s1 = fma(k1, fabs(fma(-0.5, rk1, fv[3])), k0 * fabs(fma(-0.5, rk1, fv[2])));
    double z = (b4 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, b4 ? s0 : s1, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    // the outputs of interval t on lane t, then broadcast
    const int t = lane & 1;
    const double rgt = __shfl_sync(0xffffffffu, y, t ? 24 : 8);
    const double rat = __shfl_sync(0xffffffffu, y, (t ? 16 : 0) + (negative ? 4 : 0));
    const double rst = __shfl_sync(0xffffffffu, z, t ? 16 : 0);
    GkOut o = {0.0, 0.0, 0.0, 0.0};
    if (lane < nint) {
        const double ht = t ? h[1] : h[0];
        const double rkt = t ? rk1 : rk0;
        o.result = rkt * ht;
        o.resabs = rat * fabs(ht);
        o.resasc = rst * fabs(ht);
        o.abserr = rescale_error((rkt - rgt) * ht, o.resabs, o.resasc);
    }
    for (int u = 0; u < nint; u++) {
        out[u].result = __shfl_sync(0xffffffffu, o.result, u);
        out[u].resabs = __shfl_sync(0xffffffffu, o.resabs, u);
        out[u].resasc = __shfl_sync(0xffffffffu, o.resasc, u);
        out[u].abserr = __shfl_sync(0xffffffffu, o.abserr, u);
    }
}

// Evaluate the GK61 rule on `nint` (1 or 2) intervals [a_t, b_t] with one warp.
// Every lane returns identical values.
template <class F>
__device__ __forceinline__ void gk61_warp(const F& f, const Gk61Nodes& N, int nint, const double* a, const double* b,
                                          GkOut* out) {
    const int lane = threadIdx.x & 31;
    double h[2], fv[4];
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const double c = __dmul_rn(0.5, __dadd_rn(a[t], b[t]));
        h[t] = __dmul_rn(0.5, __dsub_rn(b[t], a[t]));
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int j = lane + 32 * m;
            fv[2 * t + m] = t < nint && j < 61 ? f(__dadd_rn(c, __dmul_rn(h[t], N.x[j]))) : 0.0;
        }
    }
    gk61_lane_sums(N, fv, nint, h, out);
}

struct QagList {  // per-warp interval list in shared memory
    double a[kQagLimit], b[kQagLimit], r[kQagLimit], e[kQagLimit];
    int slot[kQagLimit];  // node-cache slot of the interval (-1: not cached)
};

struct QagResult { double result, abserr; int ok; int nint; };

// QUADPACK's bookkeeping of a bisection: interval k (result r_i, error e_i) into halves with
// the rule results g[0], g[1]; whether to go on.  The round-off and tiny-interval tests, whose
// outcome a comparison of high words nearly always settles, are then left out.
struct QagSums {
    double area, errsum, tol;
    int n, roundoff1, roundoff2, error_type;
};
__device__ __forceinline__ bool qag_account(QagSums& q, const GkOut* g, double r_i, double e_i, double a1, double a2,
                                            double b2, double epsabs, double epsrel, int limit) {
    const double area12 = g[0].result + g[1].result, error12 = g[0].abserr + g[1].abserr;
    q.errsum += error12 - e_i;
    q.area += area12 - r_i;
    // below half of e_i the error has fallen as it should
    if (__double2hiint(error12) >= __double2hiint(e_i) - 0x00100000 && g[0].resasc != g[0].abserr &&
        g[1].resasc != g[1].abserr) {
        if (fabs(r_i - area12) <= 1.0e-5 * fabs(area12) && error12 >= 0.99 * e_i) q.roundoff1++;
        if (q.n >= 10 && error12 > e_i) q.roundoff2++;
    }
    const double t = epsrel * fabs(q.area);  // fmax(epsabs, t)
    q.tol = bits_of(t) > bits_of(epsabs) && bits_of(t) <= 0x7ff0000000000000LL ? t : epsabs;
    const bool more = q.errsum > q.tol;
    if (more) {
        if (q.roundoff1 >= 6 || q.roundoff2 >= 20) q.error_type = 2;
        const int h1 = __double2hiint(fabs(a1)), h2 = __double2hiint(fabs(a2));
        if (h1 <= h2 + 1 || h2 < 0x01000000) {  // else |a1| is well above |a2|, and that above 1e-303
            const double tiny = (1 + 100 * DBL_EPSILON) * (fabs(a2) + 1000 * DBL_MIN);
            if (fabs(a1) <= tiny && fabs(b2) <= tiny) q.error_type = 3;
        }
    }
    q.n++;
    return q.n < limit && !q.error_type && more;
}

// QUADPACK QAG (Piessens et al. 1983) with the 61-point rule, run by one warp:
// bisect the interval with the largest error estimate until the summed error is
// below max(epsabs, epsrel |area|); QUADPACK's round-off and tiny-interval checks.
// Same decisions as the GSL-based reference path (delta_tot_table.c:404,597).
template <class F>
__device__ QagResult qag_warp(const F& f, const Gk61Nodes& N, QagList& L, double a, double b, double epsabs,
                              double epsrel, int limit) {
    const int lane = threadIdx.x & 31;
    QagResult R;
    GkOut g[2];
    double aa[2] = {a, a}, bb[2] = {b, b};
    gk61_warp(f, N, 1, aa, bb, g);
    if (lane == 0) { L.a[0] = a; L.b[0] = b; L.r[0] = g[0].result; L.e[0] = g[0].abserr; }
    __syncwarp();
    double tol = fmax(epsabs, epsrel * fabs(g[0].result));
    const double round_off = 50 * DBL_EPSILON * g[0].resabs;
    R.nint = 1;
    R.result = g[0].result;
    R.abserr = g[0].abserr;
    if (g[0].abserr <= round_off && g[0].abserr > tol) { R.ok = 0; return R; }
    if ((g[0].abserr <= tol && g[0].abserr != g[0].resasc) || g[0].abserr == 0.0) { R.ok = 1; return R; }
    if (limit == 1) { R.ok = 0; return R; }
    QagSums q = {g[0].result, g[0].abserr, tol, 1, 0, 0, 0};
    bool cont;
    do {
        // argmax of the error list (lowest index on ties)
        const int n = q.n, k = warp_argmax_err(L.e, n);
        const double a_i = L.a[k], b_i = L.b[k], r_i = L.r[k], e_i = L.e[k];
        const double a1 = a_i, b1 = 0.5 * (a_i + b_i), a2 = b1, b2 = b_i;
        aa[0] = a1; bb[0] = b1; aa[1] = a2; bb[1] = b2;
        gk61_warp(f, N, 2, aa, bb, g);
        cont = qag_account(q, g, r_i, e_i, a1, a2, b2, epsabs, epsrel, limit);
        __syncwarp();
        if (lane == 0) {
            L.b[k] = b1; L.r[k] = g[0].result; L.e[k] = g[0].abserr;
            L.a[n] = a2; L.b[n] = b2; L.r[n] = g[1].result; L.e[n] = g[1].abserr;
        }
        __syncwarp();
    } while (cont);
    double sum = 0;
    if (lane == 0)
        for (int i = 0; i < q.n; i++) sum += L.r[i];
    R.result = bcast0(sum);
    R.abserr = q.errsum;
    R.nint = q.n;
    R.ok = q.errsum <= q.tol;
    __syncwarp();
    return R;
}
// ------------------------------------------------------------------ cached QAG
// QAG only ever bisects, so its intervals are dyadic subintervals of [a, b].  For the
// delta_nu integral it refines toward the upper end (log a, where J -> 1 and the newest
// history rows are): at every depth the intervals it evaluates are the two children of
// the rightmost interval of the depth above.  Those are numbered, and a functor's node_at
// serves the 61 nodes of a numbered interval from a table built once; the others pass slot -1.
// Where hybrid neutrinos cut J it oscillates, and the bisections go anywhere: all intervals
// down to some depth are numbered then.  A table of `tree` = 2^(D+1) - 1 slots down to depth D
// numbers them as a heap (slot 0 = [a, b], slot s has children 2 s + 1 and 2 s + 2), and then
// left and right child of the rightmost interval, depth after depth; D = 0 without the cut.
constexpr int kNcMaxLevels = 12;
constexpr int kNcMaxSlots = 1 + 2 * kNcMaxLevels;  // 25 intervals
constexpr int kNcNodes = kNcMaxSlots * 61;         // capacity of a node table
constexpr int kNcTreeDepth = 6, kNcTree = (2 << kNcTreeDepth) - 1;
constexpr int kNcTreeSlots = kNcTree + 2 * (kNcMaxLevels - kNcTreeDepth);

struct NcLayout {
    int nslots, tree;
};
// child slot of s (right = 0, 1)
__device__ __forceinline__ int nc_child(int s, int right, NcLayout t) {
    if (s < 0) return -1;
    int c = 2 * s + 1 + right;
    if (c >= t.tree) {  // past the heap only the rightmost intervals have children
        if (s == t.tree - 1) c = t.tree + right;
        else if (s >= t.tree && ((s - t.tree) & 1)) c = s + 1 + right;
        else return -1;
    }
    return c < t.nslots ? c : -1;
}

// Centre and half-width of an interval.  A cached one's nodes need no centre, and its half-width
// is in the table.
template <class F>
__device__ __forceinline__ void gk61_geometry(const F& f, int slot, double a, double b, double& c, double& h) {
    c = 0.0;
    if (slot >= 0) {
        h = __ldg(f.nc.half + slot);
    } else {
        c = __dmul_rn(0.5, __dadd_rn(a, b));
        h = __dmul_rn(0.5, __dsub_rn(b, a));
    }
}

// gk61_warp with interval slots
template <class F>
__device__ __forceinline__ void gk61_warp_c(const F& f, const Gk61Nodes& N, int nint, const double* a,
                                            const double* b, const int* slot, GkOut* out) {
    const int lane = threadIdx.x & 31;
    double c[2], h[2];
#pragma unroll
    for (int t = 0; t < 2; t++) gk61_geometry(f, slot[t], a[t], b[t], c[t], h[t]);
    double fv[4];
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int j = lane + 32 * m;
            fv[2 * t + m] = t < nint && j < 61 ? f.node_at(slot[t], j, c[t], h[t], N.x[j]) : 0.0;
        }
    gk61_lane_sums(N, fv, nint, h, out);
}

// qag_warp with interval slots (same decisions)
template <class F>
__device__ QagResult qag_warp_c(const F& f, const Gk61Nodes& N, QagList& L, double a, double b, double epsabs,
                                double epsrel, int limit) {
    const int lane = threadIdx.x & 31;
    QagResult R;
    GkOut g[2];
    double aa[2] = {a, a}, bb[2] = {b, b};
    int ss[2] = {f.nc.lay.nslots > 0 ? 0 : -1, -1};
    gk61_warp_c(f, N, 1, aa, bb, ss, g);
    if (lane == 0) { L.a[0] = a; L.b[0] = b; L.r[0] = g[0].result; L.e[0] = g[0].abserr; L.slot[0] = ss[0]; }
    __syncwarp();
    double tol = fmax(epsabs, epsrel * fabs(g[0].result));
    const double round_off = 50 * DBL_EPSILON * g[0].resabs;
    R.nint = 1;
    R.result = g[0].result;
    R.abserr = g[0].abserr;
    if (g[0].abserr <= round_off && g[0].abserr > tol) { R.ok = 0; return R; }
    if ((g[0].abserr <= tol && g[0].abserr != g[0].resasc) || g[0].abserr == 0.0) { R.ok = 1; return R; }
    if (limit == 1) { R.ok = 0; return R; }
    QagSums q = {g[0].result, g[0].abserr, tol, 1, 0, 0, 0};
    int n = 1, cont = 0;
    do {
        const int k = warp_argmax_err(L.e, n);
        const double a_i = L.a[k], b_i = L.b[k], r_i = L.r[k], e_i = L.e[k];
        const int s_i = L.slot[k];
        const double a1 = a_i, b1 = 0.5 * (a_i + b_i), a2 = b1, b2 = b_i;
        aa[0] = a1; bb[0] = b1; aa[1] = a2; bb[1] = b2;
        ss[0] = nc_child(s_i, 0, f.nc.lay);
        ss[1] = nc_child(s_i, 1, f.nc.lay);
        gk61_warp_c(f, N, 2, aa, bb, ss, g);
        // QUADPACK's bookkeeping on lane 0 (its FP64 is not repeated on 32 lanes)
        cont = 0;
        __syncwarp();
        if (lane == 0) {
            cont = qag_account(q, g, r_i, e_i, a1, a2, b2, epsabs, epsrel, limit);
            L.b[k] = b1; L.r[k] = g[0].result; L.e[k] = g[0].abserr; L.slot[k] = ss[0];
            L.a[n] = a2; L.b[n] = b2; L.r[n] = g[1].result; L.e[n] = g[1].abserr; L.slot[n] = ss[1];
        }
        cont = __shfl_sync(0xffffffffu, cont, 0);
        __syncwarp();
        n++;
    } while (cont);
    double sum = 0;
    if (lane == 0)
        for (int i = 0; i < n; i++) sum += L.r[i];
    R.result = bcast0(sum);
    R.abserr = bcast0(q.errsum);
    R.nint = n;
    R.ok = __shfl_sync(0xffffffffu, (int)(q.errsum <= q.tol), 0);
    __syncwarp();
    return R;
}

// ------------------------------------------------------------------ block-cooperative QAG
// The same rule and decisions with the node evaluations spread over the warps of a block
// (blockDim.x = 32 * W, W = 2 or 4): thread t evaluates node t, t + 32W, ...; warp 0
// then sums them as gk61_warp_c does: the arithmetic of qag_warp_c in the same order (the compiler may contract multiply-adds differently per kernel, so the
// results agree to the last bits).  Shared scratch: QagBlockSmem.
struct QagBlockSmem {
    double fv[128];
    GkOut out[2];
    double a[2], b[2];
    int slot[2];
    int k, cont, ok;   // the interval to bisect, whether to go on, errsum <= tol
    double errsum;
};

template <class F>
__device__ __forceinline__ void gk61_block_c(const F& f, const Gk61Nodes& N, int nint, const double* a,
                                             const double* b, const int* slot, GkOut* out, QagBlockSmem& sh) {
    const int tid = threadIdx.x, lane = tid & 31;
    double c[2], h[2];
    for (int t = 0; t < 2; t++) gk61_geometry(f, slot[t], a[t], b[t], c[t], h[t]);
    const int nslots = 61 * nint;
    for (int s = tid; s < nslots; s += blockDim.x) {
        const int t = s >= 61 ? 1 : 0;
        const int j = s - 61 * t;
        sh.fv[s] = f.node_at(slot[t], j, c[t], h[t], N.x[j]);
    }
    __syncthreads();
    if (tid < 32) {  // warp 0: the sums exactly as gk61_warp_c forms them
        double fv[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const int j = lane + 32 * (m & 1), t = m >> 1;
            fv[m] = t < nint && j < 61 ? sh.fv[61 * t + j] : 0.0;
        }
        GkOut o[2];
        gk61_lane_sums(N, fv, nint, h, o);
        if (lane < nint) sh.out[lane] = o[lane];
    }
    __syncthreads();
    for (int t = 0; t < nint; t++) out[t] = sh.out[t];
}

// qag_warp_c run by a whole block: every thread follows the same decisions (they read the
// same shared list); thread 0 writes the list.
template <class F>
__device__ QagResult qag_block_c(const F& f, const Gk61Nodes& N, QagList& L, double a, double b, double epsabs,
                                 double epsrel, int limit, QagBlockSmem& sh) {
    const int tid = threadIdx.x, lane = tid & 31;
    QagResult R;
    GkOut g[2];
    double aa[2] = {a, a}, bb[2] = {b, b};
    int ss[2] = {f.nc.lay.nslots > 0 ? 0 : -1, -1};
    gk61_block_c(f, N, 1, aa, bb, ss, g, sh);
    if (tid == 0) { L.a[0] = a; L.b[0] = b; L.r[0] = g[0].result; L.e[0] = g[0].abserr; L.slot[0] = ss[0]; }
    __syncthreads();
    double tol = fmax(epsabs, epsrel * fabs(g[0].result));
    const double round_off = 50 * DBL_EPSILON * g[0].resabs;
    R.nint = 1;
    R.result = g[0].result;
    R.abserr = g[0].abserr;
    if (g[0].abserr <= round_off && g[0].abserr > tol) { R.ok = 0; return R; }
    if ((g[0].abserr <= tol && g[0].abserr != g[0].resasc) || g[0].abserr == 0.0) { R.ok = 1; return R; }
    if (limit == 1) { R.ok = 0; return R; }
    QagSums q = {g[0].result, g[0].abserr, tol, 1, 0, 0, 0};
    int n = 1;
    do {
        // warp 0 finds the interval of largest error (lowest index on ties)
        if (tid < 32) {
            const int bk = warp_argmax_err(L.e, n);
            if (lane == 0) sh.k = bk;
        }
        __syncthreads();
        const int k = sh.k;
        const double a_i = L.a[k], b_i = L.b[k], r_i = L.r[k], e_i = L.e[k];
        const int s_i = L.slot[k];
        const double a1 = a_i, b1 = 0.5 * (a_i + b_i), a2 = b1, b2 = b_i;
        aa[0] = a1; bb[0] = b1; aa[1] = a2; bb[1] = b2;
        ss[0] = nc_child(s_i, 0, f.nc.lay);
        ss[1] = nc_child(s_i, 1, f.nc.lay);
        gk61_block_c(f, N, 2, aa, bb, ss, g, sh);
        // QUADPACK's bookkeeping on thread 0
        if (tid == 0) {
            sh.cont = qag_account(q, g, r_i, e_i, a1, a2, b2, epsabs, epsrel, limit);
            L.b[k] = b1; L.r[k] = g[0].result; L.e[k] = g[0].abserr; L.slot[k] = ss[0];
            L.a[n] = a2; L.b[n] = b2; L.r[n] = g[1].result; L.e[n] = g[1].abserr; L.slot[n] = ss[1];
            sh.errsum = q.errsum;
            sh.ok = q.errsum <= q.tol;
        }
        __syncthreads();
        n++;
    } while (sh.cont);
    double sum = 0;
    if (lane == 0)
        for (int i = 0; i < n; i++) sum += L.r[i];
    R.result = bcast0(sum);
    R.abserr = sh.errsum;
    R.nint = n;
    R.ok = sh.ok;
    __syncthreads();
    return R;
}

// ------------------------------------------------------------------ block QAG with look-ahead
// qag_block_c with G - 1 levels of look-ahead.  On these integrands QAG nearly always
// bisects next the right half it has just made (the late-time end, where delta_tot and
// the free-streaming kernel change fastest).  A round that evaluates the halves of
// interval k therefore also evaluates the halves of k's right half, and so on down G levels
// (the first round: the whole interval and G - 1 levels); while the next rounds pick those
// halves, their rule results are already there and the rounds are bookkeeping only, so that
// the sequential evaluation rounds are 1/G as many.  Node values come from the same
// node_at, and each interval's sums are formed by one warp in the lane layout of a
// two-interval gk61_block_c call, so every rule result is that of qag_block_c (to the
// last bits, which the compiler's multiply-add contraction may change from kernel to
// kernel) and so is every decision.  blockDim.x = 128 G: a round's 122 G nodes in one pass.
template <int G>
struct QagSpecSmem {
    double fv[122 * G];          // group (level) g: slots [122 g, 122 g + 122)
    GkOut out[2 * G];            // group g: intervals 2 g, 2 g + 1
    double ic[2 * G], ih[2 * G]; // centre and half-width of the intervals of the next evaluation
    int isl[2 * G];              // and their node-table slots
    int k, hit, cont, ok;
    int pre_k, pre_g;            // the list entry whose halves group pre_g holds (-1: none)
    double errsum;
};

// Interval q of the next evaluation: its slot, or its geometry, formed once (one thread).
template <class S>
__device__ __forceinline__ void spec_set_interval(S& sh, int q, double a, double b, int slot) {
    sh.isl[q] = slot;
    if (slot >= 0) return;
    sh.ic[q] = __dmul_rn(0.5, __dadd_rn(a, b));
    sh.ih[q] = __dmul_rn(0.5, __dsub_rn(b, a));
}
// Groups g0 .. G - 1: the halves of [a, b] (slot), of its right half, ...
template <int G>
__device__ __forceinline__ void spec_set_halves(QagSpecSmem<G>& sh, int g0, double a, double b, int slot, NcLayout ns) {
    for (int g = g0; g < G; g++) {
        const double m = 0.5 * (a + b);
        spec_set_interval(sh, 2 * g, a, m, nc_child(slot, 0, ns));
        slot = nc_child(slot, 1, ns);
        spec_set_interval(sh, 2 * g + 1, m, b, slot);
        a = m;
    }
}

// Rule results of ng groups' intervals (n0 in {1, 2} of group 0), whose geometry is in
// sh.ic / sh.ih / sh.isl.  Warp g sums group g as gk61_block_c sums a call of that many
// intervals.
template <class S, class F>
__device__ __forceinline__ void gk61_block_groups(const F& f, const Gk61Nodes& N, int n0, int ng, S& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 122 * ng) {
        const int g = tid / 122, u = tid - 122 * g;
        const int t = u >= 61 ? 1 : 0, j = u - 61 * t;
        if (g > 0 || t < n0) {
            const int q = 2 * g + t;
            sh.fv[tid] = f.node_at(sh.isl[q], j, sh.ic[q], sh.ih[q], N.x[j]);
        }
    }
    __syncthreads();
    if (warp < ng) {
        const int ni = warp == 0 ? n0 : 2;
        const double* fvg = sh.fv + 122 * warp;
        double fv[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const int j = lane + 32 * (m & 1), t = m >> 1;
            fv[m] = t < ni && j < 61 ? fvg[61 * t + j] : 0.0;
        }
        double hh[2];
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const int q = 2 * warp + t, slot = t < ni ? sh.isl[q] : -1;
            hh[t] = slot >= 0 ? __ldg(f.nc.half + slot) : sh.ih[q];
        }
        GkOut o[2];
        gk61_lane_sums(N, fv, ni, hh, o);
        if (lane == 0) {
            sh.out[2 * warp] = o[0];
            if (ni > 1) sh.out[2 * warp + 1] = o[1];
        }
    }
    __syncthreads();
}

template <int G, class F>
__device__ QagResult qag_block_spec_c(const F& f, const Gk61Nodes& N, QagList& L, double a, double b, double epsabs,
                                      double epsrel, int limit, QagSpecSmem<G>& sh) {
    const int tid = threadIdx.x, lane = tid & 31;
    const NcLayout ns = f.nc.lay;
    QagResult R;
    const int s0 = ns.nslots > 0 ? 0 : -1;
    if (tid == 0) {  // the root, and halves ahead
        spec_set_interval(sh, 0, a, b, s0);
        spec_set_halves(sh, 1, a, b, s0, ns);
    }
    __syncthreads();
    gk61_block_groups(f, N, 1, G, sh);
    const GkOut g0 = sh.out[0];
    if (tid == 0) {
        L.a[0] = a; L.b[0] = b; L.r[0] = g0.result; L.e[0] = g0.abserr; L.slot[0] = s0;
        sh.pre_k = 0; sh.pre_g = 1;
    }
    __syncthreads();
    double tol = fmax(epsabs, epsrel * fabs(g0.result));
    const double round_off = 50 * DBL_EPSILON * g0.resabs;
    R.nint = 1;
    R.result = g0.result;
    R.abserr = g0.abserr;
    if (g0.abserr <= round_off && g0.abserr > tol) { R.ok = 0; return R; }
    if ((g0.abserr <= tol && g0.abserr != g0.resasc) || g0.abserr == 0.0) { R.ok = 1; return R; }
    if (limit == 1) { R.ok = 0; return R; }
    QagSums q = {g0.result, g0.abserr, tol, 1, 0, 0, 0};
    int n = 1;
    do {
        // warp 0 finds the interval of largest error (lowest index on ties); its lane 0
        // notes whether the halves are already evaluated and, if not, lays out the halves
        // of k, of k's right half, ...
        if (tid < 32) {
            const int bk = warp_argmax_err(L.e, n);
            if (lane == 0) {
                const bool hit = bk == sh.pre_k;
                sh.k = bk;
                sh.hit = hit;
                if (!hit) spec_set_halves(sh, 0, L.a[bk], L.b[bk], L.slot[bk], ns);
            }
        }
        __syncthreads();
        const int k = sh.k;
        if (!sh.hit) gk61_block_groups(f, N, 2, G, sh);  // block-uniform
        // QUADPACK's bookkeeping on thread 0
        if (tid == 0) {
            const int gi = sh.hit ? sh.pre_g : 0;
            const double a_i = L.a[k], b_i = L.b[k], r_i = L.r[k], e_i = L.e[k];
            const int s_i = L.slot[k];
            const double a1 = a_i, b1 = 0.5 * (a_i + b_i), a2 = b1, b2 = b_i;
            const GkOut g[2] = {sh.out[2 * gi], sh.out[2 * gi + 1]};
            sh.cont = qag_account(q, g, r_i, e_i, a1, a2, b2, epsabs, epsrel, limit);
            L.b[k] = b1; L.r[k] = g[0].result; L.e[k] = g[0].abserr; L.slot[k] = nc_child(s_i, 0, ns);
            L.a[n] = a2; L.b[n] = b2; L.r[n] = g[1].result; L.e[n] = g[1].abserr; L.slot[n] = nc_child(s_i, 1, ns);
            sh.pre_k = gi + 1 < G ? n : -1;
            sh.pre_g = gi + 1;
            sh.errsum = q.errsum;
            sh.ok = q.errsum <= q.tol;
        }
        __syncthreads();
        n++;
    } while (sh.cont);
    double sum = 0;
    if (lane == 0)
        for (int i = 0; i < n; i++) sum += L.r[i];
    R.result = bcast0(sum);
    R.abserr = sh.errsum;
    R.nint = n;
    R.ok = sh.ok;
    __syncthreads();
    return R;
}

// ------------------------------------------------------------------ block QAG, several intervals a round
// qag_block_c for integrands that oscillate (J with a momentum cut): which interval is next is
// anyone's guess, but those with a large error all have their turn.  A round that needs the halves
// of interval k evaluates those of the up to G - 1 intervals of the next largest errors as well
// and keeps their rule results until QAG picks them: next to no evaluation is wasted, and the
// sequence of decisions is qag_block_c's.  blockDim.x = 128 G.
template <int G>
struct QagMultiSmem {
    double fv[122 * G];          // as QagSpecSmem
    GkOut out[2 * G];
    double ic[2 * G], ih[2 * G];
    int isl[2 * G];
    GkOut kept[2 * 32];          // rule results of halves evaluated ahead
    signed char have[kQagLimit]; // where a list entry's are kept (-1: nowhere)
    int gk[G];                   // the groups' list entries
    int k, ng, cont, ok;
    double errsum, tol;
};

template <int G, class F>
__device__ QagResult qag_block_multi_c(const F& f, const Gk61Nodes& N, QagList& L, double a, double b, double epsabs,
                                       double epsrel, int limit, QagMultiSmem<G>& sh) {
    const int tid = threadIdx.x, lane = tid & 31;
    const NcLayout ns = f.nc.lay;
    QagResult R;
    const int s0 = ns.nslots > 0 ? 0 : -1;
    auto set_halves = [&](int g, double a, double b, int slot) {
        const double m = 0.5 * (a + b);
        spec_set_interval(sh, 2 * g, a, m, nc_child(slot, 0, ns));
        spec_set_interval(sh, 2 * g + 1, m, b, nc_child(slot, 1, ns));
    };
    if (tid == 0) {  // the root, and its halves
        spec_set_interval(sh, 0, a, b, s0);
        set_halves(1, a, b, s0);
    }
    __syncthreads();
    gk61_block_groups(f, N, 1, 2, sh);
    const GkOut g0 = sh.out[0];
    double tol = fmax(epsabs, epsrel * fabs(g0.result));
    unsigned spare = ~1u;  // (thread 0) free places of sh.kept
    if (tid == 0) {
        L.a[0] = a; L.b[0] = b; L.r[0] = g0.result; L.e[0] = g0.abserr; L.slot[0] = s0;
        sh.kept[0] = sh.out[2];
        sh.kept[1] = sh.out[3];
        sh.have[0] = 0;
        sh.tol = tol;
    }
    __syncthreads();
    const double round_off = 50 * DBL_EPSILON * g0.resabs;
    R.nint = 1;
    R.result = g0.result;
    R.abserr = g0.abserr;
    if (g0.abserr <= round_off && g0.abserr > tol) { R.ok = 0; return R; }
    if ((g0.abserr <= tol && g0.abserr != g0.resasc) || g0.abserr == 0.0) { R.ok = 1; return R; }
    if (limit == 1) { R.ok = 0; return R; }
    QagSums q = {g0.result, g0.abserr, tol, 1, 0, 0, 0};
    int n = 1;
    do {
        if (tid < 32) {
            const int bk = warp_argmax_err(L.e, n);
            int ng = 0;
            if (sh.have[bk] < 0) {
                if (lane == 0) sh.gk[0] = bk;
                ng = 1;
                const int room = __popc(__shfl_sync(0xffffffffu, spare, 0));
                // (an error below tol / 2 n is small enough to stay)
                const long long least = bits_of(sh.tol * (0.5 / n));
                while (ng < G && ng <= room) {
                    __syncwarp();
                    long long best = least;
                    int at = -1;
                    for (int i = lane; i < n; i += 32) {
                        bool taken = sh.have[i] >= 0;
                        for (int u = 0; u < ng; u++) taken = taken || sh.gk[u] == i;
                        const long long v = err_key(L.e[i]);
                        if (!taken && v > best) { best = v; at = i; }
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const long long ob = __shfl_down_sync(0xffffffffu, best, o);
                        const int oa = __shfl_down_sync(0xffffffffu, at, o);
                        if (ob > best) { best = ob; at = oa; }
                    }
                    at = __shfl_sync(0xffffffffu, at, 0);
                    if (at < 0) break;
                    if (lane == 0) sh.gk[ng] = at;
                    ng++;
                }
                __syncwarp();
                if (lane < ng) {  // a lane per group
                    const int i = sh.gk[lane];
                    set_halves(lane, L.a[i], L.b[i], L.slot[i]);
                }
            }
            if (lane == 0) {
                sh.k = bk;
                sh.ng = ng;
            }
        }
        __syncthreads();
        const int k = sh.k, ng = sh.ng;
        if (ng > 0) gk61_block_groups(f, N, 2, ng, sh);  // block-uniform
        // QUADPACK's bookkeeping on thread 0
        if (tid == 0) {
            const double a_i = L.a[k], b_i = L.b[k], r_i = L.r[k], e_i = L.e[k];
            const int s_i = L.slot[k];
            const double a1 = a_i, b1 = 0.5 * (a_i + b_i), a2 = b1, b2 = b_i;
            for (int u = 1; u < ng; u++) {
                const int p = __ffs(spare) - 1;
                spare &= spare - 1;
                sh.kept[2 * p] = sh.out[2 * u];
                sh.kept[2 * p + 1] = sh.out[2 * u + 1];
                sh.have[sh.gk[u]] = (signed char)p;
            }
            const int p = sh.have[k];
            const GkOut g[2] = {p >= 0 ? sh.kept[2 * p] : sh.out[0], p >= 0 ? sh.kept[2 * p + 1] : sh.out[1]};
            if (p >= 0) spare |= 1u << p;
            sh.cont = qag_account(q, g, r_i, e_i, a1, a2, b2, epsabs, epsrel, limit);
            L.b[k] = b1; L.r[k] = g[0].result; L.e[k] = g[0].abserr; L.slot[k] = nc_child(s_i, 0, ns);
            L.a[n] = a2; L.b[n] = b2; L.r[n] = g[1].result; L.e[n] = g[1].abserr; L.slot[n] = nc_child(s_i, 1, ns);
            sh.have[k] = sh.have[n] = -1;
            sh.tol = q.tol;
            sh.errsum = q.errsum;
            sh.ok = q.errsum <= q.tol;
        }
        __syncthreads();
        n++;
    } while (sh.cont);
    double sum = 0;
    if (lane == 0)
        for (int i = 0; i < n; i++) sum += L.r[i];
    R.result = bcast0(sum);
    R.abserr = sh.errsum;
    R.nint = n;
    R.ok = sh.ok;
    __syncthreads();
    return R;
}

}  // namespace ksp
#include "ksp_jfit.cuh"
namespace ksp {

struct StepScalars;

// ------------------------------------------------------------------ delta_nu integrand
// delta_tot_table.c:492-500: fslength(x, log a) / (a H(a)) J(k fslength / (m/kT))
// delta_tot(k, x) at x = log a_i.  Split into the part that depends only on x (and the
// instance), NodeTerms, and the per-bin rest.
struct NodeTerms {
    double g;    // fslength / (a H(a))
    double fsl;  // fslength(x, log a)
    double dx;   // x - knot[j]
    int j;       // history segment: knot[j] <= x < knot[j+1]
};

// 1 / (a H(a)) at x = log a
static __device__ __noinline__ double node_inv_aH(const Background* B, double x) {
    if (B->htab_n > 0) return exp(-x - hubble_tab_log(*B, x));
    const double ia = exp(-x);
    return ia * inv_hubble_ia(*B, x, ia);
}
// The uniform nodes of the fslength table: log a of the first, their spacing and its inverse.
struct FsGrid {
    int n;
    double x0, h, ih;
    __host__ __device__ __forceinline__ double node(int i) const { return x0 + i * h; }
    // the segment of x (a rounding across a node is harmless: the cubics meet there)
    __device__ __forceinline__ int segment(double x) const {
        const int i = (int)((x - x0) * ih);
        return i < 0 ? 0 : (i > n - 2 ? n - 2 : i);
    }
};
__host__ __device__ inline FsGrid fs_grid(int n, double loga0, double loga) {
    if (n < 2) return FsGrid{n, loga0, 0.0, 0.0};
    return FsGrid{n, loga0, (loga - loga0) / (n - 1.), (n - 1.) / (loga - loga0)};
}
// the table's spline dx past the lower node of a segment, from the values and coefficients of
// its nodes (dy: the values' difference)
__device__ __forceinline__ double fs_spline_eval(const FsGrid& g, double y0, double dy, double c0, double c1,
                                                 double dx) {
    const double bq = fma(dy, g.ih, -(g.h * (1.0 / 3.0)) * fma(2.0, c0, c1));
    const double d = (c1 - c0) * (g.ih * (1.0 / 3.0));
    return fma(dx, fma(dx, fma(dx, d, c0), bq), y0);
}
static __device__ __noinline__ NodeTerms dnu_node_terms(const Background* B, const double* fs_y, const double* fs_c,
                                                        const FsGrid& g, const double* kx, int na, double x) {
    NodeTerms t;
    const int i = g.segment(x);
    t.fsl = fs_spline_eval(g, fs_y[i], fs_y[i + 1] - fs_y[i], fs_c[i], fs_c[i + 1], x - g.node(i));
    t.j = seg_bsearch(kx, na, x);
    t.dx = x - kx[t.j];
    t.g = t.fsl * node_inv_aH(B, x);
    return t;
}

// Per-segment constants of the history knots: 1/h, h/3, 1/(3h).
struct KnotSeg {
    const double* ih;
    const double* h3;
    const double* ih3;
};

// The history row's natural spline (or linear for 2 knots) at a node: the node-independent
// part per segment of a history row, computed once per (row, call) into sb / sd by threads
// t, t+nt, ..., then three FMAs per node.
__device__ __forceinline__ void seg_poly(const double* ky, const double* kc, int na, const KnotSeg& ks, double* sb,
                                         double* sd, int t, int nt) {
    for (int j = t; j < na - 1; j += nt) {
        const double y0 = ky[j], y1 = ky[j + 1], c0 = kc[j], c1 = kc[j + 1];
        sb[j] = (y1 - y0) * __ldg(ks.ih + j) - (c1 + 2.0 * c0) * __ldg(ks.h3 + j);
        sd[j] = (c1 - c0) * __ldg(ks.ih3 + j);
    }
}
__device__ __forceinline__ double dnu_S_poly(const NodeTerms& t, const double* ky, const double* kc,
                                             const double* sb, const double* sd, int na, const KnotSeg& ks) {
    const int j = t.j;
    if (na > 2) return ky[j] + t.dx * (sb[j] + t.dx * (kc[j] + t.dx * sd[j]));
    return ky[j] + t.dx * ((ky[j + 1] - ky[j]) * __ldg(ks.ih + j));
}

// Node table of one instance for one call: nslots * 61 entries, slot-major.
struct NodeCache {
    double* g;
    double* fsl;
    double* dx;
    int* j;
    NcLayout lay;
};

// The integrand's terms at the nodes, for the adjoint.
struct DnuIntegrandC {
    const Background* B;
    double k_over_m, qc, nfl;
    const double* fs_y; const double* fs_c; FsGrid fs;
    const double* kx; const double* ky; const double* kc; int na;
    const double* sb; const double* sd;  // seg_poly of (ky, kc)
    KnotSeg ks;
    NodeCache nc;
    __device__ NodeTerms terms(int slot, int jn, double x) const {
        if (slot >= 0) {
            const int q = slot * 61 + jn;
            NodeTerms t;
            t.g = __ldg(nc.g + q);
            t.fsl = __ldg(nc.fsl + q);
            t.dx = __ldg(nc.dx + q);
            t.j = __ldg(nc.j + q);
            return t;
        }
        return dnu_node_terms(B, fs_y, fs_c, fs, kx, na, x);
    }
};

// The integrand as the integrals evaluate it.  At a node in history segment j the natural
// spline is S = A y_j + B y_{j+1} + C c_j + D c_{j+1} (c = S''/2 at the knots) with weights that
// depend on the node only, so the node table holds g A, g B, g C, g D and a bin's value is
// J (k fslength / (m / kT)) times their sum with its row: five FP64 operations and J's six,
// against fourteen with the spline's polynomial per segment and J's first table, and no
// per-bin pass over the segments.
struct NodeWeights {
    double a, b, c, d;
};
__device__ __forceinline__ NodeWeights node_weights(double g, double dx, double h, double ih, int na) {
    NodeWeights w;
    const double s = dx * ih;
    const double gs = __dmul_rn(g, s);
    w.a = __dsub_rn(g, gs);
    w.b = gs;
    const double e = na > 2 ? __dmul_rn(__dmul_rn(g, dx), 1.0 / 3.0) : 0.0;  // two knots: linear
    // C = dx (dx - 2 h / 3 - dx s / 3), D = dx (dx s - h) / 3
    w.c = __dmul_rn(e, __dsub_rn(__dmul_rn(3.0, dx), __fma_rn(dx, s, __dmul_rn(2.0, h))));
    w.d = __dmul_rn(e, __fma_rn(dx, s, -h));
    return w;
}
// Node table entry: {g A, g B}, {g C, g D}, fslength, {j, fslength as a float}; a slot's 61
// entries share a half-width.
struct NodeTable {
    const double2* ab;
    const double2* cd;
    const double* fsl;
    const int2* jf;
    const double* half;  // half-width of a slot's interval
    NcLayout lay;
};
struct DnuIntegrandW {
    const Background* B;
    const double* jt;          // J's fine table
    double kom;                // k / (m / kT)
    float komf;
    double qc, nfl;            // qc > 0: the series instead of the fit,
    const double* hyb;         // from its table (or null)
    const double* ky;          // the bin's history row and its spline coefficients
    const double* kc;
    NodeTable nc;
    // for intervals that are not in the node table
    const double* fs_y; const double* fs_c; const double* kx; const double* kih;
    const StepScalars* S;
    int na;
    __device__ __forceinline__ double value(const NodeWeights& w, double fsl, float fslf, int j) const {
        const double v = fma(w.d, kc[j + 1], fma(w.c, kc[j], fma(w.b, ky[j + 1], __dmul_rn(w.a, ky[j]))));
        return __dmul_rn(v, qc > 0 ? specialJ_cut(hyb, fsl * kom, qc, nfl)
                                   : specialJ_node(jt, fsl, fslf, kom, komf));
    }
    __device__ __forceinline__ double node_at(int slot, int jn, double c, double h, double xj) const {
        if (slot >= 0) {
            const int q = slot * 61 + jn;
            const double2 ab = __ldg(nc.ab + q), cd = __ldg(nc.cd + q);
            const int2 jf = __ldg(nc.jf + q);
            return value(NodeWeights{ab.x, ab.y, cd.x, cd.y}, __ldg(nc.fsl + q), __int_as_float(jf.y), jf.x);
        }
        return slow(__dadd_rn(c, __dmul_rn(h, xj)));
    }
    __device__ __noinline__ double slow(double x) const;  // (ksp_internal.h)
};

// Slot of the dyadic interval [a, b] of [lo, hi] in a node table (-1: not one of them), by the
// bisections QAG performs.
__device__ __forceinline__ int nc_slot_of(double a, double b, double lo, double hi, NcLayout t) {
    int s = t.nslots > 0 ? 0 : -1;
    while (s >= 0 && !(a == lo && b == hi)) {
        const double m = 0.5 * (lo + hi);
        const int right = a >= m ? 1 : 0;
        if (!right && b > m) return -1;
        if (right) lo = m;
        else hi = m;
        s = nc_child(s, right, t);
    }
    return s;
}

// Segmented sums over the lanes of a warp: runs of equal key (in lane order) are summed
// onto the run's last lane, for four values at once.
__device__ __forceinline__ void warp_seg_sum4(int key, double& a, double& b, double& c, double& d, bool& tail) {
    const int lane = threadIdx.x & 31;
    const int up = __shfl_up_sync(0xffffffffu, key, 1);
    const bool head = lane == 0 || up != key;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int my_head = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
        const double oa = __shfl_up_sync(0xffffffffu, a, dd), ob = __shfl_up_sync(0xffffffffu, b, dd);
        const double oc = __shfl_up_sync(0xffffffffu, c, dd), od = __shfl_up_sync(0xffffffffu, d, dd);
        if (lane - dd >= my_head) { a += oa; b += ob; c += oc; d += od; }
    }
    tail = lane == 31 || ((heads >> (lane + 1)) & 1u);
}

// End points of cache slot s of [a, b], by the bisections QAG performs (b1 = (a+b)/2).
__device__ __forceinline__ void nc_interval(int s, NcLayout t, double a, double b, double* lo, double* hi) {
    const int u = s - t.tree;                   // past the heap: its number there
    const int h = u < 0 ? s + 1 : t.tree;       // the heap's node (from 1) to start from
    for (int k = 30 - __clz(h); k >= 0; k--) {  // the bits after the leading one: left or right
        const double m = 0.5 * (a + b);
        if ((h >> k) & 1) a = m;
        else b = m;
    }
    if (u >= 0) {
        for (int k = 0; k < u / 2; k++) a = 0.5 * (a + b);
        const double m = 0.5 * (a + b);
        if (u & 1) a = m;
        else b = m;
    }
    *lo = a;
    *hi = b;
}
#endif  // __CUDACC__

}  // namespace ksp
