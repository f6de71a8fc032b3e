// ksp_jfit.cuh -- J(x) of the delta_nu integrand (delta_tot_table.c:417-428) evaluated
// from the piecewise polynomials of jfit_table.h (generated by gen_jtable.py): the
// octave and the top mantissa bits of x select a piece, a subtraction and seven FMAs
// evaluate it (the polynomial is stored in t = x - centre).  This
// replaces the FP64 log and exp of x^4.1811 (the FP64 rate of the GPU is 1/64 of
// FP32) at ~2e-16 relative accuracy.
#pragma once
#include <cuda_runtime.h>
#include "jfit_table.h"

// the fine table (jfine_table.h): pieces of 64 bytes, in one translation unit, handed around
// by pointer
#define KSP_JFINE_E0 (-12)
#define KSP_JFINE_PIECES 6400

namespace ksp {

static __device__ const double g_jfit[KSP_JFIT_PIECES * KSP_JFIT_STRIDE] = KSP_JFIT_TABLE_INIT;

__device__ __forceinline__ double specialJ_fit_tab(double x) {
    // x <= 0 tested on the bit pattern (+0 and the negatives are the non-positive
    // integers; a NaN, whatever its sign, goes on as the FP64 compare would let it), on
    // the integer pipe: an FP64 compare costs a warp the FP64 pipe's full time
    const long long bits = __double_as_longlong(x);
    if (bits <= 0 && (bits & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL) return 1.;
    const int e = (int)((bits >> 52) & 0x7ff) - 1023;
    if (e < KSP_JFIT_E0) {  // x < 2^-20: the x^4.1811 term is below 1e-25 relative
        const double x2 = x * x, x4 = x2 * x2, x8 = x4 * x4;
        return (1. + 0.0168 * x2 + 0.0407 * x4) / (1. + 2.1734 * x2 + 0.1467 * x8);
    }
    if (e >= KSP_JFIT_E1) return specialJ_fit(x);
    const int sub = (int)((bits >> (52 - KSP_JFIT_SUB_BITS)) & ((1 << KSP_JFIT_SUB_BITS) - 1));
    const double* p = g_jfit + (((e - KSP_JFIT_E0) << KSP_JFIT_SUB_BITS) | sub) * KSP_JFIT_STRIDE;
    const double t = x - __ldg(p);
    double v = __ldg(p + 1 + KSP_JFIT_DEG);
#pragma unroll
    for (int j = KSP_JFIT_DEG - 1; j >= 0; j--) v = fma(v, t, __ldg(p + 1 + j));
    return v;
}

// J and dJ/dx together (the adjoint): the derivative of the piece's polynomial, times
// du/dx; outside the table the formula and its derivative.
__device__ __forceinline__ void specialJ_fit_tab_d(double x, double& J, double& Jd) {
    const long long bits = __double_as_longlong(x);
    if (bits <= 0 && (bits & 0x7fffffffffffffffLL) <= 0x7ff0000000000000LL) { J = 1.; Jd = 0.; return; }
    const int e = (int)((bits >> 52) & 0x7ff) - 1023;
    if (e < KSP_JFIT_E0 || e >= KSP_JFIT_E1) {
        const double x2 = x * x, x4 = x2 * x2, x8 = x4 * x4;
        const double p = e < KSP_JFIT_E0 ? 0.0 : exp(4.1811 * log(x));
        const double N = 1. + 0.0168 * x2 + 0.0407 * x4;
        const double D = 1. + 2.1734 * x2 + 1.6787 * p + 0.1467 * x8;
        const double dN = 0.0336 * x + 0.1628 * x2 * x;
        const double dD = 4.3468 * x + 1.6787 * 4.1811 * p / x + 1.1736 * x4 * x2 * x;
        J = N / D;
        Jd = (dN * D - N * dD) / (D * D);
        return;
    }
    const int sub = (int)((bits >> (52 - KSP_JFIT_SUB_BITS)) & ((1 << KSP_JFIT_SUB_BITS) - 1));
    const double* p = g_jfit + (((e - KSP_JFIT_E0) << KSP_JFIT_SUB_BITS) | sub) * KSP_JFIT_STRIDE;
    const double t = x - __ldg(p);
    double v = __ldg(p + 1 + KSP_JFIT_DEG), dv = 0.0;
#pragma unroll
    for (int j = KSP_JFIT_DEG - 1; j >= 0; j--) {
        dv = fma(dv, t, v);
        v = fma(v, t, __ldg(p + 1 + j));
    }
    J = v;
    Jd = dv;
}

// J at the node of a bin's integral, x = fslength k / (m / kT): the piece from x in single
// precision (a piece's polynomial holds a rounding beyond its ends too), its variable
// x - centre in one multiply-add, five more for the polynomial.  Arguments below 2^-12 or from
// 2^13 on go to the first table and the formula.
__device__ __forceinline__ double specialJ_node(const double* jt, double fsl, float fslf, double kom, float komf) {
    const int idx = (int)(__float_as_uint(fslf * komf) >> 15) - ((127 + KSP_JFINE_E0) << 8);
    if ((unsigned)idx >= KSP_JFINE_PIECES) return specialJ_fit_tab(fsl * kom);
    const double2* p = reinterpret_cast<const double2*>(jt) + 4 * idx;
    const double2 p0 = __ldg(p), p1 = __ldg(p + 1), p2 = __ldg(p + 2), p3 = __ldg(p + 3);
    const double t = fma(fsl, kom, -p0.x);
    return fma(t, fma(t, fma(t, fma(t, fma(t, p3.x, p2.y), p2.x), p1.y), p1.x), p0.y);
}

// ------------------------------------------------------------------ J with a momentum cut
// Hybrid neutrinos: J is the series specialJ_sums.  Its sums A and B are smooth in x (nearest
// poles +-i), so a call tabulates them per species over x in [2^-12, 2^13), 64 pieces an
// octave, degree 6 (the interpolant's error 2e-17): 11200 evaluations of the series instead of
// one per node, and a node costs a sine, a cosine and 12 multiply-adds.  (151 bins x 100
// rows: the integrals took 3074 us term by term, 1134 with the series' sine and cosine taken
// once.)  Piece: centre, 7 coefficients of A / x, 7 of B, both over 1.5 zeta(3) (1 - nufrac_low).
constexpr int kHybE0 = -12, kHybSubBits = 6, kHybPieces = 25 << kHybSubBits, kHybStride = 16;
constexpr int kHybTable = kHybPieces * kHybStride;

// Not inlined: rare, and its sine and cosine would cost the fit's path registers.
static __device__ __noinline__ double specialJ_cut(const double* hyb, double x, double qc, double nfl) {
    const long long bits = __double_as_longlong(x);
    const int idx = (int)(bits >> (52 - kHybSubBits)) - ((1023 + kHybE0) << kHybSubBits);
    if (!hyb || bits < 0 || (unsigned)idx >= kHybPieces) return specialJ_series(x, qc, nfl);
    const double* p = hyb + (size_t)idx * kHybStride;
    const double t = x - p[0];
    double A = p[7], B = p[14];
#pragma unroll
    for (int j = 5; j >= 0; j--) {
        A = fma(A, t, p[1 + j]);
        B = fma(B, t, p[8 + j]);
    }
    double sn, cs;
    sincos(qc * x, &sn, &cs);
    return A * sn + B * cs;
}

// Pieces blk * 8 .. + 7 of the table of one species, by 64 threads: eight per piece, seven of
// them a Chebyshev node each, then a coefficient each.
__device__ __forceinline__ void hyb_table_block(double* hyb, int blk, double qc, double nfl) {
    // interpolation at cos(pi (k + 1/2) / 7), the values' differences from the centre's, folded
    // about it: even coefficients of the sums, odd ones of the differences
    static constexpr double kM[7][3] = {
        {0.0, 0.0, 0.0},
        {0.22824347439014993808, -0.79747338888240396142, 2.0765213965723365672},
        {0.23411318061389408156, -1.0200067492357776374, 4.7858935686218835559},
        {-1.5858139578511551928, 5.0751495106189256167, -5.5818117994536830292},
        {-1.6265961185809209033, 6.4913598702856732729, -12.86476375170475237},
        {1.9834685216802656936, -4.4568133128311936321, 3.574086776996707697},
        {2.0344771104577316964, -5.7004781884227065648, 8.237429649393546297}};
    const int t = threadIdx.x, k = t & 7;
    const int piece = min(blk * 8 + (t >> 3), kHybPieces - 1);
    const double lo = ldexp(1.0, kHybE0 + (piece >> kHybSubBits));
    const double h = lo * (0.5 / (1 << kHybSubBits));
    const double c = lo * (1.0 + (piece & ((1 << kHybSubBits) - 1)) * (1.0 / (1 << kHybSubBits))) + h;
    const double x = c + h * (k < 7 ? cospi((k + 0.5) / 7.0) : 0.0);
    double A, B;
    specialJ_sums(x * x, qc, exp(-qc), &A, &B);
    const double norm = 1.0 / (1.5 * kZeta3 * (1 - nfl));
    A *= norm / x;
    B *= norm;
    const unsigned all = 0xffffffffu;
    const double A3 = __shfl_sync(all, A, 3, 8), B3 = __shfl_sync(all, B, 3, 8);
    const double sgn = (k & 1) ? -1.0 : 1.0;
    double ca = 0.0, cb = 0.0;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const double a0 = __shfl_sync(all, A, q, 8) - A3, a1 = __shfl_sync(all, A, 6 - q, 8) - A3;
        const double b0 = __shfl_sync(all, B, q, 8) - B3, b1 = __shfl_sync(all, B, 6 - q, 8) - B3;
        double m = 0.0;
#pragma unroll
        for (int j = 0; j < 7; j++)
            if (j == k) m = kM[j][q];
        ca = fma(m, fma(sgn, a1, a0), ca);
        cb = fma(m, fma(sgn, b1, b0), cb);
    }
    double* p = hyb + (size_t)piece * kHybStride;
    if (k == 7) {
        p[0] = c;
        return;
    }
    const double ih = ldexp(1.0, k * (kHybSubBits + 1 - (kHybE0 + (piece >> kHybSubBits))));  // h^-k
    p[1 + k] = k == 0 ? A3 : ca * ih;
    p[8 + k] = k == 0 ? B3 : cb * ih;
}

}  // namespace ksp
