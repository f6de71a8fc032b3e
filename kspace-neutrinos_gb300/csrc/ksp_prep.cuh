// ksp_prep.cuh -- the preparation of an integrator call that does not depend on the
// current delta_cdm: the knots' spline factorisation, the fslength table and the node
// table, as device functions of one block (single calls and batches launch them over
// their own block maps).
//
// The fslength table (delta_tot_table.c:574-591) has N = 16 Na uniform nodes x_i in
// log a; fslength(x_i) = light * sum_{v >= i} s_v with s_v the integral of 1/(a^2 H) over
// segment v, and its natural spline's coefficients follow from the s_v in closed form.
// Two kernels make it: the first evaluates the segments, a block per stretch of them,
// with their suffix sums within the stretch and the stretch's total; the second adds the
// totals of the later stretches and forms the coefficients.  Nothing in it is serial in
// N, and no block is larger than 64 threads (128 in the second kernel) at a register cap of eight
// such blocks to an SM, so that the blocks find room beside the binning pass, which holds most
// of every SM.
#pragma once
#include "ksp_internal.h"

namespace ksp {

constexpr int kPrepThreads = 64;

// ------------------------------------------------------------------ segments
// The rule by the node spacing h: the 4-point Gauss-Legendre rule per segment from 5e-3 on,
// the 2-point rule below (fslength then within 1e-12, as the 4-point rule's: both are held up
// by the jump of the rho_nu tables where they give way to the series), and below 1.5e-3 one
// evaluation per node, a segment being the integral of the degree-7 interpolant through 8
// neighbouring nodes (7e-13; at wider spacings the kinks of the rho_nu tables, a knot every
// ~0.016, spread over its 8 segments: 2e-10 at h = 0.019).  An evaluation is an exp, a
// reciprocal square root and the rho_nu tables, ~60 FP64 operations (fsl_integrand).
constexpr double kFsNodeRule = 1.5e-3, kFsGauss2 = 5e-3;
constexpr int kFsNodeSegs = kPrepThreads - 7;  // segments of a block by the node rule
__host__ __device__ inline int fs_block_segs(double h) {
    return h < kFsNodeRule ? kFsNodeSegs : (h < kFsGauss2 ? kPrepThreads / 2 : kPrepThreads / 4);
}
// blocks of a table (segments 0 .. n - 2, and a last one of zero)
__host__ __device__ inline int fs_blocks(const FsGrid& g) {
    const int per = fs_block_segs(g.h);
    return (g.n + per - 1) / per;
}
// nodes per block of the second kernel: two a thread
constexpr int fs_table_blocks(int n, int threads) { return (n + 2 * threads - 1) / (2 * threads); }

#ifdef __CUDACC__
// integrals over [o, o + 1], o = 0..3, of the Lagrange basis on the nodes 0..7, x 120960
// (o = 4..6: mirrored)
static __constant__ double kNodeRule[4][8] = {
    {36799, 139849, -121797, 123133, -88547, 41499, -11351, 1375},
    {-1375, 47799, 101349, -44797, 26883, -11547, 2999, -351},
    {351, -4183, 57627, 81693, -20227, 7227, -1719, 191},
    {-191, 1879, -9531, 68323, 68323, -9531, 1879, -191}};

__device__ __noinline__ static double fsl_integrand_call(const Background& B, double x) { return fsl_integrand(B, x); }

// Block `blk` of the segments, by 64 threads: fs_seg[v] = s_v, fs_suf[v] = the sum of the
// block's s from v on, fs_tot[blk] = the block's.  f: 64 doubles of shared memory, sg: 64.
__device__ __forceinline__ void fs_eval_block(const Background& B, const FsGrid& g, double loga, int blk,
                                              double gx0, double gx1, double gw0, double gw1, double* f, double* sg,
                                              double* fs_seg, double* fs_suf, double* fs_tot) {
    const int t = threadIdx.x, Nfs = g.n;
    const double h = g.h;
    int per, v;
    double s = 0;
    if (h < kFsNodeRule) {
        per = kFsNodeSegs;
        const int first = blk * per;
        // nodes base .. base + 63, as many of the table as reach around the block's segments
        int base = first - 3;
        base = base > Nfs - kPrepThreads ? Nfs - kPrepThreads : base;
        base = base < 0 ? 0 : base;
        f[t] = base + t < Nfs ? fsl_integrand_call(B, g.node(base + t)) : 0.0;
        __syncthreads();
        v = first + t;
        if (t < per && v < Nfs - 1) {
            int st = v - 3;
            st = st > Nfs - 8 ? Nfs - 8 : st;
            st = st < 0 ? 0 : st;
            const int o = v - st;
            const double* w = kNodeRule[o < 4 ? o : 6 - o];
            const double* q = f + (st - base);
            double acc = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) acc += w[o < 4 ? k : 7 - k] * q[k];
            s = acc * (h / 120960.);
        }
    } else {
        // a segment per pair or per four threads
        const bool two = h < kFsGauss2;
        const int w = two ? 2 : 4;
        per = kPrepThreads / w;
        const int u = blk * per + t / w, q = t % w;
        double x = 0;
        if (u < Nfs - 1) {
            const double xa = g.node(u), xb = u + 1 == Nfs - 1 ? loga : g.node(u + 1);
            const double c = 0.5 * (xa + xb), hh = 0.5 * (xb - xa);
            const double gx = two ? 0.57735026918962576451 : ((q & 1) ? gx1 : gx0);  // 1 / sqrt 3
            const double gw = two ? 1.0 : ((q & 1) ? gw1 : gw0);
            x = gw * hh * fsl_integrand_call(B, 2 * q < w ? c - hh * gx : c + hh * gx);
        }
        x += __shfl_down_sync(0xffffffffu, x, 1, 4);
        if (!two) x += __shfl_down_sync(0xffffffffu, x, 2, 4);
        if (q == 0) f[t / w] = x;
        __syncthreads();
        v = blk * per + t;
        if (t < per) s = f[t];
    }
    sg[t] = t < per ? s : 0.0;
    __syncthreads();
    // suffix sums: each thread of the first warp two neighbours
    if (t < 32) {
        const double b1 = sg[2 * t + 1], b0 = sg[2 * t];
        const double own = b0 + b1;
        double r = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double n = __shfl_down_sync(0xffffffffu, r, o);
            if (t + o < 32) r += n;
        }
        double later = __shfl_down_sync(0xffffffffu, r, 1);
        if (t == 31) later = 0;
        f[2 * t + 1] = b1 + later;
        f[2 * t] = r;
        if (t == 0) fs_tot[blk] = r;
    }
    __syncthreads();
    if (t < per && v < Nfs) {
        fs_seg[v] = s;
        fs_suf[v] = f[t];
    }
}

// ------------------------------------------------------------------ table
// The totals of the stretches from the one of thread t on: suf[t] = the totals of the blocks
// t c, t c + 1, ... (c: blocks per thread), t <= 64.  suf: 65 doubles of shared memory.
__device__ __forceinline__ void fs_totals_suffix(const double* fs_tot, int nblk, double* suf) {
    const int t = threadIdx.x, c = (nblk + kPrepThreads - 1) / kPrepThreads;
    double own = 0;
    for (int b = min(nblk, (t + 1) * c) - 1; b >= t * c; b--) own += fs_tot[b];
    double r = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double n = __shfl_down_sync(0xffffffffu, r, o);
        if ((t & 31) + o < 32) r += n;
    }
    if (t >= 32) suf[t] = r;
    __syncthreads();
    if (t < 32) suf[t] = r + suf[32];
    if (t == 0) suf[kPrepThreads] = 0;
    __syncthreads();
}

struct FsTable {  // what the second kernel reads
    const double* seg;
    const double* suf;
    const double* tot;
    const double* tsuf;  // fs_totals_suffix
    FsGrid g;
    int nblk, per;
    double light;
    double cscale;       // light * 3 / h^2 / (2 sqrt 3)
};

// fslength at node i: its stretch's suffix sum and the later stretches' totals
__device__ __forceinline__ double fs_table_y(const FsTable& F, int i) {
    const int b = i / F.per, c = (F.nblk + kPrepThreads - 1) / kPrepThreads, t = b / c;
    double later = F.tsuf[t + 1];
    for (int q = min(F.nblk, (t + 1) * c) - 1; q > b; q--) later += F.tot[q];
    return F.light * (F.suf[i] + later);
}

// Spline coefficient (second derivative / 2) at node i of 0 .. Nfs-1.  The system is
// tridiag(1,4,1) c = 3 D^2 y / h^2, D^2 y_v = light (s_{v-1} - s_v) (fslength falls by light s_v
// from node v to v + 1), whose inverse on the whole line is nu^|d| / (2 sqrt 3),
// nu = sqrt 3 - 2; the ends c = 0 are met by continuing the right-hand side oddly about them,
// that is, the s evenly: s_{-1-k} = s_k, s_{n+k} = s_{n-1-k}, n = Nfs - 1.  The sums over the
// neighbours are taken over the s themselves (summation by parts: one multiply-add per
// term), D to a side: 20 where h < 0.02 (nu^20 = 4e-12 of a term below 4e-4 of fslength), 28
// elsewhere (n >= 15: the second end's continuation may reach back past the first).
//
// The two sums at a node follow from those of its neighbour by one multiply-add each, so a pair
// of nodes i, i + 1 takes the left sum of the first and the right sum of the second: c[0], c[1].
__device__ __forceinline__ double fs_table_s(const FsTable& F, int i) {
    const int n = F.g.n - 1;
    i = i < 0 ? -1 - i : i;
    i = i >= n ? 2 * n - 1 - i : i;
    i = i < 0 ? -1 - i : i;
    return F.seg[i];
}
__device__ __forceinline__ void fs_table_c2(const FsTable& F, int i, double* c) {
    const double nu = -0.26794919243112270647, k = 0.78867513459481288225;  // 1 / (1 - nu)
    double l, r;  // left sum of node i, right sum of node i + 1
    if (F.g.h < 0.02) {
        constexpr int D = 20;
        l = fs_table_s(F, i - D - 1) * k;
        r = fs_table_s(F, i + 1 + D) * k;
#pragma unroll
        for (int d = D; d >= 2; d--) {
            l = fma(nu, l, fs_table_s(F, i - d));
            r = fma(nu, r, fs_table_s(F, i + d));
        }
    } else {
        constexpr int D = 28;
        l = fs_table_s(F, i - D - 1) * k;
        r = fs_table_s(F, i + 1 + D) * k;
        for (int d = D; d >= 2; d--) {
            l = fma(nu, l, fs_table_s(F, i - d));
            r = fma(nu, r, fs_table_s(F, i + d));
        }
    }
    const double sm = fs_table_s(F, i - 1), s0 = fs_table_s(F, i), s1 = fs_table_s(F, i + 1);
    const double r0 = fma(nu, r, s1), l1 = fma(nu, l, sm);
    // the two sides' sums of nu^(d-1) D^2 y
    const double q0 = fma(1.0 - nu, l - r0, s0 - sm), q1 = fma(1.0 - nu, l1 - r, s1 - s0);
    c[0] = i == 0 ? 0.0 : F.cscale * fma(nu, q0, sm - s0);
    c[1] = i + 1 >= F.g.n - 1 ? 0.0 : F.cscale * fma(nu, q1, s0 - s1);
}

// The table of a call as the second kernel's blocks read it.  Called by a whole block of at
// least kPrepThreads threads; tsuf: kPrepThreads + 1 doubles of shared memory.
__device__ __forceinline__ FsTable fs_table(const IntegratorDev& I, const FsGrid& g, double light, double* tsuf) {
    FsTable F;
    F.seg = I.fs_seg;
    F.suf = I.fs_suf;
    F.tot = I.fs_tot;
    F.tsuf = tsuf;
    F.g = g;
    F.nblk = fs_blocks(g);
    F.per = fs_block_segs(g.h);
    F.light = light;
    F.cscale = light * (g.ih * g.ih) * 0.86602540378443864676;
    if (threadIdx.x < kPrepThreads) {
        fs_totals_suffix(I.fs_tot, F.nblk, tsuf);
    } else {
        __syncthreads();
        __syncthreads();
    }
    return F;
}

// Nodes i = 2 u, i + 1 of the table to memory; the first also to the call's scalars.
__device__ __forceinline__ void fs_table_store(const IntegratorDev& I, const FsTable& F, int u) {
    const int i = 2 * u;
    if (i >= F.g.n) return;
    double c[2];
    fs_table_c2(F, i, c);
    const double y = fs_table_y(F, i);
    I.fs_y[i] = y;
    I.fs_c[i] = c[0];
    if (i + 1 < F.g.n) {
        I.fs_y[i + 1] = i + 1 == F.g.n - 1 ? 0.0 : fs_table_y(F, i + 1);
        I.fs_c[i + 1] = c[1];
    }
    if (i == 0) {
        I.sc->fsl_A0a = y;
        I.sc->Nfs = F.g.n;
        I.sc->fs_h = F.g.h;
        I.sc->fs_ih = F.g.ih;
    }
}

// fslength at x, from the spline of the table (which falls by light s_i from node i to i + 1)
__device__ __forceinline__ double fs_table_at(const FsTable& F, double x) {
    const int i = F.g.segment(x);
    double c[2];
    fs_table_c2(F, i, c);
    return fs_spline_eval(F.g, fs_table_y(F, i), -F.light * F.seg[i], c[0], c[1], x - F.g.node(i));
}

// ------------------------------------------------------------------ knots
// Rows i0 .. i1 - 1 of the factorised natural-spline system of the knots x[0..Na-1]: the pivot
// d_i = b_i - h_i^2 / d_{i-1}, b_i = 2 (h_i + h_{i+1}), h_i = x_{i+1} - x_i, as a quotient
// of two-term recurrences p / q carried from 28 rows before i0 (an error in a pivot shrinks
// by 4 or more per row, so the start does not show), with two divisions per row at its end.
// knot(j): knot j.
template <class X>
__device__ __forceinline__ void knot_rows(const X& knot, int i0, int i1, double* invdiag, double* fac) {
    int r = i0 > 28 ? i0 - 28 : 0;
    double x1 = knot(r + 1), x2 = knot(r + 2);
    double h0 = x1 - knot(r), h1 = x2 - x1;
    double p = 2.0 * (h0 + h1), q = 1.0, pp = 0, qp = 0;
    for (;;) {
        if (r >= i0) {
            invdiag[r] = q / p;
            if (r > 0) fac[r] = h0 * (qp / pp);
        }
        if (++r >= i1) return;
        pp = p;
        qp = q;
        x1 = x2;
        x2 = knot(r + 2);
        h0 = h1;
        h1 = x2 - x1;
        p = 2.0 * (h0 + h1) * pp - h0 * h0 * qp;
        q = pp;
        if ((r & 7) == 0) {  // both back to their first size
            p /= q;
            q = 1.0;
        }
    }
}
template <class X>
__device__ __forceinline__ void knot_row(const X& knot, int i, double* invdiag, double* fac) {
    knot_rows(knot, i, i + 1, invdiag, fac);
}

// ------------------------------------------------------------------ nodes
// Node q = 61 slot + jn of the node table: its log a, and the half-width of its interval.
__device__ __forceinline__ double nc_node_x(int q, NcLayout lay, double loga0, double loga, double* half) {
    const int slot = q / 61, jn = q - 61 * slot;
    double lo, hi;
    nc_interval(slot, lay, loga0, loga, &lo, &hi);
    const double c = __dmul_rn(0.5, __dadd_rn(lo, hi));
    const double h = __dmul_rn(0.5, __dsub_rn(hi, lo));
    *half = h;
    return __dadd_rn(c, __dmul_rn(h, gk61_x(jn)));
}

// The same solve as spline_solve_scan with all T threads of a block (T a multiple of 32):
// warp scans of the affine maps, combined over the warps through sh (2 * T / 32 doubles of
// shared memory).  x, fac, invdiag: the knots and their factorised system (knot_row).
template <int T>
__device__ __forceinline__ void spline_solve_block(const double* x, const double* fac, const double* invdiag, int m,
                                                   double* sc, double* sh) {
    constexpr int NW = T / 32;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int per = (m + T - 1) / T;
    const int u0 = min(m, t * per), u1 = min(m, u0 + per);
    // forward: z_u = r_u - fac_u z_{u-1} (fac_0 = 0)
    double A = 1.0, B = 0.0;
    for (int u = u0; u < u1; u++) {
        const double f = u > 0 ? fac[u] : 0.0;
        B = sc[u + 1] - f * B;
        A = -f * A;
    }
    double pa = A, pb = B;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double qa = __shfl_up_sync(0xffffffffu, pa, d), qb = __shfl_up_sync(0xffffffffu, pb, d);
        if (lane >= d) {
            pb = pa * qb + pb;
            pa = pa * qa;
        }
    }
    if (lane == 31) {
        sh[2 * warp] = pa;
        sh[2 * warp + 1] = pb;
    }
    __syncthreads();
    double win = 0.0;  // z entering this warp's stretch
    for (int w = 0; w < warp; w++) win = sh[2 * w] * win + sh[2 * w + 1];
    double ea = __shfl_up_sync(0xffffffffu, pa, 1), eb = __shfl_up_sync(0xffffffffu, pb, 1);
    double zin = lane == 0 ? win : ea * win + eb;
    for (int u = u0; u < u1; u++) {
        const double f = u > 0 ? fac[u] : 0.0;
        zin = sc[u + 1] - f * zin;
        sc[u + 1] = zin;
    }
    __syncthreads();
    // backward: c_u = (z_u - off_u c_{u+1}) * invdiag_u, c_m = 0
    A = 1.0;
    B = 0.0;
    for (int u = u1 - 1; u >= u0; u--) {
        const double off = u < m - 1 ? x[u + 2] - x[u + 1] : 0.0;
        const double iv = invdiag[u];
        B = (sc[u + 1] - off * B) * iv;
        A = -off * iv * A;
    }
    pa = A;
    pb = B;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double qa = __shfl_down_sync(0xffffffffu, pa, d), qb = __shfl_down_sync(0xffffffffu, pb, d);
        if (lane + d < 32) {
            pb = pa * qb + pb;
            pa = pa * qa;
        }
    }
    if (lane == 0) {
        sh[2 * warp] = pa;
        sh[2 * warp + 1] = pb;
    }
    __syncthreads();
    win = 0.0;
    for (int w = NW - 1; w > warp; w--) win = sh[2 * w] * win + sh[2 * w + 1];
    ea = __shfl_down_sync(0xffffffffu, pa, 1);
    eb = __shfl_down_sync(0xffffffffu, pb, 1);
    double cin = lane == 31 ? win : ea * win + eb;
    for (int u = u1 - 1; u >= u0; u--) {
        const double off = u < m - 1 ? x[u + 2] - x[u + 1] : 0.0;
        cin = (sc[u + 1] - off * cin) * invdiag[u];
        sc[u + 1] = cin;
    }
    __syncthreads();
}

// Natural cubic spline of y on the knots x (n >= 3) by a block of T threads: c = S''/2 at the
// knots.  fac, invdiag: n doubles of scratch each; sh as spline_solve_block's.
template <int T>
__device__ __forceinline__ void natural_spline_block(const double* x, const double* y, int n, double* c, double* fac,
                                                     double* invdiag, double* sh) {
    const int t = threadIdx.x;
    auto knot = [&](int j) { return x[j]; };
    // a thread's rows side by side: one run-up for them (a row at a time, strided, 300 knots are 10
    // run-ups of 28 steps on one FP64 pipe)
    const int per = (n - 2 + T - 1) / T, u0 = t * per, u1 = min(u0 + per, n - 2);
    if (u0 < u1) knot_rows(knot, u0, u1, invdiag, fac);
    for (int u = t; u < n - 2; u += T) {
        c[u + 1] = 3.0 * ((y[u + 2] - y[u + 1]) / (x[u + 2] - x[u + 1]) - (y[u + 1] - y[u]) / (x[u + 1] - x[u]));
    }
    __syncthreads();
    spline_solve_block<T>(x, fac, invdiag, n - 2, c, sh);
    if (t == 0) {
        c[0] = 0.0;
        c[n - 1] = 0.0;
    }
    __syncthreads();
}
#endif  // __CUDACC__

}  // namespace ksp
