// ksp_integrator.cu -- the linear-response neutrino integrator on the GPU.
//
//   k_rho_points / k_rho_splines  Omega_nu(a) tables (omega_nu_single.c:117-153)
//   k_nufrac_low                hybrid-neutrino fractions (omega_nu_single.c:214-240)
//   k_update_row                update_delta_tot (delta_tot_table.c:177-191)
//   k_delta_tot_init            delta_tot_init's per-bin part (delta_tot_table.c:94-129)
//   k_prep_eval, k_prep_tables  a call's preparation in two kernels (ksp_prep.cuh): the
//                               scalars, the factorised knot spline system, the fslength
//                               table (delta_tot_table.c:574-591: sums of fixed-order
//                               segment integrals over the 16*Na uniform nodes replace 16*Na
//                               adaptive integrals), the integrand's bin-independent terms on
//                               QAG's right spine (hybrid neutrinos: on all shallow intervals),
//                               the natural spline of every history row
//   k_row_update                a prepared step's provisional row, with the binning pass's
//                               normalisation
//   k_dnu_qag                   one warp per (species, bin): history row staged into
//                               shared memory by a TMA bulk copy, then QAG/GK61 of the
//                               delta_nu time integral (delta_tot_table.c:492-500,592-599)
//   k_dnu_qag_blk               the same with a block per task (few tasks), bisection levels
//                               or intervals evaluated ahead
//   k_combine / k_finish        species sum, row commit, NaN check, clamp, ratio table
#include <cuda_runtime.h>
#include <stdio.h>
#include "ksp_internal.h"
#include "ksp_prep.cuh"
#include "jfine_table.h"
#include "ksp_ptx.cuh"

namespace ksp {

static __device__ const __align__(16) double g_jfine[KSP_JFINE_PIECES * KSP_JFINE_STRIDE] = KSP_JFINE_TABLE_INIT;
static_assert(KSP_JFINE_SUB_BITS == 8 && KSP_JFINE_DEG == 5 && KSP_JFINE_STRIDE == 8, "specialJ_node");
const double* jfine_table() {
    void* p = nullptr;
    return cudaGetSymbolAddress(&p, g_jfine) == cudaSuccess ? static_cast<const double*>(p) : nullptr;
}

// ------------------------------------------------------------------ background tables
struct RhoIntegrand {  // omega_nu_single.c:89-96
    double amnu, kT;
    __device__ double operator()(double q) const {
        const double epsilon = sqrt(q * q + amnu * amnu);
        const double f0 = 1. / (exp(q / kT) + 1);
        return q * q * epsilon * f0;
    }
};

// one warp per (species, table point): rhonu[i] = qag(...)/a^4 * conversion
__global__ void k_rho_points(Background* B, unsigned* status) {
    __shared__ Gk61Nodes N;
    extern __shared__ unsigned char smraw[];
    QagList* lists = reinterpret_cast<QagList*>(smraw);
    gk61_fill(N, threadIdx.x, blockDim.x);
    __syncthreads();
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int task = blockIdx.x * nw + warp;
    const int s = task / kNRhoTab, i = task % kNRhoTab;
    if (s >= kNuSpecies) return;
    RhoTable& T = B->tab[s];
    if (!B->deg[s] || !T.has_table) return;
    RhoIntegrand f{T.mnu * exp(T.loga[i]), B->kBtnu};
    QagResult r = qag_warp(f, N, lists[warp], 0.0, 500 * B->kBtnu, 0.0, 1e-9, kQagLimit);
    if ((threadIdx.x & 31) == 0) {
        const double ea = exp(T.loga[i]);
        T.rhonu[i] = r.result / (ea * ea * ea * ea) * B->conv;
        if (!r.ok) atomicOr(status, kStGsl);
    }
}

// a block per species: the table's natural spline and its segments' polynomials (one thread per
// species swept the system in 574 us)
constexpr int kSplineThreads = 128;
__global__ void __launch_bounds__(kSplineThreads) k_rho_splines(Background* B) {
    __shared__ double fac[kNRhoTab], inv[kNRhoTab], sh[2 * kSplineThreads / 32];
    RhoTable& T = B->tab[blockIdx.x];
    if (threadIdx.x == 0) T.imnu = 1.0 / T.mnu;
    if (!B->deg[blockIdx.x] || !T.has_table) return;
    natural_spline_block<kSplineThreads>(T.loga, T.rhonu, kNRhoTab, T.c, fac, inv, sh);
    // the node-independent terms of cspline_seg, per segment
    for (int i = threadIdx.x; i + 1 < kNRhoTab; i += kSplineThreads) {
        const double h = T.loga[i + 1] - T.loga[i];
        T.sb[i] = (T.rhonu[i + 1] - T.rhonu[i]) / h - h * (T.c[i + 1] + 2.0 * T.c[i]) / 3.0;
        T.sd[i] = (T.c[i + 1] - T.c[i]) / (3.0 * h);
    }
    if (threadIdx.x == 0) T.inv_dx = (kNRhoTab - 1) / (T.loga[kNRhoTab - 1] - T.loga[0]);
}

void launch_background_tables(Background* dB, double a0, cudaStream_t st, unsigned* status) {
    (void)a0;
    // a warp per block: the 200 integrals of one mass state spread over the SMs' FP64 pipes (four
    // warps per block used 50 of 152 SMs: 52 us, 47 so)
    const int warps = 1;
    const int tasks = kNuSpecies * kNRhoTab;
    k_rho_points<<<(tasks + warps - 1) / warps, 32 * warps, warps * sizeof(QagList), st>>>(dB, status);
    k_rho_splines<<<kNuSpecies, kSplineThreads, 0, st>>>(dB);
}

// Natural cubic spline of log H on n uniform knots (spacing h), as per-segment
// polynomial coefficients (y_i, b_i, c_i, d_i): one thread (a one-time set-up).
__global__ void k_hubble_table(const double* H, int n, double h, double* coef, double* m) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    // second derivatives: m[i-1] + 4 m[i] + m[i+1] = 6 (y[i+1] - 2 y[i] + y[i-1]) / h^2,
    // m[0] = m[n-1] = 0 (Thomas algorithm; coef[4i+1] holds the modified diagonal ratio)
    double* cp = coef;  // scratch for the forward sweep, overwritten below
    m[0] = 0;
    m[n - 1] = 0;
    double prev_c = 0, prev_d = 0;
    for (int i = 1; i < n - 1; i++) {
        const double r = 6.0 * (log(H[i + 1]) - 2.0 * log(H[i]) + log(H[i - 1])) / (h * h);
        const double den = 4.0 - prev_c;
        const double ci = 1.0 / den;
        const double di = (r - prev_d) / den;
        cp[4 * i] = ci;
        cp[4 * i + 1] = di;
        prev_c = ci;
        prev_d = di;
    }
    for (int i = n - 2; i >= 1; i--) m[i] = cp[4 * i + 1] - cp[4 * i] * m[i + 1];
    for (int i = 0; i < n - 1; i++) {
        const double y0 = log(H[i]), y1 = log(H[i + 1]);
        coef[4 * i] = y0;
        coef[4 * i + 1] = (y1 - y0) / h - h * (2.0 * m[i] + m[i + 1]) / 6.0;
        coef[4 * i + 2] = 0.5 * m[i];
        coef[4 * i + 3] = (m[i + 1] - m[i]) / (6.0 * h);
    }
}
void launch_hubble_table(const double* H, int n, double h, double* coef, double* scratch, cudaStream_t st) {
    k_hubble_table<<<1, 32, 0, st>>>(H, n, h, coef, scratch);
}

// natural spline of one table of n >= 3 knots; scratch: 2 n
__global__ void __launch_bounds__(kSplineThreads) k_spline1(const double* x, const double* y, double* c,
                                                            double* scratch, int n) {
    __shared__ double sh[2 * kSplineThreads / 32];
    natural_spline_block<kSplineThreads>(x, y, n, c, scratch, scratch + n, sh);
}
void launch_spline_coeffs(const double* x, const double* y, double* c, double* scratch, int n, cudaStream_t st) {
    k_spline1<<<1, kSplineThreads, 0, st>>>(x, y, c, scratch, n);
}

struct FermiDirac {  // omega_nu_single.c:207-210
    __device__ double operator()(double x) const { return x * x / (exp(x) + 1); }
};

// omega_nu_single.c:214-228 (qag limit 100) and :230-240
__global__ void k_nufrac_low(Background* B, double light, double vcrit, unsigned* status) {
    __shared__ Gk61Nodes N;
    __shared__ QagList L[kNuSpecies];
    gk61_fill(N, threadIdx.x, blockDim.x);
    __syncthreads();
    const int s = threadIdx.x >> 5;
    if (s >= kNuSpecies) return;
    const double qc = B->mnu[s] * vcrit / light / B->kBtnu;
    QagResult r = qag_warp(FermiDirac{}, N, L[s], 0.0, qc, 0.0, 1e-6, 100);
    if ((threadIdx.x & 31) == 0) {
        B->nufrac_low[s] = r.result / (1.5 * kZeta3);
        if (!r.ok) atomicOr(status, kStGsl);
    }
}
void launch_nufrac_low(Background* dB, double light, double vcrit, cudaStream_t st, unsigned* status) {
    k_nufrac_low<<<1, 32 * kNuSpecies, 0, st>>>(dB, light, vcrit, status);
}

// nufrac_low(qc) of n momenta (omega_nu_single.c:214-228): a warp per value
__global__ void k_nufrac_low_values(const double* qc, int n, double* out, unsigned* status) {
    __shared__ Gk61Nodes N;
    __shared__ QagList L[4];
    gk61_fill(N, threadIdx.x, blockDim.x);
    __syncthreads();
    const int w = threadIdx.x >> 5;
    const int i = blockIdx.x * 4 + w;
    if (i >= n) return;
    QagResult r = qag_warp(FermiDirac{}, N, L[w], 0.0, qc[i], 0.0, 1e-6, 100);
    if ((threadIdx.x & 31) == 0) {
        out[i] = r.result / (1.5 * kZeta3);
        if (!r.ok) atomicOr(status, kStGsl);
    }
}
void launch_nufrac_low_values(const double* qc, int n, double* out, unsigned* status, cudaStream_t st) {
    if (n > 0) k_nufrac_low_values<<<(n + 3) / 4, 128, 0, st>>>(qc, n, out, status);
}

// specialJ of n arguments (the device function the integrator uses)
__global__ void k_special_j(const double* x, int n, double qc, double nfl, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = specialJ(x[i], qc, nfl);
}
void launch_special_j(const double* x, int n, double qc, double nufrac_low, double* out, cudaStream_t st) {
    if (n > 0) k_special_j<<<(n + 127) / 128, 128, 0, st>>>(x, n, qc, nufrac_low, out);
}

// ------------------------------------------------------------------ history rows
// delta_tot_table.c:177-191: row `row` = get_delta_tot(dnu, dcdm) at a
__global__ void k_update_row(IntegratorDev I, int nk, int row, double a, double loga, const double* dcdm,
                             const double* dnu) {
    __shared__ double s3[3];
    const Background& B = *I.B;
    if (threadIdx.x == 0) {
        s3[0] = omega_nu_nopart(B, a) * (a * a * a);
        s3[1] = omega_nu(B, 1);
        s3[2] = particle_nu_fraction(B, a, 0);
        if (blockIdx.x == 0) I.scalefact[row] = loga;
    }
    __syncthreads();
    const double Omeganonu = I.sc->Omeganonu;
    for (int ik = blockIdx.x * blockDim.x + threadIdx.x; ik < nk; ik += gridDim.x * blockDim.x)
        I.dtot[(size_t)ik * I.ld + row] = get_delta_tot(dnu[ik], dcdm[ik], s3[0], Omeganonu, s3[1], s3[2]);
}
void launch_update_row(const IntegratorDev& I, int nk, int row, double a, double loga, const double* dcdm,
                       const double* dnu, cudaStream_t st) {
    k_update_row<<<(nk + 255) / 256, 256, 0, st>>>(I, nk, row, a, loga, dcdm, dnu);
}

// the same row from the call's scalars (after k_prep_eval), delta_nu_last and delta_cdm
__global__ void k_update_row_s(IntegratorDev I, int nk, int row) {
    const StepScalars& S = *I.sc;
    for (int ik = blockIdx.x * blockDim.x + threadIdx.x; ik < nk; ik += gridDim.x * blockDim.x)
        I.dtot[(size_t)ik * I.ld + row] =
            get_delta_tot(I.nu_last[ik], I.dcdm[ik], S.OmegaNua3, S.Omeganonu, S.OmegaNu1, S.partnu);
}
void launch_update_row_scalars(const IntegratorDev& I, int nk, int row, cudaStream_t st) {
    k_update_row_s<<<(nk + 255) / 256, 256, 0, st>>>(I, nk, row);
}

// delta_tot_table.c:94-129: transfer spline, first row (fresh start), delta_nu_init
__global__ void k_delta_tot_init(IntegratorDev I, int nk, const double* wavenum, const double* dcdm, int fresh,
                                 double TimeTransfer) {
    __shared__ double s4[4];
    const Background& B = *I.B;
    if (threadIdx.x == 0) {
        s4[0] = omega_nu_nopart(B, TimeTransfer) * (TimeTransfer * TimeTransfer * TimeTransfer);
        s4[1] = omega_nu(B, 1);
        s4[2] = particle_nu_fraction(B, TimeTransfer, 0);
        s4[3] = I.sc->Omeganonu;
        // k beyond the transfer table (delta_tot_table.c:113-114)
        if (log(wavenum[nk - 1]) > I.t_logk[I.ntrans - 1]) atomicOr(I.status, kStKmax);
    }
    __syncthreads();
    const double OmegaNua3 = s4[0], OmegaNu1 = s4[1], Omeganonu = s4[3];
    const double OmegaMa = Omeganonu + OmegaNua3;
    for (int ik = blockIdx.x * blockDim.x + threadIdx.x; ik < nk; ik += gridDim.x * blockDim.x) {
        const double lk = log(wavenum[ik]);
        double T;
        if (lk < I.t_logk[0] || lk > I.t_logk[I.ntrans - 1]) {
            atomicOr(I.status, kStGsl);  // GSL interpolation domain error -> 2001
            T = 0;
        } else {
            const int i = seg_bsearch(I.t_logk, I.ntrans, lk);
            T = cspline_seg(I.t_logk, I.t_T, I.t_c, i, lk);
        }
        double* row = I.dtot + (size_t)ik * I.ld;
        if (fresh) row[0] = get_delta_tot(dcdm[ik] * T, dcdm[ik], OmegaNua3, Omeganonu, OmegaNu1, s4[2]);
        I.nu_init[ik] = row[0] * OmegaMa / (OmegaMa - OmegaNua3 + T * OmegaNua3) * fabs(T);
        I.wavenum[ik] = wavenum[ik];
    }
}
void launch_delta_tot_init(const IntegratorDev& I, int nk, const double* wavenum, const double* dcdm, int fresh,
                           double TimeTransfer, cudaStream_t st) {
    k_delta_tot_init<<<(nk + 255) / 256, 256, 0, st>>>(I, nk, wavenum, dcdm, fresh, TimeTransfer);
}

// ------------------------------------------------------------------ preparation of a call
// Two kernels instead of the eight (scalars, segments, sums, coefficients, nodes, rows, first
// row, species sum) whose launches and one-thread stretches were 120 of the 163 us of a call
// with 64 bins and 16 rows.  Blocks by role; every role is parallel.
struct GL4 { double x[2], w[2]; };  // positive half of the 4-point Gauss-Legendre rule
struct PrepArgs {
    StepScalars S;                 // the call's scalars
    double loga, loga0;
    FsGrid fs;                     // its n, nodes: 0 without a table
    int Na, nodes;
    int start_row, write_knot;
    int knot_blocks, fs_blocks, node_blocks, hyb_blocks;  // hyb_blocks: per species
    int in_blocks;
    CallInput in;
};

// Block 0: the call's scalars to the device.  Then the knots' spacings and factorised spline system
// x = scalefact[0..Na-1] (shared by every row; rows below `start_row` were factorised by an
// earlier call with the same leading knots and are kept), the fslength segments, J's tables
// where hybrid neutrinos cut it, and the part of the node table that needs no fslength.
__global__ void __launch_bounds__(kPrepThreads, 8) k_prep_eval(IntegratorDev I, PrepArgs P, GL4 gl) {
    __shared__ double f[kPrepThreads], sg[kPrepThreads];
    ptx::dep_launch();
    const int t = threadIdx.x, Na = P.Na;
    int b = blockIdx.x;
    if (b == 0) {
        if (t == 0) {
            *I.sc = P.S;
            *I.qag_max = 0;  // this call's QAG statistics start from zero
            *I.qag_total = 0;
            if (P.write_knot) I.scalefact[Na - 1] = P.loga;  // the provisional knot
            if (Na > 1 && no_number(P.loga)) atomicOr(I.status, kStGsl);  // as QAG would end
        }
        return;
    }
    b--;
    if (b < P.in_blocks) {  // the call's inputs, across the host's link
        const int i = b * kPrepThreads + t;
        if (i < P.in.n) P.in.k[i] = P.in.src[i];
        else if (i < 2 * P.in.n) P.in.dcdm[i - P.in.n] = P.in.src[i];
        return;
    }
    b -= P.in_blocks;
    if (b < P.knot_blocks) {
        const double* x = I.scalefact;
        auto knot = [&](int j) { return P.write_knot && j == Na - 1 ? P.loga : x[j]; };
        const int i = b * kPrepThreads + t;
        if (i + 1 < Na) {
            const double h = knot(i + 1) - knot(i);
            I.knot_invh[i] = 1.0 / h;
            I.knot_h3[i] = h / 3.0;
            I.knot_ih3[i] = 1.0 / (3.0 * h);
        }
        if (i < Na - 2 && i >= P.start_row) knot_row(knot, i, I.knot_invdiag, I.knot_fac);
        return;
    }
    b -= P.knot_blocks;
    if (b < P.fs_blocks) {
        fs_eval_block(*I.B, P.fs, P.loga, b, gl.x[0], gl.x[1], gl.w[0], gl.w[1], f, sg, I.fs_seg, I.fs_suf,
                      I.fs_tot);
        return;
    }
    b -= P.fs_blocks;
    if (b < kNuSpecies * P.hyb_blocks) {
        const int mi = b / P.hyb_blocks;
        if (P.S.qc[mi] > 0 && I.B->deg[mi] > 0)
            hyb_table_block(I.hyb + (size_t)mi * kHybTable, b - mi * P.hyb_blocks, P.S.qc[mi], I.B->nufrac_low[0]);
        return;
    }
    b -= kNuSpecies * P.hyb_blocks;
    const int q = b * kPrepThreads + t;
    if (q >= P.nodes) return;
    double half;
    I.nc_inv[q] = node_inv_aH(I.B, nc_node_x(q, NcLayout{I.nc_slots, I.nc_tree}, P.loga0, P.loga, &half));
}

// The fslength table, the node table, and the row splines.
//
// Rows (RowsMode): a history row's natural spline is linear in the row, and the
// provisional (last) knot enters the spline system through its last right-hand side only, so
//   c = c_base + (y_new - y_base) c_unit,
// with c_base the coefficients of the row whose last knot is y_base (the knot before it)
// and c_unit those of a unit last knot with all other knots zero.  Both depend only on
// the committed rows and the knots: kRowsBase solves them beside the binning pass
// (row nk: c_unit).  After it, k_row_update forms y_new (update_delta_tot,
// delta_tot_table.c:177-191) from this step's delta_cdm and adds the correction, in
// place of the solve.  y_new - y_base is one step's growth of delta_tot, so the sum does
// not cancel.  The solves work in place in the coefficient rows (global memory,
// L1-cached): the binning pass holds nearly all of every SM's shared memory.
constexpr int kTableThreads = 128;
__global__ void __launch_bounds__(kTableThreads, 8)
    k_prep_tables(IntegratorDev I, PrepArgs P, int rows, int nk, int update_row, FinalizeArgs fin) {
    __shared__ double tsuf[kPrepThreads + 1], sh[2 * kTableThreads / 32];
    ptx::dep_wait();
    ptx::dep_launch();
    const int t = threadIdx.x, Na = P.Na;
    int b = blockIdx.x;
    const int nrow = rows == kRowsBase ? nk + 1 : (rows == kRowsFull ? nk : 0);
    if (b < nrow) {
        if (fin.active && b < nk && t == kTableThreads - 1) finalize_keff(fin, b);
        const int m = Na - 2;  // unknowns c[1..m]
        const double* ih = I.knot_invh;
        double* c;
        if (b == nk) {
            c = I.coef_unit;
            for (int u = t; u < m; u += kTableThreads) c[u + 1] = u == m - 1 ? 3.0 * ih[m] : 0.0;
        } else {
            double* y = I.dtot + (size_t)b * I.ld;
            c = I.coef + (size_t)b * I.ld;
            if (update_row >= 0) {
                if (t == 0) {
                    const StepScalars& S = *I.sc;
                    y[update_row] =
                        get_delta_tot(I.nu_last[b], I.dcdm[b], S.OmegaNua3, S.Omeganonu, S.OmegaNu1, S.partnu);
                }
                __syncthreads();
            }
            for (int u = t; u < m; u += kTableThreads) {
                // (base: the last knot taken equal to the one before)
                const double y2 = rows == kRowsBase && u == m - 1 ? y[m] : y[u + 2];
                c[u + 1] = 3.0 * ((y2 - y[u + 1]) * ih[u + 1] - (y[u + 1] - y[u]) * ih[u]);
            }
        }
        if (m < 1) return;
        __syncthreads();
        spline_solve_block<kTableThreads>(I.scalefact, I.knot_fac, I.knot_invdiag, m, c, sh);
        if (t == 0) {
            c[0] = 0.0;
            c[Na - 1] = 0.0;
        }
        return;
    }
    b -= nrow;
    const FsTable F = fs_table(I, P.fs, P.S.light, tsuf);
    const int table_blocks = fs_table_blocks(P.fs.n, kTableThreads);
    if (b < table_blocks) {
        fs_table_store(I, F, b * kTableThreads + t);
        return;
    }
    const int q = (b - table_blocks) * kTableThreads + t;
    if (q >= P.nodes) return;
    double half;
    const double x = nc_node_x(q, NcLayout{I.nc_slots, I.nc_tree}, P.loga0, P.loga, &half);
    const double fsl = fs_table_at(F, x);
    const double* kx = I.scalefact;
    const int j = seg_bsearch(kx, Na, x);
    nc_store(I, q, fsl, I.nc_inv[q], x - kx[j], j, kx[j + 1] - kx[j], I.knot_invh[j], Na, half);
}

// block per bin: this bin's delta_cdm (a deferred normalisation), the provisional row
// `row` = Na - 1, and its spline as c_base + (y_new - y_base) c_unit
__global__ void k_row_update(IntegratorDev I, int nk, int Na, int row, FinalizeArgs fin) {
    __shared__ double s_dy;
    const int ik = blockIdx.x;
    if (threadIdx.x == 0) {
        if (fin.active) {
            double p;
            I.dcdm[ik] = finalize_power(fin, ik, &p);
            if (fin.power_out) fin.power_out[ik] = p;
        }
        const StepScalars& S = *I.sc;
        double* y = I.dtot + (size_t)ik * I.ld;
        const double yn = get_delta_tot(I.nu_last[ik], I.dcdm[ik], S.OmegaNua3, S.Omeganonu, S.OmegaNu1, S.partnu);
        y[row] = yn;
        s_dy = yn - y[Na - 2];
    }
    __syncthreads();
    const double dy = s_dy;
    double* c = I.coef + (size_t)ik * I.ld;
    for (int k = 1 + threadIdx.x; k < Na - 1; k += blockDim.x) c[k] = fma(dy, __ldg(I.coef_unit + k), c[k]);
}

// ------------------------------------------------------------------ delta_nu integral
// Shared memory per CTA: Gk61Nodes | per warp: QagList, row[ld], coef[ld] | mbarriers
__global__ void __launch_bounds__(128) k_dnu_qag(IntegratorDev I, int nk, int Na, int nspec, int4 spec_ids) {
    extern __shared__ __align__(16) unsigned char sm[];
    Gk61Nodes& N = *reinterpret_cast<Gk61Nodes*>(sm);
    const size_t off = (sizeof(Gk61Nodes) + 15) & ~size_t(15);
    const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t per_warp = sizeof(QagList) + 2 * sizeof(double) * I.ld;
    unsigned char* wbase = sm + off + warp * per_warp;
    QagList& L = *reinterpret_cast<QagList*>(wbase);
    double* row = reinterpret_cast<double*>(wbase + sizeof(QagList));
    double* rc = row + I.ld;
    uint64_t* mybar = reinterpret_cast<uint64_t*>(sm + off + nw * per_warp) + warp;

    gk61_fill(N, threadIdx.x, blockDim.x);
    if (lane == 0) ptx::mbar_init(mybar, 1);
    ptx::mbar_init_fence();
    __syncthreads();

    const StepScalars& S = *I.sc;
    const int ntask = nspec * nk;
    const unsigned row_bytes = (unsigned)(((Na + 1) & ~1) * sizeof(double));
    unsigned phase = 0;
    int my_max = 0;
    long long my_tot = 0;
    for (int task = blockIdx.x * nw + warp; task < ntask; task += gridDim.x * nw) {
        const int si = task / nk, ik = task % nk;
        const int mi = si == 0 ? spec_ids.x : (si == 1 ? spec_ids.y : spec_ids.z);
        const double k = I.kq ? I.kq[ik] : I.wavenum[ik];
        double val = lane == 0 ? dnu_initial(I, S, ik, mi, k) : 0.0;
        if (!S.skip_integral && Na > 1 && S.inv_m[mi] > 0) {
            // stage the history row and its spline coefficients (TMA bulk copies)
            __syncwarp();
            if (lane == 0) {
                // order this warp's earlier generic reads of the buffers before the async writes
                ptx::fence_async_smem();
                ptx::mbar_expect_tx(mybar, Na > 2 ? 2 * row_bytes : row_bytes);
                ptx::bulk_g2s(row, I.dtot + (size_t)ik * I.ld, row_bytes, mybar);
                if (Na > 2) ptx::bulk_g2s(rc, I.coef + (size_t)ik * I.ld, row_bytes, mybar);
            }
            if (Na == 2 && lane < 2) rc[lane] = 0.0;  // linear: no coefficients
            const bool got = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(mybar, phase));  // warp-uniform
            phase ^= 1;
            if (!got) {
                if (lane == 0) atomicOr(I.status, kStTimeout);
                // wait (bounded) for the copy still in flight before leaving
                ptx::mbar_wait_bounded(mybar, phase ^ 1);
                return;
            }
            __syncwarp();
            const DnuIntegrandW f = dnu_integrand_w(I, S, mi, k * S.inv_m[mi], row, rc, Na);
            QagResult r = qag_warp_c(f, N, L, S.loga0, S.loga, 0.0, S.relerr, kQagLimit);
            val += S.prefac * r.result;
            if (I.ivals) {  // keep the final subdivision for the adjoint
                double* dst = I.ivals + ((size_t)mi * I.nk_alloc + ik) * kQagLimit * 2;
                for (int q = lane; q < r.nint; q += 32) {
                    dst[2 * q] = L.a[q];
                    dst[2 * q + 1] = L.b[q];
                }
                if (lane == 0) I.nivals[(size_t)mi * I.nk_alloc + ik] = r.nint;
            }
            if (!r.ok && lane == 0) atomicOr(I.status, kStGsl);
            my_max = max(my_max, r.nint);
            my_tot += r.nint;
        }
        if (lane == 0) I.dnu_s[(size_t)mi * I.nk_alloc + ik] = val;
    }
    if (lane == 0 && my_tot) {
        atomicMax(I.qag_max, my_max);
        atomicAdd(reinterpret_cast<unsigned long long*>(I.qag_total), (unsigned long long)my_tot);
    }
}

// One (species, bin) task per block of 4 G warps: the same integral as k_dnu_qag with the
// GK61 nodes of each step spread over the block and G - 1 bisection levels evaluated ahead
// (qag_block_spec_c: the same decisions, sums equal to the last bits).  For calls with few tasks, where one warp
// per task leaves the SMs' FP64 pipes idle between the long dependent chains of a single
// warp and the sequential QAG rounds set the time.
// G: levels of a round; -G: intervals of a round (qag_block_multi_c; 0: blocks of 2 or 4 warps and qag_block_c, no look-ahead).
// upd.row >= 0: a prepared step's provisional row (k_row_update's arithmetic, per task, while
// the row is on its way, instead of a launch of its own before this one: 7 us).
// Shared memory: Gk61Nodes | row[ld] | coef[ld] | QagList | QagSpecSmem or QagBlockSmem | mbarrier
struct RowUpdate {
    int row;
    FinalizeArgs fin;
};
constexpr int qag_blk_threads(int G) { return G > 0 ? 128 * G : (G < 0 ? -128 * G : 128); }
template <int G, bool MULTI = (G < 0)>
struct QagBlkSmemOf { typedef QagSpecSmem<G> type; };
template <int G>
struct QagBlkSmemOf<G, true> { typedef QagMultiSmem<-G> type; };
template <>
struct QagBlkSmemOf<0, false> { typedef QagBlockSmem type; };

template <int G>
__global__ void __launch_bounds__(qag_blk_threads(G), 512 / qag_blk_threads(G))
    k_dnu_qag_blk(IntegratorDev I, int nk, int Na, int nspec, int4 spec_ids, RowUpdate upd) {
    typedef typename QagBlkSmemOf<G>::type Smem;
    extern __shared__ __align__(16) unsigned char sm[];
    ptx::dep_wait();
    ptx::dep_launch();
    Gk61Nodes& N = *reinterpret_cast<Gk61Nodes*>(sm);
    size_t off = (sizeof(Gk61Nodes) + 15) & ~size_t(15);
    double* row = reinterpret_cast<double*>(sm + off);
    double* rc = row + I.ld;
    off += 2 * sizeof(double) * I.ld;
    QagList& L = *reinterpret_cast<QagList*>(sm + off);
    off += (sizeof(QagList) + 15) & ~size_t(15);
    Smem& sh = *reinterpret_cast<Smem*>(sm + off);
    off += (sizeof(Smem) + 15) & ~size_t(15);
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + off);
    __shared__ double s_y, s_dy;  // the provisional value, and what it adds
    const int tid = threadIdx.x;
    const StepScalars& S = *I.sc;
    // Blocks take the tasks from the last: the high-k bins of the last species, among the
    // deepest QAG subdivisions, start first, and the blocks that wait for a free slot
    // (more tasks than resident blocks) get the shallow low-k bins of the first species.
    const int task = nspec * nk - 1 - (int)blockIdx.x, si = task / nk, ik = task % nk;
    const int mi = si == 0 ? spec_ids.x : (si == 1 ? spec_ids.y : spec_ids.z);
    const double k = I.kq ? I.kq[ik] : I.wavenum[ik];
    const bool integrate = !S.skip_integral && Na > 1 && S.inv_m[mi] > 0;  // block-uniform
    // Thread 0: the copies of the history row and its spline coefficients, in flight while the
    // block fills its tables, and the provisional value; another warp's first thread leaves the
    // initial-condition term where the integral will be added.
    if (tid == 32) I.dnu_s[(size_t)mi * I.nk_alloc + ik] = dnu_initial(I, S, ik, mi, k);
    if (tid == 0) {
        ptx::mbar_init(bar, 1);
        ptx::mbar_init_fence();
        if (integrate) {
            const unsigned row_bytes = (unsigned)(((Na + 1) & ~1) * sizeof(double));
            ptx::fence_async_smem();
            ptx::mbar_expect_tx(bar, Na > 2 ? 2 * row_bytes : row_bytes);
            ptx::bulk_g2s(row, I.dtot + (size_t)ik * I.ld, row_bytes, bar);
            if (Na > 2) ptx::bulk_g2s(rc, I.coef + (size_t)ik * I.ld, row_bytes, bar);
            else rc[0] = rc[1] = 0.0;  // linear: no coefficients
        }
        if (upd.row >= 0) {
            double d;
            if (upd.fin.active) {
                double p;
                d = finalize_power(upd.fin, ik, &p);
                if (si == 0) {
                    I.dcdm[ik] = d;
                    if (upd.fin.power_out) upd.fin.power_out[ik] = p;
                }
            } else {
                d = I.dcdm[ik];
            }
            s_y = get_delta_tot(I.nu_last[ik], d, S.OmegaNua3, S.Omeganonu, S.OmegaNu1, S.partnu);
            s_dy = s_y - I.dtot[(size_t)ik * I.ld + Na - 2];
        }
    }
    gk61_fill(N, tid, blockDim.x);
    __syncthreads();
    if (!integrate) return;
    if (!__syncthreads_and(ptx::mbar_wait_bounded(bar, 0))) {
        if (tid == 0) atomicOr(I.status, kStTimeout);
        ptx::mbar_wait_bounded(bar, 0);  // the copies still in flight
        return;
    }
    if (upd.row >= 0) {
        const double dy = s_dy;
        for (int j = 1 + tid; j < Na - 1; j += blockDim.x) rc[j] = fma(dy, __ldg(I.coef_unit + j), rc[j]);
        if (tid == 0) row[Na - 1] = s_y;
        __syncthreads();
    }
    const DnuIntegrandW f = dnu_integrand_w(I, S, mi, k * S.inv_m[mi], row, rc, Na);
    QagResult r;
    if constexpr (G < 0) r = qag_block_multi_c(f, N, L, S.loga0, S.loga, 0.0, S.relerr, kQagLimit, sh);
    else if constexpr (G > 0) r = qag_block_spec_c(f, N, L, S.loga0, S.loga, 0.0, S.relerr, kQagLimit, sh);
    else r = qag_block_c(f, N, L, S.loga0, S.loga, 0.0, S.relerr, kQagLimit, sh);
    if (I.ivals) {  // keep the final subdivision for the adjoint
        double* dst = I.ivals + ((size_t)mi * I.nk_alloc + ik) * kQagLimit * 2;
        for (int q = tid; q < r.nint; q += blockDim.x) {
            dst[2 * q] = L.a[q];
            dst[2 * q + 1] = L.b[q];
        }
        if (tid == 0) I.nivals[(size_t)mi * I.nk_alloc + ik] = r.nint;
    }
    if (tid == 0) {
        // (thread 32 wrote the initial-condition term, before a barrier)
        I.dnu_s[(size_t)mi * I.nk_alloc + ik] += S.prefac * r.result;
        if (!r.ok) atomicOr(I.status, kStGsl);
        atomicMax(I.qag_max, r.nint);
        atomicAdd(reinterpret_cast<unsigned long long*>(I.qag_total), (unsigned long long)r.nint);
    }
}

template <int G>
static size_t dnu_qag_blk_smem(int ld) {
    return ((sizeof(Gk61Nodes) + 15) & ~size_t(15)) + 2 * sizeof(double) * ld + ((sizeof(QagList) + 15) & ~size_t(15)) +
           ((sizeof(typename QagBlkSmemOf<G>::type) + 15) & ~size_t(15)) + sizeof(uint64_t);
}

// delta_tot_table.c:155-170: combine the species
__global__ void k_combine(IntegratorDev I, int nk) {
    const int ik = blockIdx.x * blockDim.x + threadIdx.x;
    if (ik >= nk) return;
    const StepScalars& S = *I.sc;
    double acc = 0;
    for (int mi = 0; mi < kNuSpecies; mi++)
        if (S.wnu[mi] != 0.0) acc += I.dnu_s[(size_t)mi * I.nk_alloc + ik] * S.wnu[mi];
    I.dnu[ik] = acc;
}

// Gauss-Legendre nodes by Newton iteration on P_n (positive half)
static void gl_nodes(int n, double* X, double* Wt) {
    for (int i = 0; i < n / 2; i++) {
        double x = cos(3.14159265358979323846 * (i + 0.75) / (n + 0.5)), dp = 0;
        for (int it = 0; it < 100; it++) {
            double p0 = 1, p1 = x;
            for (int k = 2; k <= n; k++) {
                const double p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
                p0 = p1;
                p1 = p2;
            }
            dp = n * (x * p1 - p0) / (x * x - 1);
            const double dx = p1 / dp;
            x -= dx;
            if (fabs(dx) < 1e-16) break;
        }
        X[i] = x;
        Wt[i] = 2 / ((1 - x * x) * dp * dp);
    }
}

// fslength(logai, logaf) = light * int_{logai}^{logaf} dlna / (a^2 H(a)) (delta_tot_table.c:378-407)
// for n intervals, a warp each: the interval is cut into segments of at most 0.01 in
// log a, each integrated with the 8-point Gauss-Legendre rule (the integrand is smooth on
// a scale of ~1 in log a, so the rule error is far below double rounding); lanes take
// segments in turn and the warp sums them.  0 where logai >= logaf, as the reference.
struct GL8 {
    double x[8], w[8];
};
__global__ void k_fslength_values(const Background* B, const double* lai, const double* laf, int n, double light,
                                  GL8 gl, double* out) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= n) return;
    const double a0 = lai[i], a1 = laf[i];
    double acc = 0;
    if (a0 < a1) {
        const int nseg = (int)ceil((a1 - a0) / 0.01);
        const double h = (a1 - a0) / nseg;
        for (int sgi = lane; sgi < nseg; sgi += 32) {
            const double c = a0 + (sgi + 0.5) * h;
            double sseg = 0;
            for (int q = 0; q < 8; q++) {
                const double la = c + 0.5 * h * gl.x[q];
                const double a = exp(la);
                sseg += gl.w[q] / (a * (a * hubble(*B, a, la)));
            }
            acc += 0.5 * h * sseg;
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) out[i] = a0 < a1 ? light * acc : 0.0;
}
void launch_fslength_values(const Background* dB, const double* logai, const double* logaf, int n, double light,
                            double* out, cudaStream_t st) {
    static GL8 gl;
    static bool have = false;
    if (!have) {
        double X[4], Wt[4];  // the positive half; nodes come in +-x pairs
        gl_nodes(8, X, Wt);
        for (int q = 0; q < 4; q++) {
            gl.x[2 * q] = X[q];
            gl.x[2 * q + 1] = -X[q];
            gl.w[2 * q] = gl.w[2 * q + 1] = Wt[q];
        }
        have = true;
    }
    if (n > 0) k_fslength_values<<<(n + 3) / 4, 128, 0, st>>>(dB, logai, logaf, n, light, gl, out);
}
static GL4 gl4_host() {
    GL4 g;
    gl_nodes(4, g.x, g.w);
    return g;
}

size_t dnu_qag_smem(int ld, int wpb) {
    return ((sizeof(Gk61Nodes) + 15) & ~size_t(15)) + wpb * (sizeof(QagList) + 2 * sizeof(double) * ld) +
           wpb * sizeof(uint64_t);
}

static int sm_count_i() {
    static const int n = [] {
        int dev = 0, c = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
        return c > 0 ? c : 1;
    }();
    return n;
}

// Blocks per role of a call's preparation.
void launch_integrator_prepare(const IntegratorDev& I, const Background& B, const StepScalars& S, int Na, double a,
                               double loga, double loga0, double TimeTransfer, int start_row, int write_knot,
                               bool scalars_only, RowsMode rows, int nk, int update_row, const FinalizeArgs* fin,
                               cudaStream_t st, const CallInput& in) {
    static const GL4 gl = gl4_host();
    PrepArgs P{};
    P.S = S;
    call_scalars(B, a, loga, loga0, TimeTransfer, Na, P.S);
    P.loga = loga;
    P.loga0 = loga0;
    P.Na = Na;
    P.start_row = start_row < 0 ? 0 : start_row;
    P.write_knot = write_knot;
    if (scalars_only) {  // block 0
        k_prep_eval<<<1, kPrepThreads, 0, st>>>(I, P, gl);
        return;
    }
    P.in = in;
    P.in_blocks = (2 * in.n + kPrepThreads - 1) / kPrepThreads;
    P.knot_blocks = (Na - 1 + kPrepThreads - 1) / kPrepThreads;
    if (!no_interval(loga0, loga)) {  // the fslength table also gives fslength(log a0, log a)
        P.fs = fs_grid(16 * (Na > 1 ? Na : 1), loga0, loga);
        P.fs_blocks = fs_blocks(P.fs);
        P.nodes = Na > 1 ? I.nc_slots * 61 : 0;
        P.node_blocks = (P.nodes + kPrepThreads - 1) / kPrepThreads;
        if (I.hyb && P.S.partnu > 0 && !P.S.skip_integral) P.hyb_blocks = kHybPieces / 8;
    }
    const int roles = P.in_blocks + P.knot_blocks + P.fs_blocks + kNuSpecies * P.hyb_blocks + P.node_blocks;
    k_prep_eval<<<1 + roles, kPrepThreads, 0, st>>>(I, P, gl);
    const int nrow = rows == kRowsBase ? nk + 1 : (rows == kRowsFull && (Na > 2 || update_row >= 0) ? nk : 0);
    const int blocks = nrow + fs_table_blocks(P.fs.n, kTableThreads) +
                       (P.nodes + kTableThreads - 1) / kTableThreads;
    if (blocks <= 0) return;
    const int mode = nrow > 0 ? (int)rows : (int)kRowsNone;
    const FinalizeArgs f = fin ? *fin : FinalizeArgs{};
    // As a dependent the kernel starts 2-3 us earlier, but several blocks to an SM then spread
    // unevenly (as launch_dnu_qag_blk's): calls of 400 to 512 bins, 430 to 560 blocks, 101, 125,
    // 137 us as dependents and 98, 122, 131 after it; of 200 to 300 bins 85 and 84 to 87.
    if (2 * blocks > 5 * sm_count_i())
        k_prep_tables<<<blocks, kTableThreads, 0, st>>>(I, P, mode, nk, update_row, f);
    else
        launch_dependent(k_prep_tables, blocks, kTableThreads, 0, st, I, P, mode, nk, update_row, f);
}

// The rest, after the rows' splines: the integrals, the species sum.
// One block per task; false: the history row does not fit shared memory.
template <int G>
static bool launch_dnu_qag_blk(const IntegratorDev& I, int nk, int Na, int nspec, int4 spec_ids, const RowUpdate& upd,
                               int threads, cudaStream_t st) {
    const size_t smem = dnu_qag_blk_smem<G>(I.ld);
    if (smem > 227 * 1024 - 256) return false;
    raise_dynamic_smem_limit(reinterpret_cast<const void*>(k_dnu_qag_blk<G>));
    // Small blocks not as dependents: the up to eight an SM takes spread unevenly over the SMs if
    // they come up while the kernel before is still there (1221 tasks of 2 warps: a call of 138 us
    // as dependents, 125 so; of 8 warps, two to an SM, 4-5 us are won instead).
    if constexpr (G == 0)
        k_dnu_qag_blk<G><<<nspec * nk, threads, smem, st>>>(I, nk, Na, nspec, spec_ids, upd);
    else
        launch_dependent(k_dnu_qag_blk<G>, nspec * nk, threads, smem, st, I, nk, Na, nspec, spec_ids, upd);
    return true;
}

void launch_integrator_rest(const IntegratorDev& I, int nk, int Na, int nspec, const int* spec_ids,
                            int warps_per_block, cudaStream_t st, int qag_split, int update_row, bool defer_combine,
                            const FinalizeArgs* fin, bool base_ready, bool rows_stored) {
    RowUpdate upd{};
    upd.row = -1;
    if (update_row >= 0 && base_ready) {
        upd.row = update_row;
        if (fin && fin->active) upd.fin = *fin;
        if (rows_stored) {  // for a reader after the integrals
            k_row_update<<<nk, 128, 0, st>>>(I, nk, Na, update_row, upd.fin);
            upd.row = -1;
        }
    } else if (update_row >= 0) {
        // a history of two knots: no splines
        if (fin && fin->active)
            launch_finalize_power(fin->bin_sum, fin->F0sq, fin->count, fin->ksum, fin->compact_bins, nk, fin->BoxSize,
                                  fin->power_out, fin->keff_out, fin->dcdm_out, fin->keffphys_out, st);
        launch_update_row_scalars(I, nk, update_row, st);
    }
    int wpb = warps_per_block < 1 ? 1 : (warps_per_block > 4 ? 4 : warps_per_block);
    while (wpb > 1 && dnu_qag_smem(I.ld, wpb) > 227 * 1024 - 256) wpb--;
    const size_t smem = dnu_qag_smem(I.ld, wpb);
    static bool attr_set = false;
    if (!attr_set) {
        raise_dynamic_smem_limit(reinterpret_cast<const void*>(k_dnu_qag));
        attr_set = true;
    }
    const int ntask = nspec * nk;
    if (ntask > 0) {
        const int nsm = sm_count_i();
        // a block per task: with no more tasks than SMs 12 warps and two levels of look-ahead
        // (split 12; a call of 64, 100, 150 bins 62, 71, 78 us, with 8 warps and one level 64, 74,
        // 82; three levels 65, 75, 77; but 200 bins 86 against 82), 8 warps and one level (split 8)
        // below 4 tasks per SM (512 tasks 105 us; 4 warps without look-ahead 115, 2 117), 2 warps
        // from there (750, 900, 1221, 1536 tasks 103, 107, 125, 137 us; 4 warps 115, 126, 139, 160;
        // a warp per task, split 1, 108, 107, 127, 140).  Where hybrid neutrinos cut J the next
        // interval is anyone's guess: two intervals a round by their errors (151 bins 228 us; one
        // 256, one and a level of look-ahead 310, three 222 but 60 bins 216 against 214)
        const int split = qag_split > 0 ? qag_split : (ntask <= nsm ? 12 : (ntask < 4 * nsm ? 8 : 2));
        const bool cut = qag_split <= 0 && I.nc_tree > 1;
        const int4 sp = make_int4(spec_ids[0], spec_ids[1], spec_ids[2], 0);
        const bool done =
            cut          ? launch_dnu_qag_blk<-2>(I, nk, Na, nspec, sp, upd, 256, st)
            : split >= 12 ? launch_dnu_qag_blk<3>(I, nk, Na, nspec, sp, upd, 384, st)
            : split >= 8 ? launch_dnu_qag_blk<2>(I, nk, Na, nspec, sp, upd, 256, st)
            : split > 1  ? launch_dnu_qag_blk<0>(I, nk, Na, nspec, sp, upd, split >= 4 ? 128 : 64, st)
                         : false;
        if (!done) {
            if (upd.row >= 0) k_row_update<<<nk, 128, 0, st>>>(I, nk, Na, upd.row, upd.fin);
            const int blocks = (ntask + wpb - 1) / wpb;
            k_dnu_qag<<<blocks, 32 * wpb, smem, st>>>(I, nk, Na, nspec,
                                                      make_int4(spec_ids[0], spec_ids[1], spec_ids[2], 0));
        }
    }
    if (!defer_combine) k_combine<<<(nk + 255) / 256, 256, 0, st>>>(I, nk);
}

// ------------------------------------------------------------------ end of an update
// commit_row >= 0: overwrite that row with the final delta_tot (delta_tot_table.c:229-233);
// -1: the provisional row is dropped; -2: delta_nu_last is returned as is (the
// same-scale-factor path, delta_tot_table.c:209-213: no NaN check, no clamp);
// -3: a differentiable step: like -1 but delta_nu_last is left unchanged.
__global__ void k_finish(IntegratorDev I, int nk, int commit_row, double a, double loga, const double* keff,
                         double* dnu_out, double* logk_out, double* ratio_out, CorrTable corr, double* norm_out,
                         int combine, int logk_ready, unsigned* status_out) {
    ptx::dep_wait();
    ptx::dep_launch();
    const StepScalars& S = *I.sc;
    const bool pass = commit_row == -2;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (commit_row >= 0) I.scalefact[commit_row] = loga;
        if (norm_out) *norm_out = S.kspace_prefac;
    }
    const double norm = S.kspace_prefac;
    // delta_nu of bin ik: k_combine's species sum (same arithmetic) or the combined value
    auto dnu_of = [&](int ik) -> double {
        if (!combine) return I.dnu[ik];
        double acc = 0;
        for (int mi = 0; mi < kNuSpecies; mi++)
            if (S.wnu[mi] != 0.0) acc += I.dnu_s[(size_t)mi * I.nk_alloc + ik] * S.wnu[mi];
        return acc;
    };
    // Bin ik's slope needs bin ik+1's final value: recomputed here rather than read back,
    // so the bins are independent and spread over many blocks (their FP64 logs and
    // divisions would otherwise queue on one SM).
    for (int ik = blockIdx.x * blockDim.x + threadIdx.x; ik < nk; ik += gridDim.x * blockDim.x) {
        const double v = dnu_of(ik);
        if (combine) I.dnu[ik] = v;
        double out = v;
        if (!pass) {
            if (commit_row != -3) I.nu_last[ik] = v;
            if (commit_row >= 0)
                I.dtot[(size_t)ik * I.ld + commit_row] =
                    get_delta_tot(v, I.dcdm[ik], S.OmegaNua3, S.Omeganonu, S.OmegaNu1, S.partnu);
            if (isnan(v)) atomicOr(I.status, kStDnuNaN);
            out = v < 0 ? 0.0 : v;  // delta_tot_table.c:246-247
        }
        dnu_out[ik] = out;
        if (keff) {
            const double lk = logk_ready ? logk_out[ik] : log(keff[ik]);
            const double r = out / I.dcdm[ik];
            if (logk_out && !logk_ready) logk_out[ik] = lk;
            if (ratio_out) ratio_out[ik] = r;
            if (corr.xf) {
                corr.xf[ik] = (float)lk;
                corr.rn[ik] = (float)(norm * r);
                double sl = 0;
                if (ik + 1 < nk) {
                    const double v1 = dnu_of(ik + 1);
                    const double out1 = pass ? v1 : (v1 < 0 ? 0.0 : v1);
                    const double lk1 = logk_ready ? logk_out[ik + 1] : log(keff[ik + 1]);
                    const double r1 = out1 / I.dcdm[ik + 1];
                    sl = norm * (r1 - r) / (lk1 - lk);
                }
                corr.sn[ik] = (float)sl;
                if (!isfinite(norm * r) || !isfinite(sl)) atomicOr(I.status, kStGridNaN);
            }
        }
    }
    if (status_out) deliver_status(I.status, I.done, status_out);
}

void launch_finish_update(const IntegratorDev& I, int nk, int commit_row, double a, double loga,
                          const double* keff, double* dnu_out, double* logk_out, double* ratio_out,
                          CorrTable corr, double* norm_out, cudaStream_t st, bool combine, bool logk_ready,
                          unsigned* status_out) {
    launch_dependent(k_finish, (nk + 31) / 32 > 0 ? (nk + 31) / 32 : 1, 32, 0, st, I, nk, commit_row, a, loga, keff,
                     dnu_out, logk_out, ratio_out, corr, norm_out, combine ? 1 : 0, logk_ready ? 1 : 0, status_out);
}

}  // namespace ksp
