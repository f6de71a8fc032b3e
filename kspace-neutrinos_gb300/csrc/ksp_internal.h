// ksp_internal.h -- host-visible structures and kernel launchers shared by the
// translation units of libkspace_gb300.so.  Not part of the public C ABI.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "ksp_device.cuh"

namespace ksp {

// Scalars of one integrator call at scale factor a (delta_tot_table.c:153-172,507-548,
// interface_common.c:139-145), formed by call_scalars.
struct StepScalars {
    double a, loga, loga0;           // inputs (logs taken on the host, as the reference does)
    double light, prefac, Omeganonu; // delta_tot_table.c:52-57
    double OmegaNua3, OmegaNu1, partnu;  // get_delta_tot coefficients at a (:179-181)
    double Omega_nu_tot;             // get_omega_nu_nopart(a) (:155)
    double omeganu[kNuSpecies];      // deg * omega_nu_single(a, mi) (:162)
    double wnu[kNuSpecies];          // omeganu / Omega_nu_tot: the species' weights (0: none)
    double inv_m[kNuSpecies];        // 1 / (m / kT) of the mass inside J (0: massless)
    double qc[kNuSpecies];           // the momentum cut of J's series (0: the fit)
    double fsl_A0a;                  // fslength(log a0, log a) (:522)
    double deriv_prefac;             // a0 * H(a0)/c * a0 (:524)
    double relerr;                   // 1e-6, loosened for hybrid neutrinos (:547)
    double partnu_now;               // particle_nu_fraction(a, 0) (:539)
    double kspace_prefac;            // interface_common.c:139-145
    double fs_h, fs_ih;              // spacing of the fslength table's nodes, and its inverse
    int skip_integral;               // particles carry everything (:542-543), or no_interval
    int Na, Nfs;
};

// The arrays of a node table.
struct NcNodes {
    double2 *ab, *cd;
    int2* jf;
    double *g, *fsl, *dx, *inv;
    int* j;
    double* half;
    int slots, tree;
};

// One integrator instance (the reference's delta_tot_table + omega_nu + transfer table).
struct IntegratorDev {
    NcNodes nodes() const {
        return NcNodes{nc_ab, nc_cd, nc_jf, nc_g, nc_fsl, nc_dx, nc_inv, nc_j, nc_half, nc_slots, nc_tree};
    }
    void set_nodes(const NcNodes& t) {
        nc_ab = t.ab; nc_cd = t.cd; nc_jf = t.jf; nc_g = t.g; nc_fsl = t.fsl; nc_dx = t.dx; nc_inv = t.inv;
        nc_j = t.j; nc_half = t.half; nc_slots = t.slots; nc_tree = t.tree;
    }
    Background* B;                   // device
    int nk_alloc, namax, ld;         // ld: padded row length of the history table
    double* scalefact;               // [namax]
    double* dtot;                    // [nk_alloc][ld]
    double* coef;                    // [nk_alloc][ld]  spline coefficients of each row
    double* nu_init;                 // [nk_alloc]
    double* nu_last;                 // [nk_alloc]
    double* wavenum;                 // [nk_alloc]
    const double* kq;                // k of the bins of the current call (the reference integrates at
                                     // the wavenum argument, delta_tot_table.c:526,593); null = wavenum
    double* dcdm;                    // [nk_alloc] sqrt(P_cdm) of the current call
    double* dnu_s;                   // [kNuSpecies][nk_alloc] per-species delta_nu
    double* dnu;                     // [nk_alloc] combined
    double* knot_invdiag;            // [namax] factorised spline system of the knots
    double* knot_fac;                // [namax]
    double* knot_invh;               // [namax] 1/(x_{i+1}-x_i)
    double* knot_h3;                 // [namax] (x_{i+1}-x_i)/3
    double* knot_ih3;                // [namax] 1/(3 (x_{i+1}-x_i))
    double* nc_g;                    // [kNcNodes] node table of the delta_nu integrand (NodeCache)
    double* nc_fsl;
    double* nc_dx;
    int* nc_j;
    double2* nc_ab;                  // [kNcNodes] the same as weights of the row (NodeTable)
    double2* nc_cd;
    int2* nc_jf;
    double* nc_half;                 // [kNcMaxSlots]
    unsigned* done;                  // blocks of k_finish that are through (0 between calls)
    const double* jt;                // J's fine table (one per device)
    double* hyb;                     // optional: [kNuSpecies][kHybTable] the tables of J with a cut
    int nc_slots, nc_tree;           // slots of the node table in use (0 = none), and its heap's (NcLayout)
    double* fs_y;                    // [fs_cap]
    double* fs_c;                    // [fs_cap]
    double* fs_seg;                  // [fs_cap] integrals of 1/(a^2 H) over the table's segments
    double* fs_suf;                  // [fs_cap] their suffix sums within a block's stretch
    double* fs_tot;                  // [fs_cap / 16 + 1] the stretches' totals
    double* nc_inv;                  // [kNcNodes] 1/(a H) at the nodes
    int fs_cap;
    double* t_logk;                  // transfer table [ntrans]
    double* t_T;
    double* t_c;
    int ntrans;
    StepScalars* sc;                 // device scalars
    unsigned* status;                // device status bits
    int* qag_max;                    // diagnostics: max intervals of any bin in the last call
    long long* qag_total;
    double* ivals;                   // optional: final QAG intervals [kNuSpecies][nk_alloc][kQagLimit][2]
    int* nivals;                     // [kNuSpecies][nk_alloc]
    double* coef_unit;               // [ld] spline coefficients of a unit provisional (last) knot,
                                     // the other knots zero (kRowsBase)
};

// Whether a call at log a has nothing to integrate: at a0 the interval is empty, before a0
// fslength, a factor of the integrand, is zero (delta_tot_table.c:394-396), and an end that is no
// finite number is refused (no_number).  No fslength table and no node table is made then, and
// the integrals read neither.
KSP_HD bool no_number(double loga) { return !isfinite(loga); }
KSP_HD bool no_interval(double loga0, double loga) { return !(loga > loga0) || no_number(loga); }

// What the integrals and the species sum need of a species, from its omeganu, Omega_nu_tot and
// partnu.
KSP_HD void species_scalars(const Background& B, int mi, StepScalars& S) {
    const double mnubykT = B.mnu_J[mi] / B.kBtnu;
    S.wnu[mi] = B.deg[mi] > 0 ? S.omeganu[mi] / S.Omega_nu_tot : 0.0;
    S.inv_m[mi] = mnubykT > 0 ? 1.0 / mnubykT : 0.0;
    S.qc[mi] = S.partnu > 0 ? B.vcrit * mnubykT : 0.0;
}

// The part of StepScalars that a call sets (the rest is set with the table): on the host
// for a single call, where it takes about a microsecond beside the launches (on the device
// it was a chain of some 60 dependent FP64 divisions, 12 us of each call).
inline void call_scalars(const Background& B, double a, double loga, double loga0, double TT, int Na, StepScalars& S) {
    const double om_a = omega_nu(B, a), om_1 = omega_nu(B, 1), partnu = particle_nu_fraction(B, a, 0);
    const double nop = om_a - om_1 * partnu / (a * a * a);  // omega_nu_nopart (omega_nu_single.c:69-74)
    S.a = a;
    S.loga = loga;
    S.loga0 = loga0;
    S.Na = Na;
    S.OmegaNua3 = nop * (a * a * a);
    S.OmegaNu1 = om_1;
    S.partnu = partnu;
    S.Omega_nu_tot = nop;
    for (int mi = 0; mi < kNuSpecies; mi++) {
        S.omeganu[mi] = B.deg[mi] > 0 ? B.deg[mi] * omega_nu_single(B, a, mi) : 0.0;
        species_scalars(B, mi, S);
    }
    S.deriv_prefac = TT * (hubble(B, TT) / S.light) * TT;
    S.relerr = 1e-6;
    S.partnu_now = partnu;
    S.skip_integral = no_interval(loga0, loga) ? 1 : 0;
    if (S.partnu_now > 0) {
        if (1 - S.partnu_now < 1e-3) S.skip_integral = 1;
        S.relerr /= (1. + 1e-5 - S.partnu_now);
    }
    S.kspace_prefac = nop / (S.Omeganonu / (a * a * a) + (om_a - nop));
    S.fsl_A0a = 0;
    S.Nfs = 0;
}

#ifdef __CUDACC__
// The same on the device, for batches: the scalars of a call at a (delta_tot_table.c:153-172,
// 507-548, interface_common.c:139-145), by one warp: the background evaluations, which are
// long FP64 dependency chains, run on different lanes; lane 0 combines them.
__device__ __forceinline__ void call_scalars_warp(const Background& B, double a, double loga, double loga0,
                                                  double TT, int Na, StepScalars& S) {
    const int lane = threadIdx.x & 31;
    double v = 0.0;
    if (lane == 0) v = omega_nu(B, a);
    else if (lane == 1) v = omega_nu(B, 1);
    else if (lane < 2 + kNuSpecies) v = B.deg[lane - 2] > 0 ? B.deg[lane - 2] * omega_nu_single(B, a, lane - 2) : 0.0;
    else if (lane == 2 + kNuSpecies) v = hubble(B, TT);
    const double om_a = __shfl_sync(0xffffffffu, v, 0);
    const double om_1 = __shfl_sync(0xffffffffu, v, 1);
    double om_s[kNuSpecies];
    for (int mi = 0; mi < kNuSpecies; mi++) om_s[mi] = __shfl_sync(0xffffffffu, v, 2 + mi);
    const double h_tt = __shfl_sync(0xffffffffu, v, 2 + kNuSpecies);
    if (lane != 0) return;
    const double partnu = particle_nu_fraction(B, a, 0);
    const double nop = om_a - om_1 * partnu / (a * a * a);  // omega_nu_nopart (omega_nu_single.c:69-74)
    S.a = a;
    S.loga = loga;
    S.loga0 = loga0;
    S.Na = Na;
    S.OmegaNua3 = nop * (a * a * a);
    S.OmegaNu1 = om_1;
    S.partnu = partnu;
    S.Omega_nu_tot = nop;
    for (int mi = 0; mi < kNuSpecies; mi++) {
        S.omeganu[mi] = om_s[mi];
        species_scalars(B, mi, S);
    }
    S.deriv_prefac = TT * (h_tt / S.light) * TT;
    S.relerr = 1e-6;
    S.partnu_now = partnu;
    S.skip_integral = no_interval(loga0, loga) ? 1 : 0;
    if (S.partnu_now > 0) {
        if (1 - S.partnu_now < 1e-3) S.skip_integral = 1;
        S.relerr /= (1. + 1e-5 - S.partnu_now);
    }
    S.kspace_prefac = nop / (S.Omeganonu / (a * a * a) + (om_a - nop));
}

// Solve the natural-spline system of the knots (factorised by knot_row) for the
// right-hand side sc[1..m], m = Na - 2, in place, with all 32 lanes of a warp: both
// substitutions are linear recurrences z_u = r_u - f_u z_{u-1} and c_u = (z_u - o_u c_{u+1}) /
// d_u, i.e. chains of affine maps; each lane composes the maps of its stretch of rows, a
// warp scan composes the stretches, and each lane then replays its stretch from the
// value entering it.
__device__ __forceinline__ void spline_solve_scan(const IntegratorDev& I, int m, double* sc) {
    const int lane = threadIdx.x & 31;
    const double* x = I.scalefact;
    const int per = (m + 31) / 32;
    const int u0 = min(m, lane * per), u1 = min(m, u0 + per);
    // forward: z_u = r_u - fac_u z_{u-1} (fac_0 = 0)
    double A = 1.0, B = 0.0;
    for (int u = u0; u < u1; u++) {
        const double f = u > 0 ? I.knot_fac[u] : 0.0;
        B = sc[u + 1] - f * B;
        A = -f * A;
    }
    double pa = A, pb = B;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {  // inclusive scan of the maps, left to right
        const double qa = __shfl_up_sync(0xffffffffu, pa, d), qb = __shfl_up_sync(0xffffffffu, pb, d);
        if (lane >= d) {
            pb = pa * qb + pb;
            pa = pa * qa;
        }
    }
    double zin = __shfl_up_sync(0xffffffffu, pb, 1);  // z entering this stretch (z_{-1} = 0)
    if (lane == 0) zin = 0.0;
    for (int u = u0; u < u1; u++) {
        const double f = u > 0 ? I.knot_fac[u] : 0.0;
        zin = sc[u + 1] - f * zin;
        sc[u + 1] = zin;
    }
    __syncwarp();
    // backward: c_u = (z_u - off_u c_{u+1}) * invdiag_u, c_m = 0
    A = 1.0;
    B = 0.0;
    for (int u = u1 - 1; u >= u0; u--) {
        const double off = u < m - 1 ? x[u + 2] - x[u + 1] : 0.0;
        const double iv = I.knot_invdiag[u];
        B = (sc[u + 1] - off * B) * iv;
        A = -off * iv * A;
    }
    pa = A;
    pb = B;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {  // right to left
        const double qa = __shfl_down_sync(0xffffffffu, pa, d), qb = __shfl_down_sync(0xffffffffu, pb, d);
        if (lane + d < 32) {
            pb = pa * qb + pb;
            pa = pa * qa;
        }
    }
    double cin = __shfl_down_sync(0xffffffffu, pb, 1);  // c entering from the right
    if (lane == 31) cin = 0.0;
    __syncwarp();
    for (int u = u1 - 1; u >= u0; u--) {
        const double off = u < m - 1 ? x[u + 2] - x[u + 1] : 0.0;
        cin = (sc[u + 1] - off * cin) * I.knot_invdiag[u];
        sc[u + 1] = cin;
    }
    __syncwarp();
}

// The delta_nu integrand of one (species, bin) with the instance's node table; knots,
// row and rc may be staged copies (shared memory) of the instance's arrays.
// sb, sd: seg_poly of (row, rc), filled by the caller
// k_over_m = k / (m / kT) given: the integral
// kernels form those divisions on one lane per task and broadcast them
__device__ __forceinline__ DnuIntegrandC dnu_integrand_pre(const IntegratorDev& I, const StepScalars& S,
                                                           double k_over_m, double qc,
                                                           const double* knots, const double* row, const double* rc,
                                                           const double* sb, const double* sd, int Na) {
    DnuIntegrandC f;
    f.B = I.B; f.k_over_m = k_over_m; f.qc = qc; f.nfl = I.B->nufrac_low[0];
    f.fs_y = I.fs_y; f.fs_c = I.fs_c; f.fs = FsGrid{S.Nfs, S.loga0, S.fs_h, S.fs_ih};
    f.kx = knots; f.ky = row; f.kc = rc; f.na = Na;
    f.sb = sb; f.sd = sd;
    f.ks = KnotSeg{I.knot_invh, I.knot_h3, I.knot_ih3};
    f.nc = NodeCache{I.nc_g, I.nc_fsl, I.nc_dx, I.nc_j, {I.nc_slots, I.nc_tree}};
    return f;
}
__device__ __forceinline__ DnuIntegrandC dnu_integrand(const IntegratorDev& I, const StepScalars& S, double k,
                                                       double mnubykT, double qc, const double* knots,
                                                       const double* row, const double* rc, const double* sb,
                                                       const double* sd, int Na) {
    return dnu_integrand_pre(I, S, k / mnubykT, qc, knots, row, rc, sb, sd, Na);
}
// The integrand of one (species mi, bin) from its row and spline coefficients (shared memory).
__device__ __forceinline__ DnuIntegrandW dnu_integrand_w(const IntegratorDev& I, const StepScalars& S, int mi, double kom,
                                                         const double* row, const double* rc, int Na) {
    DnuIntegrandW f;
    f.B = I.B; f.jt = I.jt; f.kom = kom; f.komf = (float)kom;
    f.qc = S.qc[mi]; f.nfl = I.B->nufrac_low[0];
    f.hyb = I.hyb ? I.hyb + (size_t)mi * kHybTable : nullptr;
    f.ky = row; f.kc = rc;
    f.nc = NodeTable{I.nc_ab, I.nc_cd, I.nc_fsl, I.nc_jf, I.nc_half, {I.nc_slots, I.nc_tree}};
    f.fs_y = I.fs_y; f.fs_c = I.fs_c; f.kx = I.scalefact; f.kih = I.knot_invh;
    f.S = &S; f.na = Na;
    return f;
}
// A node outside the node table: its terms evaluated here, then the same arithmetic.
__device__ __noinline__ inline double DnuIntegrandW::slow(double x) const {
    const FsGrid g{S->Nfs, S->loga0, S->fs_h, S->fs_ih};
    const NodeTerms t = dnu_node_terms(B, fs_y, fs_c, g, kx, na, x);
    return value(node_weights(t.g, t.dx, kx[t.j + 1] - kx[t.j], kih[t.j], na), t.fsl, (float)t.fsl, t.j);
}
// Node q of the node table, in an interval of half-width `half`.
__device__ __forceinline__ void nc_store(const IntegratorDev& I, int q, double fsl, double inv_aH, double dx, int j,
                                         double h, double ih, int Na, double half) {
    if (q % 61 == 0) I.nc_half[q / 61] = half;
    const double g = fsl * inv_aH;
    const NodeWeights w = node_weights(g, dx, h, ih, Na);
    I.nc_g[q] = g;
    I.nc_fsl[q] = fsl;
    I.nc_dx[q] = dx;
    I.nc_j[q] = j;
    I.nc_ab[q] = make_double2(w.a, w.b);
    I.nc_cd[q] = make_double2(w.c, w.d);
    I.nc_jf[q] = make_int2(j, __float_as_int((float)fsl));
}
// The initial-condition term of one (species, bin) task (delta_tot_table.c:525-535).
__device__ __forceinline__ double dnu_initial(const IntegratorDev& I, const StepScalars& S, int ik, int mi, double k) {
    const double specJ0 = specialJ_fit_tab(k * S.fsl_A0a * (S.inv_m[mi] > 0 ? S.inv_m[mi] : 1.0));
    return specJ0 * I.nu_init[ik] * (1. + S.deriv_prefac * S.fsl_A0a);
}
#endif

// Interpolation table for the grid correction (delta_pow.c:19-37), float, per
// non-empty bin, plus the bin -> compact index map.
// K1's normalisation of one compact bin (powerspectrum.c:98-115 + interface_gadget.c:
// 96-100): P = sum / |F(0)|^2 / count, keff = sum|k| / count (grid units), delta_cdm =
// sqrt(P L^3), keff in physical units.  k_finalize_power applies it to every bin; the
// step's row-spline kernel applies it to its bin when the binning pass deferred it.
struct FinalizeArgs {
    const double* bin_sum;
    const double* F0sq;
    const long long* count;
    const double* ksum;
    const int* compact_bins;
    double BoxSize;
    double* power_out;
    double* keff_out;
    double* dcdm_out;
    double* keffphys_out;
    int active;  // 0: nothing to do
    // formed on the host, as the reference forms them there (interface_gadget.c:84,96-99):
    // scale = BoxSize^-3 (pow), kfac = 2 pi / BoxSize
    double scale, kfac;
    double* logk_out;  // log of the physical keff (finalize_keff)
};
// What a call's last kernel leaves in pinned host memory: a spectrum ([nk] power, then [nk]
// keff), and the status word from the last of its blocks to end (they count themselves in done,
// 0 between calls).
struct HostOut {
    double* out = nullptr;
    unsigned* status_out = nullptr;
    const unsigned* status = nullptr;
    unsigned* done = nullptr;
};
#ifdef __CUDACC__
// The status word to the host from the last block (of one warp) of a kernel to end.
__device__ __forceinline__ void deliver_status(const unsigned* status, unsigned* done, unsigned* out) {
    __threadfence();
    __syncwarp();
    if (threadIdx.x == 0 && atomicInc(done, gridDim.x - 1) == gridDim.x - 1) {
        __threadfence();
        *out = *reinterpret_cast<const volatile unsigned*>(status);
    }
}
// the part that depends on the sums, and the part that is the geometry's alone (a prepared
// step forms the latter beside the binning pass); p: the bin's power, returned: delta_cdm
__device__ __forceinline__ double finalize_power(const FinalizeArgs& f, int c, double* p_out) {
    const int b = f.compact_bins[c];
    double p = f.bin_sum[b];
    p /= *f.F0sq;
    p /= (double)f.count[b];
    *p_out = p;
    return sqrt(p / f.scale);
}
__device__ __forceinline__ void finalize_keff(const FinalizeArgs& f, int c) {
    const int b = f.compact_bins[c];
    const double ke = f.ksum[b] / (double)f.count[b], kp = ke * f.kfac;
    if (f.keff_out) f.keff_out[c] = ke;
    if (f.keffphys_out) f.keffphys_out[c] = kp;
    if (f.logk_out) f.logk_out[c] = log(kp);
}
__device__ __forceinline__ void finalize_bin(const FinalizeArgs& f, int c) {
    double p;
    const double d = finalize_power(f, c, &p);
    if (f.power_out) f.power_out[c] = p;
    if (f.dcdm_out) f.dcdm_out[c] = d;
    finalize_keff(f, c);
}
#endif

struct CorrTable {
    float* xf;   // log k of node j
    float* rn;   // norm * ratio_j
    float* sn;   // norm * (ratio_{j+1}-ratio_j)/(logk_{j+1}-logk_j)
    int nk;
};

// Raise a kernel's dynamic shared-memory limit to the most a block may have beside the
// kernel's own static shared memory (the device's opt-in maximum minus it), once per
// kernel and device (ksp_api.cu).  A fixed 227 KB request fails for a kernel with static
// shared memory, and the failure would surface as the error of a later, unrelated launch.
int raise_dynamic_smem_limit(const void* kernel);

// ---- integrator launchers (ksp_integrator.cu)
void launch_background_tables(Background* dB, double a0, cudaStream_t st, unsigned* status);
// natural cubic spline coefficients c[n] of y on the knots x, n >= 3; scratch[2 n]
void launch_spline_coeffs(const double* x, const double* y, double* c, double* scratch, int n, cudaStream_t st);
// J's fine table on the current device
const double* jfine_table();
void launch_nufrac_low(Background* dB, double light, double vcrit, cudaStream_t st, unsigned* status);
// natural cubic spline of log H on n uniform knots of spacing h: coef[4 (n-1)], scratch[n]
void launch_hubble_table(const double* H, int n, double h, double* coef, double* scratch, cudaStream_t st);
// nufrac_low (omega_nu_single.c:214-228) of n momenta, a warp each
void launch_nufrac_low_values(const double* qc, int n, double* out, unsigned* status, cudaStream_t st);
// specialJ (delta_tot_table.c:457-463) of n arguments
void launch_special_j(const double* x, int n, double qc, double nufrac_low, double* out, cudaStream_t st);
// fslength (delta_tot_table.c:394-407) of n intervals [logai, logaf], a warp each
void launch_fslength_values(const Background* dB, const double* logai, const double* logaf, int n, double light,
                            double* out, cudaStream_t st);
// update_delta_tot (delta_tot_table.c:177-191) for row `row` at scale factor a
void launch_update_row(const IntegratorDev& I, int nk, int row, double a, double loga, const double* dcdm,
                       const double* dnu, cudaStream_t st);
// delta_tot_init part that needs the device (delta_tot_table.c:94-129)
void launch_delta_tot_init(const IntegratorDev& I, int nk, const double* wavenum, const double* dcdm,
                           int fresh, double TimeTransfer, cudaStream_t st);
// A call's preparation (scalars, knot factorisation, fslength and node tables) and, with
// it, the splines of the history rows.
// start_row: leading rows of the knot factorisation still valid from an earlier call;
// write_knot stores the provisional knot log a
enum RowsMode {
    kRowsNone,  // no row splines
    kRowsBase,  // before the provisional row is known (beside the binning pass): every row's
                // spline with its last knot equal to the one before, and that of a unit last
                // knot; launch_integrator_rest adds the provisional row as a correction
    kRowsFull   // every row's spline; update_row >= 0: after writing the provisional row
                // `update_row` (update_delta_tot, from delta_nu_last and delta_cdm)
};
// in: a call's k and delta_cdm in pinned host memory, read by the preparation itself
struct CallInput {
    const double* src = nullptr;  // [n] k, then [n] delta_cdm
    double* k = nullptr;
    double* dcdm = nullptr;
    int n = 0;
};
// S: the table's scalars (light, prefac, Omeganonu); B: the background's host copy
// fin (kRowsBase): the binning pass's normalisation, whose geometry part (keff) is formed here
void launch_integrator_prepare(const IntegratorDev& I, const Background& B, const StepScalars& S, int Na, double a,
                               double loga, double loga0, double TimeTransfer, int start_row, int write_knot,
                               bool scalars_only, RowsMode rows, int nk, int update_row, const FinalizeArgs* fin,
                               cudaStream_t st, const CallInput& in = CallInput{});
// The rest: the integrals and the species sum (get_delta_nu_combined,
// delta_tot_table.c:153-172, writes I.dnu).
// update_row >= 0: with a prepared step's provisional row first (base_ready: kRowsBase ran);
// qag_split: warps per (species, bin) task (1, 2, 4, 8 or 12; 0 = chosen by the task count)
// defer_combine: leave the species sum to launch_finish_update(..., combine = true)
void launch_integrator_rest(const IntegratorDev& I, int nk, int Na, int nspec, const int* spec_ids,
                            int warps_per_block, cudaStream_t st, int qag_split, int update_row = -1,
                            bool defer_combine = false, const FinalizeArgs* fin = nullptr,
                            bool base_ready = false, bool rows_stored = false);
size_t dnu_qag_smem(int ld, int wpb);
// end of get_delta_nu_update (delta_tot_table.c:226-248) + interface_common.c:134-146:
// delta_nu_last, committed row, NaN check, clamp, ratio/log k/kspace_prefac, grid table
// combine: the species sum first; logk_ready: logk_out holds the logs already
void launch_finish_update(const IntegratorDev& I, int nk, int commit_row, double a, double loga,
                          const double* keff, double* dnu_out, double* logk_out, double* ratio_out,
                          CorrTable corr, double* norm_out, cudaStream_t st, bool combine = false,
                          bool logk_ready = false, unsigned* status_out = nullptr);

// ---- adjoint (ksp_adjoint.cu)
struct AdjBinsHost {
    const double* node_sum; const double* pnu_bar; const double* dnu; const double* dcdm; const double* power;
    const long long* count; const int* compact; const double* F0sq;
    double* dprov_bar; double* rbar; double* Q; double* dc_sum;
    double norm, L3, fcdm;
    int nk, ld;  // dprov_bar has stride ld
};
size_t dnu_adj_smem(int ld, int wpb);

// ---- grid launchers (ksp_grid.cu)
struct GridGeom {
    int N, nrbins, slab0, nslab;
    long long nmodes;               // nslab * N * (N/2+1)
    int* thresh;                    // device [nrbins+1]: min k^2 of each bin
    float* w1;                      // device [N/2+1]: 1-D inverse CIC window (float)
    int* cmap;                      // device [nrbins]: bin -> compact index (-1 empty)
    float bin_c1;                   // binsperunit * ln2 / 2 (approximate bin estimate)
    unsigned* runtab = nullptr;     // device run table of the binning pass (or null)
    int run_Rp = 0;                 // its row length: runs per grid row, rounded up to 4
    int run_K = 0;                  // modes per run
    int beside = 0;                 // the integrator's preparation runs beside this binning pass
};
// the run table of a geometry (ksp_stream.cu): 0 built, 1 not applicable (2^15 bins or
// more, or over 1 GiB), -1 error
int build_run_table(GridGeom& g, cudaStream_t st);
// histogram of weighted mode counts over integer k^2 for the slab range
void launch_k2_histogram(int N, int slab0, int nslab, unsigned long long* hist, cudaStream_t st);
// K1: per-bin sum of w |F|^2 W^4 (double), and |F(0)|^2 when slab0 == 0
// returns 0 (TMA kernel), 1 (plain kernel) or -2 (launch error)
int launch_bin_power(const GridGeom& g, const float* grid, double* bin_sum, double* F0sq, unsigned* status, int tma,
                     int rows_per_cta, int stages, cudaStream_t st);
// K3: grid *= 1 + norm * interp(log k)
// Every variant leaves the grid as it is when the status word holds an error (kStAbort).
int launch_apply_correction(const GridGeom& g, float* grid, CorrTable corr, float lnscale, unsigned* status, int tma,
                            int rows_per_cta, int stages, cudaStream_t st, const float* in = nullptr,
                            const HostOut& host = HostOut{}, bool* delivered = nullptr);
// normalisation of K1's sums into P(k), delta_cdm, keff (powerspectrum.c:98-115,
// interface_gadget.c:96-100)
void launch_finalize_power(const double* bin_sum, const double* F0sq, const long long* count, const double* ksum,
                           const int* compact_bins, int nk, double BoxSize, double* power_out, double* keff_out,
                           double* dcdm_out, double* keffphys_out, cudaStream_t st,
                           const HostOut& host = HostOut{});

struct GridGeom;
void launch_adj_reduce(const GridGeom& gg, CorrTable corr, float lnscale, const float* gbar, const float* x,
                       double* node_sum, cudaStream_t st);
void launch_adj_rows(const IntegratorDev& I, const AdjBinsHost& h, const double* unit, const double* umass,
                     double* Dbar, double* mbar, int nk, int Na, int nspec, const int* spec_ids, cudaStream_t st);
void launch_adj_bins2(const AdjBinsHost& h, cudaStream_t st);
void launch_dnu_adj(const IntegratorDev& I, double* unit, double* umass, const double* ivals,
                    const int* nivals, int recompute, int nk, int Na, int nspec, const int* spec_ids, int wpb,
                    cudaStream_t st);
void launch_adj_grid(const GridGeom& gg, CorrTable corr, float lnscale, const float* gbar, const float* x, float* xbar,
                     const double* Q, const double* dc_sum, const double* F0sq, cudaStream_t st);

}  // namespace ksp
