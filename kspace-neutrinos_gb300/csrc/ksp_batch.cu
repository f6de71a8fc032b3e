// ksp_batch.cu -- many independent integrator instances advanced by one launch sequence.
//
// Every instance is a complete integrator (its own cosmology and masses, transfer table,
// history of its own length, its own k bins).  One batched call performs, for every
// instance, the same arithmetic as the single-instance kernels of ksp_integrator.cu --
// which follow get_delta_nu_update, delta_tot_table.c:193-250 -- so each instance's
// delta_nu is the one a single-instance call returns:
//   kb_prologue     block per instance: provisional history row (:222), call scalars,
//                   knot factorisation of the history spline
//   kb_fs_eval      a block per stretch of an instance's fslength segments
//   kb_tables       the fslength tables and the node tables of the integrand
//   kb_dtot_coeffs  thread per (instance, bin): history-row spline coefficients
//   kb_dnu_qag      persistent warps that pull (instance, species, bin) tasks from an
//                   atomic queue; knots, row and coefficients staged into shared memory
//                   by TMA bulk copies; QAG with the 61-point Gauss-Kronrod rule
//   kb_finish       thread per (instance, bin): species sum, commit, NaN check, clamp
//   kb_corr         block per bound grid: correction table (interface_common.c:134-146)
// All kernels run on fixed launch shapes and read the call's totals from device memory,
// so one captured CUDA graph serves every call.
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>
#include "ksp_batch.h"
#include "ksp_prep.cuh"
#include "ksp_ptx.cuh"

namespace ksp {

// largest i in [0, n) with off[i] <= v (off ascending, off[0] = 0)
__device__ __forceinline__ int owner_of(const int* off, int n, int v) {
    int lo = 0, hi = n;
    while (hi > lo + 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(off + mid) <= v) lo = mid; else hi = mid;
    }
    return lo;
}

constexpr int kBatchSmallBlocks = 4 * 152;

// ------------------------------------------------------------------ prologue
// The call scalars, update_delta_tot's provisional row (as k_update_row) and the knot
// factorisation.
__global__ void kb_prologue(BatchDev b) {
    if (blockIdx.x == 0 && threadIdx.x == 0) b.hdr->counter = 0;
    for (int i = blockIdx.x; i < b.M; i += gridDim.x) {
        const BatchCall& P = b.calls[i];
        __syncthreads();  // the previous instance's scalars are complete
        if (!P.active) continue;
        const IntegratorDev& I = b.insts[i];
        StepScalars& S = *I.sc;
        const double a = P.a;
        const int Na = P.Na;
        const bool integrate = P.commit_row != -2;
        if (threadIdx.x < 32) call_scalars_warp(*I.B, a, P.loga, P.loga0, P.TimeTransfer, integrate ? Na : 1, S);
        if (threadIdx.x == 0 && integrate) I.scalefact[Na - 1] = P.loga;
        __syncthreads();
        if (!integrate) continue;
        const double OmegaNua3 = S.OmegaNua3, OmegaNu1 = S.OmegaNu1, partnu = S.partnu, Omeganonu = S.Omeganonu;
        for (int ik = threadIdx.x; ik < P.nk; ik += blockDim.x)
            I.dtot[(size_t)ik * I.ld + Na - 1] =
                get_delta_tot(I.nu_last[ik], I.dcdm[ik], OmegaNua3, Omeganonu, OmegaNu1, partnu);
        const double* xk = I.scalefact;
        for (int j = threadIdx.x; j + 1 < Na; j += blockDim.x) {
            const double h = xk[j + 1] - xk[j];
            I.knot_invh[j] = 1.0 / h;
            I.knot_h3[j] = h / 3.0;
            I.knot_ih3[j] = 1.0 / (3.0 * h);
        }
        auto knot = [&](int j) { return xk[j]; };
        for (int r = (P.start_row < 0 ? 0 : P.start_row) + threadIdx.x; r < Na - 2; r += blockDim.x)
            knot_row(knot, r, I.knot_invdiag, I.knot_fac);
        if (threadIdx.x == 0 && P.nfs == 0) {
            S.fsl_A0a = 0.0;
            S.Nfs = 0;
        }
    }
}

// ------------------------------------------------------------------ fslength table
struct GL4b { double x[2], w[2]; };

// the stretches of all instances' segments (flat, so that instances of any length balance),
// as k_prep_eval
__global__ void __launch_bounds__(kPrepThreads) kb_fs_eval(BatchDev b, GL4b gl) {
    __shared__ double f[kPrepThreads], sg[kPrepThreads];
    const int total = b.hdr->total_segs;
    for (int g = blockIdx.x; g < total; g += gridDim.x) {
        const int i = owner_of(b.fs_off, b.M, g);
        const BatchCall& P = b.calls[i];
        const IntegratorDev& I = b.insts[i];
        __syncthreads();  // the previous stretch's shared arrays
        fs_eval_block(*I.B, P.nfs, P.loga0, P.loga, g - __ldg(b.fs_off + i), gl.x[0], gl.x[1], gl.w[0], gl.w[1], f, sg,
                      I.fs_seg, I.fs_suf, I.fs_tot);
    }
}

// the fslength tables and the node tables, 128 nodes per block, as k_prep_tables
__global__ void __launch_bounds__(kBatchTable) kb_tables(BatchDev b) {
    __shared__ double tsuf[kPrepThreads + 1];
    const int total = b.hdr->total_fsc;
    for (int g = blockIdx.x; g < total; g += gridDim.x) {
        const int i = owner_of(b.fsc_off, b.M, g);
        const BatchCall& P = b.calls[i];
        const IntegratorDev& I = b.insts[i];
        int blk = g - __ldg(b.fsc_off + i);
        __syncthreads();  // the previous table's sums
        const FsTable F = fs_table(I, P.nfs, P.loga0, P.loga, I.sc->light, tsuf);
        const int table_blocks = (P.nfs + kBatchTable - 1) / kBatchTable;
        if (blk < table_blocks) {
            const int n = blk * kBatchTable + threadIdx.x;
            if (n >= P.nfs) continue;
            I.fs_x[n] = fs_node(n, P.nfs, P.loga0, P.loga);
            const double y = fs_table_y(F, n);
            I.fs_y[n] = y;
            I.fs_c[n] = fs_table_c(F, n);
            if (n == 0) {
                I.sc->fsl_A0a = y;
                I.sc->Nfs = P.nfs;
            }
            continue;
        }
        const int q = (blk - table_blocks) * kBatchTable + threadIdx.x;
        if (q >= b.nc_slots * 61) continue;
        double half;
        const double x = nc_node_x(q, P.loga0, P.loga, &half);
        const double fsl = fs_table_at(F, P.loga0, P.loga, x);
        const int j = seg_bsearch(I.scalefact, P.Na, x);
        nc_store(I, q, fsl, node_inv_aH(I.B, x), x - I.scalefact[j], j, I.scalefact[j + 1] - I.scalefact[j], P.Na, half);
    }
}

// ------------------------------------------------------------------ history splines
// thread per (instance, bin): the same substitutions as k_dtot_coeffs, each thread
// sweeping its own row in global memory.  With a million rows in flight the latency of
// the strided loads is hidden by parallelism, which a warp-per-row solve (one active
// lane per row) cannot match at this size.
__global__ void kb_dtot_coeffs(BatchDev b) {
    const int total = b.hdr->total_bins;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        const int i = owner_of(b.bin_off, b.M, g);
        const int ik = g - __ldg(b.bin_off + i);
        const BatchCall& P = b.calls[i];
        const int Na = P.Na;
        if (!P.active || P.commit_row == -2 || Na <= 2) continue;
        const IntegratorDev& I = b.insts[i];
        const double* y = I.dtot + (size_t)ik * I.ld;
        double* c = I.coef + (size_t)ik * I.ld;
        const double* ih = I.knot_invh;
        const int m = Na - 2;
        double prev = 0;
        for (int k = 0; k < m; k++) {
            double r = 3.0 * ((y[k + 2] - y[k + 1]) * ih[k + 1] - (y[k + 1] - y[k]) * ih[k]);
            if (k > 0) r -= I.knot_fac[k] * prev;
            prev = r;
            c[k + 1] = r;
        }
        c[0] = 0.0;
        c[Na - 1] = 0.0;
        double next = c[m] * I.knot_invdiag[m - 1];
        c[m] = next;
        const double* x = I.scalefact;
        for (int k = m - 1; k-- > 0;) {
            const double off = x[k + 2] - x[k + 1];
            next = (c[k + 1] - off * next) * I.knot_invdiag[k];
            c[k + 1] = next;
        }
    }
}

size_t batch_qag_smem(int ldmax, int wpb) {
    return ((sizeof(Gk61Nodes) + 15) & ~size_t(15)) + wpb * (sizeof(QagList) + 2 * sizeof(double) * ldmax) +
           wpb * sizeof(uint64_t);
}

// Shared memory: Gk61Nodes | per warp: QagList, row[ldmax], coef[ldmax] | mbarriers
__global__ void __launch_bounds__(128) kb_dnu_qag(BatchDev b) {
    extern __shared__ __align__(16) unsigned char sm[];
    Gk61Nodes& N = *reinterpret_cast<Gk61Nodes*>(sm);
    const size_t off = (sizeof(Gk61Nodes) + 15) & ~size_t(15);
    const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t per_warp = sizeof(QagList) + 2 * sizeof(double) * b.ldmax;
    unsigned char* wbase = sm + off + warp * per_warp;
    QagList& L = *reinterpret_cast<QagList*>(wbase);
    double* row = reinterpret_cast<double*>(wbase + sizeof(QagList));
    double* rc = row + b.ldmax;
    uint64_t* mybar = reinterpret_cast<uint64_t*>(sm + off + nw * per_warp) + warp;
    gk61_fill(N, threadIdx.x, blockDim.x);
    if (lane == 0) ptx::mbar_init(mybar, 1);
    ptx::mbar_init_fence();
    __syncthreads();
    const int total = b.hdr->total_tasks;
    unsigned phase = 0;
    for (;;) {
        int task = 0;
        if (lane == 0) task = atomicAdd(&b.hdr->counter, 1);
        task = __shfl_sync(0xffffffffu, task, 0);
        if (task >= total) break;
        const int i = owner_of(b.task_off, b.M, task);
        const int loc = task - __ldg(b.task_off + i);
        const BatchCall& P = b.calls[i];
        const IntegratorDev& I = b.insts[i];
        const int nk = P.nk;
        const int si = loc / nk, ik = loc - si * nk;
        const int mi = P.spec[si];
        const StepScalars& S = *I.sc;
        const int Na = P.Na;
        const double k = I.wavenum[ik];
        const bool integrate = !S.skip_integral && Na > 1 && S.inv_m[mi] > 0;
        if (integrate) {
            __syncwarp();
            if (lane == 0) {
                const unsigned bytes = (unsigned)(((Na + 1) & ~1) * sizeof(double));
                ptx::fence_async_smem();
                ptx::mbar_expect_tx(mybar, Na > 2 ? 2 * bytes : bytes);
                ptx::bulk_g2s(row, I.dtot + (size_t)ik * I.ld, bytes, mybar);
                if (Na > 2) ptx::bulk_g2s(rc, I.coef + (size_t)ik * I.ld, bytes, mybar);
            }
            if (Na == 2 && lane < 2) rc[lane] = 0.0;  // linear: no coefficients
        }
        double val = lane == 0 ? dnu_initial(I, S, ik, mi, k) : 0.0;
        if (integrate) {
            const bool got = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(mybar, phase));  // warp-uniform
            phase ^= 1;
            if (!got) {
                if (lane == 0) atomicOr(I.status, kStTimeout);
                ptx::mbar_wait_bounded(mybar, phase ^ 1);  // the copies still in flight
                return;
            }
            __syncwarp();
            const DnuIntegrandW f = dnu_integrand_w(I, S, mi, k * S.inv_m[mi], row, rc, Na);
            const QagResult r = qag_warp_c(f, N, L, S.loga0, S.loga, 0.0, S.relerr, kQagLimit);
            val += S.prefac * r.result;
            if (!r.ok && lane == 0) atomicOr(I.status, kStGsl);
        }
        if (lane == 0) I.dnu_s[(size_t)mi * I.nk_alloc + ik] = val;
    }
}

// ------------------------------------------------------------------ finish
// k_combine + k_finish for every bin of every instance
__global__ void kb_finish(BatchDev b) {
    const int total = b.hdr->total_bins;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        const int i = owner_of(b.bin_off, b.M, g);
        const int ik = g - __ldg(b.bin_off + i);
        const BatchCall& P = b.calls[i];
        if (!P.active) continue;
        const IntegratorDev& I = b.insts[i];
        const StepScalars& S = *I.sc;
        double out;
        if (P.commit_row == -2) {
            out = I.nu_last[ik];  // same scale factor: delta_nu_last as it is
            I.dnu[ik] = out;
        } else {
            double v = 0;
            for (int mi = 0; mi < kNuSpecies; mi++)
                if (S.wnu[mi] != 0.0) v += I.dnu_s[(size_t)mi * I.nk_alloc + ik] * S.wnu[mi];
            I.dnu[ik] = v;
            if (!P.dry) I.nu_last[ik] = v;
            if (P.commit_row >= 0 && !P.dry) {
                if (ik == 0) I.scalefact[P.commit_row] = P.loga;
                I.dtot[(size_t)ik * I.ld + P.commit_row] =
                    get_delta_tot(v, I.dcdm[ik], S.OmegaNua3, S.Omeganonu, S.OmegaNu1, S.partnu);
            }
            if (isnan(v)) atomicOr(I.status, kStDnuNaN);
            out = v < 0 ? 0.0 : v;
        }
        b.dnu_pool[__ldg(b.bin_off + i) + ik] = out;
    }
}

// correction tables of the bound grids (the table part of k_finish)
__global__ void kb_corr(BatchDev b, const BatchGridCorr* grids, int ngrid) {
    for (int gi = blockIdx.x; gi < ngrid; gi += gridDim.x) {
        const BatchGridCorr G = grids[gi];
        const BatchCall& P = b.calls[G.inst];
        if (!P.active) continue;
        const IntegratorDev& I = b.insts[G.inst];
        const double norm = I.sc->kspace_prefac;
        const double* dnu_out = b.dnu_pool + b.bin_off[G.inst];
        const int nk = P.nk;
        if (threadIdx.x == 0 && G.norm_out) *G.norm_out = norm;
        for (int j = threadIdx.x; j < nk; j += blockDim.x) {
            const double lk = log(G.keff[j]);
            const double r = dnu_out[j] / I.dcdm[j];
            G.corr.xf[j] = (float)lk;
            G.corr.rn[j] = (float)(norm * r);
            double s = 0;
            if (j + 1 < nk) {
                const double lk1 = log(G.keff[j + 1]);
                const double r1 = dnu_out[j + 1] / I.dcdm[j + 1];
                s = norm * (r1 - r) / (lk1 - lk);
            }
            G.corr.sn[j] = (float)s;
            if (!isfinite(norm * r) || !isfinite(s)) atomicOr(I.status, kStGridNaN);
        }
    }
}

// ------------------------------------------------------------------ launchers
static void gl_nodes_b(int n, double* X, double* Wt) {  // Newton on P_n, positive half
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

void batch_set_attributes() {
    raise_dynamic_smem_limit(reinterpret_cast<const void*>(kb_dnu_qag));
}

void launch_batch_update(const BatchDev& b, cudaStream_t st) {
    static GL4b gl;
    static bool init = false;
    if (!init) {
        gl_nodes_b(4, gl.x, gl.w);
        init = true;
    }
    const int nb = kBatchSmallBlocks;
    kb_prologue<<<b.M < nb ? b.M : nb, 128, 0, st>>>(b);
    kb_fs_eval<<<4 * nb, kPrepThreads, 0, st>>>(b, gl);
    kb_tables<<<2 * nb, kBatchTable, 0, st>>>(b);
    kb_dtot_coeffs<<<nb, 128, 0, st>>>(b);
    kb_dnu_qag<<<b.qag_blocks, 32 * b.wpb, batch_qag_smem(b.ldmax, b.wpb), st>>>(b);
    kb_finish<<<nb, 256, 0, st>>>(b);
}

void launch_batch_corr(const BatchDev& b, const BatchGridCorr* g, int ngrid, cudaStream_t st) {
    if (ngrid > 0) kb_corr<<<ngrid, 256, 0, st>>>(b, g, ngrid);
}

}  // namespace ksp
