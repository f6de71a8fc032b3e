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
//   kb_dtot_coeffs  warp per 32 bins of an instance: history-row spline coefficients
//   kb_dnu_qag      persistent warps that pull (instance, species, bin) tasks from an
//                   atomic queue; row and coefficients staged into shared memory by
//                   TMA bulk copies; QAG with the 61-point Gauss-Kronrod rule
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
        if (threadIdx.x == 0 && integrate) {
            I.scalefact[Na - 1] = P.loga;
            if (Na > 1 && no_number(P.loga)) atomicOr(I.status, kStGsl);
        }
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
        if (threadIdx.x == 0 && P.fs.n == 0) {
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
        fs_eval_block(*I.B, P.fs, P.loga, g - __ldg(b.fs_off + i), gl.x[0], gl.x[1], gl.w[0], gl.w[1], f, sg,
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
        const FsTable F = fs_table(I, P.fs, I.sc->light, tsuf);
        const int table_blocks = fs_table_blocks(P.fs.n, kBatchTable);
        if (blk < table_blocks) {
            fs_table_store(I, F, blk * kBatchTable + threadIdx.x);
            continue;
        }
        const int q = (blk - table_blocks) * kBatchTable + threadIdx.x;
        if (q >= b.nc_slots * 61) continue;
        double half;
        const double x = nc_node_x(q, NcLayout{b.nc_slots, 1}, P.loga0, P.loga, &half);
        const double fsl = fs_table_at(F, x);
        const int j = seg_bsearch(I.scalefact, P.Na, x);
        nc_store(I, q, fsl, node_inv_aH(I.B, x), x - I.scalefact[j], j, I.scalefact[j + 1] - I.scalefact[j],
                 I.knot_invh[j], P.Na, half);
    }
}

// ------------------------------------------------------------------ history splines
// A warp per 32 rows of one instance, a lane per row, 32 knots at a time: the rows' next 32
// values are on their way to shared memory (lane = knot: whole lines) while the lanes step
// through the present ones.  With g_k = r_k / diag_k the forward step is
//   g_k = A_k (y_{k+2} - y_{k+1}) + B_k (y_{k+1} - y_k) + W_k g_{k-1}
// and the backward one c_k = g_k + V_k c_{k+1}, the factors of a knot formed by one lane for
// all rows: five FP64 operations per knot and row, which is the bound (a row by the warp's
// scans costs twice that, a thread per row with its row in global memory waits for every
// knot: 256 members 687 us, now 330 to 380).
constexpr int kRowTile = 32, kRowPitch = kRowTile + 1, kRowWarps = 4;
struct RowSmem {
    double y[2][32 * kRowPitch];  // [row][knot of the tile], a pitch free of bank conflicts
    double2 ab[kRowTile], wv[kRowTile];
};
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(ptx::smem_u32(dst)), "l"(src) : "memory");
}
__global__ void __launch_bounds__(32 * kRowWarps) kb_dtot_coeffs(BatchDev b) {
    extern __shared__ __align__(16) unsigned char sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    RowSmem& sh = reinterpret_cast<RowSmem*>(sm)[warp];
    const int total = b.hdr->total_rows;
    for (int g = blockIdx.x * kRowWarps + warp; g < total; g += gridDim.x * kRowWarps) {
        const int i = owner_of(b.row_off, b.M, g);
        const BatchCall& P = b.calls[i];
        const IntegratorDev& I = b.insts[i];
        const int Na = P.Na, m = Na - 2, nt = (m + kRowTile - 1) / kRowTile;  // Na > 2
        const int r0 = 32 * (g - __ldg(b.row_off + i)), nr = min(32, P.nk - r0);
        const double* y = I.dtot + (size_t)r0 * I.ld;
        double* c = I.coef + (size_t)r0 * I.ld;
        const int my = min(lane, nr - 1);
        // knots k0 + 2 .. k0 + 33 of the rows (the unknowns k0 + 1 .. k0 + 32 with them)
        auto fetch = [&](int t, const double* src, int first, int buf) {
            const int k = kRowTile * t + lane;
            if (k < m)
                for (int r = 0; r < nr; r++)
                    cp_async8(&sh.y[buf][r * kRowPitch + lane], src + (size_t)r * I.ld + first + k);
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        auto arrived = [&](bool later) {
            if (later) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
        };
        // the factors of unknown k (of a tile, by its lane; zero past the last): what they are made
        // of is read a tile ahead
        double kinv, kih0, kih1, kx0, kx1, kx2;
        auto knots = [&](int t) {
            const int k = min(max(kRowTile * t + lane, 0), m - 1);
            kinv = I.knot_invdiag[k];
            kih0 = I.knot_invh[k];
            kih1 = I.knot_invh[k + 1];
            kx0 = I.scalefact[k];
            kx1 = I.scalefact[k + 1];
            kx2 = I.scalefact[k + 2];
        };
        auto factors = [&](int t) {
            const bool in = kRowTile * t + lane < m;
            const double i3 = 3.0 * kinv;
            sh.ab[lane] = in ? make_double2(i3 * kih1, -i3 * kih0) : make_double2(0.0, 0.0);
            sh.wv[lane] = in ? make_double2((kx0 - kx1) * kinv, (kx1 - kx2) * kinv) : make_double2(0.0, 0.0);
        };
        auto store = [&](int t, int buf) {
            const int k = kRowTile * t + lane;
            if (k < m)
                for (int r = 0; r < nr; r++) c[(size_t)r * I.ld + 1 + k] = sh.y[buf][r * kRowPitch + lane];
            __threadfence_block();  // read back by an asynchronous copy
        };
        __syncwarp();  // the previous group's reads
        fetch(0, y, 2, 0);
        knots(0);
        const double* yr = y + (size_t)my * I.ld;
        double y1 = yr[1], d0 = y1 - yr[0], gp = 0.0;
        for (int t = 0; t < nt; t++) {
            const int buf = t & 1, n = min(kRowTile, m - kRowTile * t);
            if (t + 1 < nt) fetch(t + 1, y, 2, buf ^ 1);
            factors(t);
            knots(t + 1 < nt ? t + 1 : t - 1);  // (the last tile turns round)
            arrived(t + 1 < nt);
            __syncwarp();
            double* q = sh.y[buf] + my * kRowPitch;
            if (lane < nr) {
                // (four knots' operands are read while the four before are worked on)
                double2 ab[4];
                double w[4], y2[4];
                auto operands = [&](int k) {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        ab[u] = sh.ab[k + u];
                        w[u] = sh.wv[k + u].x;
                        y2[u] = q[k + u];
                    }
                };
                operands(0);
                for (int k = 0; k < n; k += 4) {
                    double r[4], v[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const double d1 = y2[u] - y1;
                        r[u] = fma(ab[u].x, d1, ab[u].y * d0);
                        v[u] = w[u];
                        y1 = y2[u];
                        d0 = d1;
                    }
                    operands(k + 4 < kRowTile ? k + 4 : 0);
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        gp = fma(v[u], gp, r[u]);
                        q[k + u] = k + u < n ? gp : 0.0;
                    }
                }
            }
            __syncwarp();
            if (t + 1 < nt) store(t, buf);  // the last one stays
            __syncwarp();
        }
        double next = 0.0;
        for (int t = nt - 1; t >= 0; t--) {
            const int buf = t & 1, n = min(kRowTile, m - kRowTile * t);
            if (t > 0) fetch(t - 1, c, 1, buf ^ 1);
            if (t < nt - 1) {
                factors(t);
                knots(t - 1);
            }
            arrived(t > 0);
            __syncwarp();
            double* q = sh.y[buf] + my * kRowPitch;
            if (lane < nr) {
                double v[4], gk[4];
                auto operands = [&](int k) {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        v[u] = sh.wv[k + u].y;
                        gk[u] = q[k + u];
                    }
                };
                operands((n - 1) & ~3);
                for (int k = (n - 1) & ~3; k >= 0; k -= 4) {
                    double r[4], p[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        p[u] = v[u];
                        r[u] = gk[u];
                    }
                    operands(k >= 4 ? k - 4 : 0);
#pragma unroll
                    for (int u = 3; u >= 0; u--) {
                        next = fma(p[u], next, r[u]);
                        q[k + u] = next;
                    }
                }
            }
            __syncwarp();
            store(t, buf);
            __syncwarp();
        }
        if (lane < nr) c[(size_t)lane * I.ld] = c[(size_t)lane * I.ld + Na - 1] = 0.0;
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
    raise_dynamic_smem_limit(reinterpret_cast<const void*>(kb_dtot_coeffs));
}

// The tables keep the FP64 pipes busy, the prologue and the row splines wait for their serial
// chains: side by side, segments | prologue (and the binning of bound grids before it), then
// tables | splines (a call of 256 members: 3853 us one after the other, 3720 so).
cudaError_t launch_batch_segments(const BatchDev& b, const BatchStreams& s) {
    static const GL4b gl = [] {
        GL4b g;
        gl_nodes_b(4, g.x, g.w);
        return g;
    }();
    cudaError_t e = cudaEventRecord(s.start, s.main);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s.side, s.start, 0);
    if (e == cudaSuccess) kb_fs_eval<<<4 * kBatchSmallBlocks, kPrepThreads, 0, s.side>>>(b, gl);
    return e;
}
cudaError_t launch_batch_update(const BatchDev& b, const BatchStreams& s) {
    const int nb = kBatchSmallBlocks;
    const cudaStream_t st = s.main;
    kb_prologue<<<b.M < nb ? b.M : nb, 128, 0, st>>>(b);
    cudaError_t e = cudaEventRecord(s.prologue, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s.side, s.prologue, 0);
    kb_tables<<<2 * nb, kBatchTable, 0, s.side>>>(b);
    if (e == cudaSuccess) e = cudaEventRecord(s.tables, s.side);
    kb_dtot_coeffs<<<nb, 32 * kRowWarps, kRowWarps * sizeof(RowSmem), st>>>(b);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, s.tables, 0);
    if (e != cudaSuccess) return e;
    kb_dnu_qag<<<b.qag_blocks, 32 * b.wpb, batch_qag_smem(b.ldmax, b.wpb), st>>>(b);
    kb_finish<<<nb, 256, 0, st>>>(b);
    return cudaPeekAtLastError();
}

void launch_batch_corr(const BatchDev& b, const BatchGridCorr* g, int ngrid, cudaStream_t st) {
    if (ngrid > 0) kb_corr<<<ngrid, 256, 0, st>>>(b, g, ngrid);
}

}  // namespace ksp
