// Jacobi-CG with the system resident on chip (included by cg.cu): the CTA's rows of the
// matrix stay in shared memory and its parts of the Krylov vectors in registers for the
// whole solve.  Only z, which other CTAs gather, goes through global memory (L2).
//
// For systems that fit (152 x 210 KB of shared memory: about 375,000 rows of a hex mesh in
// FP64, 560,000 in FP32).  There an iteration of the streaming kernels is bound by latency:
// tiles that pass through a shared-memory ring although they never leave the chip's reach,
// and two grid reductions, each a chain of L2 round trips.  Here an iteration is
//   S  w = A z, p = z + beta p, q = w + beta q, p.q     (matrix and own z from shared memory)
//   X  x += alpha p, r -= alpha q, z = M^-1 r, r.r, r.z (registers only)
// with one all-to-all grid sum each (grid_all.cuh).  Rows are dealt to all SMs, one warp a
// 32-row slice, R slices a warp.  Same recurrences, FMA order within a row, stopping test
// and reported figures as k_cg_pipe / k_cg_mixed_pipe.
//
// Measured, us per iteration, streaming kernels before -> here: 13,824 rows of a hex mesh in
// FP64 13.2 -> 6.1 (two sums of 2 us, the FP64 latencies of a row and of alpha; an idle thread
// forms 1 / rho during the first sum), 256,000 rows 19.3 -> 12.8 (5.7 us of it FP64 pipe);
// 262,144 rows in FP32 16.2 -> 7.7.  The line to the streaming kernels is the shared memory: there is no size
// that fits and was faster streamed.
#pragma once

#include "grid_all.cuh"

namespace sysu {
namespace {

constexpr int CR_NT = 512;                     // 16 warps: enough for the FP64 pipe, few to reduce
constexpr unsigned CR_SMEM = 210 * 1024;       // dynamic shared memory a CTA may take

// channels of the grid sums (grid_all.cuh)
enum CgChannel { CH_PQ = 0, CH_RZ = 1, CH_RR = 3, CH_INIT = 4, CH_UPD = 7 };

struct CgResArgs {
    SellView A;             // FP64 values
    const float *val32;     // FP32 values (mixed)
    const double *b;
    double *x;
    double *z;              // FP64 exchange vector
    float *z32;             // FP32 exchange vector (mixed)
    double omega;           // Jacobi weight; jacobi 0: no preconditioner
    int jacobi;
    int x0_zero;
    unsigned long long *slots;
    SolveInfo *info;
    int maxit;
    double eps, inner_tol;
    unsigned long long *ts;
    int ld;                 // rows a CTA has room for (the stride of its matrix columns)
    const SolveInfo *gate;  // as CgPipeArgs::gate
};

// The CTA's matrix rows in shared memory, column-major (entry k of local row j at k ld + j).
// Columns inside the CTA's own rows become local indices, the others ~column.
template <class V>
struct ResMatrix {
    V *val, *z;
    int *col;
    int ld;
    __device__ ResMatrix(int wmax, int ld_) : ld(ld_) {
        val = reinterpret_cast<V *>(g_slots);
        z = val + (size_t)wmax * ld;
        col = reinterpret_cast<int *>(z + ld);
    }
};

// w = A z for local row j with wd entries: the CTA's own z from shared memory, the others'
// from global memory; up to 8 gathers in flight, FMAs in entry order
template <class V>
__device__ __forceinline__ V res_row(const ResMatrix<V> &M, int j, int wd, const V *zg) {
    V xv[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (k < wd) {
            const int c = M.col[k * M.ld + j];
            xv[k] = c >= 0 ? M.z[c] : zg[~c];
        }
    V acc = wd > 0 ? M.val[j] * xv[0] : (V)0;
#pragma unroll
    for (int k = 1; k < 8; ++k)
        if (k < wd) acc = fma_t(M.val[k * M.ld + j], xv[k], acc);
    for (int k = 8; k < wd; ++k) {
        const int c = M.col[k * M.ld + j];
        acc = fma_t(M.val[k * M.ld + j], c >= 0 ? M.z[c] : zg[~c], acc);
    }
    return acc;
}

// Loads the CTA's rows R0 .. R0+nrow-1; wd[u] = entries of the thread's u-th row (0: none).
template <class V, int R>
__device__ __forceinline__ void res_load(const ResMatrix<V> &M, const SellView &A, const V *val, int R0, int nrow,
                                         int (&wd)[R]) {
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int j = threadIdx.x + u * CR_NT;
        wd[u] = 0;
        if (j >= nrow) continue;
        const int s = (R0 + j) >> 5;
        const int e = __ldg(A.sl_ptr + s) + (j & 31);
        wd[u] = __ldg(A.sl_w + s);
        for (int k = 0; k < wd[u]; ++k) {
            const int c = __ldg(A.col + e + 32 * k);
            M.val[k * M.ld + j] = val[e + 32 * k];
            M.col[k * M.ld + j] = (unsigned)(c - R0) < (unsigned)nrow ? c - R0 : ~c;
        }
    }
}

template <int R>
__global__ void __launch_bounds__(CR_NT, 1) k_cg_res(CgResArgs a, int wmax) {
    if (a.gate && a.gate->status[0] != DEV_STALLED) return;  // the same word for every block
    const int it_before = a.gate ? a.gate->iters[0] : 0;
    const int tid = threadIdx.x;
    int *err = &a.info->err;
    const int sb = (int)((long long)a.A.nslices * blockIdx.x / gridDim.x);
    const int se = (int)((long long)a.A.nslices * (blockIdx.x + 1) / gridDim.x);
    const int R0 = sb * 32, nrow = min(se * 32, a.A.n) - R0;
    AllCtx c = all_ctx(a.slots);
    all_init();
    const ResMatrix<double> M(wmax, a.ld);
    int wd[R];
    res_load<double, R>(M, a.A, a.A.val, R0, nrow, wd);
    double x[R], r[R], p[R], q[R], d[R];
    double v3[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int j = tid + u * CR_NT;
        x[u] = r[u] = p[u] = q[u] = d[u] = 0.0;
        if (j >= nrow) continue;
        const int i = R0 + j;
        d[u] = a.jacobi ? a.omega / M.val[j] : 1.0;
        const double bi = a.b[i];
        double ax = 0.0;
        if (!a.x0_zero) {
            x[u] = a.x[i];
            ax = row_dot(a.A, i, a.x);
        }
        r[u] = bi - ax;
        const double z = d[u] * r[u];
        M.z[j] = z;
        a.z[i] = z;
        v3[0] = fma(bi, bi, v3[0]);
        v3[1] = fma(r[u], r[u], v3[1]);
        v3[2] = fma(r[u], z, v3[2]);
    }
    if (!all_sum<3>(v3, CH_INIT, c, err)) return;
    // thread-0 scalar state in shared memory
    __shared__ double s_bb, s_rr, s_rho, s_thr, s_unit, s_inv;
    __shared__ int s_bias, s_rr_est;
    if (tid == 0) {
        s_bb = g_ax_sum[0] == 0.0 ? 1.0 : g_ax_sum[0];
        s_thr = a.eps * a.eps * s_bb;
        s_rr = g_ax_sum[1];
        s_rho = g_ax_sum[2];
        g_bc[0] = stop_code(s_rr, s_thr);
        g_bc[1] = 0.0;
        // r.r estimated in FP32 in units of 2^2k ~ thr (see k_cg_pipe); 0: thr unusable
        s_bias = 0;
        s_rr_est = 0;
        if (s_thr > 0.0 && isfinite(s_thr)) {
            const int e = ilogb(s_thr);
            const int k = e >= 0 ? e / 2 : -((1 - e) / 2);  // floor(e / 2)
            if (k > -900 && k < 900) {
                s_bias = 1023 + k - 127;
                s_unit = ldexp(1.0, 2 * k);
            }
        }
    }
    __syncthreads();
    const int bias = s_bias;
    auto exact_rr = [&]() -> bool {
        double e1[1] = {0.0};
#pragma unroll
        for (int u = 0; u < R; ++u) e1[0] = fma(r[u], r[u], e1[0]);
        return all_sum<1>(e1, CH_RR, c, err);
    };
    int it = 0, status = DEV_OK;
    bool ok = true;
    for (;;) {
        const double code = g_bc[0], beta = g_bc[1];
        if (code == 1.0 || it >= a.maxit) break;
        if (code == 2.0) { status = DEV_NONFINITE; break; }
        ++it;
        stamp(a.ts, it, 0);
        double v1[1] = {0.0};
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = tid + u * CR_NT;
            if (j >= nrow) continue;
            const double w = res_row<double>(M, j, wd[u], a.z);
            p[u] = fma_t(beta, p[u], M.z[j]);
            q[u] = fma_t(beta, q[u], w);
            v1[0] = fma_t(p[u], q[u], v1[0]);
        }
        if (!all_sum<1>(v1, CH_PQ, c, err, [&](int, double pq) {
                g_bc[2] = pq == 0.0 ? 0.0 : s_rho / pq;
                g_bc[3] = pq == 0.0 ? 1.0 : 0.0;
            }, [&] { s_inv = recip(s_rho); })) { ok = false; break; }
        stamp(a.ts, it, 1);
        if (g_bc[3] != 0.0) { status = DEV_BREAKDOWN; break; }
        const double alpha = g_bc[2];
        double v2[2] = {0.0, 0.0};
        float rr32 = 0.f;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = tid + u * CR_NT;
            if (j >= nrow) continue;
            x[u] = fma_t(alpha, p[u], x[u]);
            r[u] = fma_t(-alpha, q[u], r[u]);
            const double z = d[u] * r[u];
            M.z[j] = z;
            a.z[R0 + j] = z;
            if (bias) {
                const float f = scaled_abs_f32(r[u], bias);
                rr32 = fmaf(f, f, rr32);
            } else {
                v2[0] = fma_t(r[u], r[u], v2[0]);
            }
            v2[1] = fma_t(r[u], z, v2[1]);
        }
        if (bias) v2[0] = (double)rr32;
        if (!all_sum<2>(v2, CH_RZ, c, err, [&](int k, double sum) {
                if (k == 1) {
                    g_bc[1] = quotient(sum, s_rho, s_inv);
                    s_rho = sum;
                } else if (bias) {
                    // the estimate decides only when it is clearly above the threshold
                    s_rr = sum * s_unit;
                    s_rr_est = 1;
                    g_bc[5] = s_rr >= s_thr * 1.001 ? 0.0 : 1.0;  // 1: take the exact r.r (NaN included)
                    g_bc[0] = 0.0;
                } else {
                    s_rr = sum;
                    g_bc[0] = stop_code(s_rr, s_thr);
                    g_bc[5] = 0.0;
                }
            })) { ok = false; break; }
        stamp(a.ts, it, 2);
        if (g_bc[5] != 0.0) {
            if (!exact_rr()) { ok = false; break; }
            if (tid == 0) {
                s_rr = g_ax_sum[0];
                s_rr_est = 0;
                g_bc[0] = stop_code(s_rr, s_thr);
            }
            __syncthreads();
        }
    }
    __syncthreads();
    const int est = s_rr_est;
    if (est && ok && exact_rr() && tid == 0) s_rr = g_ax_sum[0];  // the reported residual is exact
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int j = tid + u * CR_NT;
        if (j < nrow) a.x[R0 + j] = x[u];
    }
    if (blockIdx.x == 0 && tid == 0) {
        const double res = sqrt(s_rr) / sqrt(s_bb);
        if (status == DEV_OK && !(s_rr < s_thr)) status = isfinite(s_rr) ? DEV_MAXITER : DEV_NONFINITE;
        a.info->status[0] = status;
        a.info->iters[0] = it_before + it;
        a.info->res[0] = res;
    }
}

// Mixed precision (see k_cg_mixed_pipe): p, q, r and the correction e of the FP32
// recurrences in registers, the FP32 matrix in shared memory; the reliable updates read the
// FP64 matrix and x from global memory.
template <int R>
__global__ void __launch_bounds__(CR_NT, 1) k_cg_mixed_res(CgResArgs a, int wmax) {
    const int tid = threadIdx.x;
    int *err = &a.info->err;
    const int sb = (int)((long long)a.A.nslices * blockIdx.x / gridDim.x);
    const int se = (int)((long long)a.A.nslices * (blockIdx.x + 1) / gridDim.x);
    const int R0 = sb * 32, nrow = min(se * 32, a.A.n) - R0;
    AllCtx c = all_ctx(a.slots);
    all_init();
    const ResMatrix<float> M(wmax, a.ld);
    int wd[R];
    res_load<float, R>(M, a.A, a.val32, R0, nrow, wd);
    float r[R], p[R], q[R], e[R], d[R];
    __shared__ double s_bb, s_thr, s_rho, s_rz, s_rr, s_sig, s_sig_next, s_inv;
    __shared__ int s_stalls;
    {
        double r64[R], v2[2] = {0.0, 0.0};
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = tid + u * CR_NT;
            r64[u] = 0.0;
            r[u] = p[u] = q[u] = e[u] = d[u] = 0.f;
            if (j >= nrow) continue;
            const int i = R0 + j;
            d[u] = (float)(a.omega / a.A.val[__ldg(a.A.sl_ptr + (i >> 5)) + (i & 31)]);
            const double bi = a.b[i];
            r64[u] = bi - row_dot(a.A, i, a.x);
            v2[0] = fma(bi, bi, v2[0]);
            v2[1] = fma(r64[u], r64[u], v2[1]);
        }
        if (!all_sum<2>(v2, CH_INIT, c, err)) return;
        if (tid == 0) {
            s_bb = g_ax_sum[0] == 0.0 ? 1.0 : g_ax_sum[0];
            s_thr = a.eps * a.eps * s_bb;
            s_rr = g_ax_sum[1];
            s_sig = pow2_scale(s_rr);
            s_stalls = 0;
        }
        __syncthreads();
        const double sg = s_sig;
        float f2 = 0.f;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = tid + u * CR_NT;
            if (j >= nrow) continue;
            r[u] = (float)(sg * r64[u]);
            const float z = d[u] * r[u];
            M.z[j] = z;
            a.z32[R0 + j] = z;
            f2 = fmaf(r[u], z, f2);
        }
        double v1[1] = {(double)f2};
        if (!all_sum<1>(v1, CH_INIT + 2, c, err)) return;
        if (tid == 0) {
            s_rho = g_ax_sum[0];
            g_bc[0] = stop_code(s_rr, s_thr);
            g_bc[1] = 0.0;
        }
        __syncthreads();
    }
    int total = 0, nupd = 0, status = DEV_OK;
    for (;;) {
        const double code = g_bc[0];  // from the FP64 residual of the last update
        const float beta = (float)g_bc[1];
        if (code == 1.0 || total >= a.maxit) break;
        if (code == 2.0) { status = DEV_NONFINITE; break; }
        if (code == 3.0) { status = DEV_STALLED; break; }
        ++total;
        stamp(a.ts, total, 0);
        float g0 = 0.f;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = tid + u * CR_NT;
            if (j >= nrow) continue;
            const float w = res_row<float>(M, j, wd[u], a.z32);
            p[u] = fmaf(beta, p[u], M.z[j]);
            q[u] = fmaf(beta, q[u], w);
            g0 = fmaf(p[u], q[u], g0);
        }
        double v1[1] = {(double)g0};
        if (!all_sum<1>(v1, CH_PQ, c, err, [&](int, double pq) {
                g_bc[2] = pq == 0.0 ? 0.0 : s_rho / pq;
                g_bc[3] = pq == 0.0 ? 1.0 : 0.0;
            }, [&] { s_inv = recip(s_rho); })) return;
        stamp(a.ts, total, 1);
        if (g_bc[3] != 0.0) { status = DEV_BREAKDOWN; break; }
        const float alpha = (float)g_bc[2];
        float h0 = 0.f, h1 = 0.f;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = tid + u * CR_NT;
            if (j >= nrow) continue;
            e[u] = fmaf(alpha, p[u], e[u]);
            r[u] = fmaf(-alpha, q[u], r[u]);
            const float z = d[u] * r[u];
            M.z[j] = z;
            a.z32[R0 + j] = z;
            h0 = fmaf(r[u], r[u], h0);
            h1 = fmaf(r[u], z, h1);
        }
        double w2[2] = {(double)h0, (double)h1};
        if (!all_sum<2>(w2, CH_RZ, c, err, [&](int k, double sum) {
                if (k == 1) {
                    g_bc[1] = quotient(sum, s_rho, s_inv);  // the next beta, unless an update replaces r
                    s_rz = sum;
                } else {
                    // reliable update: as k_cg_mixed_pipe (the FP32 sums are in sig^2 units)
                    const double d2 = a.inner_tol * a.inner_tol, s2 = s_sig * s_sig;
                    const bool upd = sum <= d2 * s_rr * s2 || sum <= s_thr * s2 || total >= a.maxit || !(sum == sum);
                    if (upd) {
                        s_sig_next = s_sig * pow2_scale(sum);
                        g_bc[5] = 1.0 / s_sig;  // x += e / sig (a power of two: exact)
                    }
                    g_bc[4] = upd ? 1.0 : 0.0;
                }
            })) return;
        stamp(a.ts, total, 2);
        if (tid == 0 && g_bc[4] == 0.0) s_rho = s_rz;  // read again after the next sum's first barrier
        if (g_bc[4] != 0.0) {
            const double isg = g_bc[5], sn = s_sig_next;
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int j = tid + u * CR_NT;
                if (j < nrow) a.x[R0 + j] += (double)e[u] * isg;
                e[u] = 0.f;
            }
            if (!all_sync(c, err)) return;
            double v2[2] = {0.0, 0.0};
            float fz = 0.f;
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int j = tid + u * CR_NT;
                if (j >= nrow) continue;
                const int i = R0 + j;
                const double ri = a.b[i] - row_dot(a.A, i, a.x);
                r[u] = (float)(sn * ri);
                const float z = d[u] * r[u];
                M.z[j] = z;
                a.z32[i] = z;
                v2[0] = fma(ri, ri, v2[0]);
                fz = fmaf(r[u], z, fz);
            }
            v2[1] = (double)fz;
            if (!all_sum<2>(v2, CH_UPD, c, err)) return;
            if (tid == 0) {
                // the direction is kept while the updates make progress (beta in the new
                // units), else it restarts from z; three stalls hand over to FP64
                const bool stalled = !(g_ax_sum[0] < 0.25 * s_rr);
                s_stalls = stalled ? s_stalls + 1 : 0;
                s_rr = g_ax_sum[0];
                g_bc[0] = stop_code(s_rr, s_thr);
                if (g_bc[0] == 0.0 && s_stalls >= 3) g_bc[0] = 3.0;
                g_bc[1] = stalled ? 0.0 : (g_ax_sum[1] / s_rho) * (s_sig / s_sig_next);
                s_rho = g_ax_sum[1];
                s_sig = s_sig_next;
                ++nupd;
            }
            __syncthreads();
        }
    }
    if (status == DEV_BREAKDOWN) {  // keep the correction gathered so far
        const double isg = 1.0 / s_sig;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = tid + u * CR_NT;
            if (j < nrow) a.x[R0 + j] += (double)e[u] * isg;
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        const double res = sqrt(s_rr) / sqrt(s_bb);
        if (status == DEV_OK && !(s_rr < s_thr)) status = isfinite(s_rr) ? DEV_MAXITER : DEV_NONFINITE;
        a.info->status[0] = status;
        a.info->iters[0] = total;
        a.info->res[0] = res;
        a.info->refinements = nupd;
    }
}

// The resident launch of a system: CTAs, rows a thread (R) and shared memory, or R = 0
// where it does not fit.  ebytes = bytes per matrix value.
struct ResPlan {
    int G = 0, R = 0, ld = 0;
    unsigned smem = 0;
};

ResPlan plan_resident(const SellDev &A, int ebytes, int sm_cap) {
    ResPlan pl;
    const int cap = sm_cap > 0 ? std::min(sm_cap, num_sms()) : num_sms();
    const int G = std::max(1, std::min(std::min(A.nslices, cap), AX_MAX_BLOCKS));
    const int ld = 32 * ((A.nslices + G - 1) / G);
    const size_t smem = (size_t)ld * A.wmax * (ebytes + 4) + (size_t)ld * ebytes;
    const int need = (ld + CR_NT - 1) / CR_NT, most = ebytes == 8 ? 6 : 8;
    if (smem > CR_SMEM || need > most) return pl;
    pl.G = G;
    pl.R = need <= 2 ? need : (need <= 4 ? 4 : most);
    pl.ld = ld;
    pl.smem = (unsigned)smem;
    return pl;
}

template <class K>
void launch_resident(K kernel, const ResPlan &pl, CgResArgs &a, int wmax, cudaStream_t st) {
    SYSU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CR_SMEM));
    void *args[] = {&a, &wmax};
    SYSU_CUDA(cudaLaunchCooperativeKernel((const void *)kernel, dim3(pl.G), dim3(CR_NT), args, pl.smem, st));
    ++::sysu::g_launches;
}

}  // namespace
}  // namespace sysu
