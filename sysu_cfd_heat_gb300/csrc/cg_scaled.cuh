// Streaming Jacobi-CG on the symmetrically scaled system (included by cg.cu):
// S A S y = S b with S = diag(|a_ii|)^-1/2 and x = x0 + S y (both sides times -1 where the
// diagonal is negative, as the p' matrices' is).  Plain CG on it has the iterates
// of Jacobi-PCG on A (the Jacobi weight cancels), and less to do per row than the form with
// M^-1: the diagonal is 1 and needs neither an entry nor a gather, z is r, r.z is r.r, and
// M^-1 is not read.  The update of y waits for the next product phase, where p is in
// registers anyway.  Per row of a tet mesh (5 entries) and iteration
//   before:  S 200 MB / 2M rows and 8 FP64 operations, X 128 MB and 4
//   here:    S 208 MB and 8, X 56 MB and 2.
//   S  y += alpha p, w = r + A' r, p = r + beta p, q = w + beta q, p.q
//   X  r -= alpha q, r.r
// The matrix copy (off-diagonals only, scaled, with their columns) is made once per solve: one
// pass, 40 us of a 60 ms solve at 2M rows.  The stopping test stays on the true residual:
// ||r|| is estimated in FP32 from r' and sqrt(a_ii), and summed exactly in FP64 whenever the
// estimate does not clearly exceed the threshold, as in k_cg_pipe.
//
// us an iteration, form with M^-1 -> here: 2M tets FP64 67.4 -> 45.8, FP32 33.9 -> 24.2; hex
// mesh of 990,000 rows FP64 43.0 -> 30.2, FP32 25.3 -> 18.7; 504,000 tets FP64 24.5 -> 17.7.
// FP64 at 2M: the FP64 pipe takes 33 us of it, 264 MB through L2 and the two grid sums (4 us)
// the rest.  Tried and dropped: the CTA's own r in shared memory (slower: 66 us, it takes the
// L1 away), y updated in the X phase (61 us).
//
// Runs where all diagonal entries have one sign (k_sym_diag counts the others) and the Jacobi
// weight is positive; otherwise, without a preconditioner, and for the rows that sym_launch leaves
// out (cg.cu), the form with M^-1 runs.
#pragma once

#include "grid_all.cuh"

namespace sysu {
namespace {

struct CgSymArgs {
    SellView A;             // FP64 values; the pattern of the copy is this one without entry 0
    const void *val;        // scaled off-diagonals, FP64 or FP32: entry k >= 1 of a row at sl_ptr - 32 s + 32 (k - 1) + lane
    const int *col;
    const double *s;        // |a_ii|^-1/2
    const float *wt;        // |a_ii|^1/2 times a power of two
    const int *bad;         // rows whose diagonal is zero, not finite or of another sign: leave
    const double *b;
    double *x;
    void *r, *p, *q, *y;    // FP64, or FP32 (mixed)
    double *r64;            // mixed: FP64 residual
    unsigned long long *slots;
    SolveInfo *info;
    int maxit;
    double eps, inner_tol;
    unsigned long long *ts;
    CgPlan plan;
    const SolveInfo *gate;  // as CgPipeArgs::gate
};

// power of two near the reciprocal of the first diagonal entry's square root: keeps wt and
// the FP32 sums of (wt r')^2 in range whatever the scale of the matrix
__device__ __forceinline__ double sym_unit(const SellView &A) { return pow2_scale(fabs(A.val[0])); }
__device__ __forceinline__ double sym_sign(const SellView &A) { return A.val[0] < 0.0 ? -1.0 : 1.0; }

__global__ void k_sym_diag(SellView A, double *s, float *wt, int *bad, const SolveInfo *gate) {
    if (gate && gate->status[0] != DEV_STALLED) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    const double d = sym_sign(A) * A.val[A.sl_ptr[i >> 5] + (i & 31)];
    if (!(d > 0.0) || !isfinite(d)) {
        atomicAdd(bad, 1);
        s[i] = 1.0;
        wt[i] = 1.f;
        return;
    }
    const double q = rsqrt(d);
    s[i] = q;
    wt[i] = (float)(d * q * sym_unit(A));
}

template <class V>
__global__ void k_sym_scale(SellView A, const double *__restrict__ s, V *__restrict__ val, int *__restrict__ col,
                            const SolveInfo *gate) {
    if (gate && gate->status[0] != DEV_STALLED) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.nslices * 32) return;
    const int sl = i >> 5, w = A.sl_w[sl];
    int e = A.sl_ptr[sl] + (i & 31), f = e - 32 * sl;
    const double si = i < A.n ? sym_sign(A) * s[i] : 0.0;
    for (int k = 1; k < w; ++k, f += 32) {
        e += 32;
        const int c = A.col[e];
        val[f] = (V)(A.val[e] * si * s[c]);
        col[f] = c;
    }
}

// Place in its tile (first entry, relative) and width of each of the CTA's slices, of the
// matrix copy: from global memory they would put an L2 round trip in front of every tile's
// column reads and gathers.  Beyond the table (CTAs of more than 49,152 rows) they are read there.
constexpr int SYM_SLICES = 1536;
__shared__ int2 g_sym_slice[SYM_SLICES];

__device__ __forceinline__ int2 sym_slice_of(const Part &P, const SellView &A, int s) {
    const int first = s - (s - P.sb) % P.ts;  // the tile's first slice
    return make_int2(__ldg(A.sl_ptr + s) - __ldg(A.sl_ptr + first) - 32 * (s - first), __ldg(A.sl_w + s) - 1);
}
__device__ __forceinline__ void sym_slices_init(const Part &P, const SellView &A) {
    for (int s = P.sb + threadIdx.x; s < min(P.se, P.sb + SYM_SLICES); s += blockDim.x)
        g_sym_slice[s - P.sb] = sym_slice_of(P, A, s);
}

template <class V>
__device__ __forceinline__ void issue_sym_tile(const Part &P, const CgSymArgs &a, int t, unsigned char *dst,
                                               uint64_t *bar, uint64_t pol) {
    const long e0 = tile_entry_packed(P, a.A.sl_ptr, t), e1 = tile_entry_packed(P, a.A.sl_ptr, t + 1);
    const unsigned bv = (unsigned)((e1 - e0) * sizeof(V)), bc = (unsigned)((e1 - e0) * 4);
    mbar_arrive_expect_tx(bar, bv + bc);
    if (bv) {
        bulk_g2s(dst, static_cast<const V *>(a.val) + e0, bv, bar, pol);
        bulk_g2s(dst + bv, a.col + e0, bc, bar, pol);
    }
}

// Wait for a tile: the outcome is uniform per warp; false after a timed-out wait.
__device__ __forceinline__ bool sym_acquire(int slot, unsigned par, int *err) {
    if (__all_sync(FULL_MASK, mbar_test_wait(&g_full[slot], par))) return true;
    return acquire_at(slot, par, err);
}

// S phase of a consumer warp over the CTA's tiles, at most one slice a tile: returns the thread's
// partial p.q.  pend: the alpha of the last X phase, still owed to y.  Issue slots count here
// (with the place of a row computed in every tile: 400 warp instructions a row and iteration
// in FP32, S 22.3 us of the 2M-row solve, 17.3 here), so places and widths come from a table
// and rows advance by a constant.  No look-ahead: holding the next tile's gathers during this
// one's FMAs, as k_cg_pipe does, measured no faster in FP64 (50.2 us an iteration both) and
// slower in FP32 (27.6 against 25.9).
// WR: gathers held at a time; SYM_WIDE for rows so wide that a tile holds fewer slices than there
// are consumer warps, of which those beyond have none (the test, in every tile, costs the others
// 0.3 % in FP64 and 0.9 % in FP32).
constexpr int SYM_WIDE = 8;
template <class V, int WR>
__device__ __forceinline__ V sym_s_phase(const Part &P, Ring &R, const CgSymArgs &a, V beta, V pend, bool has_dir,
                                         int *err) {
    const int nt = P.nt, lane = threadIdx.x & 31;
    V *pv = static_cast<V *>(a.p), *qv = static_cast<V *>(a.q), *yv = static_cast<V *>(a.y);
    const V *rv = static_cast<const V *>(a.r);
    V pq = 0;
    int s = P.sb + (int)(threadIdx.x >> 5), i = 32 * s + lane;
    for (int t = 0; t < nt; ++t, s += P.ts, i += 32 * P.ts) {
        bool act = i < a.A.n && s < P.se;
        if (WR == SYM_WIDE) act = act && (int)(threadIdx.x >> 5) < P.ts;
        V r = 0, p = 0, q = 0, y = 0;
        int2 pl = make_int2(0, 0);
        if (act) {
            r = rv[i];
            if (has_dir) {
                p = pv[i];
                q = qv[i];
                y = yv[i];
            }
            pl = s - P.sb < SYM_SLICES ? g_sym_slice[s - P.sb] : sym_slice_of(P, a.A, s);
        }
        if (!sym_acquire(R.cslot, R.cpar, err)) break;
        if (act) {
            const int e0 = tile_entry_packed(P, a.A.sl_ptr, t), cnt = tile_entry_packed(P, a.A.sl_ptr, t + 1) - e0;
            const unsigned char *slot = cslot_ptr(R);
            const V *vs = reinterpret_cast<const V *>(slot) + pl.x + lane;
            const int *cs = reinterpret_cast<const int *>(slot + cnt * (int)sizeof(V)) + pl.x + lane;
            int c[WR];
            V g[WR];
#pragma unroll
            for (int k = 0; k < WR; ++k)
                if (k < pl.y) c[k] = cs[32 * k];
#pragma unroll
            for (int k = 0; k < WR; ++k)
                if (k < pl.y) g[k] = rv[c[k]];
            V w = r;
#pragma unroll
            for (int k = 0; k < WR; ++k)
                if (k < pl.y) w = fma_t(vs[32 * k], g[k], w);
            for (int k = WR; k < pl.y; ++k) w = fma_t(vs[32 * k], rv[cs[32 * k]], w);
            yv[i] = fma_t(pend, p, y);
            p = fma_t(beta, p, r);
            q = fma_t(beta, q, w);
            pv[i] = p;
            qv[i] = q;
            pq = fma_t(p, q, pq);
        }
        release(R);
    }
    return pq;
}

// X phase over the CTA's rows: r -= alpha q, r.r (of the scaled r) and the FP32 estimate of
// the true r.r; RB rows a thread a step with their loads before the arithmetic.
template <int NT, int RB>
__device__ __forceinline__ void sym_x_phase(int R0, int R1, double alpha, const double *__restrict__ qv,
                                            const float *__restrict__ wt, double *__restrict__ rv, double &rho,
                                            float &est, int bias) {
    for (int i = R0 + (int)threadIdx.x; i < R1; i += RB * NT) {
        double q[RB], r[RB];
        float w[RB];
#pragma unroll
        for (int u = 0; u < RB; ++u) {
            const int j = i + u * NT;
            if (j < R1) {
                q[u] = qv[j];
                r[u] = rv[j];
                w[u] = wt[j];
            }
        }
#pragma unroll
        for (int u = 0; u < RB; ++u) {
            const int j = i + u * NT;
            if (j < R1) {
                r[u] = fma_t(-alpha, q[u], r[u]);
                rv[j] = r[u];
                const float f = scaled_abs_f32(r[u], bias) * w[u];
                est = fmaf(f, f, est);
                rho = fma_t(r[u], r[u], rho);
            }
        }
    }
}

template <int NT, int RB>
__device__ __forceinline__ void sym_x_phase32(int R0, int R1, float alpha, const float *__restrict__ qv,
                                              const float *__restrict__ wt, float *__restrict__ rv, float &rho,
                                              float &rr) {
    for (int i = R0 + (int)threadIdx.x; i < R1; i += RB * NT) {
        float q[RB], r[RB], w[RB];
#pragma unroll
        for (int u = 0; u < RB; ++u) {
            const int j = i + u * NT;
            if (j < R1) {
                q[u] = qv[j];
                r[u] = rv[j];
                w[u] = wt[j];
            }
        }
#pragma unroll
        for (int u = 0; u < RB; ++u) {
            const int j = i + u * NT;
            if (j < R1) {
                r[u] = fmaf(-alpha, q[u], r[u]);
                rv[j] = r[u];
                const float f = r[u] * w[u];
                rr = fmaf(f, f, rr);
                rho = fmaf(r[u], r[u], rho);
            }
        }
    }
}

// Threads a CTA, us an iteration: FP64 2M tets 512 48.7, 640 45.8, 768 48.8 (hex mesh of
// 990,000 rows 30.0, 30.2, 32.6); FP32 640 26.7, 768 24.9, 896 24.8 (19.1, 18.7, 19.4).
constexpr int SYM_NT = 640, SYM_NT32 = 768;

template <int WR>
__global__ void __launch_bounds__(SYM_NT, 1) k_cg_sym(CgSymArgs a) {
    constexpr int NT = SYM_NT;
    if (a.gate && a.gate->status[0] != DEV_STALLED) return;  // the same words for every block
    if (*a.bad) return;
    const int it_before = a.gate ? a.gate->iters[0] : 0;
    const int tid = threadIdx.x;
    const bool prod = is_producer();
    int *err = &a.info->err;
    AllCtx gc = all_ctx(a.slots);
    all_init();
    const Part P = make_part(a.A.n, a.A.nslices, a.plan.ts);
    const int nt = P.nt, R0 = P.sb * 32, R1 = min(P.se * 32, a.A.n);
    const double sgn = sym_sign(a.A);
    double *r = static_cast<double *>(a.r), *p = static_cast<double *>(a.p), *y = static_cast<double *>(a.y);
    const double *q = static_cast<const double *>(a.q);
    Ring R;
    sym_slices_init(P, a.A);
    ring_init(R, a.plan, P, a.A.sl_ptr, true);
    auto issue = [&](int t, unsigned char *dst, uint64_t *bar, uint64_t pol) {
        issue_sym_tile<double>(P, a, t, dst, bar, pol);
    };
    if (prod) producer_tiles(R, 0, issue, err);  // the first tiles land during the initial residual
    double v3[3] = {0.0, 0.0, 0.0};
    for (int i = R0 + tid; i < R1; i += NT) {
        const double bi = a.b[i], ri = bi - row_dot(a.A, i, a.x), rsc = sgn * a.s[i] * ri;
        r[i] = rsc;
        v3[0] = fma(bi, bi, v3[0]);
        v3[1] = fma(ri, ri, v3[1]);
        v3[2] = fma(rsc, rsc, v3[2]);
    }
    __shared__ double s_bb, s_rr, s_rho, s_thr, s_unit;
    __shared__ int s_bias, s_rr_est;
    if (!all_sum<3>(v3, CH_INIT, gc, err)) { drain(R); return; }
    if (tid == 0) {
        s_bb = g_ax_sum[0] == 0.0 ? 1.0 : g_ax_sum[0];
        s_thr = a.eps * a.eps * s_bb;
        s_rr = g_ax_sum[1];
        s_rho = g_ax_sum[2];
        g_bc[0] = stop_code(s_rr, s_thr);
        g_bc[1] = 0.0;
        // the estimate of r.r in units of 2^2k / unit^2, 2^2k ~ thr unit^2 (bias 0: thr unusable)
        s_bias = 0;
        s_rr_est = 0;
        const double u = sym_unit(a.A), th = s_thr * u * u;
        if (th > 0.0 && isfinite(th)) {
            const int e = ilogb(th);
            const int k = e >= 0 ? e / 2 : -((1 - e) / 2);  // floor(e / 2)
            if (k > -900 && k < 900) {
                s_bias = 1023 + k - 127;
                s_unit = ldexp(1.0, 2 * k) / (u * u);
            }
        }
    }
    __syncthreads();
    const int bias = s_bias;
    // the true r.r in FP64: r = r' / s, 1 / s = a_ii s
    auto exact_rr = [&]() -> bool {
        double e1[1] = {0.0};
        for (int i = R0 + tid; i < R1; i += NT) {
            const double d = a.A.val[a.A.sl_ptr[i >> 5] + (i & 31)], ri = r[i] * (d * a.s[i]);  // up to its sign
            e1[0] = fma(ri, ri, e1[0]);
        }
        return all_sum<1>(e1, CH_RR, gc, err);
    };
    long long base = 0;  // job index of the running S phase's first tile
    double pend = 0.0;   // alpha p is owed to y
    int it = 0, status = DEV_OK;
    bool ok = true;
    for (;;) {
        const double code = g_bc[0], beta = g_bc[1];
        if (code == 1.0 || it >= a.maxit) break;
        if (code == 2.0) { status = DEV_NONFINITE; break; }
        ++it;
        stamp(a.ts, it, 0);
        double v1[1] = {0.0};
        if (prod) producer_tiles(R, base + nt, issue, err);
        else v1[0] = sym_s_phase<double, WR>(P, R, a, beta, pend, it > 1, err);
        base += nt;
        pend = 0.0;
        if (!all_sum<1>(v1, CH_PQ, gc, err, [&](int, double pq) {
                g_bc[2] = pq == 0.0 ? 0.0 : s_rho / pq;
                g_bc[3] = pq == 0.0 ? 1.0 : 0.0;
            }) || fail_flag()) { ok = false; break; }
        stamp(a.ts, it, 1);
        if (g_bc[3] != 0.0) { status = DEV_BREAKDOWN; break; }
        const double alpha = g_bc[2];
        pend = alpha;
        if (prod) producer_tiles(R, 0, issue, err);  // the next S phase's tiles
        double v2[2] = {0.0, 0.0};
        float est = 0.f;
        sym_x_phase<NT, 4>(R0, R1, alpha, q, a.wt, r, v2[1], est, bias);
        v2[0] = (double)est;
        if (!all_sum<2>(v2, CH_RZ, gc, err, [&](int k, double sum) {
                if (k == 1) {
                    g_bc[1] = quotient(sum, s_rho, 0.0);
                    s_rho = sum;
                } else {
                    // the estimate decides only when it is clearly above the threshold
                    s_rr = sum * s_unit;
                    s_rr_est = 1;
                    g_bc[5] = bias && isfinite(sum) && s_rr >= s_thr * 1.001 ? 0.0 : 1.0;  // 1: take the exact r.r
                    g_bc[0] = 0.0;
                }
            }) || fail_flag()) { ok = false; break; }
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
    drain(R);
    __syncthreads();
    const int est = s_rr_est;
    // the reported residual is the exact one (not after a failed wait, when the blocks no longer meet)
    if (est && ok && !fail_flag() && exact_rr() && tid == 0) s_rr = g_ax_sum[0];
    if (it > 0)
        for (int i = R0 + tid; i < R1; i += NT) a.x[i] = fma(a.s[i], fma(pend, p[i], y[i]), a.x[i]);
    __syncthreads();
    if (blockIdx.x == 0 && tid == 0) {
        const double res = sqrt(s_rr) / sqrt(s_bb);
        if (status == DEV_OK && !(s_rr < s_thr)) status = isfinite(s_rr) ? DEV_MAXITER : DEV_NONFINITE;
        a.info->status[0] = status;
        a.info->iters[0] = it_before + it;
        a.info->res[0] = res;
    }
}

// Mixed precision (see k_cg_mixed_pipe): r', p, q and the correction y in FP32, in units of
// sig (a power of two, sig ||r'|| ~ 1 after each reliable update); x += S y / sig in FP64 and
// the FP64 residual b - A x at each update, on which convergence is decided.
template <int WR>
__global__ void __launch_bounds__(SYM_NT32, 1) k_cg_mixed_sym(CgSymArgs a) {
    if (*a.bad) return;  // the same word for every block
    const int tid = threadIdx.x;
    const bool prod = is_producer();
    int *err = &a.info->err;
    AllCtx gc = all_ctx(a.slots);
    all_init();
    const Part P = make_part(a.A.n, a.A.nslices, a.plan.ts);
    const int nt = P.nt, R0 = P.sb * 32, R1 = min(P.se * 32, a.A.n);
    const double sgn = sym_sign(a.A);
    float *r = static_cast<float *>(a.r), *p = static_cast<float *>(a.p), *y = static_cast<float *>(a.y);
    const float *q = static_cast<const float *>(a.q);
    Ring R;
    sym_slices_init(P, a.A);
    ring_init(R, a.plan, P, a.A.sl_ptr, true);
    auto issue = [&](int t, unsigned char *dst, uint64_t *bar, uint64_t pol) {
        issue_sym_tile<float>(P, a, t, dst, bar, pol);
    };
    if (prod) producer_tiles(R, 0, issue, err);
    __shared__ double s_bb, s_thr, s_rho, s_rs, s_rr, s_sig, s_sig_next, s_u2;
    __shared__ int s_stalls;
    // FP64 residual of the initial guess, then its scaled FP32 copy
    double v3[3] = {0.0, 0.0, 0.0};
    for (int i = R0 + tid; i < R1; i += SYM_NT32) {
        const double bi = a.b[i], ri = bi - row_dot(a.A, i, a.x), rsc = sgn * a.s[i] * ri;
        a.r64[i] = rsc;
        v3[0] = fma(bi, bi, v3[0]);
        v3[1] = fma(ri, ri, v3[1]);
        v3[2] = fma(rsc, rsc, v3[2]);
    }
    if (!all_sum<3>(v3, CH_INIT, gc, err)) { drain(R); return; }
    if (tid == 0) {
        s_bb = g_ax_sum[0] == 0.0 ? 1.0 : g_ax_sum[0];
        s_thr = a.eps * a.eps * s_bb;
        s_rr = g_ax_sum[1];
        s_sig = pow2_scale(g_ax_sum[2]);
        const double u = sym_unit(a.A);
        s_u2 = u * u;
        s_stalls = 0;
    }
    __syncthreads();
    {
        const double sg = s_sig;
        float f2 = 0.f;
        for (int i = R0 + tid; i < R1; i += SYM_NT32) {
            const float rf = (float)(sg * a.r64[i]);
            r[i] = rf;
            f2 = fmaf(rf, rf, f2);
        }
        double v1[1] = {(double)f2};
        if (!all_sum<1>(v1, CH_RR, gc, err)) { drain(R); return; }
        if (tid == 0) {
            s_rho = g_ax_sum[0];
            g_bc[0] = stop_code(s_rr, s_thr);
            g_bc[1] = 0.0;
        }
        __syncthreads();
    }
    long long base = 0;
    float pend = 0.f;   // alpha p is owed to y
    int total = 0, nupd = 0, status = DEV_OK;
    bool fresh = true;  // p, q and y start anew
    for (;;) {
        const double code = g_bc[0];  // from the FP64 residual of the last update
        const float beta = (float)g_bc[1];
        if (code == 1.0 || total >= a.maxit) break;
        if (code == 2.0) { status = DEV_NONFINITE; break; }
        if (code == 3.0) { status = DEV_STALLED; break; }
        ++total;
        stamp(a.ts, total, 0);
        float g0 = 0.f;
        if (prod) producer_tiles(R, base + nt, issue, err);
        else g0 = sym_s_phase<float, WR>(P, R, a, beta, pend, !fresh, err);
        fresh = false;
        base += nt;
        pend = 0.f;
        double v1[1] = {(double)g0};
        if (!all_sum<1>(v1, CH_PQ, gc, err, [&](int, double pq) {
                g_bc[2] = pq == 0.0 ? 0.0 : s_rho / pq;
                g_bc[3] = pq == 0.0 ? 1.0 : 0.0;
            }) || fail_flag()) break;
        stamp(a.ts, total, 1);
        if (g_bc[3] != 0.0) { status = DEV_BREAKDOWN; break; }
        const float alpha = (float)g_bc[2];
        pend = alpha;
        if (prod) producer_tiles(R, 0, issue, err);
        float h0 = 0.f, h1 = 0.f;
        sym_x_phase32<SYM_NT32, 4>(R0, R1, alpha, q, a.wt, r, h1, h0);
        double w2[2] = {(double)h0, (double)h1};
        if (!all_sum<2>(w2, CH_RZ, gc, err, [&](int k, double sum) {
                if (k == 1) {
                    g_bc[1] = sum / s_rho;  // the next beta, unless an update replaces r
                    s_rs = sum;
                } else {
                    // reliable update once the FP32 residual fell by inner_tol since the last
                    // one, when it looks converged, or at the iteration cap (the sum is the true
                    // r.r in sig^2 unit^2)
                    const double d2 = a.inner_tol * a.inner_tol, s2 = s_sig * s_sig * s_u2;
                    const bool upd = sum <= d2 * s_rr * s2 || sum <= s_thr * s2 || total >= a.maxit || !isfinite(sum);
                    g_bc[4] = upd ? 1.0 : 0.0;
                }
            }) || fail_flag()) break;
        stamp(a.ts, total, 2);
        if (g_bc[4] == 0.0) {
            if (tid == 0) s_rho = s_rs;  // read again after the next sum's first barrier
        } else {
            if (tid == 0) s_sig_next = s_sig * pow2_scale(s_rs);  // from the FP32 r'.r'
            __syncthreads();
            const double isg = 1.0 / s_sig, sn = s_sig_next;  // powers of two: exact
            for (int i = R0 + tid; i < R1; i += SYM_NT32) {
                a.x[i] = fma(a.s[i] * isg, (double)fmaf(pend, p[i], y[i]), a.x[i]);
                y[i] = 0.f;
            }
            pend = 0.f;
            if (!all_sync(gc, err)) break;
            double u[2] = {0.0, 0.0};
            float fz = 0.f;
            for (int i = R0 + tid; i < R1; i += SYM_NT32) {
                const double ri = a.b[i] - row_dot(a.A, i, a.x);
                const float rf = (float)(sn * sgn * (a.s[i] * ri));
                r[i] = rf;
                u[0] = fma(ri, ri, u[0]);
                fz = fmaf(rf, rf, fz);
            }
            u[1] = (double)fz;
            if (!all_sum<2>(u, CH_UPD, gc, err)) break;
            if (tid == 0) {
                // the direction is kept while the updates make progress (beta in the new
                // units), else it restarts from r; three stalls hand over to FP64
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
    drain(R);
    __syncthreads();
    if (status == DEV_BREAKDOWN) {  // keep the correction gathered so far
        const double isg = 1.0 / s_sig;
        for (int i = R0 + tid; i < R1; i += SYM_NT32) a.x[i] = fma(a.s[i] * isg, (double)fmaf(pend, p[i], y[i]), a.x[i]);
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

}  // namespace
}  // namespace sysu
