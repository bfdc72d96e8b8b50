// Jacobi-preconditioned CG on a caller-owned device CSR matrix that allocates
// nothing: its scratch (z, the inverse diagonal, the exchange area of the grid
// sums and the status words) lives in one file-scope device array,
// g_noalloc_scratch, of fixed size.
//
// Who needs it: callers that cannot call cudaMalloc -- host applications that
// own all device memory through their own pool and do not let libraries
// allocate behind their back, and time-critical loops that must not pay
// cudaMalloc/cudaFree, which synchronise the whole device.  Such a caller
// passes its own device buffers for the matrix, b and x, and this entry point
// uses only the static array besides them.
//
// Limits and rules (also in include/sysu_cfd.h):
// * at most SYSU_NOALLOC_MAX_ROWS rows (262,144); larger systems are rejected;
// * the array costs 4.2 MB on every GPU that loads the library, until exit;
// * all calls share the array and it keeps the last call's contents: each call
//   clears what must start at zero (exchange area, status words) itself;
//   calls that overlap on the GPU (two streams, two threads) race on it;
// * every call looks up the array's device address (cudaGetSymbolAddress,
//   which allocates nothing) with the calling thread's device current, so a
//   cudaDeviceReset between calls is harmless; the first call on a device
//   also queries the cooperative-launch occupancy once and caches it;
// * every call waits for its stream (it reads the iteration count, residual
//   and status back), so it cannot be captured into a CUDA graph: a call on a
//   capturing stream is refused with SYSU_ERR_INPUT before anything is queued;
// * the CSR arrays are the caller's: a row pointer that decreases, a column
//   outside 0..n-1 or a row without a nonzero diagonal is reported as
//   SYSU_ERR_INPUT (first offending row in the message) and such entries are
//   never used to index x.  The caller must still make rowptr[n] no larger
//   than the length of d_col and d_val.
#include <cuda_runtime.h>

#include <cmath>
#include <cstddef>
#include <mutex>
#include <string>

#include "../../include/sysu_cfd.h"
#include "grid_all.cuh"

namespace {

constexpr int NA_MAX_ROWS = 262144;
constexpr int NA_KB = 256;                 // threads of the check kernel
constexpr int NA_NT = 512;                 // threads of a solver CTA
constexpr int NA_ROWS = 4;                 // rows a thread at most
constexpr unsigned NA_SMEM = 200 * 1024;   // matrix entries a CTA keeps in shared memory
constexpr int NA_ENTRIES = NA_SMEM / 12;
constexpr int NA_CL_ROWS = 16 * NA_NT;     // up to here one cluster of at most 16 CTAs solves the system

// what a malformed CSR row was found to hold (low two bits of NaHeader::bad)
enum NaBad : int { NA_BAD_NONE = 0, NA_BAD_ROWPTR = 1, NA_BAD_COL = 2, NA_BAD_DIAG = 3 };

struct NaHeader {  // at the start of the array, cleared by every call
    int unused;
    int wide;  // the rows of a CTA of the cluster do not fit its shared memory: it has not run
    int err;
    int status;
    int iters;
    int pad;
    double res;
    // lowest malformed row and what it holds, as (row << 2) | NaBad, kept by
    // atomicMin; all ones (set by the host before each call) when none is
    unsigned long long bad;
};

// layout in doubles: header (64 B) | z | dinv | exchange area of the grid sums
constexpr size_t NA_HDR = 16;
static_assert(sizeof(NaHeader) <= NA_HDR * sizeof(double), "NaHeader must fit its slot");
constexpr size_t NA_SLOTS = NA_HDR + 2 * (size_t)NA_MAX_ROWS;
constexpr size_t NA_DOUBLES = NA_SLOTS + sysu::AX_WORDS;

static __device__ __align__(256) double g_noalloc_scratch[NA_DOUBLES];

struct NaArgs {
    int n;
    const int *rowptr, *col;
    const double *val, *b;
    double *x;
    double omega;
    int maxit;
    double eps;
    double *base;  // device address of g_noalloc_scratch
    int cluster;   // CTAs of the cluster that is to solve the system; 0: the whole GPU does
};

// First row of block o of G: whole groups of 32.
__device__ __forceinline__ int na_first_row(int n, int o, int G) {
    return min(n, 32 * (int)((long long)((n + 31) / 32) * o / G));
}

constexpr unsigned long long NA_GOOD = ~0ull;

__device__ __forceinline__ void na_report(NaHeader *h, int row, int kind) {
    atomicMin(&h->bad, ((unsigned long long)row << 2) | (unsigned long long)kind);
}

// D^-1 scaled by omega, and the checks of the caller's CSR: rows whose pointer
// decreases, columns outside 0..n-1 and rows without a nonzero diagonal are
// recorded in the header (lowest row) instead of being used.  Says also whether the cluster
// can hold the matrix.
__global__ void k_na_dinv(NaArgs a) {
    NaHeader *h = reinterpret_cast<NaHeader *>(a.base);
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    if (i < a.cluster &&
        (long long)a.rowptr[na_first_row(a.n, i + 1, a.cluster)] - a.rowptr[na_first_row(a.n, i, a.cluster)] >
            NA_ENTRIES)
        h->wide = 1;
    int k0 = a.rowptr[i], k1 = a.rowptr[i + 1];
    double d = 0.0;
    int kind = NA_BAD_NONE;
    if (k0 < 0 || k1 < k0) {
        kind = NA_BAD_ROWPTR;
    } else {
        for (int k = k0; k < k1; ++k) {
            int c = a.col[k];
            if ((unsigned)c >= (unsigned)a.n) { kind = NA_BAD_COL; break; }
            if (c == i) d += a.val[k];
        }
        if (kind == NA_BAD_NONE && !(d != 0.0 && isfinite(d))) kind = NA_BAD_DIAG;
    }
    if (kind != NA_BAD_NONE) {
        na_report(h, i, kind);
        d = 1.0;
    }
    a.base[NA_HDR + (size_t)NA_MAX_ROWS + i] = a.omega / d;
}

// Same recurrences as the SELL persistent CG (Templates Fig. 2.5, Jacobi) with w = A z and
// q = w + beta q in place of the product of p, so that an iteration has two grid-wide steps.
// Row i's product takes its entries in the caller's order.
//
// One CTA per SM owns a contiguous range of rows: their vectors in registers, their part of
// the caller's CSR in shared memory when it fits (17,066 entries a CTA, so always for the
// 7-entry rows of a hex mesh; without a cluster a CTA whose rows hold more reads the caller's arrays).  z, which
// other CTAs gather, is the only vector in memory.  Latency bounds it at every size up to the
// limit: two sums (grid_all.cuh) and an FP64 division an iteration.  1,716 rows on 7 blocks
// of 256 threads, with three barriers and FP64 shuffle trees, square roots and divisions in
// every thread, took 12.7 us an iteration; on 54 CTAs here 6.1 (238,080 rows: 12.4).
// CL: the grid is one cluster.  z lies in its CTAs' shared memory, the columns there are turned
// into shared addresses of the cluster, and the sums meet at the cluster's barrier: one sum
// (CgScalars) and a barrier, 3.9 us; with the two sums 0.7 more.  Over the whole GPU the form with
// one sum was not faster (6.9 against 6.8 at 32,768 rows, 7.5 against 7.2 at 60,680): three values
// at once and a bare barrier take as long as the two sums.
template <int R, bool CL>
__global__ void __launch_bounds__(NA_NT, 1) k_na_cg(NaArgs a) {
    NaHeader *h = reinterpret_cast<NaHeader *>(a.base);
    double *zg = a.base + NA_HDR;
    const double *dinv = zg + NA_MAX_ROWS;
    const int n = a.n, tid = threadIdx.x;
    // k_na_dinv ran before this launch on the same stream: every block reads the
    // same check result, so on a malformed matrix all leave together, before any
    // row loop or barrier
    if (__ldcg(&h->bad) != NA_GOOD || (CL && __ldcg(&h->wide))) return;
    const int groups = (n + 31) / 32;
    const int R0 = na_first_row(n, blockIdx.x, gridDim.x), R1 = na_first_row(n, blockIdx.x + 1, gridDim.x);
    sysu::AllCtx c = sysu::all_ctx(reinterpret_cast<unsigned long long *>(a.base + NA_SLOTS));
    sysu::ClCtx cl = sysu::cl_ctx();
    if (CL) sysu::cl_sync();  // every block has started before its shared memory is written to
    else sysu::all_init();
    auto sum = [&](auto &v, int ch, auto fin) {
        if (!CL) return sysu::all_sum(v, ch, c, &h->err, fin);
        sysu::cl_sum(v, cl, fin);
        return true;
    };
    const int NT = CL ? (int)blockDim.x : NA_NT;
    extern __shared__ __align__(16) unsigned char na_smem[];
    // CL: this block's z, and where the cluster keeps row j's
    __shared__ double zs[CL ? R * NA_NT : 1];
    auto at = [&](int j) {
        const int g = j >> 5, G = (int)gridDim.x;
        int o = (int)(((long long)(g + 1) * G - 1) / groups);
        return sysu::cl_addr(zs + (j - 32 * (int)((long long)groups * o / G)), o);
    };
    const int E0 = a.rowptr[R0], nent = a.rowptr[R1] - E0;
    const bool res = CL || nent <= NA_ENTRIES;
    double *sval = reinterpret_cast<double *>(na_smem);
    int *scol = reinterpret_cast<int *>(sval + (res ? nent : 0));
    if (res) {
        for (int k = tid; k < nent; k += NT) {
            sval[k] = a.val[E0 + k];
            scol[k] = CL ? (int)at(a.col[E0 + k]) : a.col[E0 + k];
        }
    }
    const double *mv = res ? sval : a.val + E0;
    const int *mc = res ? scol : a.col + E0;
    auto zat = [&](int e) {
        if (!CL) return zg[mc[e]];
        return sysu::cl_load((unsigned)mc[e]);
    };
    __shared__ double s_rr, s_rho, s_thr, s_bb, s_alpha, s_beta, s_inv;
    __shared__ sysu::CgScalars S;
    __shared__ int s_brk, s_end;  // s_end: 1 converged, 2 the residual is not finite, 0 go on
    auto end_code = [&](double rr) {
        return sysu::stop_below(rr, s_thr, a.eps, s_bb) ? 1 : sysu::finite_bits(rr) ? 0 : 2;
    };
    double x[R], r[R], p[R], q[R], d[R];
    int e0[R], len[R];
    double v3[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int i = R0 + tid + u * NT;
        x[u] = r[u] = p[u] = q[u] = d[u] = 0.0;
        e0[u] = len[u] = 0;
        if (i >= R1) continue;
        const int k0 = a.rowptr[i], k1 = a.rowptr[i + 1];
        e0[u] = k0 - E0;
        len[u] = k1 - k0;
        double s = 0.0;
        for (int k = k0; k < k1; ++k) s = fma(a.val[k], a.x[a.col[k]], s);
        const double bi = a.b[i];
        x[u] = a.x[i];
        d[u] = dinv[i];
        r[u] = bi - s;
        const double z = d[u] * r[u];
        if (CL) zs[i - R0] = z;
        else zg[i] = z;
        v3[0] = fma(bi, bi, v3[0]);
        v3[1] = fma(r[u], r[u], v3[1]);
        v3[2] = fma(r[u], z, v3[2]);
    }
    if (!sum(v3, 0, [&](int k, double s) {
            if (k == 0) {
                s_bb = s == 0.0 ? 1.0 : s;
                s_thr = sysu::stop_threshold(a.eps, s_bb);
            } else if (k == 1) {
                s_rr = s;
            } else {
                s_rho = s;
                s_beta = 0.0;
                sysu::cg_first(S);
            }
        })) return;
    auto product = [&](int u) {  // row u of A z
        double w = 0.0;
        int k = 0;
        for (; k + 4 <= len[u]; k += 4) {  // four entries' loads before their FMAs
            const int e = e0[u] + k;
            const double g0 = zat(e), g1 = zat(e + 1), g2 = zat(e + 2), g3 = zat(e + 3);
            w = fma(mv[e], g0, w);
            w = fma(mv[e + 1], g1, w);
            w = fma(mv[e + 2], g2, w);
            w = fma(mv[e + 3], g3, w);
        }
        for (; k < len[u]; ++k) w = fma(mv[e0[u] + k], zat(e0[u] + k), w);
        return w;
    };
    int it = 0, status = sysu::DEV_OK;
    while (CL) {  // one sum and one barrier an iteration
        double w[R], v[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int u = 0; u < R; ++u) {
            w[u] = 0.0;
            if (len[u] == 0) continue;
            w[u] = product(u);
            const double z = d[u] * r[u];
            v[0] = fma(r[u], r[u], v[0]);
            v[1] = fma(r[u], z, v[1]);
            v[2] = fma(w[u], z, v[2]);
        }
        sysu::cl_sum(v, cl, [&](int k, double s) {
            if (k == 0) {
                s_rr = s;
                s_end = end_code(s);
            } else if (k == 1) {
                S.gamma = s;
            } else {
                S.delta = s;
            }
        });
        if (s_end == 1 || it >= a.maxit) break;
        if (s_end == 2) { status = sysu::DEV_NONFINITE; break; }
        ++it;
        if (tid == 0) sysu::cg_scalars(S);
        __syncthreads();
        if (S.den == 0.0) { status = sysu::DEV_BREAKDOWN; break; }
        const double alpha = S.alpha, beta = S.beta;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int i = R0 + tid + u * NT;
            if (i >= R1) continue;
            p[u] = fma(beta, p[u], d[u] * r[u]);
            q[u] = fma(beta, q[u], w[u]);
            x[u] = fma(alpha, p[u], x[u]);
            r[u] = fma(-alpha, q[u], r[u]);
            zs[i - R0] = d[u] * r[u];
        }
        sysu::cl_sync([&] { sysu::cg_next(S); });
    }
    if (!CL) {  // (the first sums are taken by different warps)
        if (tid == 0) s_end = end_code(s_rr);
        __syncthreads();
    }
    while (!CL && s_end != 1 && it < a.maxit) {
        if (s_end == 2) { status = sysu::DEV_NONFINITE; break; }
        ++it;
        const double beta = s_beta;
        double v1[1] = {0.0};
#pragma unroll
        for (int u = 0; u < R; ++u) {
            if (len[u] == 0) continue;
            const double w = product(u);
            p[u] = fma(beta, p[u], d[u] * r[u]);
            q[u] = fma(beta, q[u], w);
            v1[0] = fma(p[u], q[u], v1[0]);
        }
        if (!sysu::all_sum(v1, 3, c, &h->err, [&](int, double pq) {
                s_brk = pq == 0.0;
                s_alpha = pq == 0.0 ? 0.0 : s_rho / pq;
            }, [&] { s_inv = sysu::recip(s_rho); })) return;
        if (s_brk) { status = sysu::DEV_BREAKDOWN; break; }
        const double alpha = s_alpha;
        double v2[2] = {0.0, 0.0};
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int i = R0 + tid + u * NT;
            if (i >= R1) continue;
            x[u] = fma(alpha, p[u], x[u]);
            r[u] = fma(-alpha, q[u], r[u]);
            const double z = d[u] * r[u];
            zg[i] = z;
            v2[0] = fma(r[u], r[u], v2[0]);
            v2[1] = fma(r[u], z, v2[1]);
        }
        if (!sysu::all_sum(v2, 4, c, &h->err, [&](int k, double s) {
                if (k == 0) {
                    s_rr = s;
                    s_end = end_code(s);
                } else {
                    s_beta = sysu::quotient(s, s_rho, s_inv);
                    s_rho = s;
                }
            })) return;
    }
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int i = R0 + tid + u * NT;
        if (i < R1) a.x[i] = x[u];
    }
    if (blockIdx.x == 0 && tid == 0) {
        if (status == sysu::DEV_OK && s_end != 1) status = s_end == 0 ? sysu::DEV_MAXITER : sysu::DEV_NONFINITE;
        h->status = status;
        h->iters = it;
        h->res = sqrt(s_rr) / sqrt(s_bb);
    }
}

thread_local std::string g_na_err;
std::mutex g_na_mu;
int g_na_blocks[64] = {0};   // SMs of a device, 0: not asked yet
int g_na_cluster[64] = {0};  // CTAs of its largest cluster of the solver

int na_fail(int code, const std::string &m) {
    g_na_err = m;
    return code;
}

}  // namespace

extern "C" {

int sysu_csr_cg_noalloc(int n, const int *d_rowptr, const int *d_col, const double *d_val, const double *d_b,
                        double *d_x, int maxit, double eps, double omega, void *stream, int *iters, double *res,
                        int *status) {
    if (n < 1 || n > NA_MAX_ROWS)
        return na_fail(SYSU_ERR_INPUT, "sysu_csr_cg_noalloc: n = " + std::to_string(n) + " is outside 1.." +
                                           std::to_string(NA_MAX_ROWS) + " (the size of the static scratch)");
    if (!d_rowptr || !d_col || !d_val || !d_b || !d_x) return na_fail(SYSU_ERR_INPUT, "null device pointer");
    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return na_fail(SYSU_ERR_CUDA, "device ordinal out of range");
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(st, &cap);
    if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("cudaStreamIsCapturing: ") + cudaGetErrorString(e));
    if (cap != cudaStreamCaptureStatusNone)
        return na_fail(SYSU_ERR_INPUT, "sysu_csr_cg_noalloc waits for its stream to read the result back and "
                                       "cannot run on a stream that is being captured");
    // the array's device address in the current context: looked up on every call
    // (it allocates nothing), so a context torn down and re-created between calls
    // never leaves a stale address behind
    void *ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    double *base = static_cast<double *>(ptr);
    int blocks;
    {
        std::lock_guard<std::mutex> lock(g_na_mu);
        if (!g_na_blocks[dev]) {  // once per device: cooperative-launch occupancy
            int per_sm = 0, sms = 0, coop = 0;
            const void *kernels[] = {(const void *)k_na_cg<1, false>, (const void *)k_na_cg<2, false>,
                                     (const void *)k_na_cg<NA_ROWS, false>};
            for (const void *k : kernels) {
                if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NA_SMEM);
                int ps = 0;
                if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, k, NA_NT, NA_SMEM);
                per_sm = k == kernels[0] || ps < per_sm ? ps : per_sm;
            }
            const void *clk = (const void *)k_na_cg<1, true>;
            if (e == cudaSuccess) e = cudaFuncSetAttribute(clk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)NA_SMEM);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(clk, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
            if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("device query: ") + cudaGetErrorString(e));
            if (!coop || per_sm < 1) return na_fail(SYSU_ERR_CUDA, "cooperative launch unavailable");
            if ((long long)sms * NA_NT * NA_ROWS < NA_MAX_ROWS)
                return na_fail(SYSU_ERR_CUDA, "the device has too few SMs for the solver");
            // the largest cluster the device takes, 0: none
            for (int cs = sysu::CL_MAX; cs >= 1 && !g_na_cluster[dev]; cs /= 2) {
                cudaLaunchAttribute at{};
                at.id = cudaLaunchAttributeClusterDimension;
                at.val.clusterDim.x = (unsigned)cs;
                at.val.clusterDim.y = at.val.clusterDim.z = 1;
                cudaLaunchConfig_t lc{};
                lc.gridDim = dim3(cs);
                lc.blockDim = dim3(NA_NT);
                lc.dynamicSmemBytes = NA_SMEM;
                lc.attrs = &at;
                lc.numAttrs = 1;
                int fit = 0;
                if (cudaOccupancyMaxActiveClusters(&fit, k_na_cg<1, true>, &lc) == cudaSuccess && fit > 0)
                    g_na_cluster[dev] = cs;
            }
            (void)cudaGetLastError();
            g_na_blocks[dev] = sms < sysu::AX_MAX_BLOCKS ? sms : sysu::AX_MAX_BLOCKS;
        }
        blocks = g_na_blocks[dev];
    }
    const int groups = (n + 31) / 32;
    const int G = groups < blocks ? groups : blocks;
    const int need = (32 * ((groups + G - 1) / G) + NA_NT - 1) / NA_NT;  // rows a thread
    // One cluster where a thread a row suffices: CTAs of 128 rows, one warp a scheduler, up to 16
    // of them, then more rows each.  Cluster against whole GPU, us an iteration: 512 rows 3.7 and
    // 5.9, 1,716 rows 3.9 and 6.1, 4,096 rows 4.4 and 6.0, 8,000 rows 5.8 and 6.0; with two rows a
    // thread and two sums 13,824 rows took 8.5 when the whole GPU took 6.8.  A matrix that the
    // cluster's shared memory does not hold (16 x 17,066 entries at most; k_na_dinv says so, and the
    // call launches again) goes to the whole GPU: 4,096 rows of 101 entries 11.6, 8,192 of 61 9.1,
    // where the cluster reading the caller's arrays took 54 and 47 and the form before it 46 and 32.
    int cluster = 0;
    if (n <= NA_CL_ROWS && g_na_cluster[dev] > 0) {
        cluster = 1;
        while (cluster < g_na_cluster[dev] && 4 * cluster < groups) cluster *= 2;
    }
    const int rows = cluster ? 32 * ((groups + cluster - 1) / cluster) : 0;
    if (rows > NA_NT) cluster = 0;
    const int threads = rows < 128 ? 128 : rows;
    NaArgs a{n, d_rowptr, d_col, d_val, d_b, d_x, omega, maxit, eps, base, cluster};
    // what must start at zero: the exchange area of the grid sums and the status words;
    // the malformed-row key starts at all ones (no row found)
    e = cudaMemsetAsync(base, 0, offsetof(NaHeader, bad), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(base + NA_SLOTS, 0, sysu::AX_WORDS * sizeof(double), st);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(reinterpret_cast<char *>(base) + offsetof(NaHeader, bad), 0xff, sizeof(unsigned long long),
                            st);
    if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
    k_na_dinv<<<(n + NA_KB - 1) / NA_KB, NA_KB, 0, st>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    void *args[] = {&a};
    const void *kern = need <= 1 ? (const void *)k_na_cg<1, false>
                                 : need <= 2 ? (const void *)k_na_cg<2, false> : (const void *)k_na_cg<NA_ROWS, false>;
    NaHeader h;
    auto whole_gpu = [&] { return cudaLaunchCooperativeKernel(kern, dim3(G), dim3(NA_NT), args, NA_SMEM, st); };
    auto read_back = [&] {
        cudaError_t r = cudaMemcpyAsync(&h, base, sizeof(NaHeader), cudaMemcpyDeviceToHost, st);
        return r == cudaSuccess ? cudaStreamSynchronize(st) : r;
    };
    if (cluster) {
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)cluster;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3(cluster);
        lc.blockDim = dim3(threads);
        lc.dynamicSmemBytes = NA_SMEM;
        lc.stream = st;
        lc.attrs = &at;
        lc.numAttrs = 1;
        e = cudaLaunchKernelEx(&lc, k_na_cg<1, true>, a);
    } else {
        e = whole_gpu();
    }
    if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("cooperative launch: ") + cudaGetErrorString(e));
    e = read_back();
    if (e == cudaSuccess && cluster && h.wide && h.bad == NA_GOOD) {
        e = whole_gpu();
        if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("cooperative launch: ") + cudaGetErrorString(e));
        e = read_back();
    }
    if (e != cudaSuccess) return na_fail(SYSU_ERR_CUDA, std::string("read-back: ") + cudaGetErrorString(e));
    if (h.bad != NA_GOOD) {
        static const char *what[] = {"", "a row pointer that decreases", "a column index outside 0..n-1",
                                     "no nonzero finite diagonal entry"};
        return na_fail(SYSU_ERR_INPUT, "sysu_csr_cg_noalloc: malformed CSR matrix: row " +
                                           std::to_string(h.bad >> 2) + " has " + what[h.bad & 3]);
    }
    if (iters) *iters = h.iters;
    if (res) *res = h.res;
    if (status) *status = h.err ? sysu::DEV_BARRIER_TIMEOUT : h.status;
    return SYSU_OK;
}

const char *sysu_noalloc_last_error(void) { return g_na_err.c_str(); }

}  // extern "C"
