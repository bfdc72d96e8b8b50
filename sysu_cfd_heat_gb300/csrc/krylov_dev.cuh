// Device and host helpers shared by the Krylov translation units (included
// once per .cu file; everything sits in an anonymous namespace).
#pragma once

#include <algorithm>
#include <cstdint>
#include <initializer_list>

#include "exact_sum.cuh"
#include "krylov.hpp"

namespace sysu {
namespace {

constexpr int KB = 256;
constexpr int NVMAX = 6;

struct RedCtx {
    double *partials;
    int G;
    int parity;
};

// Exact deterministic grid sums of NV <= XS_NVMAX values per thread
// (exact_sum.cuh); the sums are valid in thread 0 only.  Per-block partials are
// (exponent, 128-bit sum, nonfinite flag) in four 64-bit words, double
// buffered, so that a block that runs ahead to the next sum cannot overwrite
// values another block is still reading; rc.partials must hold 2 * XS_NVMAX * G * 4 words.
constexpr int XS_NVMAX = 3;
__shared__ long long g_xs_smem[XS_NVMAX * 32 * 4];

template <int NV>
__device__ __forceinline__ bool grid_sum_t0(double (&v)[NV], RedCtx &rc, GridBarrier *gb, int *err) {
    static_assert(NV <= XS_NVMAX, "grid_sum_t0: too many values");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        int E, nf;
        I128 S;
        xs_warp(v[k], E, S, nf);
        if (lane == 0) {
            long long *q = g_xs_smem + (k * 32 + warp) * 4;
            q[0] = E;
            q[1] = (long long)S.lo;
            q[2] = S.hi;
            q[3] = nf;
        }
    }
    __syncthreads();
    long long *buf = reinterpret_cast<long long *>(rc.partials) + (size_t)rc.parity * XS_NVMAX * rc.G * 4;
    rc.parity ^= 1;
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            int e = 0, f = 0;
            I128 s{0ull, 0ll};
            if (lane < nw) {
                const long long *q = g_xs_smem + (k * 32 + lane) * 4;
                e = (int)q[0];
                s.lo = (unsigned long long)q[1];
                s.hi = q[2];
                f = (int)q[3];
            }
            int E, nf;
            I128 S;
            xs_combine(e, s, f, 0, E, S, nf);
            if (lane == 0) {
                long long *o = buf + ((size_t)k * rc.G + blockIdx.x) * 4;
                o[0] = E;
                o[1] = (long long)S.lo;
                o[2] = S.hi;
                o[3] = nf;
            }
        }
    }
    if (!grid_sync(gb, err)) return false;
    if (warp == 0) {
        // every lane loads its blocks' partials in one pass (16-byte loads), for
        // up to XS_LANE_BLOCKS * 32 blocks at a time
        constexpr int XS_LANE_BLOCKS = 5;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const longlong2 *pk = reinterpret_cast<const longlong2 *>(buf + (size_t)k * rc.G * 4);
            int E = 0, f = 0;
            I128 t{0ull, 0ll};
            for (int c0 = 0; c0 < rc.G; c0 += 32 * XS_LANE_BLOCKS) {
                longlong2 q0[XS_LANE_BLOCKS], q1[XS_LANE_BLOCKS];
#pragma unroll
                for (int j = 0; j < XS_LANE_BLOCKS; ++j) {
                    int blk = c0 + lane + 32 * j;
                    if (blk < rc.G) {
                        q0[j] = __ldcg(pk + 2 * blk);      // exponent, low word
                        q1[j] = __ldcg(pk + 2 * blk + 1);  // high word, flag
                    } else {
                        q0[j] = make_longlong2(0, 0);
                        q1[j] = make_longlong2(0, 0);
                    }
                }
                int em = 0;
#pragma unroll
                for (int j = 0; j < XS_LANE_BLOCKS; ++j)
                    if (q0[j].y != 0 || q1[j].x != 0) em = max(em, (int)q0[j].x);
                int Ec = __reduce_max_sync(FULL_MASK, em);
                if (Ec > E) {  // rescale what earlier chunks summed (rare: more than 160 blocks)
                    t = xs_sar(t, Ec - E);
                    E = Ec;
                }
#pragma unroll
                for (int j = 0; j < XS_LANE_BLOCKS; ++j) {
                    f |= (int)q1[j].y;
                    I128 sb{(unsigned long long)q0[j].y, q1[j].x};
                    if (sb.lo != 0 || sb.hi != 0) t = xs_add(t, xs_sar(sb, E - (int)q0[j].x + XS_G));
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t = xs_add(t, xs_shfl_xor(t, o));
            int nf = __reduce_or_sync(FULL_MASK, f);
            if (lane == 0) v[k] = xs_to_double(E, t, nf, XS_G);
        }
    }
    return true;
}

// scalars broadcast from thread 0 to the block
__shared__ double g_bc[8];

// A power of two s with s^2 rr in [1, 4) (1 when rr is zero or not finite).
// The FP32 inner solves of the mixed-precision forms work on s r, so residuals
// that have become tiny (or huge) in FP64 neither underflow nor overflow in
// FP32; scaling by a power of two is exact.
__device__ __forceinline__ double pow2_scale(double rr) {
    if (!(rr > 0.0) || !isfinite(rr)) return 1.0;
    const int e = ilogb(rr);
    const int h = e >= 0 ? e / 2 : -((1 - e) / 2);  // floor(e / 2)
    return ldexp(1.0, -h);
}

// One SELL row: the loads of four entries are issued before their FMAs, so a
// thread keeps several independent gathers in flight (rows hold 4-7 entries).
__device__ __forceinline__ double row_dot(const SellView &A, int i, const double *__restrict__ x) {
    int s = i >> 5;
    int e = A.sl_ptr[s] + (i & 31);
    int w = A.sl_w[s];
    double acc = 0.0;
    int k = 0;
    for (; k + 4 <= w; k += 4, e += 128) {
        int c0 = __ldg(A.col + e), c1 = __ldg(A.col + e + 32), c2 = __ldg(A.col + e + 64), c3 = __ldg(A.col + e + 96);
        double a0 = __ldg(A.val + e), a1 = __ldg(A.val + e + 32), a2 = __ldg(A.val + e + 64), a3 = __ldg(A.val + e + 96);
        double x0 = x[c0], x1 = x[c1], x2 = x[c2], x3 = x[c3];
        acc += a0 * x0;
        acc += a1 * x1;
        acc += a2 * x2;
        acc += a3 * x3;
    }
    for (; k < w; ++k, e += 32) acc += __ldg(A.val + e) * x[__ldg(A.col + e)];
    return acc;
}


__global__ void k_jacobi_dinv(SellView A, double omega, int jacobi, double *dinv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    if (!jacobi) {
        dinv[i] = 1.0;
        return;
    }
    double d = A.val[A.sl_ptr[i >> 5] + (i & 31)];
    dinv[i] = omega / d;
}

__global__ void k_zero(double *x, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = 0.0;
}

// Phase timestamps for profiling: block 0 records %globaltimer at the phase
// boundaries of the first PHASE_TS_ITERS iterations (4 per iteration).
constexpr int PHASE_TS_ITERS = 64;
__device__ __forceinline__ void stamp(unsigned long long *ts, int it, int k) {
    if (ts && blockIdx.x == 0 && threadIdx.x == 0 && it >= 1 && it <= PHASE_TS_ITERS) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        ts[(it - 1) * 4 + k] = t;
    }
}

__device__ __forceinline__ float4 ld4(const float *p, int j) { return reinterpret_cast<const float4 *>(p)[j]; }
__device__ __forceinline__ void st4(float *p, int j, float4 v) { reinterpret_cast<float4 *>(p)[j] = v; }

// Non-persistent kernels: thread 0 of every block publishes its block's NV
// totals to part[block][NV] and counts its arrival; the last block to arrive
// adds all partials up (every thread of that block loads a strided share, then
// a block reduction in a fixed order).  Returns true in exactly one thread
// (thread 0 of the last block), which then holds the totals in v.  sm: NV * 8
// doubles of shared memory (blocks of at most 256 threads).
template <int NV>
__device__ bool grid_sums_publish(double (&v)[NV], double *part, unsigned *cnt, double *sm) {
    __shared__ int s_last;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) part[(size_t)blockIdx.x * NV + k] = v[k];
        __threadfence();
        unsigned prev = atomicAdd(cnt, 1u);
        s_last = prev == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    double t[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) t[k] = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < NV; ++k) t[k] += __ldcg(part + (size_t)b * NV + k);
    block_sum_t0<NV>(t, sm);
    if (threadIdx.x != 0) return false;
    *cnt = 0;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = t[k];
    return true;
}

// Grid sums of FP64 per-thread values (block sum in FP64).
template <int NV>
__device__ bool grid_sums(double (&v)[NV], double *part, unsigned *cnt) {
    __shared__ double sm[NV * 8];
    block_sum_t0<NV>(v, sm);
    return grid_sums_publish<NV>(v, part, cnt, sm);
}

// One step of the warp's butterfly over NV values with the values dealt out: a lane keeps
// the half of the values that its side of the step owns and adds its partner's, so NV values
// cost about NV additions instead of 5 NV.  The additions are those of the butterfly of each
// value (xor 16, 8, 4, 2, 1): the same bits.  Returns how many values a lane still holds.
template <int NV>
__device__ __forceinline__ double deal_sum(const double (&v)[NV], int o) {
    const int lane = threadIdx.x & 31;
    if constexpr (NV == 1) {
        double s = v[0];
        for (; o > 0; o >>= 1) s += __shfl_xor_sync(FULL_MASK, s, o);
        return s;
    } else {
        constexpr int H = (NV + 1) / 2;  // the lower side keeps values 0..H-1, the upper H..NV-1
        const bool up = (lane & o) != 0;
        double k[H];
#pragma unroll
        for (int j = 0; j < H; ++j) {
            const double lo = v[j], hi = H + j < NV ? v[H + j] : 0.0;
            const double other = __shfl_xor_sync(FULL_MASK, up ? lo : hi, o);
            k[j] = (up ? hi : lo) + other;
        }
        return deal_sum<H>(k, o >> 1);
    }
}
// lane that holds value k's sum after deal_sum<NV>
template <int NV>
__device__ __forceinline__ int deal_lane(int k, int o = 16) {
    if constexpr (NV == 1) {
        return 0;
    } else {
        constexpr int H = (NV + 1) / 2;
        return k < H ? deal_lane<H>(k, o >> 1) : o + deal_lane<H>(k - H, o >> 1);
    }
}

// Grid sums of FP32 per-thread partials, for blocks of up to 256 threads: true in every thread of
// the last block to arrive, which finds the sums in g_gt_sum.  The warp sums stay in FP32 (a
// fixed butterfly, so the total is the same on every run); only the warp totals go to FP64 for
// the block and grid sums.  An FP64 shuffle tree in every thread runs on GB300's FP64 pipe
// (1/64 of the FP32 rate): 6 FP64 operations per value and thread took 10-20 us of a 2M-row
// vector pass.  What is left is the tail after the last block's arrival, a chain of FP64
// additions of 65 clocks each: values side by side, a lane each or dealt over the lanes, not
// one after the other in one thread, and callers work their scalars out with a thread a
// component.  The order of each value's additions (warp butterflies, then the warps one after
// the other) is part of the results: BiCGSTAB amplifies a last bit to 1e-9 of the solution.  On 262,144 rows k_m3_upd (six sums, three components' scalars) went
// from 21.8 to 12.8 us, k_m3_at from 17.0 to 11.4 and k_fcg_upd from 11.1 to 8.1.
__shared__ double g_gt_warp[NVMAX * 8], g_gt_sum[NVMAX];

template <int NV>
__device__ bool grid_totals_f(const float (&f)[NV], double *part, unsigned *cnt) {
    static_assert(NV <= NVMAX && NV * 8 <= 64, "grid_totals_f: too many values");
    __shared__ float sm[NV * 8];
    __shared__ int s_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5, G = gridDim.x;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        float g = f[k];
        for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(FULL_MASK, g, o);
        if (lane == 0) sm[k * 8 + warp] = g;
    }
    __syncthreads();
    if (tid < NV) {
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += (double)sm[tid * 8 + w];
        part[(size_t)tid * G + blockIdx.x] = s;
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        s_last = atomicAdd(cnt, 1u) == (unsigned)G - 1u;
    }
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    double t[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) t[k] = 0.0;
    for (int b = tid; b < G; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < NV; ++k) t[k] += __ldcg(part + (size_t)k * G + b);
    const double w = deal_sum<NV>(t, 16);
#pragma unroll
    for (int k = 0; k < NV; ++k)
        if (lane == deal_lane<NV>(k)) g_gt_warp[k * 8 + warp] = w;
    __syncthreads();
    if (tid < NV) {
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += g_gt_warp[tid * 8 + w];
        g_gt_sum[tid] = s;
    }
    if (tid == 0) *cnt = 0;
    __syncthreads();
    return true;
}

int g_num_sms = 0;

int num_sms() {
    if (!g_num_sms) {
        int dev;
        SYSU_CUDA(cudaGetDevice(&dev));
        SYSU_CUDA(cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev));
        int coop = 0;
        SYSU_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        if (!coop) throw CaseError{"device does not support cooperative launch"};
    }
    return g_num_sms;
}

template <class K>
int coresident_blocks(K kernel, int block = KB) {
    int per_sm = 0;
    SYSU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0));
    if (per_sm < 1) throw CaseError{"persistent Krylov kernel cannot be resident"};
    return per_sm * num_sms();
}

SellView view(const SellDev &A, const double *val) {
    return SellView{A.n, A.nslices, A.sl_ptr.get(), A.sl_w.get(), A.col.get(), val};
}

int grid_for(int n, int max_blocks, int block = KB) {
    int want = (n + block - 1) / block;
    return std::max(1, std::min(want, max_blocks));
}

// the vector phases of the CG kernels use 16-byte loads
void check_aligned16(std::initializer_list<const void *> ptrs) {
    for (const void *p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) % 16 != 0) throw CaseError{"CG vectors must be 16-byte aligned"};
}


}  // namespace
}  // namespace sysu
