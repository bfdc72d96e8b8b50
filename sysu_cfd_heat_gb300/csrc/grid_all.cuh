// Grid-wide sums and barriers of the persistent kernels that run at most one CTA per SM.
//
// What bounds a small solve is not its rows but the chain of dependent steps in a grid
// reduction: combine the warps, publish, wait for all blocks, read the partials, combine
// them.  On the 24^3 cavity's p' system (13,824 rows) an iteration has two of these.
//  - Sums are exact as in exact_sum.cuh, but a term is cut into six 24-bit limbs at
//    absolute limb positions (its exponent / 24), so aligning two numbers moves whole limbs
//    and a warp adds them with six redux.sync instead of five rounds of 128-bit shuffles,
//    shifts and carries.
//  - The blocks' sums meet in L2: each limb is one 64-bit word that every block adds to (one
//    red instruction of eight lanes), with an arrival count in the word's top byte.  A block
//    polls the eight words of a value, one 64-byte line, and has the total with the last
//    arrival; integer adds commute, so every run and every block sees the same bits.  The
//    words are never cleared: a block keeps their previous totals and takes the difference.
//    All blocks must add at the same limb positions: those of the previous sum at the same
//    place in the code (its channel).  Where some block's sum lies above them, or all lie more
//    than one limb below, every block sees it from the marks in the eighth word; they then
//    exchange their positions and add again.
//  - The barrier that orders the blocks' data runs beside it in another warp: a counter that
//    grows monotonically (a block adds 1 without waiting for the old value and polls for its
//    own target), with the fences that release and acquire.
// Tried and dropped: partials in slots read by every block after the counter (3.2 us a sum
// on 152 blocks), slots that every block polls (2.5 us for a bare barrier against 1.2 us
// through the counter), a mailbox of every block in every block (3.4 us).
#pragma once

#include "exact_sum.cuh"

namespace sysu {

constexpr int AX_NVMAX = 3;
constexpr int AX_MAX_BLOCKS = 255;  // the arrival count has 8 bits

// 64-bit words of a launch's exchange area: the counter, two sets of
// AX_NVMAX groups of accumulators, and a limb position a block and value.  Zero when the
// launch starts.
constexpr size_t AX_LINE = 128;  // accumulators 1 KB apart: at 128 B a sum of two values took 2.5 instead of 2.2 us
constexpr size_t AX_WORDS = AX_LINE + 2 * AX_NVMAX * AX_LINE + AX_NVMAX * (AX_MAX_BLOCKS + 1);
constexpr int AX_CHANNELS = 24;     // sums of a kernel that keep their limb positions apart

#ifdef __CUDACC__
namespace {

struct AllCtx {
    unsigned *count;
    unsigned long long *words;  // accumulators
    unsigned long long *pos;    // limb positions
    int G;
    unsigned target;            // counter value that completes the last operation; its tag
    int parity;
};

__device__ __forceinline__ AllCtx all_ctx(unsigned long long *area) {
    return AllCtx{reinterpret_cast<unsigned *>(area), area + AX_LINE, area + AX_LINE + 2 * AX_NVMAX * AX_LINE,
                  (int)gridDim.x, 0u, 0};
}

// A sum in progress: value = sum_j l[j] 2^(24 (P - 2 + j) - 1075).  A term of biased
// exponent e has P = e / 24 and occupies l[2..5]; l[0..1] keep the 48 bits below the
// largest term's last place that smaller terms reach into (what lies below is cut:
// less than 2^-100 of the largest term).
struct AxNum {
    int l[6];
    int P;
};

__shared__ __align__(16) int g_ax_warp[AX_NVMAX * 32 * 8];  // warp sums: limbs, P, nonfinite flag
__shared__ double g_ax_sum[AX_NVMAX];         // the sums, valid for the whole block after a call
__shared__ unsigned long long g_ax_prev[2][AX_NVMAX][8];  // the accumulators' last totals
__shared__ int g_ax_ref[AX_CHANNELS];         // limb position of a channel's next sum
__shared__ int g_ax_keep[AX_CHANNELS];        // sums for which it may not fall
__shared__ int g_ax_bad;

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned ld_relaxed32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Call once per launch, before the first operation, with all threads.
__device__ __forceinline__ void all_init() {
    for (int i = threadIdx.x; i < 2 * AX_NVMAX * 8; i += blockDim.x) (&g_ax_prev[0][0][0])[i] = 0ull;
    for (int i = threadIdx.x; i < AX_CHANNELS; i += blockDim.x) {
        g_ax_ref[i] = -1;
        g_ax_keep[i] = 0;
    }
    if (threadIdx.x == 0) g_ax_bad = 0;
    __syncthreads();
}

constexpr int AX_LIMB = (1 << 24) - 1;

// limbs moved down by d positions (P grows by d)
__device__ __forceinline__ void ax_down(AxNum &a, int d) {
    if (d & 1) {
#pragma unroll
        for (int j = 0; j < 6; ++j) a.l[j] = j + 1 < 6 ? a.l[j + 1] : 0;
    }
    if (d & 2) {
#pragma unroll
        for (int j = 0; j < 6; ++j) a.l[j] = j + 2 < 6 ? a.l[j + 2] : 0;
    }
    if (d & 4) {
#pragma unroll
        for (int j = 0; j < 6; ++j) a.l[j] = j + 4 < 6 ? a.l[j + 4] : 0;
    }
    if (d >= 6) {
#pragma unroll
        for (int j = 0; j < 6; ++j) a.l[j] = 0;
    }
}

// l[0..4] into [0, 2^24), the rest into the signed l[5]
__device__ __forceinline__ void ax_carry(AxNum &a) {
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        a.l[j + 1] += a.l[j] >> 24;
        a.l[j] &= AX_LIMB;
    }
}

__device__ __forceinline__ AxNum ax_term(double x, int &nonfinite) {
    unsigned long long m;
    bool neg;
    const int e = xs_split(x, m, neg, nonfinite);
    AxNum a;
    a.P = e / 24;
    const int s = e - 24 * a.P;
    const unsigned long long lo = m << s;
    const unsigned hi = s ? (unsigned)(m >> (64 - s)) : 0u;
    a.l[0] = a.l[1] = 0;
    a.l[2] = (int)lo & AX_LIMB;
    a.l[3] = (int)(lo >> 24) & AX_LIMB;
    a.l[4] = (int)((unsigned)(lo >> 48) | (hi << 16)) & AX_LIMB;
    a.l[5] = (int)(hi >> 8);
    if (neg) {
#pragma unroll
        for (int j = 2; j < 6; ++j) a.l[j] = -a.l[j];
    }
    return a;
}

// Sum over the warp's lanes of numbers with |l[j]| <= 2^24 (l[5] < 2^20), on every lane;
// the limbs of the result are below 2^29 and not carried.
__device__ __forceinline__ void ax_warp_sum(AxNum &a) {
    const int P = (int)__reduce_max_sync(FULL_MASK, (unsigned)a.P);
    if (!__all_sync(FULL_MASK, a.P == P)) ax_down(a, P - a.P);
    a.P = P;
#pragma unroll
    for (int j = 0; j < 6; ++j) a.l[j] = __reduce_add_sync(FULL_MASK, a.l[j]);
}

// sum_j l[j] 2^(24 (ref - 3 + j) - 1075) as FP64, correctly rounded; |l[j]| < 2^38, so that two limbs
// make a signed 64-bit group.  The largest come from ax_grid: limbs of carried block sums, at most
// 2^24 in size, from up to AX_MAX_BLOCKS blocks.
static_assert(AX_MAX_BLOCKS <= 1 << 13, "a limb's total over the blocks must stay below 2^38");
__device__ __forceinline__ double ax_to_double(const long long (&l)[7], int ref) {
    constexpr unsigned long long M48 = 0xFFFFFFFFFFFFull;
    // 48-bit groups g0..g2 in [0, 2^48) and the signed rest g3
    long long c = l[0] + (l[1] << 24);
    unsigned long long g0 = (unsigned long long)c & M48;
    c = (c >> 48) + l[2] + (l[3] << 24);
    unsigned long long g1 = (unsigned long long)c & M48;
    c = (c >> 48) + l[4] + (l[5] << 24);
    unsigned long long g2 = (unsigned long long)c & M48;
    long long g3 = (c >> 48) + l[6];
    const bool neg = g3 < 0;
    if (neg) {
        g0 = (g0 ^ M48) + 1;
        g1 = (g1 ^ M48) + (g0 >> 48);
        g2 = (g2 ^ M48) + (g1 >> 48);
        g3 = ~g3 + (long long)(g2 >> 48);
        g0 &= M48;
        g1 &= M48;
        g2 &= M48;
    }
    int sc = 24 * (ref - 3) - 1075;
    unsigned sticky = 0;
    if (g3 != 0) {  // the upper three groups, the lowest as a sticky bit
        sticky = g0 != 0;
        g0 = g1;
        g1 = g2;
        g2 = (unsigned long long)g3;
        sc += 48;
    }
    unsigned long long hi, lo;  // value = (hi 2^64 + lo) 2^sc
    if (g2 >> 32) {
        hi = (g2 << 16) | (g1 >> 32);
        lo = (g1 << 32) | (g0 >> 16) | (unsigned long long)((g0 & 0xFFFFu) != 0 || sticky);
        sc += 16;
    } else {
        hi = (g2 << 32) | (g1 >> 16);
        lo = (g1 << 48) | g0 | sticky;
    }
    if ((hi | lo) == 0) return 0.0;
    if (hi == 0) {
        hi = lo;
        lo = 0;
        sc -= 64;
    }
    const int z = __clzll((long long)hi);
    if (z) {
        hi = (hi << z) | (lo >> (64 - z));
        lo <<= z;
    }
    // value = 1.f 2^(sc + 127 - z): 53 bits of hi, the rest decides the rounding
    unsigned long long mant = hi >> 11;
    const unsigned rest = (unsigned)(hi & 0x7FF);
    if (rest > 0x400u || (rest == 0x400u && (lo != 0 || (mant & 1)))) ++mant;
    const int ex = sc + 127 - z + 1023;
    double d;
    if (ex >= 1 && ex < 0x7FE) {
        d = __longlong_as_double((long long)(((unsigned long long)ex << 52) + (mant - (1ull << 52))));
    } else {  // beyond FP64's normal range
        d = __ull2double_rn(mant);
        const int s = sc + 127 - z - 52;
        const int s1 = max(-1000, min(1000, s / 2)), s2 = max(-1000, min(1000, s - s / 2));
        d *= __longlong_as_double((long long)(s1 + 1023) << 52);
        d *= __longlong_as_double((long long)(s2 + 1023) << 52);
    }
    return neg ? -d : d;
}

// Waits until every block has arrived.
__device__ __forceinline__ bool ax_wait(const AllCtx &c) {
    long long spins = 0;
    while ((int)(ld_relaxed32(c.count) - c.target) < 0)
        if (++spins > BARRIER_SPIN_LIMIT) return false;
    return true;
}
__device__ __forceinline__ void ax_arrive(const AllCtx &c) {
    asm volatile("red.add.relaxed.gpu.global.u32 [%0], 1;" ::"l"(c.count) : "memory");
}
__device__ __forceinline__ void ax_fail(int *err) {
    *reinterpret_cast<volatile int *>(&g_ax_bad) = 1;
    atomicExch(err, (int)DEV_BARRIER_TIMEOUT);
}

// The sum over all blocks of the block sums `a` (carried; the same in every lane of the
// calling warp) of value k: in lane 0.  nf: the block saw a value that is not finite.
__device__ __forceinline__ double ax_grid(const AxNum &a, int nf, int k, int ch, const AllCtx &c, int *err) {
    const int lane = threadIdx.x & 31;
    unsigned long long *w = c.words + (size_t)(c.parity * AX_NVMAX + k) * AX_LINE + (lane & 7);
    unsigned long long prev = g_ax_prev[c.parity][k][lane & 7], diff = 0;
    int ref = g_ax_ref[ch], keep = g_ax_keep[ch];
    constexpr long long BIAS = 1ll << 34;  // keeps a contribution positive
    bool ok = true;
    for (;;) {
        // limbs ref - 3 .. ref + 3 in lanes 0..6, the marks in lane 7
        const int d = ref - a.P, idx = lane - 1 + d;
        int lv = 0;
#pragma unroll
        for (int j = 0; j < 6; ++j) lv = idx == j ? a.l[j] : lv;
        if (d < 0) lv = 0;
        unsigned long long add = (1ull << 56) + (unsigned long long)((long long)lv + BIAS);
        if (lane == 7)
            add = (1ull << 56) + (nf ? 1u : 0u) + (d < 0 ? 1ull << 16 : 0ull) + (d == 0 || d == 1 ? 1ull << 32 : 0ull);
        if (lane < 8) asm volatile("red.add.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w), "l"(add) : "memory");
        long long spins = 0;
        for (;;) {
            const unsigned long long cur = ld_relaxed64(w);
            diff = cur - prev;
            if (__all_sync(FULL_MASK, (int)(diff >> 56) == c.G)) {
                prev = cur;
                break;
            }
            if (++spins > BARRIER_SPIN_LIMIT) { ok = false; break; }
        }
        const unsigned long long marks = __shfl_sync(FULL_MASK, diff, 7);
        if (!ok || (((marks >> 16) & 0xFFFFu) == 0 && ((marks >> 32) & 0xFFFFu) != 0)) break;
        // some block's sum lies above the limbs, or all lie so far below that their own
        // would be cut: the largest position of all blocks
        unsigned long long *pos = c.pos + (size_t)k * (AX_MAX_BLOCKS + 1);
        if (lane == 0)
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(pos + blockIdx.x),
                         "l"(((unsigned long long)c.target << 32) | (unsigned)a.P)
                         : "memory");
        int P = 0;
        for (int b = lane; b < c.G && ok; b += 32) {
            unsigned long long q;
            long long n = 0;
            while ((unsigned)((q = ld_relaxed64(pos + b)) >> 32) != c.target)
                if (++n > BARRIER_SPIN_LIMIT) { ok = false; break; }
            P = max(P, (int)(unsigned)q);
        }
        ok = __all_sync(FULL_MASK, ok);
        if (!ok) break;
        ref = (int)__reduce_max_sync(FULL_MASK, (unsigned)P);
        keep = 64;
    }
    if (lane < 8) g_ax_prev[c.parity][k][lane] = prev;
    const long long v = (long long)(diff & ((1ull << 56) - 1)) - c.G * BIAS;
    long long l[7];
#pragma unroll
    for (int j = 0; j < 7; ++j) l[j] = __shfl_sync(FULL_MASK, v, j);
    const bool nan = (__shfl_sync(FULL_MASK, (unsigned)diff, 7) & 0xFFFFu) != 0;
    const double s = nan ? __longlong_as_double(0x7FF8000000000000ll) : ax_to_double(l, ref);
    if (lane == 0) {
        // the next sum's position: the total's, which the terms of a sum without
        // cancellation do not exceed
        const int P = ((int)(__double_as_longlong(s) >> 52) & 0x7FF) / 24;
        if (!nan && (P > ref || keep == 0)) g_ax_ref[ch] = P;
        else g_ax_ref[ch] = ref;
        g_ax_keep[ch] = max(keep - 1, 0);
        if (!ok) ax_fail(err);
    }
    return s;
}

// Each warp's sums of NV values per thread, to g_ax_warp.
template <int NV>
__device__ __forceinline__ void ax_warps(const double (&v)[NV]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        int *q = g_ax_warp + (k * 32 + warp) * 8;
        if (!__any_sync(FULL_MASK, v[k] != 0.0)) {  // warps without rows have nothing to add
            if (lane < 8) q[lane] = 0;
            continue;
        }
        int f = 0;
        AxNum a = ax_term(v[k], f);
        ax_warp_sum(a);
        const int nf = __any_sync(FULL_MASK, f);
        if (lane == 0) {
            int4 *o = reinterpret_cast<int4 *>(q);
            o[0] = make_int4(a.l[0], a.l[1], a.l[2], a.l[3]);
            o[1] = make_int4(a.l[4], a.l[5], a.P, nf);
        }
    }
}

// The block's sum of value k, carried, and whether a value was not finite: in every lane of
// the calling warp.
__device__ __forceinline__ AxNum ax_block(int k, int &nf) {
    const int lane = threadIdx.x & 31;
    AxNum a{{0, 0, 0, 0, 0, 0}, 0};
    int f = 0;
    if (lane < (int)(blockDim.x >> 5)) {  // lane w holds warp w's
        const int4 *q = reinterpret_cast<const int4 *>(g_ax_warp + (k * 32 + lane) * 8);
        const int4 u = q[0], w = q[1];
        a = AxNum{{u.x, u.y, u.z, u.w, w.x, w.y}, w.z};
        f = w.w;
    }
    ax_carry(a);
    ax_warp_sum(a);
    ax_carry(a);
    nf = __any_sync(FULL_MASK, f);
    return a;
}

// Exact sums of NV values per thread over the grid, and a barrier: what any thread wrote
// before the call, every thread may read after it.  Value k is combined by warp k, whose
// lane 0 calls fin(k, sum) before the block goes on (what it writes to shared memory, every
// thread may read after the call); idle() runs meanwhile in a thread with nothing to do (a
// division that the next step needs); the last warp orders the block's data: the block needs
// NV + 1 warps.  ch: the first of the NV channels of this place in the code.
struct AxNone {
    __device__ void operator()() const {}
};

template <int NV, class Fin, class Idle = AxNone>
__device__ __forceinline__ bool all_sum(const double (&v)[NV], int ch, AllCtx &c, int *err, Fin &&fin,
                                        Idle &&idle = Idle()) {
    static_assert(NV <= AX_NVMAX, "all_sum: too many values");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    ax_warps<NV>(v);
    c.target += (unsigned)c.G;
    c.parity ^= 1;
    __syncthreads();
    if (warp == nw - 1) {
        if (lane == 0) {
            fence_gpu();  // releases what the block's threads wrote before the __syncthreads
            ax_arrive(c);
            if (!ax_wait(c)) ax_fail(err);
            fence_gpu();  // acquires what the other blocks released
        }
        __syncwarp();
    } else if (warp < NV) {
        int f;
        const AxNum a = ax_block(warp, f);
        const double s = ax_grid(a, f, warp, ch + warp, c, err);
        if (lane == 0) fin(warp, s);
    } else if (warp == NV && lane == 0) {
        idle();
    }
    __syncthreads();
    return *reinterpret_cast<volatile int *>(&g_ax_bad) == 0;
}

// the sums into g_ax_sum
template <int NV>
__device__ __forceinline__ bool all_sum(const double (&v)[NV], int ch, AllCtx &c, int *err) {
    return all_sum<NV>(v, ch, c, err, [](int k, double s) { g_ax_sum[k] = s; });
}

// Barrier alone.
__device__ __forceinline__ bool all_sync(AllCtx &c, int *err) {
    c.target += (unsigned)c.G;
    __syncthreads();
    if (threadIdx.x == 0) {
        fence_gpu();
        ax_arrive(c);
        if (!ax_wait(c)) ax_fail(err);
        fence_gpu();
    }
    __syncthreads();
    return *reinterpret_cast<volatile int *>(&g_ax_bad) == 0;
}

// a / b by way of the reciprocal that an idle thread formed earlier, so that what stands in the
// chain of an iteration is a multiplication (a division takes 840 clocks).  recip: 0 where 1 / b
// is not a normal number (|b| below 2^-1021: it may be infinite where a / b is not); there the
// quotient is divided, and 0 / b is 0 also where b has underflowed to 0: CG then starts a new
// direction instead of losing x to 0 / 0.
__device__ __forceinline__ double recip(double b) {
    const int e = (__double2hiint(b) >> 20) & 0x7FF;  // |b| in [2^-1021, 2^1021), by integer tests
    return e >= 2 && e < 2044 ? 1.0 / b : 0.0;
}
__device__ __forceinline__ double quotient(double a, double b, double inv_b) {
    if (__double2hiint(inv_b) != 0) return a * inv_b;
    asm volatile("");  // a branch: the division is not to be formed beside the product
    return a == 0.0 ? 0.0 : a / b;
}

// The stopping test ||r|| / ||b|| < eps, on the squares where thr = stop_threshold(eps, bb) > 0 (a
// square root takes 2,600 clocks, a division 840).  0: eps is not positive, or eps^2 ||b||^2 leaves
// the range of normal numbers, and the norms themselves are compared.
__device__ __forceinline__ double stop_threshold(double eps, double bb) {
    const double thr = eps * eps * bb;
    return eps > 0.0 && thr >= 0x1p-1022 && isfinite(thr) ? thr : 0.0;
}
// (rr >= 0 or NaN and thr >= 0 compare as integers: an FP64 comparison waits 64 clocks)
__device__ __forceinline__ bool stop_below(double rr, double thr, double eps, double bb) {
    const long long t = __double_as_longlong(thr);
    if (t != 0) return __double_as_longlong(rr) < t;
    asm volatile("");  // a branch: the roots are not to be formed beside the comparison
    return eps > 0.0 && sqrt(rr) / sqrt(bb) < eps;
}
__device__ __forceinline__ bool finite_bits(double v) { return ((__double2hiint(v) >> 20) & 0x7FF) != 0x7FF; }

// ---- the same for a grid that is one thread-block cluster ----------------------
// The blocks write their sums into each other's shared memory and meet at the cluster's
// hardware barrier: 0.6 us a sum where the accumulators in L2 take 2 (16 blocks).  The totals
// have the same bits.
constexpr int CL_MAX = 16;

struct ClCtx {
    int G, rank, parity;
};

__shared__ __align__(16) int g_cl_slot[2][AX_NVMAX][CL_MAX][8];

__device__ __forceinline__ ClCtx cl_ctx() { return ClCtx{(int)gridDim.x, (int)blockIdx.x, 0}; }

// address of this block's shared variable p in block `rank` of the cluster
__device__ __forceinline__ unsigned cl_addr(const void *p, int rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ double cl_load(unsigned a) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cl_store(unsigned a, int x, int y, int z, int w) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w)
                 : "memory");
}
// Barrier of the cluster's threads: what any of them wrote before, all may read after, and
// what idle() writes to shared memory, the block's threads (by a barrier of their own).
__device__ __forceinline__ void cl_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <class Idle>
__device__ __forceinline__ void cl_sync(Idle &&idle) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (threadIdx.x == 32) idle();
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    __syncthreads();
}

// all_sum over the cluster; at least NV warps a block.
template <int NV, class Fin>
__device__ __forceinline__ void cl_sum(const double (&v)[NV], ClCtx &c, Fin &&fin) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ax_warps<NV>(v);
    __syncthreads();
    if (warp < NV) {
        int f;
        const AxNum a = ax_block(warp, f);
        if (lane < c.G) {
            const unsigned q = cl_addr(g_cl_slot[c.parity][warp][c.rank], lane);
            cl_store(q, a.l[0], a.l[1], a.l[2], a.l[3]);
            cl_store(q + 16, a.l[4], a.l[5], a.P, f);
        }
    }
    cl_sync();
    if (warp < NV) {
        AxNum a{{0, 0, 0, 0, 0, 0}, 0};
        int f = 0;
        if (lane < c.G) {
            const int4 *q = reinterpret_cast<const int4 *>(g_cl_slot[c.parity][warp][lane]);
            const int4 u = q[0], w = q[1];
            a = AxNum{{u.x, u.y, u.z, u.w, w.x, w.y}, w.z};
            f = w.w;
        }
        ax_warp_sum(a);
        f = __any_sync(FULL_MASK, f);
        const long long l[7] = {0, a.l[0], a.l[1], a.l[2], a.l[3], a.l[4], a.l[5]};
        const double s = f ? __longlong_as_double(0x7FF8000000000000ll) : ax_to_double(l, a.P);
        if (lane == 0) fin(warp, s);
    }
    c.parity ^= 1;
    __syncthreads();
}

// ---- CG with one sum an iteration ----------------------------------------------
// Chronopoulos and Gear's form of CG's two scalars: with w = A z, gamma = r.z, delta = w.z,
//     beta = gamma / gamma_old,   alpha = gamma / (delta - beta gamma / alpha_old)
// (p.q in the denominator: r is orthogonal to the old z), so both sums and the residual's are
// taken at once and an iteration has one sum and one bare barrier.  The quotients that only
// the next iteration needs are formed by an idle thread during the barrier.
struct CgScalars {
    double gamma, delta, beta, alpha, den;
    double old_gamma, inv_gamma, inv_alpha;  // of the iteration before
};

__device__ __forceinline__ void cg_first(CgScalars &S) {  // beta = 0 and nothing taken off delta
    S.old_gamma = __longlong_as_double(0x7FF0000000000000ll);
    S.inv_gamma = S.inv_alpha = 0.0;
}
__device__ __forceinline__ void cg_scalars(CgScalars &S) {
    S.beta = quotient(S.gamma, S.old_gamma, S.inv_gamma);
    S.den = fma(-(S.beta * S.inv_alpha), S.gamma, S.delta);
    S.alpha = S.den == 0.0 ? 0.0 : S.gamma / S.den;
}
__device__ __forceinline__ void cg_next(CgScalars &S) {
    S.old_gamma = S.gamma;
    S.inv_gamma = recip(S.gamma);
    S.inv_alpha = S.gamma == 0.0 ? 0.0 : quotient(S.den, S.gamma, S.inv_gamma);
}

}  // namespace
#endif  // __CUDACC__

}  // namespace sysu
