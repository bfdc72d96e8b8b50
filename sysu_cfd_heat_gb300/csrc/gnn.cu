// Learned preconditioner (see gnn.hpp): network forward / backward on the
// tensor cores, Adam, and flexible CG with fallback to Jacobi.
//
// Network kernels work on tiles of 128 rows, one thread per row, four warps
// per CTA; warp w of a tile owns SELL slice 4t + w, so matrix loads are the
// coalesced SELL-32 pattern, and thread t's row is TMEM lane t of the MMA
// accumulator.  A thread gathers its row's neighbours (FP32 accumulation of
// BF16 activations), writes its operand row to shared memory, one elected
// thread issues the MMAs, the commit arrives on an mbarrier (bounded wait),
// and every thread reads its own accumulator row back for the epilogue.
//
// Reductions (scale, loss, the flexible-CG scalars) are per-block partial
// sums that the last block to finish adds up in block order, so results are
// run-to-run deterministic; so are the parameter gradients (per-CTA records,
// summed in a fixed order by the Adam kernel).
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <random>

#include "gnn.hpp"
#include "graph_loop.hpp"
#include "krylov_dev.cuh"
#include "umma.cuh"

namespace sysu {
namespace {

constexpr int GT = 128;  // rows per tile = threads per CTA of the network kernels
constexpr int FB = 256;  // threads per block of the flat kernels
constexpr uint32_t IDESC_F = umma::idesc_bf16_f32(128, 32);   // forward: 128 x 32, K = 64
constexpr uint32_t IDESC_B1 = umma::idesc_bf16_f32(128, 64);  // backward, input gradient: 128 x 64, K = 32
// backward, weight gradient: 128 x 32, K = 128, both operands MN-major
constexpr uint32_t IDESC_B2 = umma::idesc_bf16_f32(128, 32) | umma::IDESC_A_MN | umma::IDESC_B_MN;

constexpr int FWD_G = 2048 + 32;  // forward: a group of the operand tile
constexpr int FWD_SMEM = 8 * FWD_G + 4096 + 136 * 4 + 16;
// backward: X tile, weights, transposition tiles, dpre tile (the 32 bytes between its groups
// spread a row's four groups over the banks), parameters and sums
constexpr int BWD_X = 32768, BWD_W = 4096, BWD_T = 16384, BWD_DG = 2048 + 32, BWD_D = 4 * BWD_DG;
constexpr int BWD_SMEM = BWD_X + BWD_W + BWD_T + BWD_D + (96 + 256) * 4 + 16;
// The backward kernel holds 128 TMEM columns; requesting this much shared
// memory caps it at three resident CTAs per SM (384 of 512 columns).
constexpr int BWD_SMEM_REQ = 64 * 1024;
static_assert(BWD_SMEM <= BWD_SMEM_REQ, "backward shared-memory layout");

struct GView {
    int n;
    const int *sl_ptr, *sl_w, *col;
    const float *val;
    const float *dinv;
};

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t bf_pack(float a, float b) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(a)) |
           ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(b)) << 16);
}

// The flexible-CG kernels accumulate each thread's rows (a handful) in FP32 and
// hand those partials to grid_totals_f (FP32 warp sums, FP64 block and grid
// sums): per-row FP64 arithmetic and conversions run on GB300's FP64 pipe (1/64
// of the FP32 rate) and took half of these kernels' time.  Convergence is
// decided on the FP64 residual b - A x.

// ---------------------------------------------------------------- forward --

struct NetArgs {
    GView g;
    const float *r;
    const float *inv_s_p, *s_p;
    const uint16_t *wbf;  // this layer's BF16 weights (Wt[32][64] at +0)
    const float *prm;
    int layer;
    const uint16_t *hin;
    uint16_t *hout, *mout;
    uint32_t *mask;
    float *aw;
    float *z;
    const float *zbase;  // multigrid form: z = zbase + network output
    float skip;          // weight of the Jacobi term u in the decoder (1 as a whole preconditioner)
    const float *qprev;
    FcgState *fs;
    double *part;
    int *err;
};

// What bounds this kernel is its gathers: a row's neighbours, 64 bytes of BF16 features each.
// TR, the rows of a tile:
//   128  a thread gathers and finishes its own row; 28 warps an SM hide the latencies.
//   32   four lanes take a row, 16 bytes each, and the four warps eight rows each; eight
//        neighbours' features are in flight and the next eight columns on their way.  The
//        MMA's other 96 rows go unused, and one warp finishes the 32 rows.  For levels of a few
//        thousand rows, where 128-row tiles leave most SMs without work and the time is one
//        thread's chain of gathers: 7 to 9 us a layer where that took 16 to 18 (second coarse
//        level of a 264,000-cell tetrahedral mesh).
// The operand tile is stored as groups of 8 features, byte(r, c) = (c / 8) * FWD_G + 16 r +
// 2 (c % 8); the 32 bytes between groups keep a row's four lanes on different banks, and the
// new features leave through it, four lanes a row (126,720 rows, four layers: 64 -> 61 us).
template <bool L1, bool TRAIN, bool DEC, int TR>
__global__ void __launch_bounds__(GT) k_gnn_fwd(NetArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *sX = smem;          // [h, m]: 8 groups of 8 features x 128 rows
    uint8_t *sB = smem + 8 * FWD_G;  // Wt: 32 outputs x 64 inputs
    float *sprm = reinterpret_cast<float *>(sB + 4096);  // bias, e, c, w_d, b_d
    uint64_t *bar = reinterpret_cast<uint64_t *>(sprm + 136);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q4 = lane & 3, l8 = 8 * warp + (lane >> 2);  // 32-row tiles: this lane's chunk and row
    const int s0 = TR == 128 ? 32 * warp : 0;              // the warp's slice in the tile
    if (a.fs && (a.fs->done || !a.fs->use_gnn)) return;

    for (int q = tid; q < 32 * 8; q += GT) {
        int o = q >> 3, c = q & 7;
        uint4 w = *reinterpret_cast<const uint4 *>(a.wbf + o * 64 + c * 8);
        *reinterpret_cast<uint4 *>(sB + ((o >> 3) * 8 + c) * 128 + (o & 7) * 16) = w;
    }
    const float *lp = a.prm + GNN_OFF_LAYER + a.layer * GNN_LAYER_STRIDE;
    if (tid < 32) {
        sprm[tid] = lp[2048 + tid];
        sprm[32 + tid] = a.prm[GNN_OFF_ENC + tid];
        sprm[64 + tid] = a.prm[GNN_OFF_ENC + 32 + tid];
        sprm[96 + tid] = a.prm[GNN_OFF_DEC + tid];
        if (tid == 0) sprm[128] = a.prm[GNN_OFF_DEC + 32];
    }
    if (warp == 0) umma::tmem_alloc(tslot, 32);
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    umma::fence_smem_to_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;
    const float inv_s = *a.inv_s_p, s_net = *a.s_p;
    const int n = a.g.n, ntiles = (n + TR - 1) / TR;
    const uint32_t x0 = umma::smem_addr(sX), b0 = umma::smem_addr(sB);
    const bool rows = TR == 128 || warp == 0;                // has a row a thread
    uint8_t *xrow = sX + tid * 16;                           // this thread's row
    uint8_t *xchunk = sX + q4 * FWD_G + l8 * 16;             // 32-row tiles: this lane's chunk
    float zq = 0.f;
    int it = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
        const int row0 = t * TR + s0;  // the warp's slice
        const int row = row0 + lane;
        const bool valid = row < n;
        int base = 0, w = 0;
        if (row0 < n) {
            base = a.g.sl_ptr[row0 >> 5];
            w = a.g.sl_w[row0 >> 5];
        }
        const float di = valid ? a.g.dinv[row] : 0.f;
        uint32_t hs[16];  // the row's h (BF16 pairs)
        if (L1 && rows) {
            float ui = 0.f, ai = 0.f, wi = 0.f;
            if (valid) {
                float su = 0.f, sw = 0.f;
#pragma unroll 4
                for (int k = 1; k < w; ++k) {
                    int pos = base + k * 32 + lane;
                    int j = a.g.col[pos];
                    float v = a.g.val[pos];
                    su += v * (a.g.dinv[j] * a.r[j]);
                    sw += v;
                }
                ai = di * su * inv_s;
                wi = di * sw;
                ui = di * a.r[row] * inv_s;
                if (TRAIN) {
                    a.aw[2 * (size_t)row] = ai;
                    a.aw[2 * (size_t)row + 1] = wi;
                }
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t m[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int c = 8 * g + 2 * e;
                    const float e0 = sprm[32 + c], e1 = sprm[33 + c], c0 = sprm[64 + c], c1 = sprm[65 + c];
                    hs[4 * g + e] = valid ? bf_pack(ui * e0 + c0, ui * e1 + c1) : 0u;
                    m[e] = bf_pack(ai * e0 + wi * c0, ai * e1 + wi * c1);
                }
                *reinterpret_cast<uint4 *>(xrow + g * FWD_G) =
                    make_uint4(hs[4 * g], hs[4 * g + 1], hs[4 * g + 2], hs[4 * g + 3]);
                *reinterpret_cast<uint4 *>(xrow + (4 + g) * FWD_G) = make_uint4(m[0], m[1], m[2], m[3]);
            }
        }
        if (!L1 && TR == 128) {
            float mv[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) mv[c] = 0.f;
#pragma unroll
            for (int c = 0; c < 16; ++c) hs[c] = 0u;
            if (valid) {
                const uint4 *hp = reinterpret_cast<const uint4 *>(a.hin + (size_t)row * 32);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint4 h4 = __ldg(hp + q);
                    hs[4 * q] = h4.x;
                    hs[4 * q + 1] = h4.y;
                    hs[4 * q + 2] = h4.z;
                    hs[4 * q + 3] = h4.w;
                }
                // two neighbours per step: eight 16-byte loads in flight per thread
                for (int k = 1; k < w; k += 2) {
                    const int pos = base + k * 32 + lane;
                    const bool two = k + 1 < w;
                    const int j0 = a.g.col[pos];
                    const float v0 = a.g.val[pos];
                    const int j1 = two ? a.g.col[pos + 32] : j0;
                    const float v1 = two ? a.g.val[pos + 32] : 0.f;
                    const uint4 *p0 = reinterpret_cast<const uint4 *>(a.hin + (size_t)j0 * 32);
                    const uint4 *p1 = reinterpret_cast<const uint4 *>(a.hin + (size_t)j1 * 32);
                    uint4 x[4], y[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        x[q] = __ldg(p0 + q);
                        y[q] = __ldg(p1 + q);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t xw[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
                        const uint32_t yw[4] = {y[q].x, y[q].y, y[q].z, y[q].w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            mv[8 * q + 2 * e] += v0 * bf_lo(xw[e]) + v1 * bf_lo(yw[e]);
                            mv[8 * q + 2 * e + 1] += v0 * bf_hi(xw[e]) + v1 * bf_hi(yw[e]);
                        }
                    }
                }
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t m[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) m[e] = bf_pack(mv[8 * g + 2 * e] * di, mv[8 * g + 2 * e + 1] * di);
                const uint4 m4 = make_uint4(m[0], m[1], m[2], m[3]);
                *reinterpret_cast<uint4 *>(xrow + g * FWD_G) =
                    make_uint4(hs[4 * g], hs[4 * g + 1], hs[4 * g + 2], hs[4 * g + 3]);
                *reinterpret_cast<uint4 *>(xrow + (4 + g) * FWD_G) = m4;
                if (TRAIN && valid) reinterpret_cast<uint4 *>(a.mout + (size_t)row * 32)[g] = m4;
            }
        }
        if (!L1 && TR == 32) {
            const uint16_t *hq = a.hin + 8 * q4;
            const bool in = row0 + l8 < n;
            float mv[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) mv[e] = 0.f;
            int c[8];
            float v[8];
            // columns and values of the row's neighbours k .. k + 7, past the last one the row itself
            // with weight 0 (another row's features may be infinite)
            auto entries = [&](int k) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    c[i] = in ? row0 + l8 : 0;
                    v[i] = 0.f;
                    if (in && k + i < w) {
                        c[i] = a.g.col[base + (k + i) * 32 + l8];
                        v[i] = a.g.val[base + (k + i) * 32 + l8];
                    }
                }
            };
            entries(1);
            uint4 h = make_uint4(0, 0, 0, 0);
            if (in) h = __ldg(reinterpret_cast<const uint4 *>(hq + (size_t)(row0 + l8) * 32));
            // eight gathers in flight, the next eight neighbours' columns on their way
            for (int k = 1; k < w; k += 8) {
                uint4 x[8];
                float u[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    x[i] = __ldg(reinterpret_cast<const uint4 *>(hq + (size_t)c[i] * 32));
                    u[i] = v[i];
                }
                entries(k + 8);
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    const uint32_t xw[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
                    const uint32_t yw[4] = {x[i + 1].x, x[i + 1].y, x[i + 1].z, x[i + 1].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        mv[2 * e] += u[i] * bf_lo(xw[e]) + u[i + 1] * bf_lo(yw[e]);
                        mv[2 * e + 1] += u[i] * bf_hi(xw[e]) + u[i + 1] * bf_hi(yw[e]);
                    }
                }
            }
            const float d = __shfl_sync(FULL_MASK, di, l8);
            uint32_t m[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) m[e] = in ? bf_pack(mv[2 * e] * d, mv[2 * e + 1] * d) : 0u;
            const uint4 m4 = make_uint4(m[0], m[1], m[2], m[3]);
            *reinterpret_cast<uint4 *>(xchunk) = h;
            *reinterpret_cast<uint4 *>(xchunk + 4 * FWD_G) = m4;
            if (TRAIN && in) *reinterpret_cast<uint4 *>(a.mout + (size_t)(row0 + l8) * 32 + 8 * q4) = m4;
        }
        umma::fence_smem_to_async();
        umma::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            umma::fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                umma::mma_bf16(tmem, umma::smem_desc(x0 + kk * 2 * FWD_G, FWD_G, 128),
                               umma::smem_desc(b0 + kk * 256, 128, 1024), IDESC_F, kk > 0);
            umma::commit(bar);
        }
        __syncwarp();
        bool fail = !mbar_wait(bar, it & 1);
        if (__syncthreads_or(fail)) {
            if (tid == 0) atomicExch(a.err, (int)DEV_BARRIER_TIMEOUT);
            break;
        }
        umma::fence_after_sync();
        if (rows) {
            float pre[32];
            umma::ld32(tmem + ((uint32_t)(warp * 32) << 16), pre);
            if (!L1 && TR == 32) {
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const uint4 h = *reinterpret_cast<const uint4 *>(xrow + g * FWD_G);
                    hs[4 * g] = h.x;
                    hs[4 * g + 1] = h.y;
                    hs[4 * g + 2] = h.z;
                    hs[4 * g + 3] = h.w;
                }
            }
            uint32_t ho[16];
            uint32_t mbits = 0;
#pragma unroll
            for (int c = 0; c < 32; c += 2) {
                float p0 = pre[c] + sprm[c], p1 = pre[c + 1] + sprm[c + 1];
                float h0 = bf_lo(hs[c >> 1]) + fmaxf(p0, 0.f);
                float h1 = bf_hi(hs[c >> 1]) + fmaxf(p1, 0.f);
                mbits |= (p0 > 0.f ? 1u : 0u) << c;
                mbits |= (p1 > 0.f ? 1u : 0u) << (c + 1);
                ho[c >> 1] = bf_pack(h0, h1);
            }
            if (!DEC || TRAIN) {  // rows to chunks through the tile (this warp's rows only)
#pragma unroll
                for (int g = 0; g < 4; ++g)
                    *reinterpret_cast<uint4 *>(xrow + g * FWD_G) =
                        make_uint4(ho[4 * g], ho[4 * g + 1], ho[4 * g + 2], ho[4 * g + 3]);
                __syncwarp();
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    if (row0 + 8 * s + (lane >> 2) < n)
                        *reinterpret_cast<uint4 *>(a.hout + (size_t)(row0 + 8 * s + (lane >> 2)) * 32 + 8 * q4) =
                            *reinterpret_cast<const uint4 *>(sX + q4 * FWD_G + (s0 + 8 * s + (lane >> 2)) * 16);
            }
            if (valid) {
                if (TRAIN) a.mask[row] = mbits;
                if (DEC) {
                    float acc = sprm[128];
#pragma unroll
                    for (int c = 0; c < 32; c += 2) acc += sprm[96 + c] * bf_lo(ho[c >> 1]) + sprm[97 + c] * bf_hi(ho[c >> 1]);
                    float u = di * a.r[row] * inv_s;
                    float zi = s_net * (a.skip * u + acc);
                    if (a.zbase) zi += a.zbase[row];
                    a.z[row] = zi;
                    if (a.qprev) zq = fmaf(zi, a.qprev[row], zq);
                }
            }
        }
        // the tile's rows are read before the next tile's are written
        if (TR == 128) __syncwarp();
        else __syncthreads();
    }
    if (DEC && a.fs) {
        const float fv[1] = {zq};
        if (grid_totals_f<1>(fv, a.part, &a.fs->cnt[0]) && threadIdx.x == 0) a.fs->zq = g_gt_sum[0];
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_free(tmem, 32);
}

// --------------------------------------------------------------- backward --

struct BwdArgs {
    GView g;
    float sgn;
    int kind;
    const float *r;
    const float *inv_s_p, *s_p;
    const uint16_t *wbf;
    const float *prm;
    int layer;
    const uint16_t *hprev, *mcur;
    const uint32_t *mask;
    const float *aw;
    const uint16_t *h4;
    const float *y;
    const GnnScalars *sc;
    const float *dIn, *gIn;
    float *dOut, *gOut;
    float *rec;
    int *err;
};

__device__ __forceinline__ float4 f4_add(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// The warp's 32 rows (a thread a row, 32 values each) to chunks: out[s] holds values
// 4 (lane % 8) .. + 3 of row 4 s + lane / 8.  tile: the warp's 4 KB of shared memory; the
// 16-byte pieces of a row are swapped about by the row's number, so that neither side has
// bank conflicts.
__device__ __forceinline__ void rows_to_chunks(const float *v, float4 *out, uint8_t *tile, int lane) {
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4 *>(tile + lane * 128 + ((q ^ (lane & 7)) << 4)) =
            make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int r = 4 * s + (lane >> 3);
        out[s] = *reinterpret_cast<const float4 *>(tile + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
    }
}

// What bounds this kernel is the traffic of its gathers and streams through L1 and L2 (some
// 700 bytes a row and layer) and, before, the work of feeding the tensor core.  Rows move as
// chunks: eight lanes take one row's 32 FP32 features, 16 bytes each, so a load touches four
// lines where a thread a row touches 32; only the accumulator, a row a lane, goes through
// shared memory to chunks (rows_to_chunks).  The weight gradient's contraction runs over rows,
// so its operands are the transposes of X and of dpre: both are read as MN-major operands from
// the row-by-row tiles, and dpre's tile serves the input gradient's MMA as K-major operand as
// well; nothing is transposed by 2-byte stores (96 a thread and tile), and BF16 activations go
// from memory to the tile unconverted.  126,720 rows of a 7-point graph: 55 -> 33 us a
// middle layer, 48 -> 29 the first, 34 -> 18 the last.
// Encoder and decoder gradients are summed over a tile's rows pairwise, then over the tiles.
template <bool TOP, bool L1>
__global__ void __launch_bounds__(GT, 3) k_gnn_bwd(BwdArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *sX = smem;                         // [X, 1, 0]: 16 groups of 8 features x 128 rows x 16 bytes
    uint8_t *sW = smem + BWD_X;                 // W: 64 inputs x 32 outputs (K = 32)
    uint8_t *sT = sW + BWD_W;                   // 4 KB a warp: accumulator rows to chunks
    uint8_t *sD = sT + BWD_T;                   // dpre: 4 groups of 8 outputs x 128 rows x 16 bytes, padded
    float *sprm = reinterpret_cast<float *>(sD + BWD_D);  // e, c, w_d
    float *sred = sprm + 96;                              // [4 warps][64]
    uint64_t *bar = reinterpret_cast<uint64_t *>(sprm + 96 + 256);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q8 = lane & 7, r4 = lane >> 3;  // chunk of a row, row within a step of four

    for (int q = tid; q < 64 * 4; q += GT) {
        int i = q >> 2, c = q & 3;
        uint4 w = *reinterpret_cast<const uint4 *>(a.wbf + 2048 + i * 32 + c * 8);
        *reinterpret_cast<uint4 *>(sW + ((i >> 3) * 4 + c) * 128 + (i & 7) * 16) = w;
    }
    // features 64 (1: the bias gradient; rows past the end have dpre = 0) and 65 .. 127 (0)
    for (int g = 8; g < 16; ++g)
        *reinterpret_cast<uint4 *>(sX + g * 2048 + tid * 16) = make_uint4(g == 8 ? 0x3F80u : 0u, 0, 0, 0);
    if (tid < 32) {
        sprm[tid] = a.prm[GNN_OFF_ENC + tid];
        sprm[32 + tid] = a.prm[GNN_OFF_ENC + 32 + tid];
        sprm[64 + tid] = a.prm[GNN_OFF_DEC + tid];
    }
    if (warp == 0) umma::tmem_alloc(tslot, 128);
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    umma::fence_smem_to_async();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;
    const float inv_s = *a.inv_s_p, s_net = *a.s_p;
    const int n = a.g.n, ntiles = (n + GT - 1) / GT;
    const uint32_t x0 = umma::smem_addr(sX), w0 = umma::smem_addr(sW), d0 = umma::smem_addr(sD);
    const double den = TOP ? a.sc->loss_den : 1.0;
    const float gscale = TOP ? (float)(2.0 / (den > 0.0 ? den : 1.0)) : 0.f;
    // sums over the CTA's rows: TOP: the decoder's weights (this lane's chunk) and bias;
    // L1: the encoder's e and c (this lane's chunk)
    float4 acc_a = make_float4(0.f, 0.f, 0.f, 0.f), acc_b = acc_a;
    float acc_s = 0.f;
    int it = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
        const int row0 = t * GT + warp * 32;  // the warp's rows: one slice
        const int row = row0 + lane;
        const bool valid = row < n;
        float4 delta[8];
        float ui = 0.f, ai = 0.f, wi = 0.f, di = 0.f;
        uint32_t mbits = 0;
        int base = 0, w = 0;
        if (row0 < n) {
            base = a.g.sl_ptr[row0 >> 5];
            w = a.g.sl_w[row0 >> 5];
        }
        if (valid) {
            di = a.g.dinv[row];
            mbits = a.mask[row];
        }
        if (TOP) {
            float gs = 0.f;
            if (valid) {
                float gz;
                if (a.kind == 0) {
                    gz = gscale * a.y[row];
                } else {
                    float sy = 0.f;
                    for (int k = 0; k < w; ++k) {
                        int pos = base + k * 32 + lane;
                        sy += a.g.val[pos] * a.y[a.g.col[pos]];
                    }
                    gz = gscale * a.sgn * sy;
                }
                gs = gz * s_net;
            }
            const float4 wd = *reinterpret_cast<const float4 *>(sprm + 64 + 4 * q8);
            float4 pair[8];
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const int r = 4 * s + r4;
                const float gr = __shfl_sync(FULL_MASK, gs, r);
                delta[s] = make_float4(gr * wd.x, gr * wd.y, gr * wd.z, gr * wd.w);
                uint2 h = make_uint2(0, 0);
                if (row0 + r < n) h = *reinterpret_cast<const uint2 *>(a.h4 + (size_t)(row0 + r) * 32 + 4 * q8);
                pair[s] = make_float4(gr * bf_lo(h.x), gr * bf_hi(h.x), gr * bf_lo(h.y), gr * bf_hi(h.y));
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                for (int s = 0; s < o; ++s) pair[s] = f4_add(pair[s], pair[s + o]);
            acc_a = f4_add(acc_a, pair[0]);
            acc_s += gs;
        } else {
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const int r = row0 + 4 * s + r4;
                delta[s] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < n) delta[s] = *reinterpret_cast<const float4 *>(a.dIn + (size_t)r * 32 + 4 * q8);
            }
            int cn = 0;
            float vn = 0.f;
            if (valid && w > 1) {
                cn = a.g.col[base + 32 + lane];
                vn = a.g.val[base + 32 + lane];
            }
            for (int k = 1; k < w; ++k) {
                const int c = cn;
                const float v = vn;
                if (valid && k + 1 < w) {
                    cn = a.g.col[base + (k + 1) * 32 + lane];
                    vn = a.g.val[base + (k + 1) * 32 + lane];
                }
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const int j = __shfl_sync(FULL_MASK, c, 4 * s + r4);
                    const float vj = __shfl_sync(FULL_MASK, v, 4 * s + r4);
                    const float4 g4 = *reinterpret_cast<const float4 *>(a.gIn + (size_t)j * 32 + 4 * q8);
                    delta[s].x += vj * g4.x;
                    delta[s].y += vj * g4.y;
                    delta[s].z += vj * g4.z;
                    delta[s].w += vj * g4.w;
                }
            }
        }
        // the operand tiles
        if (L1) {
            if (valid) {
                ai = a.aw[2 * (size_t)row];
                wi = a.aw[2 * (size_t)row + 1];
                ui = di * a.r[row] * inv_s;
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t h[4], m[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int c = 8 * g + 2 * e;
                    h[e] = valid ? bf_pack(ui * sprm[c] + sprm[32 + c], ui * sprm[c + 1] + sprm[33 + c]) : 0u;
                    m[e] = bf_pack(ai * sprm[c] + wi * sprm[32 + c], ai * sprm[c + 1] + wi * sprm[33 + c]);
                }
                *reinterpret_cast<uint4 *>(sX + g * 2048 + tid * 16) = make_uint4(h[0], h[1], h[2], h[3]);
                *reinterpret_cast<uint4 *>(sX + (4 + g) * 2048 + tid * 16) = make_uint4(m[0], m[1], m[2], m[3]);
            }
        } else {
            // eight rows of 64 bytes a load
            const int g = lane >> 3;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int r = 8 * s + (lane & 7);
                uint4 h = make_uint4(0, 0, 0, 0), m = h;
                if (row0 + r < n) {
                    h = *reinterpret_cast<const uint4 *>(a.hprev + (size_t)(row0 + r) * 32 + 8 * g);
                    m = *reinterpret_cast<const uint4 *>(a.mcur + (size_t)(row0 + r) * 32 + 8 * g);
                }
                *reinterpret_cast<uint4 *>(sX + g * 2048 + (warp * 32 + r) * 16) = h;
                *reinterpret_cast<uint4 *>(sX + (4 + g) * 2048 + (warp * 32 + r) * 16) = m;
            }
        }
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const int r = 4 * s + r4;
            const uint32_t mb = __shfl_sync(FULL_MASK, mbits, r) >> (4 * q8);
            const uint2 dp = make_uint2(bf_pack(mb & 1u ? delta[s].x : 0.f, mb & 2u ? delta[s].y : 0.f),
                                        bf_pack(mb & 4u ? delta[s].z : 0.f, mb & 8u ? delta[s].w : 0.f));
            *reinterpret_cast<uint2 *>(sD + (q8 >> 1) * BWD_DG + (warp * 32 + r) * 16 + (q8 & 1) * 8) = dp;
        }
        umma::fence_smem_to_async();
        umma::fence_before_sync();
        __syncthreads();
        if (tid == 0) {
            umma::fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
                umma::mma_bf16(tmem, umma::smem_desc(d0 + kk * 2 * BWD_DG, BWD_DG, 128),
                               umma::smem_desc(w0 + kk * 256, 128, 512), IDESC_B1, kk > 0);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
                umma::mma_bf16(tmem + 64, umma::smem_desc(x0 + kk * 256, 128, 2048),
                               umma::smem_desc(d0 + kk * 256, 128, BWD_DG), IDESC_B2, it > 0 || kk > 0);
            umma::commit(bar);
        }
        __syncwarp();
        bool fail = !mbar_wait(bar, it & 1);
        if (__syncthreads_or(fail)) {
            if (tid == 0) atomicExch(a.err, (int)DEV_BARRIER_TIMEOUT);
            break;
        }
        umma::fence_after_sync();
        uint8_t *tile = sT + warp * 4096;
        const uint32_t lb = (uint32_t)(warp * 32) << 16;
        {
            float acc[32];
            float4 dx[8];
            umma::ld32(tmem + lb, acc);
            rows_to_chunks(acc, dx, tile, lane);
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                delta[s] = f4_add(delta[s], dx[s]);
                const int r = row0 + 4 * s + r4;
                if (!L1 && r < n) *reinterpret_cast<float4 *>(a.dOut + (size_t)r * 32 + 4 * q8) = delta[s];
            }
            umma::ld32(tmem + lb + 32, acc);
            rows_to_chunks(acc, dx, tile, lane);
            if (!L1) {
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const int r = row0 + 4 * s + r4;
                    const float d = __shfl_sync(FULL_MASK, di, 4 * s + r4);
                    if (r < n)
                        *reinterpret_cast<float4 *>(a.gOut + (size_t)r * 32 + 4 * q8) =
                            make_float4(d * dx[s].x, d * dx[s].y, d * dx[s].z, d * dx[s].w);
                }
            } else {
                // encoder: h0 = u e + c, m1 = a e + w c; rows past the end count as zero
                float4 ce[8];
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const int r = 4 * s + r4;
                    const bool in = row0 + r < n;
                    const float u = __shfl_sync(FULL_MASK, ui, r), aa = __shfl_sync(FULL_MASK, ai, r),
                                ww = __shfl_sync(FULL_MASK, wi, r);
                    const float4 h = in ? delta[s] : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float4 m = in ? dx[s] : make_float4(0.f, 0.f, 0.f, 0.f);
                    ce[s] = make_float4(u * h.x + aa * m.x, u * h.y + aa * m.y, u * h.z + aa * m.z, u * h.w + aa * m.w);
                    dx[s] = make_float4(h.x + ww * m.x, h.y + ww * m.y, h.z + ww * m.z, h.w + ww * m.w);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                    for (int s = 0; s < o; ++s) {
                        ce[s] = f4_add(ce[s], ce[s + o]);
                        dx[s] = f4_add(dx[s], dx[s + o]);
                    }
                acc_a = f4_add(acc_a, ce[0]);
                acc_b = f4_add(acc_b, dx[0]);
            }
        }
        umma::fence_before_sync();
    }
    // weight and bias gradients of this CTA from the accumulator (rows 0..64)
    float *rec = a.rec + (size_t)blockIdx.x * GNN_NPARAM_PAD;
    float *lrec = rec + GNN_OFF_LAYER + a.layer * GNN_LAYER_STRIDE;
    __syncthreads();
    umma::fence_after_sync();
    if (warp < 3) {
        float dw[32];
        umma::ld32(tmem + ((uint32_t)(warp * 32) << 16) + 64, dw);
#pragma unroll
        for (int o = 0; o < 32; ++o) dw[o] = it > 0 ? dw[o] : 0.f;
        if (warp < 2) {
            float4 ch[8];
            rows_to_chunks(dw, ch, sT + warp * 4096, lane);
#pragma unroll
            for (int s = 0; s < 8; ++s)
                *reinterpret_cast<float4 *>(lrec + (warp * 32 + 4 * s + r4) * 32 + 4 * q8) = ch[s];
        } else if (lane == 0) {
#pragma unroll
            for (int o = 0; o < 32; ++o) lrec[2048 + o] = dw[o];
        }
    }
    if (TOP || L1) {
#pragma unroll
        for (int o = 16; o >= 8; o >>= 1) {  // over the four rows of a step
            acc_a = f4_add(acc_a, make_float4(__shfl_xor_sync(FULL_MASK, acc_a.x, o), __shfl_xor_sync(FULL_MASK, acc_a.y, o),
                                              __shfl_xor_sync(FULL_MASK, acc_a.z, o), __shfl_xor_sync(FULL_MASK, acc_a.w, o)));
            if (L1)
                acc_b = f4_add(acc_b, make_float4(__shfl_xor_sync(FULL_MASK, acc_b.x, o), __shfl_xor_sync(FULL_MASK, acc_b.y, o),
                                                  __shfl_xor_sync(FULL_MASK, acc_b.z, o), __shfl_xor_sync(FULL_MASK, acc_b.w, o)));
        }
        if (TOP)
            for (int o = 16; o > 0; o >>= 1) acc_s += __shfl_xor_sync(FULL_MASK, acc_s, o);
        if (r4 == 0) {
            *reinterpret_cast<float4 *>(sred + warp * 64 + 4 * q8) = acc_a;
            *reinterpret_cast<float4 *>(sred + warp * 64 + 32 + 4 * q8) = TOP ? make_float4(acc_s, 0.f, 0.f, 0.f) : acc_b;
        }
        __syncthreads();
        if (tid < 64) {
            float v = sred[tid] + sred[64 + tid] + sred[128 + tid] + sred[192 + tid];
            if (TOP) {
                if (tid <= 32) rec[GNN_OFF_DEC + tid] = v;
            } else {
                rec[GNN_OFF_ENC + tid] = v;
            }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == 0) umma::tmem_free(tmem, 128);
}

// ------------------------------------------------------- loss, Adam, misc --

__global__ void k_gnn_loss(GView g, float sgn, int kind, const float *z, const float *e, float *y, double *part,
                           GnnScalars *sc) {
    double v[2] = {0.0, 0.0};
    for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < g.n; row += gridDim.x * blockDim.x) {
        const int sl = row >> 5, lane = row & 31;
        const int base = g.sl_ptr[sl], w = g.sl_w[sl];
        float st = 0.f, se = 0.f;
        for (int k = 0; k < w; ++k) {
            int pos = base + k * 32 + lane;
            int j = g.col[pos];
            float av = g.val[pos];
            st += av * (z[j] - e[j]);
            se += av * e[j];
        }
        st *= sgn;
        se *= sgn;
        y[row] = st;
        if (kind == 0) {
            v[0] += (double)(z[row] - e[row]) * st;
            v[1] += (double)e[row] * se;
        } else {
            v[0] += (double)st * st;
            v[1] += (double)se * se;
        }
    }
    if (grid_sums<2>(v, part, &sc->cnt[1])) {
        sc->loss_num = v[0];
        sc->loss_den = v[1];
    }
}

__global__ void k_gnn_scale(GView g, const float *r, double *part, GnnScalars *sc) {
    double v[1] = {0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += gridDim.x * blockDim.x) {
        double u = (double)g.dinv[i] * r[i];
        v[0] += u * u;
    }
    if (grid_sums<1>(v, part, &sc->cnt[0])) {
        double s = sqrt(v[0] / (double)g.n);
        sc->s = (float)s;
        sc->inv_s = s > 0.0 ? (float)(1.0 / s) : 0.f;
    }
}

// Sum the per-CTA gradient records; update (Adam) or just report.  What bounds it is the FP64
// pipe (a conversion and an addition a record and parameter, 64 clocks a warp each): a warp's
// 32 parameters are split over the block's eight warps, each summing every eighth record, so
// that all the SMs' pipes work and eight loads are in flight.  One thread a parameter, record
// after record, took 87 us for 456 records; this takes 22.  corr1, corr2: 1 - beta^t.  The
// first thread also files the loss of the step.
constexpr int ADAM_P = 32, ADAM_W = 8;

__global__ void __launch_bounds__(ADAM_P * ADAM_W)
    k_gnn_adam(const float *rec, int nrec, float *p, float *m, float *v, uint16_t *wbf, float *grad_out, double lr,
               double corr1, double corr2, int update, const GnnScalars *sc, double *loss_out) {
    __shared__ double part[ADAM_W][ADAM_P];
    const int c = threadIdx.x & (ADAM_P - 1), w = threadIdx.x / ADAM_P;
    const int q = blockIdx.x * ADAM_P + c;
    double g = 0.0;
    if (q < GNN_NPARAM) {
        const float *rq = rec + q;
        int b = w;
        for (; b + 7 * ADAM_W < nrec; b += 8 * ADAM_W) {
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = rq[(size_t)(b + i * ADAM_W) * GNN_NPARAM_PAD];
#pragma unroll
            for (int i = 0; i < 8; ++i) g += x[i];
        }
        for (; b < nrec; b += ADAM_W) g += rq[(size_t)b * GNN_NPARAM_PAD];
    }
    part[w][c] = g;
    __syncthreads();
    if (w != 0) return;
    if (q == 0) *loss_out = sc->loss_den > 0.0 ? sc->loss_num / sc->loss_den : 0.0;
    if (q >= GNN_NPARAM) return;
#pragma unroll
    for (int i = 1; i < ADAM_W; ++i) g += part[i][c];
    if (grad_out) grad_out[q] = (float)g;
    if (!update) return;
    const double b1 = 0.9, b2 = 0.999, eps = 1e-8;
    double mq = b1 * m[q] + (1.0 - b1) * g;
    double vq = b2 * v[q] + (1.0 - b2) * g * g;
    m[q] = (float)mq;
    v[q] = (float)vq;
    double mh = mq / corr1, vh = vq / corr2;
    float pn = (float)(p[q] - lr * mh / (sqrt(vh) + eps));
    p[q] = pn;
    int rel = q - GNN_OFF_LAYER;
    if (rel >= 0 && rel < GNN_LAYERS * GNN_LAYER_STRIDE && rel % GNN_LAYER_STRIDE < 2048) {
        int l = rel / GNN_LAYER_STRIDE, k = rel % GNN_LAYER_STRIDE, in = k / 32, o = k % 32;
        uint16_t b = __bfloat16_as_ushort(__float2bfloat16_rn(pn));
        wbf[l * GNN_WBF_LAYER + o * 64 + in] = b;
        wbf[l * GNN_WBF_LAYER + 2048 + in * 32 + o] = b;
    }
}

__global__ void k_gnn_refresh(const float *p, uint16_t *wbf) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= GNN_LAYERS * 2048) return;
    int l = q / 2048, k = q % 2048, in = k / 32, o = k % 32;
    uint16_t b = __bfloat16_as_ushort(__float2bfloat16_rn(p[GNN_OFF_LAYER + l * GNN_LAYER_STRIDE + k]));
    wbf[l * GNN_WBF_LAYER + o * 64 + in] = b;
    wbf[l * GNN_WBF_LAYER + 2048 + in * 32 + o] = b;
}

__global__ void k_gnn_dinv(int n, const int *sl_ptr, const double *val, float *dinv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d = val[sl_ptr[i >> 5] + (i & 31)];
    dinv[i] = d != 0.0 ? (float)(1.0 / d) : 0.f;
}

// training pair from a partial solve: r = b - A x1, e = xs - x1 (x1 == nullptr: 0)
__global__ void k_pair_from(GView g, const double *val64, const double *b, const double *x1, const double *xs,
                            float *r, float *e) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    double ri = b[i], ei = xs[i];
    if (x1) {
        const int sl = i >> 5, lane = i & 31;
        const int base = g.sl_ptr[sl], w = g.sl_w[sl];
        double ax = 0.0;
        for (int k = 0; k < w; ++k) {
            int pos = base + k * 32 + lane;
            ax += val64[pos] * x1[g.col[pos]];
        }
        ri -= ax;
        ei -= x1[i];
    }
    r[i] = (float)ri;
    e[i] = (float)ei;
}

__global__ void k_to_f32(int n, const double *a, float *b) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = (float)a[i];
}
__global__ void k_post_jacobi(int n, const float *z2, const float *w, const float *t, float *z) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) z[i] = z2[i] + w[i] * t[i];
}

__global__ void k_to_f64(int n, const float *a, double *b) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = (double)a[i];
}

// ----------------------------------------------------------- flexible CG --

struct FcgArgs {
    GView g;      // FP32 matrix
    const double *val64;
    float sgn;
    const double *b;
    double *x;
    float *r, *z, *p, *q, *e;
    FcgState *fs;
    double *part;
    double inner_tol2;
    int stall_max;
};

// Row i of the FP32 matrix times x, the column indices and values of four
// entries loaded before their gathers (the sum runs in entry order, as a plain
// loop's); default cache policy, so the matrix stays in L2 between the kernels
// of an iteration that read it
__device__ __forceinline__ float sell_dot32(const GView &g, int i, const float *x) {
    const int lane = i & 31;
    int e = g.sl_ptr[i >> 5] + lane;
    const int w = g.sl_w[i >> 5];
    float acc = 0.f;
    int k = 0;
    for (; k + 4 <= w; k += 4, e += 128) {
        const int c0 = g.col[e], c1 = g.col[e + 32], c2 = g.col[e + 64], c3 = g.col[e + 96];
        const float v0 = g.val[e], v1 = g.val[e + 32], v2 = g.val[e + 64], v3 = g.val[e + 96];
        const float x0 = x[c0], x1 = x[c1], x2 = x[c2], x3 = x[c3];
        acc += v0 * x0;
        acc += v1 * x1;
        acc += v2 * x2;
        acc += v3 * x3;
    }
    for (; k < w; ++k, e += 32) acc += g.val[e] * x[g.col[e]];
    return acc;
}

__device__ __forceinline__ double spmv64_row(const GView &g, const double *val64, const double *x, int row) {
    const int sl = row >> 5, lane = row & 31;
    const int base = g.sl_ptr[sl], w = g.sl_w[sl];
    double s = 0.0;
    for (int k = 0; k < w; ++k) {
        int pos = base + k * 32 + lane;
        s += val64[pos] * x[g.col[pos]];
    }
    return s;
}

__global__ void k_fcg_init(FcgArgs a, int x0_zero, double eps, int maxit, int use_gnn) {
    double v[3] = {0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.g.n; i += gridDim.x * blockDim.x) {
        double bi = a.b[i];
        double ri = x0_zero ? bi : bi - spmv64_row(a.g, a.val64, a.x, i);
        a.r[i] = (float)ri;
        a.e[i] = 0.f;
        double u = (double)a.g.dinv[i] * ri;
        v[0] += bi * bi;
        v[1] += ri * ri;
        v[2] += u * u;
    }
    if (grid_sums<3>(v, a.part, &a.fs->cnt[0])) {
        FcgState *f = a.fs;
        f->bnorm2 = v[0];
        f->eps2 = v[0] > 0.0 ? eps * eps * v[0] : eps * eps;
        f->rr = f->rr_upd = f->rr_best = v[1];
        double s = sqrt(v[2] / (double)a.g.n);
        f->s = (float)s;
        f->inv_s = s > 0.0 ? (float)(1.0 / s) : 0.f;
        f->res = v[0] > 0.0 ? sqrt(v[1] / v[0]) : sqrt(v[1]);
        f->iters = 0;
        f->refinements = 0;
        f->status = DEV_OK;
        f->done = v[1] <= f->eps2 ? 1 : 0;
        f->use_gnn = use_gnn;
        f->stall = 0;
        f->restart = 1;
        f->need_update = 0;
        f->fallback_at = -1;
        f->maxit = maxit;
        f->loops = 0;
        f->zq = f->pq = f->pq_prev = f->pr = f->alpha = 0.0;
    }
}

// x = 0 for a zero initial guess (before k_fcg_init reads it).
__global__ void k_fcg_zero(int n, double *x) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = 0.0;
}

__global__ void k_fcg_jacobi(FcgArgs a) {
    if (a.fs->done || a.fs->use_gnn) return;
    float f0 = 0.f;
    const bool rs = a.fs->restart;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.g.n; i += gridDim.x * blockDim.x) {
        float zi = a.g.dinv[i] * a.r[i];
        a.z[i] = zi;
        if (!rs) f0 += zi * a.q[i];
    }
    const float fv[1] = {f0};
    if (grid_totals_f<1>(fv, a.part, &a.fs->cnt[0]) && threadIdx.x == 0) a.fs->zq = g_gt_sum[0];
}

// multigrid form, finest level after the coarse correction z2: t = r - A z2, then
// either (network off) z = z2 + w t and z.q_prev for the flexible beta, or
// (network on) t for the network and its scale s2 = rms(D^-1 t)
__global__ void k_fcg_mgfine(FcgArgs a, const float *z2, float *t, const float *w, int fine_net) {
    if (a.fs->done) return;
    const bool net = fine_net && a.fs->use_gnn, rs = a.fs->restart;
    float f0 = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.g.n; i += gridDim.x * blockDim.x) {
        const float ti = a.r[i] - sell_dot32(a.g, i, z2);
        if (net) {
            t[i] = ti;
            const float u = a.g.dinv[i] * ti;
            f0 += u * u;
        } else {
            const float zi = z2[i] + w[i] * ti;
            a.z[i] = zi;
            if (!rs) f0 += zi * a.q[i];
        }
    }
    const float fv[1] = {f0};
    if (grid_totals_f<1>(fv, a.part, &a.fs->cnt[0]) && threadIdx.x == 0) {
        const double *v = g_gt_sum;
        if (net) {
            double s = sqrt(v[0] / (double)a.g.n);
            a.fs->s2 = (float)s;
            a.fs->inv_s2 = s > 0.0 ? (float)(1.0 / s) : 0.f;
        } else {
            a.fs->zq = v[0];
        }
    }
}

// network as a coarse level's post-smoother: t = r - A zp on that level, and
// (network on) the network's input scale s2 = rms(D^-1 t) into the finest-level
// flexible CG's state
__global__ void k_lvl_resid(GView g, const float *r, const float *zp, float *t, FcgState *fs, double *part) {
    if (fs->done) return;
    const bool net = fs->use_gnn;  // written by other launches only: uniform here
    float f0 = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += gridDim.x * blockDim.x) {
        const int base = g.sl_ptr[i >> 5], wd = g.sl_w[i >> 5], lane = i & 31;
        float az = 0.f;
        for (int k = 0; k < wd; ++k) {
            int pos = base + k * 32 + lane;
            az += g.val[pos] * zp[g.col[pos]];
        }
        const float ti = r[i] - az;
        t[i] = ti;
        if (net) {
            const float u = g.dinv[i] * ti;
            f0 += u * u;
        }
    }
    if (!net) return;
    const float fv[1] = {f0};
    if (grid_totals_f<1>(fv, part, &fs->cnt[3]) && threadIdx.x == 0) {
        const double *v = g_gt_sum;
        double s = sqrt(v[0] / (double)g.n);
        fs->s2 = (float)s;
        fs->inv_s2 = s > 0.0 ? (float)(1.0 / s) : 0.f;
    }
}

// the Jacobi post-smoothing step of that level while the network is off
__global__ void k_lvl_jacobi(int n, const float *zp, const float *w, const float *t, float *z, const FcgState *fs) {
    if (fs->done || fs->use_gnn) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) z[i] = zp[i] + w[i] * t[i];
}

// r = b - A x1 (FP64) rounded to FP32; x1 == nullptr: r = b
__global__ void k_res32(GView g, const double *val64, const double *b, const double *x1, float *r) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += gridDim.x * blockDim.x) {
        double ri = b[i];
        if (x1) {
            const int base = g.sl_ptr[i >> 5], wd = g.sl_w[i >> 5], lane = i & 31;
            for (int k = 0; k < wd; ++k) {
                int pos = base + k * 32 + lane;
                ri -= val64[pos] * x1[g.col[pos]];
            }
        }
        r[i] = (float)ri;
    }
}

__global__ void k_fcg_dir(FcgArgs a) {
    if (a.fs->done) return;
    const bool rs = a.fs->restart;
    const double beta = rs ? 0.0 : a.fs->zq / a.fs->pq_prev;
    const float bf = (float)beta;
    float f0 = 0.f, f1 = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.g.n; i += gridDim.x * blockDim.x) {
        const float az = sell_dot32(a.g, i, a.z);
        float qi = rs ? az : az - bf * a.q[i];
        float pi = rs ? a.z[i] : a.z[i] - bf * a.p[i];
        a.q[i] = qi;
        a.p[i] = pi;
        f0 += pi * qi;
        f1 += pi * a.r[i];
    }
    const float fv[2] = {f0, f1};
    if (grid_totals_f<2>(fv, a.part, &a.fs->cnt[1]) && threadIdx.x == 0) {
        const double *v = g_gt_sum;
        FcgState *f = a.fs;
        double pq = v[0], pr = v[1];
        double alpha = pr / pq;
        bool bad = !((double)a.sgn * pq > 0.0) || !isfinite(alpha);
        f->pq = pq;
        f->pr = pr;
        if (bad) {
            f->alpha = 0.0;
            f->restart = 1;
            if (f->use_gnn) {
                f->use_gnn = 0;
                f->fallback_at = f->iters;
            } else {
                f->status = DEV_BREAKDOWN;
                f->need_update = 1;
            }
        } else {
            f->alpha = alpha;
            f->restart = 0;
        }
    }
}

// e += alpha p, r -= alpha q; r.r and |D^-1 r|^2.  Four rows a thread with
// 16-byte loads (the arrays are whole allocations, 16-byte aligned): a pure
// vector pass, where one row a thread left it at half of HBM.
__device__ __forceinline__ void fcg_upd_row(float al, float &r, float &e, float p, float q, float d, float &f0,
                                            float &f1) {
    if (al != 0.f) {
        e += al * p;
        r -= al * q;
    }
    const float u = d * r;
    f0 += r * r;
    f1 += u * u;
}

__global__ void k_fcg_upd(FcgArgs a) {
    if (a.fs->done) return;
    const float al = (float)a.fs->alpha;
    float f0 = 0.f, f1 = 0.f;
    const int n4 = a.g.n >> 2, T = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (int j = t0; j < n4; j += T) {
        float4 r = ld4(a.r, j), e = ld4(a.e, j);
        const float4 p = ld4(a.p, j), q = ld4(a.q, j), d = ld4(a.g.dinv, j);
        fcg_upd_row(al, r.x, e.x, p.x, q.x, d.x, f0, f1);
        fcg_upd_row(al, r.y, e.y, p.y, q.y, d.y, f0, f1);
        fcg_upd_row(al, r.z, e.z, p.z, q.z, d.z, f0, f1);
        fcg_upd_row(al, r.w, e.w, p.w, q.w, d.w, f0, f1);
        if (al != 0.f) {
            st4(a.e, j, e);
            st4(a.r, j, r);
        }
    }
    for (int i = 4 * n4 + t0; i < a.g.n; i += T) {
        float r = a.r[i], e = a.e[i];
        fcg_upd_row(al, r, e, a.p[i], a.q[i], a.g.dinv[i], f0, f1);
        if (al != 0.f) {
            a.e[i] = e;
            a.r[i] = r;
        }
    }
    const float fv[2] = {f0, f1};
    if (grid_totals_f<2>(fv, a.part, &a.fs->cnt[2]) && threadIdx.x == 0) {
        const double *v = g_gt_sum;
        FcgState *f = a.fs;
        f->iters += 1;
        f->rr = v[0];
        if (f->use_gnn) {  // the network's input scale (an FP64 root and a division: 1.8 us of the tail)
            double s = sqrt(v[1] / (double)a.g.n);
            f->s = (float)s;
            f->inv_s = s > 0.0 ? (float)(1.0 / s) : 0.f;
        }
        f->pq_prev = f->pq;
        if (v[0] < f->rr_best) {
            f->rr_best = v[0];
            f->stall = 0;
        } else {
            f->stall += 1;
        }
        if (f->use_gnn && f->stall >= a.stall_max) {
            f->use_gnn = 0;
            f->restart = 1;
            f->fallback_at = f->iters;
        }
        if (v[0] <= a.inner_tol2 * f->rr_upd || v[0] <= f->eps2 || f->iters >= f->maxit || !isfinite(v[0]))
            f->need_update = 1;
    }
}

__global__ void k_fcg_rel1(FcgArgs a) {
    if (a.fs->done || !a.fs->need_update) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.g.n; i += gridDim.x * blockDim.x) {
        a.x[i] += (double)a.e[i];
        a.e[i] = 0.f;
    }
}

__global__ void k_fcg_rel2(FcgArgs a) {
    if (a.fs->done || !a.fs->need_update) return;
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.g.n; i += gridDim.x * blockDim.x) {
        double ri = a.b[i] - spmv64_row(a.g, a.val64, a.x, i);
        a.r[i] = (float)ri;
        double u = (double)a.g.dinv[i] * ri;
        v[0] += ri * ri;
        v[1] += u * u;
    }
    if (grid_sums<2>(v, a.part, &a.fs->cnt[3])) {
        FcgState *f = a.fs;
        f->refinements += 1;
        f->rr = f->rr_upd = f->rr_best = v[0];
        f->stall = 0;
        f->res = f->bnorm2 > 0.0 ? sqrt(v[0] / f->bnorm2) : sqrt(v[0]);
        double s = sqrt(v[1] / (double)a.g.n);
        f->s = (float)s;
        f->inv_s = s > 0.0 ? (float)(1.0 / s) : 0.f;
        f->need_update = 0;
        if (!isfinite(v[0])) {
            f->done = 1;
            f->status = DEV_NONFINITE;
        } else if (v[0] <= f->eps2) {
            f->done = 1;
            f->status = DEV_OK;
        } else if (f->status == DEV_BREAKDOWN || f->iters >= f->maxit) {
            f->done = 1;
            if (f->status != DEV_BREAKDOWN) f->status = DEV_MAXITER;
        }
    }
}

__global__ void k_fcg_info(const FcgState *f, SolveInfo *info) {
    info->status[0] = f->status;
    info->iters[0] = f->iters;
    info->res[0] = f->res;
    info->refinements = f->refinements;
    info->err = 0;
}

int blocks_flat(int n) { return std::max(1, std::min((n + FB - 1) / FB, num_sms() * 8)); }

}  // namespace

void GnnPrecond::drop_graphs() {
    for (SolveGraph &g : graphs_) {
        if (g.exec) cudaGraphExecDestroy(g.exec);
        g = SolveGraph{};
    }
}

void GnnPrecond::attach_multigrid(AggMultigrid *mg) {
    if (mg && (!mg->ready() || !bound() || mg->level_rows(0) != n_))
        throw CaseError{"multigrid: hierarchy not built for the bound matrix"};
    drop_graphs();
    mg_ = mg;
    if (mg_ && z2_.size() < (size_t)n_) {
        z2_.alloc(n_);
        t_.alloc(n_);
    }
}

void GnnPrecond::transform_pair(int k, cudaStream_t st) {
    if (!mg_) return;
    mg_->smoother_pair(pr_.get() + (size_t)k * n_, pe_.get() + (size_t)k * n_, st);
}

void GnnPrecond::bind(const SellDev &A, const double *val64, const float *val32, cudaStream_t st) {
    drop_graphs();
    mg_ = nullptr;
    A_ = &A;
    val64_ = val64;
    val32_ = val32;
    n_ = A.n;
    ntiles_ = (n_ + GT - 1) / GT;
    static bool attr = false;
    if (!attr) {
        SYSU_CUDA(cudaFuncSetAttribute(k_gnn_bwd<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM_REQ));
        SYSU_CUDA(cudaFuncSetAttribute(k_gnn_bwd<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM_REQ));
        SYSU_CUDA(cudaFuncSetAttribute(k_gnn_bwd<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM_REQ));
        attr = true;
    }
    // forward: as many co-resident CTAs as registers and shared memory allow
    // (the gather is latency-bound).  Computed from the kernel's attributes:
    // the runtime's occupancy query reports one CTA per SM for kernels that
    // allocate tensor memory.
    cudaFuncAttributes fa{};
    SYSU_CUDA(cudaFuncGetAttributes(&fa, k_gnn_fwd<false, true, true, 128>));
    int by_regs = 65536 / std::max(1, fa.numRegs * GT);
    int by_smem = (227 * 1024) / (FWD_SMEM + (int)fa.sharedSizeBytes + 1024);
    int occ = std::max(1, std::min(std::min(by_regs, by_smem), 8));
    if (fwd_per_sm > 0) occ = fwd_per_sm;
    // 32-row tiles up to two CTAs an SM (9,728 rows on 152 SMs).  Four layers and their flat
    // kernels on a 7-point graph, 32-row against 128-row tiles: 1,300 rows 24.6 and 30.7 us,
    // 4,096 rows 26.6 and 30.7, 13,824 rows 32.8 and 31.8; wider rows gain more.
    small_ = (n_ + 31) / 32 <= num_sms() * 2;
    gfwd_ = std::max(1, std::min(small_ ? (n_ + 31) / 32 : ntiles_, num_sms() * occ));
    gtiles_ = std::max(1, std::min(ntiles_, num_sms() * 3));
    gflat_ = blocks_flat(n_);
    const size_t n = (size_t)n_;
    dinv_.alloc(n);
    refresh(st);
    double d0 = 0.0;  // the matrix's sign (entry 0 is row 0's diagonal)
    SYSU_CUDA(cudaMemcpyAsync(&d0, val64_, sizeof(double), cudaMemcpyDeviceToHost, st));
    SYSU_CUDA(cudaStreamSynchronize(st));
    sgn_ = d0 < 0.0 ? -1.0f : 1.0f;
    if (p_.size() == 0) {
        p_.alloc(GNN_NPARAM_PAD);
        m_.alloc(GNN_NPARAM_PAD);
        v_.alloc(GNN_NPARAM_PAD);
        wbf_.alloc(GNN_LAYERS * GNN_WBF_LAYER);
        p_.zero(st);
        m_.zero(st);
        v_.zero(st);
        wbf_.zero(st);
        sc_.alloc(1);
        fs_.alloc(1);
        sc_.zero(st);
        fs_.zero(st);
        losses_.alloc(1 << 16);
        err_.alloc(1);
        err_.zero(st);
    }
    rec_.alloc((size_t)gtiles_ * GNN_NPARAM_PAD);
    part_.alloc((size_t)std::max(std::max(gtiles_, gfwd_), gflat_) * 4);
    H_.alloc(5 * n * 32);
    M_.alloc(4 * n * 32);
    mask_.alloc(4 * n);
    aw_.alloc(2 * n);
    dA_.alloc(n * 32);
    gA_.alloc(n * 32);
    dB_.alloc(n * 32);
    gB_.alloc(n * 32);
    for (DevBuf<float> *b : {&z32_, &y32_, &r32_, &e32_, &p32_, &q32_, &x32_}) b->alloc(n);
    pr_.alloc((size_t)capacity_ * n);
    pe_.alloc((size_t)capacity_ * n);
    r64_.alloc(n);
    count_ = next_ = 0;
}

// New values of the bound matrix (same pattern and the same sign convention,
// which bind read): the Jacobi weights.  No host round trip, so a refresh can be
// part of a captured outer iteration.
void GnnPrecond::refresh(cudaStream_t st) {
    k_gnn_dinv<<<(n_ + FB - 1) / FB, FB, 0, st>>>(n_, A_->sl_ptr.get(), val64_, dinv_.get());
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
}

void GnnPrecond::refresh_bf16(cudaStream_t st) {
    k_gnn_refresh<<<(GNN_LAYERS * 2048 + FB - 1) / FB, FB, 0, st>>>(p_.get(), wbf_.get());
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
}

void GnnPrecond::init_params(unsigned long long seed, cudaStream_t st) {
    std::vector<float> h(GNN_NPARAM_PAD, 0.f);
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<float> U(-1.f, 1.f);
    for (int c = 0; c < 64; ++c) h[GNN_OFF_ENC + c] = U(rng);
    const float a = std::sqrt(6.0f / 96.0f) * 0.5f;
    for (int l = 0; l < GNN_LAYERS; ++l)
        for (int k = 0; k < 2048; ++k) h[GNN_OFF_LAYER + l * GNN_LAYER_STRIDE + k] = a * U(rng);
    set_params(h.data(), st);
}

void GnnPrecond::set_params(const float *host, cudaStream_t st) {
    if (!p_.size()) throw CaseError{"learned preconditioner: bind a matrix first"};
    p_.upload(host, GNN_NPARAM, st);
    SYSU_CUDA(cudaStreamSynchronize(st));
    refresh_bf16(st);
    reset_adam(st);
}

void GnnPrecond::get_params(float *host, cudaStream_t st) {
    p_.download(host, GNN_NPARAM, st);
    SYSU_CUDA(cudaStreamSynchronize(st));
}

void GnnPrecond::reset_adam(cudaStream_t st) {
    m_.zero(st);
    v_.zero(st);
    adam_t_ = 0;
}

static GView gview(const SellDev &A, const float *val32, const float *dinv) {
    return GView{A.n, A.sl_ptr.get(), A.sl_w.get(), A.col.get(), val32, dinv};
}

void GnnPrecond::scale_of(const float *r32, cudaStream_t st) {
    k_gnn_scale<<<gflat_, FB, 0, st>>>(gview(*A_, val32_, dinv_.get()), r32, part_.get(), sc_.get());
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
}

void GnnPrecond::forward(const float *r32, float *z32, bool train, FcgState *fs, const float *qprev, cudaStream_t st,
                         const float *zbase) {
    NetArgs a{};
    a.g = gview(*A_, val32_, dinv_.get());
    a.r = r32;
    a.inv_s_p = fs ? (zbase ? &fs->inv_s2 : &fs->inv_s) : &sc_.get()->inv_s;
    a.s_p = fs ? (zbase ? &fs->s2 : &fs->s) : &sc_.get()->s;
    a.zbase = zbase;
    a.skip = skip;
    a.prm = p_.get();
    a.aw = aw_.get();
    a.z = z32;
    a.qprev = qprev;
    a.fs = fs;
    a.part = part_.get();
    a.err = err_.get();
    const size_t nn = (size_t)n_ * 32;
    for (int l = 0; l < GNN_LAYERS; ++l) {
        a.layer = l;
        a.wbf = wbf_.get() + l * GNN_WBF_LAYER;
        if (train) {
            a.hin = l ? H_.get() + (size_t)l * nn : nullptr;
            a.hout = H_.get() + (size_t)(l + 1) * nn;
            a.mout = M_.get() + (size_t)l * nn;
            a.mask = mask_.get() + (size_t)l * n_;
        } else {
            a.hin = l ? H_.get() + (size_t)(l & 1 ? 1 : 2) * nn : nullptr;
            a.hout = H_.get() + (size_t)(l & 1 ? 2 : 1) * nn;
            a.mout = nullptr;
            a.mask = nullptr;
        }
        dim3 grid(gfwd_), blk(GT);
        auto run = [&](auto TR) {
            if (l == 0) {
                if (train) k_gnn_fwd<true, true, false, TR.value><<<grid, blk, FWD_SMEM, st>>>(a);
                else k_gnn_fwd<true, false, false, TR.value><<<grid, blk, FWD_SMEM, st>>>(a);
            } else if (l == GNN_LAYERS - 1) {
                if (train) k_gnn_fwd<false, true, true, TR.value><<<grid, blk, FWD_SMEM, st>>>(a);
                else k_gnn_fwd<false, false, true, TR.value><<<grid, blk, FWD_SMEM, st>>>(a);
            } else {
                if (train) k_gnn_fwd<false, true, false, TR.value><<<grid, blk, FWD_SMEM, st>>>(a);
                else k_gnn_fwd<false, false, false, TR.value><<<grid, blk, FWD_SMEM, st>>>(a);
            }
        };
        if (small_) run(std::integral_constant<int, 32>{});
        else run(std::integral_constant<int, 128>{});
        ++g_launches;
        SYSU_CUDA(cudaGetLastError());
    }
}

void GnnPrecond::backward(const float *r32, cudaStream_t st) {
    BwdArgs a{};
    a.g = gview(*A_, val32_, dinv_.get());
    a.sgn = sgn_;
    a.kind = loss_kind;
    a.r = r32;
    a.inv_s_p = &sc_.get()->inv_s;
    a.s_p = &sc_.get()->s;
    a.prm = p_.get();
    a.aw = aw_.get();
    a.h4 = H_.get() + (size_t)4 * n_ * 32;
    a.y = y32_.get();
    a.sc = sc_.get();
    a.rec = rec_.get();
    a.err = err_.get();
    const size_t nn = (size_t)n_ * 32;
    float *dbuf[2] = {dA_.get(), dB_.get()}, *gbuf[2] = {gA_.get(), gB_.get()};
    for (int l = GNN_LAYERS - 1; l >= 0; --l) {
        a.layer = l;
        a.wbf = wbf_.get() + l * GNN_WBF_LAYER;
        a.hprev = l ? H_.get() + (size_t)l * nn : nullptr;
        a.mcur = M_.get() + (size_t)l * nn;
        a.mask = mask_.get() + (size_t)l * n_;
        int in = (l + 1) & 1, out = l & 1;
        a.dIn = dbuf[in];
        a.gIn = gbuf[in];
        a.dOut = dbuf[out];
        a.gOut = gbuf[out];
        dim3 grid(gtiles_), blk(GT);
        if (l == GNN_LAYERS - 1) k_gnn_bwd<true, false><<<grid, blk, BWD_SMEM_REQ, st>>>(a);
        else if (l == 0) k_gnn_bwd<false, true><<<grid, blk, BWD_SMEM_REQ, st>>>(a);
        else k_gnn_bwd<false, false><<<grid, blk, BWD_SMEM_REQ, st>>>(a);
        ++g_launches;
        SYSU_CUDA(cudaGetLastError());
    }
}

void GnnPrecond::apply(const double *r, double *z, cudaStream_t st) {
    if (!bound()) throw CaseError{"learned preconditioner: no matrix bound"};
    int nb = (n_ + FB - 1) / FB;
    k_to_f32<<<nb, FB, 0, st>>>(n_, r, r32_.get());
    ++g_launches;
    scale_of(r32_.get(), st);
    forward(r32_.get(), z32_.get(), false, nullptr, nullptr, st);
    k_to_f64<<<nb, FB, 0, st>>>(n_, z32_.get(), z);
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
    check_err(st);
}

void GnnPrecond::post_smooth(const float *r, const float *zp, float *z, FcgState *fs, const float *w, cudaStream_t st) {
    if (!bound()) throw CaseError{"coarse-level network: no matrix bound"};
    if (t_.size() < (size_t)n_) t_.alloc(n_);
    k_lvl_resid<<<gflat_, FB, 0, st>>>(gview(*A_, val32_, dinv_.get()), r, zp, t_.get(), fs, part_.get());
    ++g_launches;
    forward(t_.get(), z, false, fs, nullptr, st, zp);
    k_lvl_jacobi<<<gflat_, FB, 0, st>>>(n_, zp, w, t_.get(), z, fs);
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
}

void GnnPrecond::residual32(const double *b, const double *x1, float *r, cudaStream_t st) {
    if (!bound()) throw CaseError{"learned preconditioner: no matrix bound"};
    k_res32<<<gflat_, FB, 0, st>>>(gview(*A_, val32_, dinv_.get()), val64_, b, x1, r);
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
}

void GnnPrecond::apply_mg(const double *r, double *z, bool use_gnn, cudaStream_t st) {
    if (!bound() || !mg_) throw CaseError{"multigrid form: no matrix bound or no hierarchy attached"};
    int nb = (n_ + FB - 1) / FB;
    k_to_f32<<<nb, FB, 0, st>>>(n_, r, r32_.get());
    ++g_launches;
    mg_->apply_fixed(r32_.get(), z2_.get(), t_.get(), nullptr, st);
    if (use_gnn) {
        scale_of(t_.get(), st);
        forward(t_.get(), z32_.get(), false, nullptr, nullptr, st, z2_.get());
    } else {
        k_post_jacobi<<<nb, FB, 0, st>>>(n_, z2_.get(), mg_->w0(), t_.get(), z32_.get());
        ++g_launches;
    }
    k_to_f64<<<nb, FB, 0, st>>>(n_, z32_.get(), z);
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
    check_err(st);
}

double GnnPrecond::time_apply(const double *r, int reps, cudaStream_t st) {
    int nb = (n_ + FB - 1) / FB;
    k_to_f32<<<nb, FB, 0, st>>>(n_, r, r32_.get());
    ++g_launches;
    scale_of(r32_.get(), st);
    forward(r32_.get(), z32_.get(), false, nullptr, nullptr, st);
    cudaEvent_t e0, e1;
    SYSU_CUDA(cudaEventCreate(&e0));
    SYSU_CUDA(cudaEventCreate(&e1));
    SYSU_CUDA(cudaEventRecord(e0, st));
    for (int i = 0; i < reps; ++i) forward(r32_.get(), z32_.get(), false, nullptr, nullptr, st);
    SYSU_CUDA(cudaEventRecord(e1, st));
    SYSU_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    check_err(st);
    return ms / std::max(reps, 1);
}

void GnnPrecond::check_err(cudaStream_t st) {
    int e = 0;
    SYSU_CUDA(cudaMemcpyAsync(&e, err_.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
    SYSU_CUDA(cudaStreamSynchronize(st));
    if (e) {
        err_.zero(st);
        throw CaseError{"learned preconditioner: a tensor-core wait timed out"};
    }
}

void GnnPrecond::add_pair(const double *r, const double *e, cudaStream_t st) {
    if (!bound()) throw CaseError{"learned preconditioner: no matrix bound"};
    int nb = (n_ + FB - 1) / FB;
    size_t off = (size_t)next_ * n_;
    k_to_f32<<<nb, FB, 0, st>>>(n_, r, pr_.get() + off);
    k_to_f32<<<nb, FB, 0, st>>>(n_, e, pe_.get() + off);
    g_launches += 2;
    SYSU_CUDA(cudaGetLastError());
    transform_pair(next_, st);
    next_ = (next_ + 1) % capacity_;
    count_ = std::min(count_ + 1, capacity_);
}

void GnnPrecond::add_pair_from(const double *b, const double *x1, const double *xs, cudaStream_t st) {
    if (!bound()) throw CaseError{"learned preconditioner: no matrix bound"};
    size_t off = (size_t)next_ * n_;
    k_pair_from<<<(n_ + FB - 1) / FB, FB, 0, st>>>(gview(*A_, val32_, dinv_.get()), val64_, b, x1, xs,
                                                  pr_.get() + off, pe_.get() + off);
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
    transform_pair(next_, st);
    next_ = (next_ + 1) % capacity_;
    count_ = std::min(count_ + 1, capacity_);
}

void GnnPrecond::train_step(int k, double lr, cudaStream_t st) {
    if (count_ == 0) throw CaseError{"learned preconditioner: no training pairs"};
    k %= count_;
    const float *r = pr_.get() + (size_t)k * n_, *e = pe_.get() + (size_t)k * n_;
    scale_of(r, st);
    forward(r, z32_.get(), true, nullptr, nullptr, st);
    k_gnn_loss<<<gflat_, FB, 0, st>>>(gview(*A_, val32_, dinv_.get()), sgn_, loss_kind, z32_.get(), e, y32_.get(),
                                      part_.get(), sc_.get());
    ++g_launches;
    backward(r, st);
    ++adam_t_;
    k_gnn_adam<<<(GNN_NPARAM + ADAM_P - 1) / ADAM_P, ADAM_P * ADAM_W, 0, st>>>(
        rec_.get(), gtiles_, p_.get(), m_.get(), v_.get(), wbf_.get(), nullptr, lr, 1.0 - std::pow(0.9, adam_t_),
        1.0 - std::pow(0.999, adam_t_), 1, sc_.get(), losses_.get() + ((adam_t_ - 1) & ((1 << 16) - 1)));
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
}

void GnnPrecond::loss_grad(int k, double *loss, float *grad_host, cudaStream_t st) {
    if (count_ == 0) throw CaseError{"learned preconditioner: no training pairs"};
    k %= count_;
    const float *r = pr_.get() + (size_t)k * n_, *e = pe_.get() + (size_t)k * n_;
    scale_of(r, st);
    forward(r, z32_.get(), true, nullptr, nullptr, st);
    k_gnn_loss<<<gflat_, FB, 0, st>>>(gview(*A_, val32_, dinv_.get()), sgn_, loss_kind, z32_.get(), e, y32_.get(),
                                      part_.get(), sc_.get());
    ++g_launches;
    backward(r, st);
    DevBuf<float> g(GNN_NPARAM);
    k_gnn_adam<<<(GNN_NPARAM + ADAM_P - 1) / ADAM_P, ADAM_P * ADAM_W, 0, st>>>(
        rec_.get(), gtiles_, p_.get(), m_.get(), v_.get(), wbf_.get(), g.get(), 0.0, 1.0, 1.0, 0, sc_.get(),
        losses_.get());
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
    g.download(grad_host, GNN_NPARAM, st);
    SYSU_CUDA(cudaMemcpyAsync(loss, losses_.get(), sizeof(double), cudaMemcpyDeviceToHost, st));
    SYSU_CUDA(cudaStreamSynchronize(st));
    check_err(st);
}

void GnnPrecond::last_losses(std::vector<double> &out, int count, cudaStream_t st) {
    count = std::min(count, std::min(adam_t_, 1 << 16));
    out.assign(count, 0.0);
    for (int i = 0; i < count; ++i) {
        int idx = (adam_t_ - count + i) & ((1 << 16) - 1);
        SYSU_CUDA(cudaMemcpyAsync(&out[i], losses_.get() + idx, sizeof(double), cudaMemcpyDeviceToHost, st));
    }
    SYSU_CUDA(cudaStreamSynchronize(st));
}

// One flexible-CG iteration (network or Jacobi preconditioner, direction,
// update, conditional reliable update) enqueued on st.
void GnnPrecond::fcg_iteration(const void *args, bool use_gnn, cudaStream_t st) {
    const FcgArgs &a = *static_cast<const FcgArgs *>(args);
    if (mg_) {
        mg_->apply_to_fine(a.r, z2_.get(), &a.fs->done, st);
        k_fcg_mgfine<<<gflat_, FB, 0, st>>>(a, z2_.get(), t_.get(), mg_->w0(), net_level == 0 ? 1 : 0);
        ++g_launches;
        if (use_gnn && net_level == 0) forward(t_.get(), a.z, false, a.fs, a.q, st, z2_.get());
    } else {
        if (use_gnn) forward(a.r, a.z, false, a.fs, a.q, st);
        k_fcg_jacobi<<<gflat_, FB, 0, st>>>(a);
    }
    k_fcg_dir<<<gflat_, FB, 0, st>>>(a);
    k_fcg_upd<<<gflat_, FB, 0, st>>>(a);
    k_fcg_rel1<<<gflat_, FB, 0, st>>>(a);
    k_fcg_rel2<<<gflat_, FB, 0, st>>>(a);
    g_launches += mg_ ? 4 : 5;
    SYSU_CUDA(cudaGetLastError());
}

// Everything a captured flexible-CG solve bakes in: its kernels' arguments, the
// caller's b, x and statistics pointers, the initial kernel's scalars and the
// attached cycle's parameters.
struct FcgKey {
    FcgArgs a;
    const double *b_in;
    double *x_out;
    SolveInfo *info;
    int x0_zero, maxit, use_gnn, chunk, gflat, net_level, post_level, hook, mg_one_launch;
    double eps, mg_gamma;
    float skip;
    const void *mg;
};

void GnnPrecond::fcg(const double *b, double *x, bool x0_zero, const KrylovOpts &o, bool use_gnn, SolveInfo *info_dev,
                     cudaStream_t st) {
    if (!bound()) throw CaseError{"learned preconditioner: no matrix bound"};
    // the iterations run over fixed buffers: b and x are copied in and out
    if (b64_.size() < (size_t)n_) {
        b64_.alloc(n_);
        x64_.alloc(n_);
    }
    FcgKey k;
    std::memset(&k, 0, sizeof(k));  // padding too: the key is compared as bytes
    FcgArgs &a = k.a;
    a.g = gview(*A_, val32_, dinv_.get());
    a.val64 = val64_;
    a.sgn = sgn_;
    a.b = b64_.get();
    a.x = x64_.get();
    a.r = r32_.get();
    a.z = z32_.get();
    a.p = p32_.get();
    a.q = q32_.get();
    a.e = e32_.get();
    a.fs = fs_.get();
    a.part = part_.get();
    a.inner_tol2 = o.inner_tol * o.inner_tol;
    a.stall_max = stall_max;
    k.b_in = b;
    k.x_out = x;
    k.info = info_dev;
    k.x0_zero = x0_zero ? 1 : 0;
    k.maxit = o.maxit;
    k.use_gnn = use_gnn ? 1 : 0;
    k.chunk = check_every;
    k.gflat = gflat_;
    k.eps = o.eps;
    k.skip = skip;
    k.mg = mg_;
    if (mg_) {
        k.net_level = net_level;
        k.post_level = mg_->post_level;
        k.hook = mg_->post_hook ? 1 : 0;
        k.mg_one_launch = mg_->one_launch ? 1 : 0;
        k.mg_gamma = mg_->gamma;
    }
    // b, x0 in; the iterations; x and the statistics out
    auto prologue = [&](cudaStream_t s) {
        SYSU_CUDA(cudaMemcpyAsync(b64_.get(), b, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
        if (!x0_zero) SYSU_CUDA(cudaMemcpyAsync(x64_.get(), x, sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
        if (x0_zero) {
            k_fcg_zero<<<(n_ + FB - 1) / FB, FB, 0, s>>>(n_, a.x);
            ++g_launches;
        }
        k_fcg_init<<<gflat_, FB, 0, s>>>(a, x0_zero ? 1 : 0, o.eps, o.maxit, use_gnn ? 1 : 0);
        ++g_launches;
        SYSU_CUDA(cudaGetLastError());
    };
    auto epilogue = [&](cudaStream_t s) {
        SYSU_CUDA(cudaMemcpyAsync(x, x64_.get(), sizeof(double) * n_, cudaMemcpyDeviceToDevice, s));
        k_fcg_info<<<1, 1, 0, s>>>(fs_.get(), info_dev);
        ++g_launches;
        SYSU_CUDA(cudaGetLastError());
    };
    // the iterations as a WHILE node: check_every a body; the body's last kernel
    // ends the loop once the solve is done, or after maxit / check_every + 8
    // bodies (the solve stops at maxit itself)
    auto enqueue = [&](cudaStream_t s) {
        prologue(s);
        const int bound = o.maxit / std::max(1, check_every) + 8;
        cudaGraphConditionalHandle loop = graph_cond_handle(s, 1);
        graph_cond_node(s, graph_side_stream(), loop, cudaGraphCondTypeWhile, [&](cudaStream_t bs) {
            for (int c = 0; c < check_every; ++c) fcg_iteration(&a, use_gnn, bs);
            graph_loop_tail(loop, &a.fs->done, &a.fs->loops, bound, bs);
        });
        epilogue(s);
    };
    if (stream_capturing(st)) {  // inside the caller's graph: errors surface in the statuses
        enqueue(st);
        return;
    }
    if (!device_loop) {
        // host-driven form, for per-kernel profiling (profilers skip the kernels of
        // graphs with conditional nodes): the same kernels, check_every
        // iterations a captured graph, the host reading `done` after each
        k.chunk = -check_every;  // a different cache entry from the device loop's
        const unsigned char *kc = reinterpret_cast<const unsigned char *>(&k);
        SolveGraph *cg = nullptr;
        for (SolveGraph &g : graphs_)
            if (g.exec && g.key.size() == sizeof(k) && std::memcmp(g.key.data(), kc, sizeof(k)) == 0) cg = &g;
        if (!cg) {
            cg = &graphs_[graph_next_];
            graph_next_ = (graph_next_ + 1) % 4;
            if (cg->exec) cudaGraphExecDestroy(cg->exec);
            *cg = SolveGraph{};
            const long before = g_launches.load();
            cudaGraph_t g;
            SYSU_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
            for (int c = 0; c < check_every; ++c) fcg_iteration(&a, use_gnn, st);
            SYSU_CUDA(cudaStreamEndCapture(st, &g));
            cg->launches = g_launches.load() - before;
            g_launches -= cg->launches;
            cudaError_t e = cudaGraphInstantiate(&cg->exec, g, 0);
            cudaGraphDestroy(g);
            SYSU_CUDA(e);
            cg->key.assign(kc, kc + sizeof(k));
        }
        prologue(st);
        int done = 0;
        for (int it = 0; it < o.maxit + check_every && !done; it += check_every) {
            SYSU_CUDA(cudaGraphLaunch(cg->exec, st));
            g_launches += cg->launches;
            SYSU_CUDA(cudaMemcpyAsync(&done, &fs_.get()->done, sizeof(int), cudaMemcpyDeviceToHost, st));
            SYSU_CUDA(cudaStreamSynchronize(st));
        }
        epilogue(st);
        if (use_gnn || (mg_ && mg_->post_hook)) check_err(st);
        return;
    }
    const unsigned char *kb = reinterpret_cast<const unsigned char *>(&k);
    SolveGraph *sg = nullptr;
    for (SolveGraph &g : graphs_)
        if (g.exec && g.key.size() == sizeof(k) && std::memcmp(g.key.data(), kb, sizeof(k)) == 0) sg = &g;
    if (!sg) {
        sg = &graphs_[graph_next_];
        graph_next_ = (graph_next_ + 1) % 4;
        if (sg->exec) cudaGraphExecDestroy(sg->exec);
        *sg = SolveGraph{};
        const long before = g_launches.load();
        cudaGraph_t g;
        SYSU_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        try {
            enqueue(st);
        } catch (...) {
            cudaGraph_t junk = nullptr;
            cudaStreamEndCapture(st, &junk);
            if (junk) cudaGraphDestroy(junk);
            throw;
        }
        SYSU_CUDA(cudaStreamEndCapture(st, &g));
        sg->launches = g_launches.load() - before;
        g_launches -= sg->launches;
        cudaError_t e = cudaGraphInstantiate(&sg->exec, g, 0);
        cudaGraphDestroy(g);
        SYSU_CUDA(e);
        sg->key.assign(kb, kb + sizeof(k));
    }
    SYSU_CUDA(cudaGraphLaunch(sg->exec, st));
    g_launches += sg->launches;
    // a network that timed out on a tensor-core wait (a grid barrier of the cycle that gave up is
    // the caller's to report: AggMultigrid::check_wait)
    if (use_gnn || (mg_ && mg_->post_hook)) check_err(st);
}

GnnPrecond::~GnnPrecond() { drop_graphs(); }

__global__ void k_bf16_to_f32(long n, const uint16_t *a, float *b) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = __uint_as_float((uint32_t)a[i] << 16);
}

void GnnPrecond::hidden(const double *r, int layer, float *host, cudaStream_t st) {
    if (!bound()) throw CaseError{"learned preconditioner: no matrix bound"};
    if (layer < 1 || layer > GNN_LAYERS) throw CaseError{"hidden: layer 1..4"};
    int nb = (n_ + FB - 1) / FB;
    k_to_f32<<<nb, FB, 0, st>>>(n_, r, r32_.get());
    ++g_launches;
    scale_of(r32_.get(), st);
    forward(r32_.get(), z32_.get(), true, nullptr, nullptr, st);
    long nn = (long)n_ * 32;
    DevBuf<float> tmp(nn);
    k_bf16_to_f32<<<(unsigned)((nn + FB - 1) / FB), FB, 0, st>>>(nn, H_.get() + (size_t)layer * nn, tmp.get());
    ++g_launches;
    SYSU_CUDA(cudaGetLastError());
    tmp.download(host, nn, st);
    SYSU_CUDA(cudaStreamSynchronize(st));
    check_err(st);
}

FcgState GnnPrecond::last_state(cudaStream_t st) {
    FcgState f;
    SYSU_CUDA(cudaMemcpyAsync(&f, fs_.get(), sizeof(FcgState), cudaMemcpyDeviceToHost, st));
    SYSU_CUDA(cudaStreamSynchronize(st));
    return f;
}

}  // namespace sysu
