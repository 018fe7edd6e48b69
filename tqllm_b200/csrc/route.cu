// Router logits and top-k routing (softmax and sigmoid + selection bias families).
// Replaces router_k / topk_k / topk_warp_k (src/experts/moe.cu:17-166,237-267) and route_k (src/experts/moe_common.cu:18-70).
// Selection rule everywhere: larger key first, lower index on ties (src/experts/moe.cpp:75-78); weights come from
// the unbiased probabilities (src/experts/moe.cpp:85-86); the renormalising sum is clamped at 6.103515625e-5
// (src/experts/moe.hpp:38) and accumulated in selection order like the host reference (src/experts/moe.cpp:103-108).
#include <cooperative_groups.h>
#include <math_constants.h>

#include "common.cuh"
#include "dec4_stage.cuh"
#include "dispatch.cuh"
#include "route_token.cuh"

namespace b2 {
namespace {

constexpr int ROUTER_TOK = 8;   // tokens one warp carries per pass over a weight row

// One warp per router row (row `experts` = the shared-gate vector), ROUTER_TOK tokens at a time, fp32 accumulation.
template <int DT>
__global__ void router_k(const float * __restrict__ w, const float * __restrict__ shared, const typename Elem<DT>::type * __restrict__ x,
                         float * __restrict__ logits, int ld, int h, int e, int rows, int n) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const float * wr = row == e ? shared : w + size_t(row) * h;
    for (int t0 = blockIdx.y * ROUTER_TOK; t0 < n; t0 += gridDim.y * ROUTER_TOK) {
        float acc[ROUTER_TOK];
#pragma unroll
        for (int c = 0; c < ROUTER_TOK; ++c) acc[c] = 0.f;
        for (int j = lane * 4; j < h; j += 128) {
            const float4 wv = *reinterpret_cast<const float4 *>(wr + j);
#pragma unroll
            for (int c = 0; c < ROUTER_TOK; ++c) {
                if (t0 + c < n) {
                    const typename Elem<DT>::type * xr = x + size_t(t0 + c) * h + j;
                    acc[c] += wv.x * Elem<DT>::to_f(xr[0]) + wv.y * Elem<DT>::to_f(xr[1]) + wv.z * Elem<DT>::to_f(xr[2]) +
                              wv.w * Elem<DT>::to_f(xr[3]);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < ROUTER_TOK; ++c) {
            float s = acc[c];
            for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
            if (lane == 0 && t0 + c < n) logits[size_t(t0 + c) * ld + row] = s;
        }
    }
}

// ---- tensor-core router ----
// logits = W x with W fp32 split exactly into three bf16 terms (hi + mid + lo = 24 significant bits) and x split into as many as
// it has bits for (bf16: itself, fp16: two, fp32: three; of the fp32 products the three whose terms lie below 2^-24 of the
// product are left out): every product is exact in fp32 and the sums are fp32, so the result is fp32-accurate (within 3e-6 of
// an fp64 dot) at a fraction of the instructions of a scalar loop (fp16, 600 tokens x 256 experts x 3072: scalar 148 us).
// The tensor core cuts its running sums off instead of rounding them, by up to an ulp per product and always the same way, so for fp16
// and fp32 rows a chain of products does not carry the sum: the leading products of 16 columns start from zero and are added with
// rounding, the others, 2^-8 of them and less, have sums of their own. Relative error against fp64 (2-norm; a scalar fp32 loop,
// one chain for all, this): h = 768 0.88e-7, 1.7e-7, 0.81e-7; 4096 1.28e-7, 3.3e-7 (fp32 4.0e-7), 0.9e-7; in router_tile_k 1.04e-7 where one chain had
// 1.37e-6 (fp32 1.68e-6). bf16 rows, whose products lost three bits of the fp32 chain from the start, keep their one chain (2.2e-7).
// One block = 16 router rows x 8 J tokens; its 16 warps split the hidden dimension and add their partial tiles in shared
// memory in warp order (a token's bits do not depend on J). J is the smallest of 1, 2, 4, 8 that takes the batch in one block or leaves
// at most a block per SM: with J = 8 one token pays for 64.
template <int DT> constexpr int x_terms() { return DT == B2MOE_BF16 ? 1 : DT == B2MOE_F16 ? 2 : 3; }
constexpr int RM_WARPS = 16, RM_PART = 8;   // warps per block (each takes a slice of the columns); partial-sum slots in shared memory
__device__ __forceinline__ void split3(float2 w, uint32_t & hi, uint32_t & mid, uint32_t & lo) {
    const __nv_bfloat16 h0 = __float2bfloat16_rn(w.x), h1 = __float2bfloat16_rn(w.y);
    const float r0 = w.x - __bfloat162float(h0), r1 = w.y - __bfloat162float(h1);
    const __nv_bfloat16 m0 = __float2bfloat16_rn(r0), m1 = __float2bfloat16_rn(r1);
    const __nv_bfloat16 l0 = __float2bfloat16_rn(r0 - __bfloat162float(m0)), l1 = __float2bfloat16_rn(r1 - __bfloat162float(m1));
    hi = uint32_t(__bfloat16_as_ushort(h0)) | (uint32_t(__bfloat16_as_ushort(h1)) << 16);
    mid = uint32_t(__bfloat16_as_ushort(m0)) | (uint32_t(__bfloat16_as_ushort(m1)) << 16);
    lo = uint32_t(__bfloat16_as_ushort(l0)) | (uint32_t(__bfloat16_as_ushort(l1)) << 16);
}
__device__ __forceinline__ void mma_bf16_acc(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (w.x, w.y) -> bf16x2 terms hi, mid, lo with hi + mid + lo = w exactly (24 significant bits); same values as split3
__device__ __forceinline__ void split3_pair(float2 w, uint32_t & hi, uint32_t & mid, uint32_t & lo) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(w.y), "f"(w.x));
    const float r0 = w.x - __uint_as_float(hi << 16), r1 = w.y - __uint_as_float(hi & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(mid) : "f"(r1), "f"(r0));
    const float q0 = r0 - __uint_as_float(mid << 16), q1 = r1 - __uint_as_float(mid & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(q1), "f"(q0));
}
// two neighbouring activations at p -> their bf16x2 terms, the largest first
template <int DT> __device__ __forceinline__ void x_pair(const typename Elem<DT>::type * p, uint32_t (&v)[x_terms<DT>()]) {
    if constexpr (DT == B2MOE_BF16) {
        v[0] = *reinterpret_cast<const uint32_t *>(p);
    } else if constexpr (DT == B2MOE_F16) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(p));
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v[0]) : "f"(f.y), "f"(f.x));
        const float r0 = f.x - __uint_as_float(v[0] << 16), r1 = f.y - __uint_as_float(v[0] & 0xffff0000u);      // at most 3 bits are left: exact as bf16
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v[1]) : "f"(r1), "f"(r0));
    } else {
        split3_pair(*reinterpret_cast<const float2 *>(p), v[0], v[1], v[2]);
    }
}
// A logit whose split products did not give a number: an infinity (or a value that rounds to one as bf16) leaves infinity minus
// infinity behind when it is split, and meets zero terms of the other operand. In a plain loop one infinite activation gives
// infinite logits of the weights' signs, as it should. A NaN ends the loop, so that rows of garbage cost little.
template <int DT> __device__ __noinline__ float plain_logit(const float * w, const typename Elem<DT>::type * x, int h) {
    float s = 0.f;
    for (int j = 0; j < h && s == s; j += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(w + j);
        s += v.x * Elem<DT>::to_f(x[j]) + v.y * Elem<DT>::to_f(x[j + 1]) + v.z * Elem<DT>::to_f(x[j + 2]) + v.w * Elem<DT>::to_f(x[j + 3]);
    }
    return s;
}
// the logit to store: the sum s of (router row, token), looked at again where fp16 or fp32 rows were split; lost: there is no sum
template <int DT> __device__ __forceinline__ float checked_logit(float s, const float * w, const float * shared, const typename Elem<DT>::type * x, int row, int tok, int e, int h, bool lost = false) {
    if (lost || (x_terms<DT>() > 1 && !isfinite(s))) return plain_logit<DT>(row == e ? shared : w + size_t(row) * h, x + size_t(tok) * h, h);
    return s;
}
template <int DT, int J>
__global__ void __launch_bounds__(RM_WARPS * 32) router_mma_k(const float * __restrict__ w, const float * __restrict__ shared,
                                                                const typename Elem<DT>::type * x, float * logits, int ld,
                                                                int h, int e, int rows, int n, int * clear) {
    constexpr int XT = x_terms<DT>(), TOK = 8 * J;
    __shared__ float part[RM_PART][16][65];
    __shared__ float tile[16][65];                                      // this block's sums over its slice of the columns
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();                    // the gridDim.z blocks that split the hidden dimension
    grid_release();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int r0 = blockIdx.x * 16, t0 = blockIdx.y * TOK;
    // The router rows are asked for into the L2 while the launch before this one ends: no value is read, so nothing that launch may write is read too early. Calls of one token
    // back to back 28.3 -> 27.0 us (512 experts x 2048), four layers of 64 tokens 651 -> 649
    if (threadIdx.x < 16 && blockIdx.y == 0 && r0 + int(threadIdx.x) < rows) {
        const int r = r0 + threadIdx.x, cols = h / int(gridDim.z);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"((r == e ? shared : w + size_t(r) * h) + int(blockIdx.z) * cols), "r"(cols * 4));
    }
    grid_wait();                                                       // x may be the output of the launch before this one
    const int ra = min(r0 + g, rows - 1), rb = min(r0 + g + 8, rows - 1);
    const float * wa = ra == e ? shared : w + size_t(ra) * h, * wb = rb == e ? shared : w + size_t(rb) * h;
    float acc[J][4];
    [[maybe_unused]] float low[J][4];                                   // fp16, fp32: the sums of all products but the leading one
#pragma unroll
    for (int j = 0; j < J; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) { acc[j][i] = 0.f; if (XT > 1) low[j][i] = 0.f; }
    const int hs = h / int(gridDim.z), h_lo = int(blockIdx.z) * hs;     // this block's columns (a multiple of 16)
    const int kper = (hs / 16 + RM_WARPS - 1) / RM_WARPS * 16;          // columns per warp, a multiple of 16
    const int k_lo = h_lo + warp * kper, k_hi = min(h_lo + hs, k_lo + kper);
#pragma unroll (XT == 1 ? 4 : 2)
    for (int k0 = k_lo; k0 < k_hi; k0 += 16) {
        uint32_t hi[4], mid[4], lo[4];
        // lane t holds columns 4 t .. 4 t + 3 of the sixteen in both operands (the sum does not care which of them the fragment calls 2 t, 2 t + 1, 2 t + 8, 2 t + 9): one load
        // a row instead of two. 504 sizes of 512 to 5120 columns: bf16 up to 64 tokens 1.06 times as fast, fp32 1.03, fp16 1.01; 64 tokens x 2048 x 512 9.3 -> 8.6 us
        const float4 va = *reinterpret_cast<const float4 *>(wa + k0 + 4 * t), vb = *reinterpret_cast<const float4 *>(wb + k0 + 4 * t);
        split3(make_float2(va.x, va.y), hi[0], mid[0], lo[0]);
        split3(make_float2(vb.x, vb.y), hi[1], mid[1], lo[1]);
        split3(make_float2(va.z, va.w), hi[2], mid[2], lo[2]);
        split3(make_float2(vb.z, vb.w), hi[3], mid[3], lo[3]);
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int tok = min(t0 + 8 * j + g, n - 1);
            struct alignas(4 * sizeof(typename Elem<DT>::type)) Four { typename Elem<DT>::type v[4]; };
            const Four xr = *reinterpret_cast<const Four *>(x + size_t(tok) * h + k0 + 4 * t);
            uint32_t b0[XT], b1[XT];
            x_pair<DT>(xr.v, b0);
            x_pair<DT>(xr.v + 2, b1);
            if constexpr (XT == 1) {                                     // smallest terms first
                mma_bf16_acc(acc[j], lo, b0[0], b1[0]);
                mma_bf16_acc(acc[j], mid, b0[0], b1[0]);
                mma_bf16_acc(acc[j], hi, b0[0], b1[0]);
            } else {
#pragma unroll
                for (int xt = XT - 1; xt >= 0; --xt) {
                    if (xt == 0 || DT == B2MOE_F16) mma_bf16_acc(low[j], lo, b0[xt], b1[xt]);
                    if (xt < 2) mma_bf16_acc(low[j], mid, b0[xt], b1[xt]);
                    if (xt > 0) mma_bf16_acc(low[j], hi, b0[xt], b1[xt]);
                }
                float lead[4] = {0.f, 0.f, 0.f, 0.f};
                mma_bf16_acc(lead, hi, b0[0], b1[0]);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[j][i] += lead[i];
            }
        }
    }
    if constexpr (XT > 1) {
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[j][i] += low[j][i];
    }
    // warps 8..15 park their sums, warps 0..7 add theirs on top (always in this order: the same bits every run)
    if (warp >= RM_PART) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
            part[warp - RM_PART][g][8 * j + 2 * t] = acc[j][0]; part[warp - RM_PART][g][8 * j + 2 * t + 1] = acc[j][1];
            part[warp - RM_PART][g + 8][8 * j + 2 * t] = acc[j][2]; part[warp - RM_PART][g + 8][8 * j + 2 * t + 1] = acc[j][3];
        }
    }
    __syncthreads();
    if (warp < RM_PART) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
            part[warp][g][8 * j + 2 * t] += acc[j][0]; part[warp][g][8 * j + 2 * t + 1] += acc[j][1];
            part[warp][g + 8][8 * j + 2 * t] += acc[j][2]; part[warp][g + 8][8 * j + 2 * t + 1] += acc[j][3];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 16 * TOK; i += blockDim.x) {
        const int r = i & 15, c = i >> 4;
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < RM_PART; ++q) s += part[q][r][c];
        tile[r][c] = s;
    }
    // the blocks of the cluster hold the sums of their column slices: block 0 adds them in block order through
    // distributed shared memory (the same bits every run) and writes the logits
    cluster.sync();
    if (blockIdx.z == 0) {
        for (int i = threadIdx.x; i < 16 * TOK; i += blockDim.x) {
            const int r = i & 15, c = i >> 4;
            if (r0 + r < rows && t0 + c < n) {
                float s = tile[r][c];
                for (unsigned z = 1; z < gridDim.z; ++z) s += cluster.map_shared_rank(&tile[0][0], z)[r * 65 + c];
                logits[size_t(t0 + c) * ld + r0 + r] = checked_logit<DT>(s, w, shared, x, r0 + r, t0 + c, e, h);
            }
        }
        // in the instance of up to eight tokens alone: the compiler gave the others other registers for it (bf16, 32 tokens x 2048 x 512: a layer 115 -> 122 us)
        if (J == 1 && clear && blockIdx.x + blockIdx.y == 0 && threadIdx.x == blockDim.x - 1) *clear = 0;
    }
    cluster.sync();                                                     // the other blocks' tiles stay alive until block 0 has read them
}

// ---- the same product for many tokens (prefill) of fp32, and of short fp16 rows: shared-memory tiles ----
// One block = 64 router rows x 128 tokens, 8 warps of 32 x 32 outputs, 32 columns per stage: both operands are split into
// their bf16 terms once per block and stage (not once per 64 tokens and warp as above) and reach the MMAs through ldmatrix. Every output is summed over the hidden dimension in
// ascending column order (terms lo, mid, hi per 16 columns; 256 columns per partial sum): the same bits every run; the leading products of a stage's two 16-column steps are added to each other, then to the partial sum (see above for the reason).
// A launch has few such tiles (2047 tokens x 256 experts: 64), and a tile alone leaves an SM waiting on its own loads: up to
// eight blocks of a cluster take a part of a tile's 256-column partial sums each and add all of them, in column order, through
// distributed shared memory, so the split changes no bit.
// Measured, one block per tile against the split: 20 of 3072 columns (fp16) 124 -> 32; (bf16, since served by router_tc_k) 32 tiles of 2048 columns
// 60 -> 21 us, 128 of 4096 columns 116 -> 127, 256 of 2048 columns 96 -> 118: from 100 tiles on, one block per tile.
constexpr int RT_ROWS = 64, RT_TOK = 128, RT_K = 32, RT_THREADS = 256, RT_LD = RT_K + 8;   // row stride in shared memory: 80 bytes, conflict-free for ldmatrix
constexpr int RT_SPLIT_BELOW = 100, RT_MAX_PARTS = 64, RT_COLS = 256, RT_PLD = RT_ROWS + 4, RT_PART = RT_TOK * RT_PLD * 4;           // columns of a partial sum; a tile of them in shared memory, [token][row]
constexpr int RT_W_STAGE = 3 * RT_ROWS * RT_LD * 2, RT_X_TERM = RT_TOK * RT_LD * 2;
template <int DT> constexpr int rt_stages_bytes() { return 2 * (RT_W_STAGE + x_terms<DT>() * RT_X_TERM); }
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
template <int DT, bool SPLIT>
__global__ void __launch_bounds__(RT_THREADS) router_tile_k(const float * __restrict__ w, const float * __restrict__ shared,
                                                             const typename Elem<DT>::type * x, float * logits, int ld, int h,
                                                             int e, int rows, int n) {
    using E = typename Elem<DT>::type;
    constexpr int XT = x_terms<DT>(), X_STAGE = XT * RT_X_TERM;
    namespace cg = cooperative_groups;
    extern __shared__ __align__(128) uint8_t rt_smem[];
    uint8_t * w_sm = rt_smem;                                          // [2 stages][3 terms][64 rows][RT_LD] bf16
    uint8_t * x_sm = rt_smem + 2 * RT_W_STAGE;                         // [2 stages][XT terms][128 tokens][RT_LD] bf16
    grid_release();
    grid_wait();                                                       // x may be the output of the launch before this one
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int r0 = blockIdx.x * RT_ROWS, t0 = blockIdx.y * RT_TOK;
    const int wr = warp >> 2, wc = warp & 3;                            // the warp's 32 rows x 32 tokens
    // the block's partial sums [p_lo, p_hi) of the tile's n_part; the last one takes the stages' place in shared memory, the others follow them
    const int n_part = (h + RT_COLS - 1) / RT_COLS, ks = gridDim.z;
    auto first_part = [&](int z) { return n_part * z / ks; };
    const int p_lo = first_part(blockIdx.z), p_hi = first_part(blockIdx.z + 1);
    // this thread's four float2 of a weight stage: row f / 16, columns 2 (f % 16), f = tid + 256 j
    const float * wsrc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int f = tid + RT_THREADS * j, row = min(r0 + (f >> 4), rows - 1);
        wsrc[j] = (row == e ? shared : w + size_t(row) * h) + 2 * (f & 15);
    }
    // this thread's 16 values of an activation stage: 16-byte pieces p = tid + 256 j, token p / PPT, piece p % PPT
    constexpr int V = 16 / int(sizeof(E)), PPT = RT_K / V, XJ = RT_TOK * PPT / RT_THREADS;
    const E * xsrc[XJ];
#pragma unroll
    for (int j = 0; j < XJ; ++j) {
        const int p = tid + RT_THREADS * j;
        xsrc[j] = x + size_t(min(t0 + p / PPT, n - 1)) * h + V * (p % PPT);
    }
    uint4 xreg[XJ];
    auto load_x = [&](int k0) {                                        // the values wait in registers to be split
#pragma unroll
        for (int j = 0; j < XJ; ++j) xreg[j] = *reinterpret_cast<const uint4 *>(xsrc[j] + k0);
    };
    auto store_x = [&](int stage) {
#pragma unroll
        for (int j = 0; j < XJ; ++j) {
            const int p = tid + RT_THREADS * j;
            uint32_t * dst = reinterpret_cast<uint32_t *>(x_sm + stage * X_STAGE + ((p / PPT) * RT_LD + V * (p % PPT)) * 2);
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
                uint32_t v[XT];
                x_pair<DT>(reinterpret_cast<const E *>(&xreg[j]) + 2 * i, v);
#pragma unroll
                for (int q = 0; q < XT; ++q) dst[q * (RT_X_TERM / 4) + i] = v[q];
            }
        }
    };
    float2 wreg[4];
    auto load_w = [&](int k0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) wreg[j] = *reinterpret_cast<const float2 *>(wsrc[j] + k0);
    };
    auto store_w = [&](int stage) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int f = tid + RT_THREADS * j;
            uint32_t hi, mid, lo;
            split3_pair(wreg[j], hi, mid, lo);
            uint32_t * dst = reinterpret_cast<uint32_t *>(w_sm + stage * RT_W_STAGE + ((f >> 4) * RT_LD + 2 * (f & 15)) * 2);
            dst[0] = hi;
            dst[RT_ROWS * RT_LD / 2] = mid;
            dst[2 * RT_ROWS * RT_LD / 2] = lo;
        }
    };
    // acc sums 256 columns at a time and is then put away: the rounding error of a long fp32 chain grows with its
    // length, and the router's tolerance against an fp64 dot (3e-6) leaves no room for a 2048-term chain
    float acc[2][4][4];
    float low[2][4][4];                                                // the sums of all products but the leading one
    [[maybe_unused]] float tot[2][4][4];                               // one block per tile: it adds the partial sums up in registers
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 4; ++c) { acc[a][b][c] = low[a][b][c] = 0.f; if (!SPLIT) tot[a][b][c] = 0.f; }
    auto part_sum = [&](int a, int b, int c) {                         // the finished partial sum, and back to zero
        const float v = acc[a][b][c] + low[a][b][c];
        acc[a][b][c] = low[a][b][c] = 0.f;
        return v;
    };
    auto put_away = [&](uint8_t * at) {
        float * part = reinterpret_cast<float *>(at);
#pragma unroll
        for (int rt = 0; rt < 2; ++rt)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    part[(32 * wc + 8 * nt + 2 * t + (c & 1)) * RT_PLD + 32 * wr + 16 * rt + g + 8 * (c >> 1)] = part_sum(rt, nt, c);
    };
    // ldmatrix addresses of this lane inside a stage: A rows 32 wr + 16 rt + (lane % 16), columns 8 (lane / 16);
    // B tokens 32 wc + 16 pr + (lane % 8) + 8 (lane / 16), columns 8 ((lane / 8) % 2)
    const uint32_t w_base = uint32_t(__cvta_generic_to_shared(w_sm)) + ((32 * wr + (lane & 15)) * RT_LD + 8 * (lane >> 4)) * 2;
    const uint32_t x_base = uint32_t(__cvta_generic_to_shared(x_sm)) + ((32 * wc + (lane & 7) + 8 * (lane >> 4)) * RT_LD + 8 * ((lane >> 3) & 1)) * 2;
    const int s_lo = p_lo * (RT_COLS / RT_K), s_hi = min(h / RT_K, p_hi * (RT_COLS / RT_K));
    load_x(s_lo * RT_K);
    load_w(s_lo * RT_K);
#pragma unroll 1
    for (int s = s_lo; s < s_hi; ++s) {
        const int buf = s & 1;
        store_w(buf);
        store_x(buf);
        __syncthreads();                                               // stage s is complete; every warp is done with stage s - 1
        if (s + 1 < s_hi) { load_x((s + 1) * RT_K); load_w((s + 1) * RT_K); }
        float lead[2][4][4];                          // the leading products of the stage's first 16 columns
#pragma unroll
        for (int kk = 0; kk < RT_K / 16; ++kk) {
            uint32_t b[XT][2][4];                                      // per term, token tiles (0, 1) and (2, 3): b0, b1 of each
#pragma unroll
            for (int q = 0; q < XT; ++q)
#pragma unroll
                for (int pr = 0; pr < 2; ++pr) ldmatrix4(b[q][pr], x_base + buf * X_STAGE + q * RT_X_TERM + (16 * pr * RT_LD + 16 * kk) * 2);
#pragma unroll
            for (int term = 2; term >= 0; --term) {                    // smallest terms first
#pragma unroll
                for (int rt = 0; rt < 2; ++rt) {
                    uint32_t a[4];
                    ldmatrix4(a, w_base + buf * RT_W_STAGE + ((term * RT_ROWS + 16 * rt) * RT_LD + 16 * kk) * 2);
#pragma unroll
                    for (int q = XT - 1; q >= 0; --q)
#pragma unroll
                        for (int nt = 0; nt < 4; ++nt)
                            if (DT != B2MOE_F32 || term + q < 3) {
                                const uint32_t b0 = b[q][nt >> 1][2 * (nt & 1)], b1 = b[q][nt >> 1][2 * (nt & 1) + 1];
                                if (term + q > 0) {
                                    mma_bf16_acc(low[rt][nt], a, b0, b1);
                                } else {
                                    float v[4] = {0.f, 0.f, 0.f, 0.f};
                                    mma_bf16_acc(v, a, b0, b1);
#pragma unroll
                                    for (int c = 0; c < 4; ++c) {
                                        if (kk == 0) lead[rt][nt][c] = v[c];
                                        else acc[rt][nt][c] += lead[rt][nt][c] + v[c];
                                    }
                                }
                            }
                }
            }
        }
        if constexpr (SPLIT) {
            if ((s & 7) == 7 && s + 1 < s_hi) put_away(rt_smem + rt_stages_bytes<DT>() + (s / 8 - p_lo) * RT_PART);
        } else if ((s & 7) == 7 || s + 1 == s_hi) {
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int c = 0; c < 4; ++c) tot[a][b][c] += part_sum(a, b, c);
        }
    }
    if constexpr (!SPLIT) {
#pragma unroll
        for (int rt = 0; rt < 2; ++rt)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int row = r0 + 32 * wr + 16 * rt + g + 8 * (c >> 1), tok = t0 + 32 * wc + 8 * nt + 2 * t + (c & 1);
                    if (row < rows && tok < n) logits[size_t(tok) * ld + row] = checked_logit<DT>(tot[rt][nt][c], w, shared, x, row, tok, e, h);
                }
        return;
    }
    __syncthreads();                                                   // every warp is done with the stages
    put_away(rt_smem);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    // every block of the cluster finishes a share of the tile's tokens; the partial sums' places in the cluster's shared memory
    // come from a table, eight loads are in flight at a time
    __shared__ uint32_t place[RT_MAX_PARTS];
    if (tid < n_part) {
        int z = 0;
        while (first_part(z + 1) <= tid) ++z;
        const int q = tid - first_part(z), last = first_part(z + 1) - first_part(z) - 1;
        const uint32_t local = uint32_t(__cvta_generic_to_shared(rt_smem)) + (q < last ? rt_stages_bytes<DT>() + q * RT_PART : 0);
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(place[tid]) : "r"(local), "r"(z));
    }
    __syncthreads();
    const int tk_lo = RT_TOK * int(blockIdx.z) / ks, tk_hi = RT_TOK * (int(blockIdx.z) + 1) / ks;
    for (int i = tid; i < (tk_hi - tk_lo) * RT_ROWS; i += RT_THREADS) {
        const int tk = tk_lo + i / RT_ROWS, r = i % RT_ROWS;
        if (t0 + tk >= n || r0 + r >= rows) continue;
        const uint32_t off = uint32_t(tk * RT_PLD + r) * 4u;
        float sum = 0.f;
        for (int q = 0; q < n_part; q += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = 0.f;
                if (q + j < n_part) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[j]) : "r"(place[q + j] + off) : "memory");
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) if (q + j < n_part) sum += v[j];
        }
        logits[size_t(t0 + tk) * ld + r0 + r] = checked_logit<DT>(sum, w, shared, x, r0 + r, t0 + tk, e, h);
    }
    cluster.sync();                                                    // the blocks' tiles stay alive until every block has read them
}

__device__ __forceinline__ void argmax_merge(float & v, int & i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

// One warp per token. p[] = unbiased probabilities, key[] = selection keys (p, or p + bias), both in shared memory.
// routes one token with one warp; p / key: e floats each of shared memory owned by the warp
template <int GATING>
__device__ __forceinline__ void route_token(const float * logits, int ld, const float * __restrict__ bias, int * __restrict__ ids,
                                            float * __restrict__ weights, float * __restrict__ shared_weights, int e, int k, int norm,
                                            float scale, int token, int lane, float * p, float * key) {
    if (k <= 32 && e <= 128) return route_token_regs<GATING, 4>(logits, ld, bias, ids, weights, shared_weights, e, k, norm, scale, token, lane, reinterpret_cast<Picked *>(p));
    if (k <= 32 && e <= 256) return route_token_regs<GATING, 8>(logits, ld, bias, ids, weights, shared_weights, e, k, norm, scale, token, lane, reinterpret_cast<Picked *>(p));
    if (k <= 32 && e <= 512) return route_token_regs<GATING, 16>(logits, ld, bias, ids, weights, shared_weights, e, k, norm, scale, token, lane, reinterpret_cast<Picked *>(p));
    const float * x = logits + size_t(token) * ld;
    if (GATING == B2MOE_SOFTMAX) {
        float m = -CUDART_INF_F;
        for (int j = lane; j < e; j += 32) m = fmaxf(m, x[j]);
        for (int d = 16; d; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
        float sum = 0.f;
        for (int j = lane; j < e; j += 32) { const float v = expf(x[j] - m); p[j] = v; sum += v; }
        for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        for (int j = lane; j < e; j += 32) { const float v = p[j] / sum; p[j] = v; key[j] = v; }
    } else {
        for (int j = lane; j < e; j += 32) {
            const float v = 1.f / (1.f + expf(-x[j]));
            p[j] = v;
            key[j] = bias ? v + bias[j] : v;
        }
    }
    __syncwarp();
    float sel_sum = 0.f;
    for (int r = 0; r < k; ++r) {
        float bv = -CUDART_INF_F;
        int bi = 0x7fffffff;
        for (int j = lane; j < e; j += 32) {
            const float v = key[j];                  // taken entries hold NaN and never compare true
            if (v > bv || (bi == 0x7fffffff && v == v)) { bv = v; bi = j; }   // ascending j: the lowest index keeps a tie
        }
        for (int d = 16; d; d >>= 1) argmax_merge(bv, bi, __shfl_xor_sync(0xffffffffu, bv, d), __shfl_xor_sync(0xffffffffu, bi, d));
        if (bi == 0x7fffffff) bi = 0;              // only when the logits themselves hold NaN
        if (lane == 0) {
            const float pv = p[bi];
            ids[size_t(token) * k + r] = bi;
            weights[size_t(token) * k + r] = pv;
            sel_sum += pv;
            key[bi] = CUDART_NAN_F;
        }
        __syncwarp();
    }
    if (lane == 0) {
        float * w = weights + size_t(token) * k;
        if (norm) {
            const float total = fmaxf(sel_sum, 6.103515625e-5f);
            for (int r = 0; r < k; ++r) w[r] = w[r] / total;
        }
        if (scale != 0.f && scale != 1.f) for (int r = 0; r < k; ++r) w[r] *= scale;
        if (shared_weights) shared_weights[token] = 1.f / (1.f + expf(-x[e]));
    }
}

template <int GATING>
__global__ void route_k(const float * logits, int ld, const float * __restrict__ bias, int * __restrict__ ids,
                        float * __restrict__ weights, float * __restrict__ shared_weights, int e, int k, int norm, float scale, int n) {
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int token = blockIdx.x * warps + warp;
    grid_release();
    grid_wait();
    if (token >= n) return;
    float * p = smem + size_t(warp) * 2 * e;
    route_token<GATING>(logits, ld, bias, ids, weights, shared_weights, e, k, norm, scale, token, lane, p, p + e);
}

// Two routings in one launch (blockIdx.y picks the set): this layer's logits and the next layer's predicted ones
// (topk_warp2_k, src/experts/moe.cu:160-166). Each token's selection is route_k's.
struct RouteSet { const float * logits; int * ids; float * weights; float * shared_weights; };
template <int GATING>
__global__ void route2_k(const RouteSet a, const RouteSet b, int ld, const float * __restrict__ bias, int e, int k, int norm, float scale, int n) {
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int token = blockIdx.x * warps + warp;
    const RouteSet & t = blockIdx.y ? b : a;
    grid_release();
    grid_wait();
    if (token >= n) return;
    float * p = smem + size_t(warp) * 2 * e;
    route_token<GATING>(t.logits, ld, bias, t.ids, t.weights, t.shared_weights, e, k, norm, scale, token, lane, p, p + e);
}

// Top-k routing and dispatch in one launch for decode-sized batches: the block's 16 warps route the tokens (round
// robin), then the same block builds the plan from the ids it just wrote. Saves a launch and a device-wide drain.
// 512 threads: the register-resident top-k keeps 32 values per lane, which a 1024-thread block's 64 registers would spill.
constexpr int RD_THREADS = 512;
template <int GATING>
__global__ void __launch_bounds__(RD_THREADS) route_dispatch_k(const float * logits, int ld, const float * __restrict__ bias,
                                                         int * __restrict__ ids, float * __restrict__ weights,
                                                         float * __restrict__ shared_weights, int e, int k, int norm, float scale, int n,
                                                         int shared_first, int shared_count, int * __restrict__ plan) {
    extern __shared__ __align__(16) float smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float * p = smem + size_t(warp) * 2 * e;
    grid_release();
    grid_wait();
    for (int token = warp; token < n; token += RD_THREADS / 32) {
        route_token<GATING>(logits, ld, bias, ids, weights, shared_weights, e, k, norm, scale, token, lane, p, p + e);
        __syncwarp();
    }
    __syncthreads();                              // the ids are written and the routing scratch is dead
    dispatch_small_body<false>(ids, n * k, e, shared_first, shared_count, plan, reinterpret_cast<unsigned short *>(smem));
}

// The same for up to RC_BLOCKS * RD_THREADS / 32 tokens, as one thread-block cluster: every block routes its share of the tokens
// (a warp per token), the cluster meets once, block 0 builds the plan from the ids and the other blocks meanwhile bring the
// layer's activation rows into the staged form of the 4-bit decode kernels (dec4_stage.cuh), which depends on the rows
// alone. One launch instead of three (top-k, dispatch, staging) on the critical path of a decode-sized layer call.
constexpr int RC_BLOCKS = 8;
struct StageJob { const void * x; int dtype, k, bits; uint8_t * rows; float * inv_scale; };     // x = nullptr: nothing to stage
template <int GATING>
__global__ void __launch_bounds__(RD_THREADS) route_cluster_k(const float * logits, int ld, const float * __restrict__ bias,
                                                        int * __restrict__ ids, float * __restrict__ weights,
                                                        float * __restrict__ shared_weights, int e, int k, int norm, float scale, int n,
                                                        int shared_first, int shared_count, int * __restrict__ plan, const StageJob st) {
    extern __shared__ __align__(16) float smem[];
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rank = int(cluster.block_rank()), nb = int(cluster.num_blocks());
    float * p = smem + size_t(warp) * 2 * e;
    grid_release();
    grid_wait();
    for (int token = rank + nb * warp; token < n; token += nb * (RD_THREADS / 32)) {
        route_token<GATING>(logits, ld, bias, ids, weights, shared_weights, e, k, norm, scale, token, lane, p, p + e);
        __syncwarp();
    }
    __threadfence();
    cluster.sync();                               // every block's ids are written and visible
    if (rank == 0) {
        dispatch_small_body<false>(ids, n * k, e, shared_first, shared_count, plan, reinterpret_cast<unsigned short *>(smem));
    } else if (st.x) {
        for (int row = (rank - 1) + (nb - 1) * warp; row < n; row += (nb - 1) * (RD_THREADS / 32))
            stage_row_warp(st.x, st.dtype, row, st.k, st.bits, st.rows, st.inv_scale, lane);
    }
}

template <int GATING>
int32_t route_launch(const float * logits, int ld, const float * bias, int * ids, float * weights, float * shared_weights, int e,
                     int k, int norm, float scale, int n, cudaStream_t s) {
    const int warps = e <= 1024 ? 4 : 1;
    const size_t smem = size_t(warps) * 2 * e * sizeof(float);
    launch_overlapped(route_k<GATING>, dim3(ceil_div(n, warps)), dim3(warps * 32), smem, s, logits, ld, bias, ids, weights, shared_weights, e, k, norm, scale, n);
    return launch_status();
}

}  // namespace

// true when the one-cluster routing launch takes this shape: a warp per token, the plan built by one block
bool route_cluster_fits(int experts, int topk, int n) {
    return n >= 1 && n <= RC_BLOCKS * (RD_THREADS / 32) && dispatch_small_path(experts, n * topk) &&
           size_t(RD_THREADS / 32) * 2 * experts * sizeof(float) <= 160 * 1024;
}
// Top-k + dispatch (+ staging of the n activation rows x[n][k] for the 4-bit decode kernels when x is given) as one cluster
// launch. *took = false and B2MOE_OK when the shape does not fit: the caller takes the separate launches.
int32_t route_plan_stage(int gating, const float * logits, int ld, const float * bias, int * ids, float * weights, float * shared_weights,
                         int experts, int topk, int norm, float scale, int n, int shared_first, int shared_count, int * plan, const void * x,
                         int x_dtype, int k, int bits, uint8_t * staged_rows, float * inv_scale, cudaStream_t s, bool * took) {
    *took = false;
    if (!route_cluster_fits(experts, topk, n)) return B2MOE_OK;
    const size_t smem = size_t(RD_THREADS / 32) * 2 * experts * sizeof(float);
    const StageJob st{x, x_dtype, k, bits, staged_rows, inv_scale};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(RC_BLOCKS);
    cfg.blockDim = dim3(RD_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = RC_BLOCKS; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_overlap ? 2 : 1;
    if (gating == B2MOE_SOFTMAX) {
        if (cudaFuncSetAttribute(route_cluster_k<B2MOE_SOFTMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return B2MOE_ERR_CUDA;
        cudaLaunchKernelEx(&cfg, route_cluster_k<B2MOE_SOFTMAX>, logits, ld, (const float *)nullptr, ids, weights, shared_weights, experts, topk, 1, scale, n,
                           shared_first, shared_count, plan, st);
    } else {
        if (cudaFuncSetAttribute(route_cluster_k<B2MOE_SIGMOID>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return B2MOE_ERR_CUDA;
        cudaLaunchKernelEx(&cfg, route_cluster_k<B2MOE_SIGMOID>, logits, ld, bias, ids, weights, (float *)nullptr, experts, topk, norm, scale, n,
                           shared_first, shared_count, plan, st);
    }
    *took = true;
    return launch_status();
}
namespace {
constexpr int ROUTER_SMS = 148;
template <typename... KArgs, typename... Args>
int32_t launch_cluster_z(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t s, Args &&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = grid.z;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_overlap ? 2 : 1;
    if (cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...) != cudaSuccess) return B2MOE_ERR_CUDA;
    return launch_status();
}
}  // namespace
}  // namespace b2
#include "router_tc.cuh"
namespace b2 {
namespace {
// clear (may be null): a word that router_mma_k sets to 0 for up to eight tokens; *cleared tells whether it does
template <int DT>
int32_t router_launch(const float * w, const float * shared, const void * xv, float * logits, int ld, int h, int e, int rows, int n, int * clear, bool * cleared, cudaStream_t s) {
    const auto * x = static_cast<const typename Elem<DT>::type *>(xv);
    // router_mma_k splits the hidden dimension over a cluster of up to 4 blocks while every block keeps at least 256 columns
    int ks = 1;
    while (ks < 4 && h % (32 * ks) == 0 && h / (2 * ks) >= 256) ks *= 2;
    auto mma_blocks = [&](int tokens) { return (long long)ceil_div(rows, 16) * ceil_div(n, tokens) * ks; };
    // 16-bit rows go to router_tc_k where router_mma_k, with its 64 tokens a block, has more than two blocks per SM, or more than one and enough rows to fill most of a tile of
    // 128. Before / router_tc_k, us: bf16 2048 columns x 512 experts, 256 tokens 17.8 / 10.1, 509 23.5 / 11.2, 4096 87 / 32; 4096 x 128, 8192 tokens 163 / 40; 3072 x 256, 2047
    // tokens 57 / 20; fp16 600 x 3072 x 256 32 / 15.5, 4096 x 2048 x 512 187 / 73, 600 x 2560 x 60 (160 blocks) 21.9 / 13.7. Not where the other kernels are more precise (2-norm against
    // fp64): bf16 below 256 tokens (1.3e-7 to 2.2e-7, the chains here 4.7e-7), fp16 below 768 columns (6.9e-8, here 7.2e-8; from there on 8.1e-8 to 1.04e-7). bf16 rows below 256 tokens
    // with more than a block per SM take the fine form instead (7.2e-8) where it costs fewer cycles; router_mma_k / fine, us: 2048 x 512, 65 tokens 15.3 / 12.9, 128 18.1 / 13.1, 255 35.4 / 13.3;
    // 3072 x 256, 200 tokens 1.5 times as fast; 2048 x 1024, 1 token 7.0 / 13.0, 16 8.0 / 14.4, 32 13.6 / 14.3, 64 18.1 / 14.8; 2048 x 4000, 1 token 20.6 / 13.9. What router_mma_k costs there is the cost of the instance that
    // it would launch: with the 64-token one's for every batch 232 sizes of up to 64 tokens took 1.23 times the better kernel's time on average, 2.25 at most; now 1276 sizes take 1.002 and 1.20 (352 of 65 to 255 tokens: 1.0025, 1.17).
    // bf16 rows between one and two blocks per SM and up to 48 router rows: the fine form (7.2e-8; router_mma_k up to 2.7e-7) where it costs fewer cycles. router_tile_k, which served them once at
    // 8.2e-7 / router_mma_k / fine, us: 2048 x 48, 1024 tokens 12.7 / 17.6 / 12.3; 1536 x 48, 1500 14.1 / 23.9 / 12.5; 1024 x 32, 2047 13.9 / 14.9 / 12.7; 256 x 32, 8192 10.5 / 12.1 / 7.8; dearer:
    // 5120 x 32, 2047 55 / 26.6 / 39. Up to 16 rows a tile of 128 stays empty: router_mma_k (1.3e-7 and more exact than the chains) where it costs less than they: 3072 x 8, 6000 tokens
    // 29 / 37, 5120 x 8, 4096 (256 blocks) 25 / 36, but 2048 x 16, 8192 35 / 19. Cycles of router_mma_k: of 64 tokens a block as fitted to 300 sizes of 256 to 5120 columns
    // when a lane loaded two columns (0.99 of 720 sizes' times since, 15 % spread), of fewer fitted to 957 sizes of 600 and more rows, on
    // the scale of the fine form's cycles (1400 to 1500 a microsecond).
    // fp16 rows stay here with few rows too, as it is the most exact (8 rows x 3072, 8192 tokens: 70 us, router_mma_k 45 at 8.9e-8; router_tile_k 93 at 9.7e-8).
    // Rows of fp32, and short ones of fp16: tiles once router_mma_k has more than two blocks per SM. router_mma_k / tiles, us: 1024 columns x 32 experts, fp16,
    // 600 tokens 8.9 / 17.7, 2047 (256 blocks) 16.8 / 18.0, 4096 (512 blocks) 32 / 18; 2560 x 60, 600 tokens (160) 22.8 / 31, 2047 (512) 46 / 32;
    // 3072 x 256, 256 tokens (256) 25 / 31, 300 (320) 36 / 31; 256 x 32 4096 tokens (128) 8.3 / 22.
    // A grid holds 65,535 blocks of tokens; what is more than that many takes the scalar loop, as everything else that does not fit.
    constexpr int GRID_Y = 65535;
    const long long blocks = mma_blocks(64);
    // the fewest tokens a block of router_mma_k that leave at most a block per SM: with 64, 64 tokens of 768 columns x 64 experts were 8 blocks
    auto fits = [&](int tokens) { return n <= tokens || mma_blocks(tokens) <= ROUTER_SMS; };
    const int mma_tokens = fits(8) ? 8 : fits(16) ? 16 : fits(32) ? 32 : 64;
    if constexpr (DT == B2MOE_F16)
        if (h % RT_K == 0 && h >= 768 && (blocks > 2 * ROUTER_SMS || (blocks > ROUTER_SMS && rows > 48)))
            return rtc::launch<DT, true>(w, shared, x, logits, ld, h, e, rows, n, s);
    if constexpr (DT == B2MOE_BF16)
        if (h % RT_K == 0 && blocks > ROUTER_SMS) {
            struct Cost { int launch, block, ten_columns; };
            const Cost c = mma_tokens <= 16 ? Cost{3000, 3500, 27} : mma_tokens == 32 ? Cost{6700, 5500, 54} : Cost{5000, 8900, 156};
            const long long mma_cycles = c.launch + mma_blocks(mma_tokens) * (c.block + (long long)c.ten_columns * (h / ks) / 10) / ROUTER_SMS;
            auto below_mma = [&](const rtc::Shape & p) { return p.cycles < mma_cycles || ceil_div(n, 64) > GRID_Y; };
            if (n >= 256 && (rows > 48 || (blocks > 2 * ROUTER_SMS && (rows > 16 || below_mma(rtc::shape_of<DT, false>(rows, n, h))))))
                return rtc::launch<DT, false>(w, shared, x, logits, ld, h, e, rows, n, s);
            if ((n < 256 || blocks <= 2 * ROUTER_SMS) && rows > 16 && below_mma(rtc::shape_of<DT, true>(rows, n, h)))
                return rtc::launch<DT, true>(w, shared, x, logits, ld, h, e, rows, n, s);
        }
    if constexpr (DT != B2MOE_BF16) if (h % RT_K == 0 && blocks > 2 * ROUTER_SMS && ceil_div(n, RT_TOK) <= GRID_Y) {
        const dim3 tiles(ceil_div(rows, RT_ROWS), ceil_div(n, RT_TOK), 1);
        const int n_part = ceil_div(h, RT_COLS), share = ceil_div(n_part, 8), ks = ceil_div(n_part, share);      // at most eight blocks, no more than the shares need
        const size_t smem = rt_stages_bytes<DT>() + size_t(share - 1) * RT_PART;
        static_assert(rt_stages_bytes<DT>() >= RT_PART, "the last partial sum takes the stages' place");
        const bool split = n_part > 1 && tiles.x * tiles.y < RT_SPLIT_BELOW && n_part <= RT_MAX_PARTS && smem <= 227 * 1024;
        const auto kernel = split ? router_tile_k<DT, true> : router_tile_k<DT, false>;
        const size_t bytes = split ? smem : size_t(rt_stages_bytes<DT>());
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)) != cudaSuccess) return B2MOE_ERR_CUDA;
        return launch_cluster_z(kernel, dim3(tiles.x, tiles.y, split ? ks : 1), RT_THREADS, bytes, s, w, shared, x, logits, ld, h, e, rows, n);
    }
    if (h % 16 == 0 && ceil_div(n, 64) <= GRID_Y) {
        if (cleared) *cleared = clear && n <= 8;
        auto launch = [&](auto kernel, int tokens) {
            return launch_cluster_z(kernel, dim3(ceil_div(rows, 16), ceil_div(n, tokens), ks), RM_WARPS * 32, 0, s, w, shared, x, logits, ld, h, e, rows, n, clear);
        };
        return mma_tokens == 8 ? launch(router_mma_k<DT, 1>, 8) : mma_tokens == 16 ? launch(router_mma_k<DT, 2>, 16) : mma_tokens == 32 ? launch(router_mma_k<DT, 4>, 32) : launch(router_mma_k<DT, 8>, 64);
    }
    router_k<DT><<<dim3(ceil_div(rows, 8), std::min(ceil_div(n, ROUTER_TOK), 64)), 256, 0, s>>>(w, shared, x, logits, ld, h, e, rows, n);
    return launch_status();
}
}  // namespace

void router_drop_step(int step) { rtc::g_drop_step = step; }

// b2moe_router; where it can (*cleared), the launch also sets *clear to 0, in order before every launch behind it
int32_t router_logits(const float * router_w, const float * shared_gate, const void * x, int32_t x_dtype, float * logits, int32_t ld, int32_t hidden, int32_t experts, int32_t n, int * clear, bool * cleared,
                      cudaStream_t s) {
    if (cleared) *cleared = false;
    if (hidden <= 0 || experts <= 0 || n <= 0 || hidden % 8 || ld < experts + (shared_gate ? 1 : 0)) return B2MOE_ERR_SHAPE;
    if (!router_w || !x || !logits) return B2MOE_ERR_NULL;
    if (!valid_dtype(x_dtype)) return B2MOE_ERR_SHAPE;
    if (!aligned16(router_w) || !aligned16(x) || (shared_gate && !aligned16(shared_gate))) return B2MOE_ERR_ALIGN;
    const int rows = experts + (shared_gate ? 1 : 0);
    if (x_dtype == B2MOE_F32) return router_launch<B2MOE_F32>(router_w, shared_gate, x, logits, ld, hidden, experts, rows, n, clear, cleared, s);
    if (x_dtype == B2MOE_BF16) return router_launch<B2MOE_BF16>(router_w, shared_gate, x, logits, ld, hidden, experts, rows, n, clear, cleared, s);
    return router_launch<B2MOE_F16>(router_w, shared_gate, x, logits, ld, hidden, experts, rows, n, clear, cleared, s);
}
}  // namespace b2

using namespace b2;

extern "C" B2MOE_API int32_t b2moe_router(const float * router_w, const float * shared_gate, const void * x, int32_t x_dtype, float * logits,
                                int32_t ld, int32_t hidden, int32_t experts, int32_t n, b2moe_stream stream) {
    return router_logits(router_w, shared_gate, x, x_dtype, logits, ld, hidden, experts, n, nullptr, nullptr, as_stream(stream));
}

extern "C" B2MOE_API int32_t b2moe_topk_softmax(const float * logits, int32_t ld, int32_t * ids, float * weights, float * shared_weights,
                                      int32_t experts, int32_t topk, int32_t n, float scale, b2moe_stream stream) {
    if (experts <= 0 || experts > 4096 || topk <= 0 || topk > experts || n <= 0 || ld < experts + (shared_weights ? 1 : 0))
        return B2MOE_ERR_SHAPE;
    if (!logits || !ids || !weights) return B2MOE_ERR_NULL;
    return route_launch<B2MOE_SOFTMAX>(logits, ld, nullptr, ids, weights, shared_weights, experts, topk, 1, scale, n, as_stream(stream));
}

extern "C" B2MOE_API int32_t b2moe_topk_softmax2(const float * logits, int32_t * ids, float * weights, float * shared_weights, const float * logits2,
                                                 int32_t * ids2, float * weights2, float * shared_weights2, int32_t ld, int32_t experts, int32_t topk,
                                                 int32_t n, float scale, b2moe_stream stream) {
    if (experts <= 0 || experts > 4096 || topk <= 0 || topk > experts || n <= 0 || ld < experts + ((shared_weights || shared_weights2) ? 1 : 0))
        return B2MOE_ERR_SHAPE;
    if (!logits || !ids || !weights || !logits2 || !ids2 || !weights2) return B2MOE_ERR_NULL;
    const int warps = experts <= 1024 ? 4 : 1;
    const size_t smem = size_t(warps) * 2 * experts * sizeof(float);
    const RouteSet a{logits, ids, weights, shared_weights}, b{logits2, ids2, weights2, shared_weights2};
    launch_overlapped(route2_k<B2MOE_SOFTMAX>, dim3(ceil_div(n, warps), 2), dim3(warps * 32), smem, as_stream(stream), a, b, ld, (const float *)nullptr,
                      experts, topk, 1, scale, n);
    return launch_status();
}

extern "C" B2MOE_API int32_t b2moe_route_sigmoid(const float * logits, int32_t ld, const float * bias, int32_t * ids, float * weights,
                                       int32_t experts, int32_t topk, int32_t norm, float scale, int32_t n, b2moe_stream stream) {
    if (experts <= 0 || experts > 4096 || topk <= 0 || topk > experts || n <= 0 || ld < experts) return B2MOE_ERR_SHAPE;
    if (!logits || !ids || !weights) return B2MOE_ERR_NULL;
    return route_launch<B2MOE_SIGMOID>(logits, ld, bias, ids, weights, nullptr, experts, topk, norm, scale, n, as_stream(stream));
}

// b2moe_topk_softmax / b2moe_route_sigmoid followed by b2moe_dispatch_range, as one launch when the batch is
// decode-sized (otherwise the separate launches); same outputs, same bits.
extern "C" B2MOE_API int32_t b2moe_route_dispatch(int32_t gating, const float * logits, int32_t ld, const float * bias, int32_t * ids,
                                                  float * weights, float * shared_weights, int32_t experts, int32_t topk, int32_t norm,
                                                  float scale, int32_t n, int32_t shared_first, int32_t shared_count, int32_t * plan,
                                                  void * workspace, size_t workspace_bytes, b2moe_stream stream) {
    if (gating != B2MOE_SOFTMAX && gating != B2MOE_SIGMOID) return B2MOE_ERR_SHAPE;
    if (experts <= 0 || experts > 4096 || topk <= 0 || topk > experts || n <= 0 || ld < experts + (shared_weights ? 1 : 0)) return B2MOE_ERR_SHAPE;
    if (shared_first < 0 || shared_count < 0 || shared_first + shared_count > n || (long long)n * topk > 0x3fffffffLL) return B2MOE_ERR_SHAPE;
    if (!logits || !ids || !weights || !plan) return B2MOE_ERR_NULL;
    const size_t smem = size_t(RD_THREADS / 32) * 2 * experts * sizeof(float);
    // one launch only while every token has a warp of its own: the single block routes its tokens RD_THREADS / 32 at a time,
    // and a token's selection rounds are a dependent chain (measured: 64 tokens, 512 experts: 53 us fused against 12 + 10 us as
    // two launches)
    if (n <= RD_THREADS / 32 && dispatch_small_path(experts, n * topk) && smem <= 160 * 1024) {
        cudaStream_t s = as_stream(stream);
        if (gating == B2MOE_SOFTMAX) {
            if (cudaFuncSetAttribute(route_dispatch_k<B2MOE_SOFTMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return B2MOE_ERR_CUDA;
            launch_overlapped(route_dispatch_k<B2MOE_SOFTMAX>, dim3(1), dim3(RD_THREADS), smem, s, logits, ld, nullptr, ids, weights, shared_weights, experts,
                              topk, 1, scale, n, shared_first, shared_count, plan);
        } else {
            if (cudaFuncSetAttribute(route_dispatch_k<B2MOE_SIGMOID>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return B2MOE_ERR_CUDA;
            launch_overlapped(route_dispatch_k<B2MOE_SIGMOID>, dim3(1), dim3(RD_THREADS), smem, s, logits, ld, bias, ids, weights, nullptr, experts, topk,
                              norm, scale, n, shared_first, shared_count, plan);
        }
        return launch_status();
    }
    if (route_cluster_fits(experts, topk, n)) {
        bool took = false;
        const int32_t rc = route_plan_stage(gating, logits, ld, bias, ids, weights, shared_weights, experts, topk, norm, scale, n, shared_first,
                                            shared_count, plan, nullptr, 0, 0, 0, nullptr, nullptr, as_stream(stream), &took);
        if (rc || took) return rc;
    }
    if (int32_t rc = gating == B2MOE_SOFTMAX ? b2moe_topk_softmax(logits, ld, ids, weights, shared_weights, experts, topk, n, scale, stream)
                                             : b2moe_route_sigmoid(logits, ld, bias, ids, weights, experts, topk, norm, scale, n, stream)) return rc;
    return b2moe_dispatch_range(ids, n, topk, experts, shared_first, shared_count, plan, workspace, workspace_bytes, stream);
}
