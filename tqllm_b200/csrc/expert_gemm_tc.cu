// Grouped expert GEMM on the 5th-generation tensor cores for every bank format: the path for batches where an expert
// sees many tokens (prefill) and the tensor-core path of the formats that have no hand-tuned decode kernel.
// Replaces the grouped prefill kernels u4h_gemm_k / k_expert_gemm / k_expert_gemm_gateup
// (src/formats/weight/quant_u4h.inc:609-774, src/formats/weight/quant.cu:286-405) with their fused SwiGLU epilogue
// (quant_u4h.inc:756-759): per expert Y_e = W_e . X_e^T over the expert's gathered token rows.
//
// One persistent block per SM; an item is (expert, tile of up to `cap` of its tokens, block of 128 weight rows): 128 rows of the
// down matrix, or 64 rows of the gate and the same 64 rows of the up matrix (row tiles of 16, gate and up alternating, so
// that both rows of an output element sit in one warp's quarter of tensor memory). Per item
//   D[128 rows][N tokens] (fp32, tensor memory) = sum over K of A[128][K] (fp16) . B[N][K] (fp16)
//   A: the weight rows, decoded from the bank's block format to fp16 by the CUDA cores and written to TENSOR MEMORY
//      (tcgen05.st.16x256b: the lane-major bank tile decodes to exactly that fragment). An A operand in shared memory costs
//      64 bytes per clock for its stores and 64 for the tensor core's reads beside 64 for B at N = 128: more than the 128 an
//      SM has, and that was the limit. Four stages of a unit (two steps of 64 columns);
//   B: the tokens' activation rows (fp16, each row scaled by a power of two, brought into slot order before the product), one TMA
//      box per unit in the 128-byte swizzled form. Copies by the threads (cp.async) need a proxy fence before the tensor core
//      may read them, and that fence waits for the copies of the later steps too: measured, the B loader then set the pace
//      (1680 cycles per step at 80 tokens). Gathering token rows by TMA (tile::gather4) costs the issuing warp 60 to 200
//      cycles per four rows and stays for calls whose scratch holds no rows in slot order;
//   two accumulators of 128 columns alternate between items of up to 128 tokens, so the epilogue of one item (SwiGLU, stores)
//   overlaps the products of the next; a wider item takes both. An item of up to 64 tokens splits its K over the two halves of
//   its accumulator (products in turn), and the epilogue adds them: half as long a chain of truncated sums (NVFP4 gate/up, relative error against
//   64 bits 3.7e-7 and 8.3e-7 in one chain); the products' pace is the same either way. In launches of narrow items (by_chunk) the halves take an even
//   number of chunks in turn, and an item of up to 32 tokens has a quarter each for their even and odd products (NVFP4, K = 2048: 1.9e-7 in halves, 1.1e-7 in quarters); a wider one too, of both accumulators,
//   where a last chunk that is not full would leave the halves uneven.
// The control warps share their schedulers with six others, so what they execute per unit bounds the block: they walk uniform
// loops, one elected lane issues, and the raw blocks and rows come in the largest boxes that fit. They are the first warps of the
// block: as the last ones they were served last (c3 decode gate/up 110 us, as the first 78).
// Warps: 0 issues tcgen05.mma, and so does 3 unless it gathers rows; 1 streams the raw blocks (256 columns of the item's eight row tiles per ring slot: one TMA box
// of the down bank, one each of gate and up, running ahead across items); 2 (when it gathers 2..7) loads B; then from 4 (8) on
// eight epilogue warps (two per TMEM lane quarter, 16-token groups in turn) and sixteen that decode A (the j-th: lane quarter j & 3, row tile
// (j >> 2) & 1 of it, every other 256-column chunk). One barrier per step says that its products are done (a commit costs the issuing thread
// 60 cycles): it frees the unit's A stage and the step's B stage. Every wait is bounded; a wait that runs out sets the plan's
// status word, and the block drains and leaves.
// The exact form (TERMS > 0; Q4_K and IQ3_S codes, where the decode kernels' precision is asked for and their eight tokens a pass are too few): A
// holds the integers sc q or (1 + 2 s)(2 n - 15), B the activations in one or two fp16 terms, every 256-column chunk has accumulators of
// its own (sets in turn), and the epilogue warps scale a chunk's sums by the rows' d in fp32 while the next one is multiplied. The mins of Q4_K
// meet the sub-block sums of the activations in one more product a chunk. Items have up to 32 tokens. Decoding costs two instructions
// less a pair of weights than with the scales in the operand, reading the sums back about 150 a scheduler and chunk.
//
// Numerics of the other form: weights are rounded to fp16 after the exact fp32 decode (relative error <= 2^-11 per weight; bf16 operands
// gave 3e-2 of the output RMS as the largest error, fp16 stays below the layer tolerance). An activation row is
// multiplied by 2^e so that its largest magnitude lies in [2^14, 2^15) and rounded to fp16: exact for bf16 inputs down
// to 2^-29 of the row maximum; the epilogue multiplies the sums (fp32) by 2^-e.
#include <type_traits>

#include "common.cuh"
#include "formats.cuh"
#include "gemm_decode.cuh"
#include "tc_ptx.cuh"
#include "tensor_map.cuh"

namespace b2 {
namespace {
using namespace tc;

constexpr int G_KS = 64;                    // columns per step (four MMAs of K = 16); a unit is two steps
constexpr int A_STAGES = 4, A_COLS = 64;    // stages of decoded A operand, a unit each, and their columns
constexpr int STEP_RING = 2 * A_STAGES;     // barriers "the products of step g are done"
constexpr int ACC_COLS = 128, A_COL0 = 2 * ACC_COLS;                // the two accumulators, then the A stages: all 512 columns
constexpr int SPLIT_COLS = ACC_COLS / 2;    // items of up to this many tokens split their K over the halves of the accumulator
constexpr int QUARTER_COLS = SPLIT_COLS / 2;  // those of up to this many over its quarters (GemmArgs::by_chunk)
constexpr int MAX_B_STAGES = 8, RAW_SLOTS = 6, MAX_CAP = 256;
constexpr int MMA_WARP = 0, RAW_WARP = 1, LOAD_WARP0 = 2, MMA_WARP1 = 3, EPI_WARPS = 8, DEC_WARPS = 16;
// warps that load rows: one with boxes (behind it the second issuer: the other roles start at a multiple of four, a TMEM lane quarter each), six gather
constexpr int load_warps(bool gather) { return gather ? 6 : 2; }
constexpr int g_threads(bool gather) { return (LOAD_WARP0 + load_warps(gather) + EPI_WARPS + DEC_WARPS) * 32; }
static_assert(EPI_WARPS * 32 == MAX_CAP, "an epilogue thread looks one token up");
static_assert(MAX_B_STAGES <= STEP_RING, "a B stage is freed by the barrier of the step that used it");
// The exact form (TERMS > 0): items of up to X_CAP tokens at every density (an expert of 100 tokens is decoded four times: 1000 tokens on 60 experts 311 us,
// 168 with the other form's items of 128); sets of sums, a chunk's each: X_CAP columns per term of the activations, then X_CAP
// of the mins; after them the mins' A operand of either group's chunk. As many sets as fit: with two of them the products waited for the epilogue warps
// (445 of 1140 cycles a unit): c2, 509 tokens 316.6 -> 313.4 us, c4, 600 tokens 670 -> 666.5. x_ring: chunks whose row constants the epilogue may still need: those are written when the products of
// the chunk two before are done, so when the sums of the chunk x_sets + 2 before are read
constexpr int X_CAP = 32;
constexpr int x_sets(bool mins, int terms) { return !mins ? 4 : terms == 1 ? 3 : 2; }
constexpr int x_set_cols(bool mins, int terms) { return X_CAP * (terms + (mins ? 1 : 0)); }
constexpr int x_ring(bool mins, int terms) { return x_sets(mins, terms) > 2 ? 8 : 4; }
constexpr int N_BARS = 3 * RAW_SLOTS + A_STAGES + STEP_RING + MAX_B_STAGES + 10;

struct GemmArgs {
    const float * aux0, * aux1, * saux0, * saux1;      // row scales of the banks (gate, up) or (down, -) and of the shared expert's (may be null)
    const float * inv_scale;                // per activation row (the fp16 rows themselves come through the tensor maps)
    int * plan;
    void * out;                             // [assignments][rows] of out_dtype
    int out_dtype;
    int rows, k, experts, topk, A;
    int cap, cap_log2, b_stages, raw_slots; // most tokens of an item; B stages; raw chunks in the ring
    int by_chunk;                           // items of up to SPLIT_COLS tokens split their K by chunks (and products), not by products: cap <= 64, an even number of chunks
    // by_chunk: an item of more tokens than this takes both accumulators, a quarter of 64 columns for each of its four sums. Rows that end inside a chunk: 32, as halves of whole chunks are uneven
    // there (K = 384: 16 and 8 products), a longer chain of truncated sums than products in turn give. Relative error against 64 bits, 50 tokens, products in turn / halves of chunks / quarters: K = 384
    // 6.90e-8 / 7.14e-8 / 6.37e-8, 896 1.03e-7 / 1.04e-7 / 7.9e-8, 1408 1.40e-7 / 1.41e-7 / 9.4e-8. Else 64: no item
    int both_above;
    int b_pair;                             // 1: the B stages are filled and freed a unit at a time, beside the A stage of the unit and through its barriers (b_stages = 2 A_STAGES)
};
// The rows' boxes: sixteen rows and multiples of them, as many as the products take (32 in launches of items of up to 256 tokens). With boxes in quarters of
// `cap` 80 tokens brought 96 rows. Layers, us: c3 prefill 626 -> 623.5, c4 prefill 974 -> 966, c5 prefill 2785 -> 2768
constexpr int BOXES = 8;
__host__ __device__ inline int box_log2(int cap) { return cap > 16 * BOXES ? 5 : 4; }
// x[i]: the activation rows, boxes of i + 1 times 1 << box_log2(cap) rows (a gathering launch: x[0], one row; the exact form: x[0], x[1], and of the sub-block sums x[2], x[3]); w: banks (gate, up) or (down, -), then the shared expert's
struct GemmMaps { CUtensorMap x[BOXES], w[4]; };

template <uint32_t T> constexpr int chunk_tiles() { return 256 / Fmt<T>::KT; }
template <uint32_t T> constexpr int chunk_bytes() { return chunk_tiles<T>() * Fmt<T>::TILE; }
// a chunk of a row tile as the raw TMA boxes see it: parts of at most 256 8-byte words; rows of K may end after any part
template <uint32_t T> constexpr int chunk_parts() { return T == T_IQ4_NL ? 4 : 2; }
template <uint32_t T> constexpr int part_words() { return chunk_bytes<T>() / chunk_parts<T>() / 8; }

// the active experts of the launch: items before it, expert, tokens, first assignment slot
struct Info { int cum, e, cnt, off; };

// what the exact form keeps beside the operands: the mins' B tiles (32 bytes a row) and the rows' constants
// (no mins: 8 KB as ever, though a float a row takes 4: those would only move the numbers of experts, 2565 and 3637, from which a block's ring holds five chunks and four)
constexpr size_t exact_smem(bool mins, int terms) {
    return !terms ? 0 : mins ? size_t(A_STAGES) * X_CAP * 32 + size_t(x_ring(true, terms)) * 128 * sizeof(float2) : size_t(8192);
}
template <uint32_t T>
constexpr size_t gemm_smem(int experts, int cap, int b_stages, int raw_slots, int terms = 0) {
    return 1024 + size_t(b_stages) * cap * 128 * (terms ? terms : 1) + exact_smem(T == T_Q4_K, terms) + size_t(8) * raw_slots * chunk_bytes<T>() + gdec::Dec<T>::TAB_BYTES +
           DEC_WARPS * gdec::Dec<T>::SCRATCH + size_t(experts + 2) * sizeof(Info) + 2 * MAX_CAP * sizeof(int2) + size_t(N_BARS) * 8 + 16;
}

// Eight values of an activation row, those of positions 8 l .. 8 l + 7 of a 64-column step (gdec::colmap): they lie in one, two
// or four runs of neighbouring columns, so a lane takes them with loads of 16, 8 or 4 bytes (16-bit types; rows are 16-byte
// aligned). xr points at the step's first column.
template <uint32_t T, int DT> __device__ __forceinline__ void load_positions(const typename Elem<DT>::type * xr, int l, float (&v)[8]) {
    using E = typename Elem<DT>::type;
    constexpr int RUN = T == T_Q4_K || T == T_IQ3S4 ? 8 : T == T_IQ4_XS || T == T_IQ4_NL ? 2 : 4, BYTES = RUN * int(sizeof(E));
    const int i = l >> 1, b = l & 1;
    float w[8];                                                        // run after run
#pragma unroll
    for (int r = 0; r < 8 / RUN; ++r) {
        const int col = RUN == 8 ? 32 * (i & 1) + 16 * (i >> 1) + 8 * b : RUN == 4 ? 8 * (2 * b + r + 4 * (i >> 1)) + 4 * (i & 1)
                                                                                : 32 * (i >> 1) + 8 * b + 2 * (i & 1) + 16 * (r & 1) + 4 * (r >> 1);
        uint32_t raw[BYTES / 4];
        if constexpr (BYTES >= 16) {
#pragma unroll
            for (int q = 0; q < BYTES / 16; ++q) *reinterpret_cast<uint4 *>(raw + 4 * q) = reinterpret_cast<const uint4 *>(xr + col)[q];
        } else if constexpr (BYTES == 8) {
            *reinterpret_cast<uint2 *>(raw) = *reinterpret_cast<const uint2 *>(xr + col);
        } else {
            raw[0] = *reinterpret_cast<const uint32_t *>(xr + col);
        }
#pragma unroll
        for (int q = 0; q < RUN; ++q) w[r * RUN + q] = Elem<DT>::to_f(reinterpret_cast<const E *>(raw)[q]);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int half = q & 4, e = q & 3;                             // positions come in two words of four values
        v[q] = RUN == 8 ? w[half + ((e & 1) << 1) + (e >> 1)] : RUN == 4 ? w[q] : w[half + 2 * (e & 1) + (e >> 1)];
    }
}
// One activation row of any dtype scaled by a power of two (largest magnitude in [2^14, 2^15)), by one warp; put(step
// column, values) gets a lane's eight positions, the inverse scale is returned. Two passes over the row: its largest
// magnitude, then (from the cache) the values.
template <uint32_t T, int DT, typename Put>
__device__ __forceinline__ float row_scaled(const typename Elem<DT>::type * xr, int k, int lane, Put put) {
    using E = typename Elem<DT>::type;
    constexpr int V = 16 / int(sizeof(E));                              // elements per 16-byte load
    float mx = 0.f;
#pragma unroll 4
    for (int j = lane * V; j < k; j += 32 * V) {
        const uint4 q = *reinterpret_cast<const uint4 *>(xr + j);
        const E * e = reinterpret_cast<const E *>(&q);
#pragma unroll
        for (int i = 0; i < V; ++i) mx = fmaxf(mx, fabsf(Elem<DT>::to_f(e[i])));
    }
    for (int d = 16; d; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    int ex = int((__float_as_uint(mx) >> 23) & 255u) - 127;              // floor(log2(mx)) for a normal mx
    ex = (mx > 0.f && mx < 3e38f) ? max(-100, min(100, ex)) : 14;
    const float scale = __uint_as_float(uint32_t(127 + 14 - ex) << 23);  // 2^(14 - ex)
#pragma unroll 2
    for (int gb = 64 * (lane >> 3); gb < k; gb += 256) {
        float v[8];
        load_positions<T, DT>(xr + gb, lane & 7, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] *= scale;
        put(gb + 8 * (lane & 7), v);
    }
    return __uint_as_float(uint32_t(127 - 14 + ex) << 23);
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
    return make_uint4(gdec::pack_h2(v[0], v[1]), gdec::pack_h2(v[2], v[3]), gdec::pack_h2(v[4], v[5]), gdec::pack_h2(v[6], v[7]));
}
template <uint32_t T, int DT, typename Put>
__device__ __forceinline__ float row_to_f16(const typename Elem<DT>::type * xr, int k, int lane, Put put) {
    return row_scaled<T, DT>(xr, k, lane, [&](int c, const float (&v)[8]) { put(c, pack8(v)); });
}
// The product behind a conversion reads the plan and the weights without waiting for the rows (gemm_tc_k), so a conversion lets it begin only once the launches
// before are complete; or at once (late = false) where its caller knows that the plan is. A layer of 8 tokens on 512 NVFP4 experts 73.3 -> 70.0 us
// (four preparations of weights and tokens: 3 to 6 % each).
__device__ __forceinline__ void rows_begin(bool late) {
    if (!late) grid_release();
    grid_wait();
    if (late) grid_release();
}
// rows in their own order: the gathered form
template <uint32_t T, int DT>
__global__ void rows_to_f16_k(const typename Elem<DT>::type * x, int rows, int k, __half * out, float * inv_scale) {
    const int lane = threadIdx.x & 31, row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    rows_begin(true);
    if (row >= rows) return;
    const float inv = row_to_f16<T, DT>(x + size_t(row) * k, k, lane, [&](int c, const uint4 & v) { *reinterpret_cast<uint4 *>(out + size_t(row) * k + c) = v; });
    if (lane == 0) inv_scale[row] = inv;
}
// rows in the order of the plan's slots (a token's row once for every assignment it has; topk = 0: row = assignment), a warp per slot
template <uint32_t T, int DT>
__global__ void rows_to_slots_k(const typename Elem<DT>::type * x, const int * plan, int experts, int A, int topk, int k,
                                __half * out, float * inv_scale, bool late) {
    const int lane = threadIdx.x & 31, slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    rows_begin(late);
    if (slot >= plan[PLAN_NGROUPED]) return;
    const int e1 = experts + 1, a = plan[PLAN_HDR + e1 + e1 + 1 + e1 + slot];
    const int row = topk == 0 ? a : a < A ? a / topk : a - A;
    const float inv = row_to_f16<T, DT>(x + size_t(row) * k, k, lane, [&](int c, const uint4 & v) { *reinterpret_cast<uint4 *>(out + size_t(slot) * k + c) = v; });
    if (lane == 0) inv_scale[slot] = inv;
}
// the slot of every grouped assignment
__global__ void slot_of_k(const int * plan, int experts, int * slot_of) {
    grid_release();
    grid_wait();
    const int slot = blockIdx.x * blockDim.x + threadIdx.x, e1 = experts + 1;
    if (slot < plan[PLAN_NGROUPED]) slot_of[plan[PLAN_HDR + e1 + e1 + 1 + e1 + slot]] = slot;
}
// the same rows, a warp per token: the row is converted once and stored into the slots of all its assignments. An assignment that
// is not grouped has no slot: what slot_of holds for it is told by the plan's own list.
template <uint32_t T, int DT>
__global__ void tokens_to_slots_k(const typename Elem<DT>::type * x, const int * plan, const int * slot_of,
                                  int experts, int n, int topk, int shared, int k, __half * out, float * inv_scale) {
    const int lane = threadIdx.x & 31, token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    rows_begin(true);
    if (token >= n) return;
    const int e1 = experts + 1, grouped = plan[PLAN_NGROUPED];
    const int * perm = plan + PLAN_HDR + e1 + e1 + 1 + e1;
    int mine = -1;                                                     // lane s: the slot of the token's s-th assignment (lane topk: the shared expert's)
    if (lane < topk + shared) {
        const int a = lane < topk ? token * topk + lane : n * topk + token, slot = slot_of[a];
        if (slot >= 0 && slot < grouped && perm[slot] == a) mine = slot;
    }
    __shared__ int list[8][32];                                        // the token's slots, for each of the block's warps
    int * slots = list[threadIdx.x >> 5];
    const unsigned live = __ballot_sync(0xffffffffu, mine >= 0);
    if (mine >= 0) slots[__popc(live & ((1u << lane) - 1u))] = mine;
    __syncwarp();
    const int count = __popc(live);
    const float inv = row_to_f16<T, DT>(x + size_t(token) * k, k, lane, [&](int c, const uint4 & v) {
        for (int i = 0; i < count; ++i) *reinterpret_cast<uint4 *>(out + size_t(slots[i]) * k + c) = v;
    });
    if (mine >= 0) inv_scale[mine] = inv;
}
// Rows of the exact form: [TERMS][rows][k] fp16, a value as one term (16-bit activations: exact down to 2^-29 of the row's largest magnitude) or as two (fp32: 22 bits), and for the mins of
// Q4_K the sums of the row's 32-column sub-blocks, divided by 32, as [rows][k / 256][16]: eight leading fp16 terms, then the eight rests.
// A lane holds eight columns of one sub-block, lanes l, l ^ 1, l ^ 4, l ^ 5 all of it.
template <uint32_t T, int DT, int TERMS, typename Slots>
__device__ __forceinline__ float exact_row(const typename Elem<DT>::type * xr, int k, int lane, __half * out, size_t plane, __half * mins, Slots each) {
    return row_scaled<T, DT>(xr, k, lane, [&](int c, const float (&v)[8]) {
        const uint4 hi = pack8(v);
        uint4 lo;
        if (TERMS == 2) {
            float r[8];
            const __half * h = reinterpret_cast<const __half *>(&hi);
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = v[i] - __half2float(h[i]);
            lo = pack8(r);
        }
        __half s0, s1;
        if (gdec::Exact<T>::MINS) {
            float s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s = (s + __shfl_xor_sync(0xffffffffu, s, 4)) * 0.03125f;
            s0 = __float2half_rn(s);
            s1 = __float2half_rn(s - __half2float(s0));
        }
        each([&](size_t slot) {
            *reinterpret_cast<uint4 *>(out + slot * k + c) = hi;
            if (TERMS == 2) *reinterpret_cast<uint4 *>(out + plane + slot * k + c) = lo;
            if (gdec::Exact<T>::MINS && (lane & 5) == 0) {
                __half * m = mins + slot * (k / 16) + 16 * (c >> 8) + 2 * (lane >> 3) + ((lane >> 1) & 1);
                m[0] = s0;
                m[8] = s1;
            }
        });
    });
}
template <uint32_t T, int DT, int TERMS>
__global__ void exact_rows_k(const typename Elem<DT>::type * x, const int * plan, int experts, int A, int topk, int k, __half * out, size_t plane,
                             __half * mins, float * inv_scale, bool late) {
    const int lane = threadIdx.x & 31, slot = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    rows_begin(late);
    int row = slot;                                                    // no plan: A rows in their own order, the gathered form
    if (plan) {
        if (slot >= plan[PLAN_NGROUPED]) return;
        const int e1 = experts + 1, a = plan[PLAN_HDR + e1 + e1 + 1 + e1 + slot];
        row = topk == 0 ? a : a < A ? a / topk : a - A;
    } else if (slot >= A) {
        return;
    }
    const float inv = exact_row<T, DT, TERMS>(x + size_t(row) * k, k, lane, out, plane, mins, [&](auto store) { store(size_t(slot)); });
    if (lane == 0) inv_scale[slot] = inv;
}

// The experts that have tokens, in order, and the items before each, into info (then the number of items): from the counts themselves, one scan by all threads of the block; returns how many.
// By way of the plan's list of them (three dependent loads), scanned by one warp, a block asked for its first chunk 2.1 us after it had begun with 75 experts, 4.7 us with 513; now 1.6 and 1.7. A function
// of its own: in the kernel it cost the decoders registers (IQ4, 24 tokens 261 -> 274 us). The caller synchronises after it.
__device__ __noinline__ int find_experts(const int * counts, int e1, int row_blocks, int cap_log2, Info * info, int2 * sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, threads = blockDim.x, * offsets = counts + e1;
    int na = 0, items = 0;
#pragma unroll 1
    for (int base = 0; base < e1; base += threads) {
        const int e = base + int(threadIdx.x), cnt = e < e1 ? counts[e] : 0, off = e < e1 ? offsets[e] : 0, mine = ((cnt + (1 << cap_log2) - 1) >> cap_log2) * row_blocks;
        int a = cnt > 0, v = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int oa = __shfl_up_sync(0xffffffffu, a, d), ov = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) { a += oa; v += ov; }
        }
        if (base > 0) __syncthreads();                                 // the sums of the round before are read
        if (lane == 31) sums[warp] = make_int2(a, v);
        __syncthreads();
        const int2 own = lane < threads / 32 ? sums[lane] : make_int2(0, 0);
        int2 w = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int oa = __shfl_up_sync(0xffffffffu, w.x, d), ov = __shfl_up_sync(0xffffffffu, w.y, d);
            if (lane >= d) { w.x += oa; w.y += ov; }
        }
        const int wa = __shfl_sync(0xffffffffu, w.x - own.x, warp), wv = __shfl_sync(0xffffffffu, w.y - own.y, warp);
        if (cnt > 0) info[na + wa + a - 1] = Info{items + wv + v - mine, e, cnt, off};
        na += __shfl_sync(0xffffffffu, w.x, 31);
        items += __shfl_sync(0xffffffffu, w.y, 31);
    }
    if (threadIdx.x == 0) info[na].cum = items;
    return na;
}

// MODE 0: act[a][r] = silu(gate_r . x_tok(a)) * (up_r . x_tok(a));  MODE 1: y[a][r] = down_r . act[a]
// TERMS > 0: the exact form: no rounding but that of the activations to TERMS fp16 terms (16-bit ones: none above 2^-29 of the row's largest) and of the fp32 sums
// F32_OUT: an instance for fp32 results and one for 16-bit ones, chosen by the call's output type. A branch at the stores, or two
// loops in one kernel, cost every fp32 caller: c3 down (80 tokens x K = 512) 262 us against 184, c5 gate/up 1305 against 1240.
// GATHER: the activation rows lie in token order.
// NARROW: two issuers (launches of items of up to 64 tokens, GemmArgs::by_chunk). What the others do not use would cost them 1 % (c3 prefill 625 -> 633 us).
template <uint32_t T, int MODE, bool F32_OUT, bool GATHER, int TERMS = 0, bool NARROW = false>
__global__ void __launch_bounds__(g_threads(GATHER), 1) gemm_tc_k(const GemmArgs p, const __grid_constant__ GemmMaps maps) {
    using D = gdec::Dec<T>;
    constexpr bool EXACT = TERMS > 0, TWO = !GATHER && (NARROW || EXACT);            // TWO: two issuers
    static_assert(!NARROW || (!GATHER && !EXACT));
    using X = gdec::Exact<EXACT ? T : uint32_t(T_Q4_K)>;
    static_assert(!EXACT || X::SCRATCH <= D::SCRATCH);
    constexpr int PLANES = EXACT ? TERMS : 1;                          // rows of B per token
    constexpr int CB = chunk_bytes<T>();
    constexpr int ITEM_TILES = MODE == 0 ? 4 : 8;                      // row tiles of one matrix that an item covers
    constexpr int LOAD_WARPS = load_warps(GATHER), EPI_WARP0 = LOAD_WARP0 + LOAD_WARPS, DEC_WARP0 = EPI_WARP0 + EPI_WARPS, G_THREADS = g_threads(GATHER);
    static_assert(EPI_WARP0 % 4 == 0 && DEC_WARP0 % 4 == 0, "warp w reaches the tensor-memory lanes of quarter w % 4");
    extern __shared__ uint8_t smem_raw[];
    // aligned by an offset and not by a cast of the rounded address: that one loses the pointer's address space, and every read of
    // the block's shared memory became a generic load with 64-bit addresses
    uint8_t * smem = smem_raw + (-saddr(smem_raw) & 1023u);
    uint8_t * b_st = smem;                                            // [b_stages][cap][128 bytes], swizzled
    uint8_t * mins_st = b_st + size_t(p.b_stages) * p.cap * 128 * PLANES;       // exact: [A stages][X_CAP][32 bytes], swizzled (only with mins); then the row constants, [x_ring][128]
    float2 * consts = reinterpret_cast<float2 *>(mins_st + (X::MINS ? A_STAGES * X_CAP * 32 : 0));
    uint8_t * raw = mins_st + exact_smem(X::MINS, TERMS);                      // [raw_slots][8 row tiles][CB]
    uint8_t * dec_tab = raw + size_t(8) * p.raw_slots * CB;           // the decoder's lookup table
    uint8_t * dec_scratch = dec_tab + D::TAB_BYTES;                   // [decode warps][SCRATCH]
    Info * info = reinterpret_cast<Info *>(dec_scratch + DEC_WARPS * D::SCRATCH);   // [na + 1]
    int2 * tok = reinterpret_cast<int2 *>(info + p.experts + 2);      // [2][MAX_CAP]: assignment (-1: none) and activation scale of an item's tokens
    uint64_t * bars = reinterpret_cast<uint64_t *>(tok + 2 * MAX_CAP);
    uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(bars + N_BARS);
    volatile int * abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int S = p.raw_slots, BS = p.b_stages;
    const uint32_t raw_full = saddr(bars), raw_empty = raw_full + 16 * RAW_SLOTS, a_full = raw_empty + 8 * RAW_SLOTS,
                   done = a_full + 8 * A_STAGES, b_full = done + 8 * STEP_RING, acc_full = b_full + 8 * MAX_B_STAGES, acc_empty = acc_full + 16,
                   drain = acc_empty + 16, tok_bar = drain + 8;
    // the exact form: as many barriers as sets and chunks of constants, in place of those that it does not need (B stages come through the A stages' barriers)
    constexpr int SETS = x_sets(X::MINS, TERMS), SET_COLS = x_set_cols(X::MINS, TERMS), MINS_COL = X_CAP * TERMS, AMINS = SETS * SET_COLS, CONSTS = x_ring(X::MINS, TERMS);
    static_assert(!EXACT || AMINS + (X::MINS ? 2 * 8 : 0) <= A_COL0, "sets of sums and two operands of mins below the A stages");
    static_assert(CONSTS <= MAX_B_STAGES && SETS <= 4 && CONSTS >= SETS + 2);
    const uint32_t const_full = b_full, set_full = tok_bar + 8, set_empty = acc_full;
    // The warp's number as a shuffle's result: the compiler then knows it, and with it the roles' branches, their loops and addresses, to be the same in the whole warp, and
    // keeps them in uniform registers: fewer instructions in every role, and products issued without moving their operands there one by one.
    // c3 decode 8 73.0 -> 66.9 us, c5 decode 24 308 -> 292 (309 with the issuing branch taken by one lane), c2 509 tokens 351 -> 323, c4 600 745 -> 685
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0);
    const int e1 = p.experts + 1;
    const int * counts = p.plan + PLAN_HDR, * offsets = counts + e1, * perm = offsets + e1 + 1 + e1;
    const int row_tiles = (p.rows + 15) >> 4, row_blocks = (row_tiles + ITEM_TILES - 1) / ITEM_TILES;
    const int ksteps = p.k / G_KS, nchunks = (ksteps + 3) >> 2;             // a last chunk may lack steps: they bring no products, but their barriers turn

    // A thread per barrier; two threads that know the tensor maps will be needed
    if (threadIdx.x < N_BARS) {
        const int i = threadIdx.x;
        int at = 2 * RAW_SLOTS, count = 1;                             // raw_full; then the others in their order
        auto next = [&](int n, int c) { if (i >= at) count = c; at += n; };
        next(RAW_SLOTS, DEC_WARPS / 2);
        next(A_STAGES, p.b_pair ? 8 + (GATHER ? LOAD_WARPS : 1) : 8);
        next(STEP_RING, 1);
        next(MAX_B_STAGES, EXACT ? 8 : GATHER ? LOAD_WARPS : 1);
        next(2, EXACT ? EPI_WARPS : NARROW ? 2 : 1);
        next(2, EPI_WARPS);
        next(1, 1);
        next(1, EPI_WARPS);
        next(4, 1);
        bar_init(saddr(bars) + 8 * i, count);
        bar_init_fence();
    }
    if (threadIdx.x == 64) *abort_flag = 0;
    if (warp == RAW_WARP && lane < (MODE == 0 ? 2 : 1)) prefetch_map(maps.w + lane);
    if (warp == LOAD_WARP0 && lane == 0) prefetch_map(maps.x);
    if (warp == MMA_WARP) tmem_alloc(saddr(tmem_slot), 512);
    // The launch before this one converts the activation rows, and began to let this one in when the plan was complete (rows_begin): only the rows are awaited
    // (grid_wait), by the warps that read them. The plan is looked through, and the first chunks are brought and decoded, meanwhile.
    auto tiles_of = [&](int cnt) { return (cnt + p.cap - 1) >> p.cap_log2; };      // an expert's tokens are spread evenly over the fewest tiles of at most `cap`
    D::init(dec_tab, threadIdx.x, G_THREADS);
    const int na = __shfl_sync(0xffffffffu, find_experts(counts, e1, row_blocks, p.cap_log2, info, tok), 0);    // (the table's first use comes later)
    fence_before();
    __syncthreads();
    fence_after();
    // All 512 columns are this block's, so they begin at column 0 of lane 0. As a constant the base saves the issuing thread an addition and
    // a move into the uniform registers per product: c5 decode 24 gate/up 196.6 -> 194.5 us, down 119 -> 115
    constexpr uint32_t tmem = 0;
    const int n_items = __shfl_sync(0xffffffffu, info[na].cum, 0);

    // item -> expert, first token slot, token count, row block; called by whole warps, with `at` = the active expert of the
    // warp's previous item (items only grow: usually one round of 32 probes)
    struct Item { int e, slot0, nv, rb; };
    auto locate = [&](int it, int & at) {
        while (true) {
            const unsigned m = __ballot_sync(0xffffffffu, at + 1 + lane < na && info[min(at + 1 + lane, na)].cum <= it);
            at += __popc(m);
            if (m != 0xffffffffu) break;
        }
        const Info f = info[at];
        const int nt = tiles_of(f.cnt), local = it - f.cum;
        Item r;
        r.e = f.e;
        int per = (f.cnt + 15) & ~15, tile = 0;
        r.rb = local;
        if (nt > 1) {                                                  // (three divisions: as many instructions as a warp's conversion of half a chunk, in every warp)
            per = ((f.cnt + nt - 1) / nt + 15) & ~15;
            r.rb = local / nt;
            tile = local - r.rb * nt;
        }
        r.slot0 = f.off + tile * per;
        r.nv = __shfl_sync(0xffffffffu, max(0, min(per, f.cnt - tile * per)), 0);      // uniform, for the products' descriptors
        return r;
    };
    auto x_row = [&](int a) { return MODE == 0 ? (a < p.A ? a / p.topk : a - p.A) : a; };
    // the smallest box that holds the item's tokens
    auto b_class = [&](int nv) { return max(nv - 1, 0) >> (EXACT ? 4 : box_log2(p.cap)); };
    const int class_rows = EXACT ? 16 : 1 << box_log2(p.cap);
    // an item that takes both accumulators
    auto takes_both = [&](int nv) { return NARROW || (GATHER && p.by_chunk) ? nv > p.both_above : nv > ACC_COLS; };
    auto give_up = [&]() { *abort_flag = 1; atomicExch(p.plan + PLAN_STATUS, 2); };
    int at = 0;

    if (warp >= EPI_WARP0 && warp < DEC_WARP0) {
        // ---- epilogue: warps q and q + 4 read TMEM lanes [32 q, 32 q + 32) = rows of the block, 16-token groups in turn.
        // What a store needs to know about its token (assignment, activation scale) lies in a table that the warps fill one
        // item ahead, and is read for eight tokens before their stores (the compiler may not move a load over a store that
        // could alias it: one load per store took 100 cycles per token, and two shuffles per token before that 140, which bound
        // every product with a short K: c3 down, 80 tokens x K = 512: 412 us, 255 with the table) ----
        const int q = warp & 3, tid = threadIdx.x - EPI_WARP0 * 32, first = 16 * ((warp - EPI_WARP0) >> 2);
        grid_wait();                                                   // the rows' scales
        const bool upper = lane >= 16;
        constexpr bool ROW_SCALE = T == T_NVFP4G;
        const uint32_t row_bytes = uint32_t(p.rows) * (F32_OUT ? 4u : 2u);
        int2 mine;
        auto fetch = [&](const Item & im) {                            // this thread's token of the item
            mine = make_int2(-1, 0);
            if (tid < im.nv) {
                mine.x = perm[im.slot0 + tid];
                mine.y = __float_as_int(p.inv_scale[GATHER ? x_row(mine.x) : im.slot0 + tid]);
            }
        };
        auto put = [&](uint32_t n) {                                   // the table of the block's n-th item; then a (bounded) meeting of the warps
            tok[(n & 1u) * MAX_CAP + tid] = mine;
            __syncwarp();
            if (lane == 0) bar_arrive(tok_bar);
            return warp_wait(tok_bar, n & 1u);
        };
        uint32_t next = 0, uses0 = 0, uses1 = 0, ic = 0;
        Item im{}, after{};
        bool ok = true;
        if (int(blockIdx.x) < n_items) { im = locate(blockIdx.x, at); fetch(im); ok = put(0); }
#pragma unroll 1
        for (int it = blockIdx.x; it < n_items && ok && !*abort_flag; it += gridDim.x, ++ic, im = after) {
            const bool wide = takes_both(im.nv);
            // sums that an item's K is split into, and the columns from one to the next
            const int parts = !NARROW && im.nv > SPLIT_COLS ? 1 : (NARROW || (GATHER && p.by_chunk)) && (wide || im.nv <= QUARTER_COLS) ? 4 : 2, part_cols = wide || parts == 2 ? SPLIT_COLS : QUARTER_COLS;
            const uint32_t h = wide ? 0 : next;
            next = wide ? 0 : next ^ 1u;
            if (it + int(gridDim.x) < n_items) { after = locate(it + gridDim.x, at); fetch(after); }
            // this lane's weight row: row tiles of a quarter are (gate, up) of the same 16 output rows, or two tiles of the down matrix
            const int row = MODE == 0 ? 16 * (im.rb * 4 + q) + (lane & 15) : 128 * im.rb + 32 * q + lane;
            [[maybe_unused]] float rs = 1.f;                           // fp32 row scale of the bank
            if (ROW_SCALE && row < p.rows) {
                const bool shared = im.e == p.experts;
                const float * ax = MODE == 0 && upper ? (shared ? p.saux1 : p.aux1) : (shared ? p.saux0 : p.aux0);
                rs = ax[size_t(shared ? 0 : im.e) * row_tiles * 16 + row];
            }
            if constexpr (!EXACT) {
                if (!warp_wait(acc_full + 8 * h, (h ? uses1 : uses0) & 1u)) { ok = false; break; }
                if (h) ++uses1; else ++uses0;
                fence_after();
            }
            const uint32_t taddr = tmem + (uint32_t(32 * q) << 16) + h * ACC_COLS;
            const int4 * t = reinterpret_cast<const int4 *>(tok + (ic & 1u) * MAX_CAP);
            char * const out = reinterpret_cast<char *>(static_cast<typename std::conditional<F32_OUT, float, uint16_t>::type *>(p.out) + row);
            const bool in = row < p.rows;
            auto store = [&](int a, float y) {
                if (!in || a < 0) return;
                if constexpr (F32_OUT) *reinterpret_cast<float *>(out + uint64_t(uint32_t(a)) * row_bytes) = y;
                else store_act(out + uint64_t(uint32_t(a)) * row_bytes, p.out_dtype, 0, y);
            };
            if constexpr (EXACT) {
                // the sums of every chunk are scaled by the row's d (and the mins' sums by its dmin) and added in fp32, 8-token groups in turn
                const int g0 = 8 * ((warp - EPI_WARP0) >> 2), lo = 16 * (b_class(im.nv) + 1);       // the second term's columns
                float sum[2][8];
#pragma unroll
                for (int i = 0; i < 16; ++i) sum[i >> 3][i & 7] = 0.f;
#pragma unroll 1
                for (int c = 0; c < nchunks; ++c, ++uses0) {
                    const uint32_t set = uses0 % SETS, at_set = tmem + (uint32_t(32 * q) << 16) + set * SET_COLS;
                    if (!warp_wait(const_full + 8 * (uses0 % CONSTS), (uses0 / CONSTS) & 1u)) { ok = false; break; }
                    float2 k;
                    if constexpr (X::MINS) k = consts[(uses0 % CONSTS) * 128 + 32 * q + lane];
                    else k.x = reinterpret_cast<const float *>(consts)[(uses0 % CONSTS) * 128 + 32 * q + lane];
                    if (!warp_wait(set_full + 8 * set, (uses0 / SETS) & 1u)) { ok = false; break; }
                    fence_after();
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (g0 + 16 * i >= im.nv) break;
                        uint32_t v[8], w[8], z[8];
                        tmem_ld8(at_set + g0 + 16 * i, v);
                        if constexpr (TERMS == 2) tmem_ld8(at_set + lo + g0 + 16 * i, w);
                        if constexpr (X::MINS) tmem_ld8(at_set + MINS_COL + g0 + 16 * i, z);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            float m = __uint_as_float(v[j]);
                            if constexpr (TERMS == 2) m += __uint_as_float(w[j]);
                            sum[i][j] = fmaf(k.x, m, sum[i][j]);
                            if constexpr (X::MINS) sum[i][j] = fmaf(k.y, __uint_as_float(z[j]), sum[i][j]);
                        }
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0) bar_arrive(set_empty + 8 * set);
                }
                if (!ok) break;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int c = g0 + 16 * g;
                    if (c >= im.nv) break;
                    int4 two[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) two[i] = t[c / 2 + i];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float v0 = sum[g][2 * i], v1 = sum[g][2 * i + 1];
                        if (MODE == 0) {
                            const float other = __shfl_xor_sync(0xffffffffu, upper ? v0 : v1, 16);
                            const float is = __int_as_float(upper ? two[i].w : two[i].y);
                            const float gv = (upper ? other : v0) * is, uv = (upper ? v1 : other) * is;
                            store(upper ? two[i].z : two[i].x, gv / (1.f + expf(-gv)) * uv);
                        } else {
                            store(two[i].x, v0 * __int_as_float(two[i].y));
                            store(two[i].z, v1 * __int_as_float(two[i].w));
                        }
                    }
                }
            } else {
#pragma unroll 1
            for (int c = first; c < im.nv; c += 32) {
                uint32_t v[16];
                if ((NARROW || GATHER) && parts == 4) {
                    // the two sums of either issuer first, so that neither's place shows in the result
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        uint32_t w[4][8];
#pragma unroll
                        for (int q4 = 0; q4 < 4; ++q4) tmem_ld8(taddr + q4 * part_cols + c + 8 * i, w[q4]);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            v[8 * i + j] = __float_as_uint((__uint_as_float(w[0][j]) + __uint_as_float(w[1][j])) + (__uint_as_float(w[2][j]) + __uint_as_float(w[3][j])));
                    }
                } else {
                    tmem_ld16(taddr + c, v);
                }
                if (parts == 2) {
                    uint32_t w[16];
                    tmem_ld16(taddr + SPLIT_COLS + c, w);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
                }
                tmem_ld_wait();
#pragma unroll
                for (int j0 = 0; j0 < 16; j0 += 8) {
                    int4 two[4];                                       // tokens j, j + 1: (assignment, scale) each
#pragma unroll
                    for (int i = 0; i < 4; ++i) two[i] = t[(c + j0) / 2 + i];
                    if (MODE == 0) {
                        // lanes l and l + 16 hold gate and up of the same row: they swap, and l finishes the even tokens, l + 16 the odd ones
                        float res[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float v0 = __uint_as_float(v[j0 + 2 * i]), v1 = __uint_as_float(v[j0 + 2 * i + 1]);
                            if (ROW_SCALE) { v0 *= rs; v1 *= rs; }
                            const float other = __shfl_xor_sync(0xffffffffu, upper ? v0 : v1, 16);
                            const float is = __int_as_float(upper ? two[i].w : two[i].y);
                            const float gv = (upper ? other : v0) * is, uv = (upper ? v1 : other) * is;
                            res[i] = __fdividef(gv, 1.f + __expf(-gv)) * uv;      // fast exp and divide: relative error about 2^-21
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) store(upper ? two[i].z : two[i].x, res[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float is0 = __int_as_float(two[i].y), is1 = __int_as_float(two[i].w);
                            store(two[i].x, __uint_as_float(v[j0 + 2 * i]) * (ROW_SCALE ? is0 * rs : is0));
                            store(two[i].z, __uint_as_float(v[j0 + 2 * i + 1]) * (ROW_SCALE ? is1 * rs : is1));
                        }
                    }
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) {
                bar_arrive(acc_empty + 8 * h);
                if (wide) bar_arrive(acc_empty + 8);
            }
            }
            ok = put(ic + 1);                                          // the other table: every warp has left the item that used it
        }
        if (!ok && lane == 0) give_up();
    } else if (warp >= DEC_WARP0) {
        // ---- A decoder: raw chunks (256 columns of one row tile) -> fp16 operand in tensor memory. The warps j < 8 and j >= 8 take
        // the block's chunks in turn, a chunk's two units in the A stages 2 (j >> 3) and the next: what a warp does once per chunk
        // (waits, scales, addresses) took as many instructions as the conversion itself when it took a unit of every chunk.
        // Steps past the end of K and units without steps are decoded from zeros and not multiplied ----
        const int j = warp - DEC_WARP0, q = j & 3, m = (j >> 2) & 1, group = j >> 3, r = 2 * q + m;      // r: row tile of the block
        uint8_t * my_scratch = dec_scratch + j * D::SCRATCH;
        const uint8_t * my_raw = raw + size_t(MODE == 0 ? 4 * m + q : r) * CB;
        const uint32_t a_addr = tmem + (uint32_t(32 * q + 16 * m) << 16) + A_COL0 + 2 * group * A_COLS;
        const uint32_t full = a_full + 16 * group, freed = done + 8 * (4 * group + 1);      // the stages' second steps: their products free them
        // Chunk c lies in slot c % S and is announced by barrier c % 2 S: a ring of S barriers with an odd S would bring a group to every other
        // phase of each, and a phase that two chunks back has completed looks like the one that the group waits for
        uint32_t turn = 0, next = group, phase = 0;                    // chunks of this warp so far; the next one's barrier and its phase
        int pos = group;                                               // the next chunk, in the current item
        bool ok = true;
#pragma unroll 1
        for (int it = blockIdx.x; it < n_items && ok && !*abort_flag; it += gridDim.x, pos -= nchunks) {
#pragma unroll 1
            for (; pos < nchunks; pos += 2, ++turn) {
                const uint32_t slot = next >= uint32_t(S) ? next - S : next;
                const uint8_t * chunk = my_raw + slot * (8 * CB);
                if (!warp_wait(raw_full + 8 * next, phase)) { ok = false; break; }
                using P = typename std::conditional<EXACT, X, D>::type;
                const typename P::Pre pre = P::prep(chunk, lane, my_scratch);
                if (P::SCRATCH) __syncwarp();
                uint32_t f[16];
                // a unit's stage is free; a unit is there (the stores of either step have landed)
                auto stage_free = [&](int u) {
                    if (turn > 0 && !warp_wait(freed + 16 * u, (turn - 1) & 1u)) return false;
                    fence_after();
                    return true;
                };
                auto unit_done = [&](int u) {
                    tmem_st_wait();
                    fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        bar_arrive(full + 8 * u);
                        if (EXACT && u == 0) bar_arrive(const_full + 8 * ((group + 2 * turn) % CONSTS));
                        if (u == 1) bar_arrive(raw_empty + 8 * slot);  // every lane is done with the slot (the syncwarp above)
                    }
                };
                // Rounded operands with scales or look-ups in the way: what a step reads from shared memory is asked for a step ahead, and the stores of the first unit are awaited
                // behind the conversion of a step of the second. Q4_K, 2047 tokens 1033 -> 1024 us a layer (runs of one side 0.4 % apart at most), IQ4, 24 tokens 318 -> 312 (2.6 %);
                // NVFP4, whose conversion has no such chain, no difference. The exact form's sums wait for its units: IQ3_S codes, 509 tokens 357, with a step ahead 362
                constexpr bool AHEAD = !EXACT && T != T_NVFP4G;
                auto first = P::template load<0>(chunk, lane, my_scratch), second = first;
                if constexpr (AHEAD) second = P::template load<1>(chunk, lane, my_scratch);
                P::template step<0>(first, lane, dec_tab, pre, f);
                if (!stage_free(0)) { ok = false; break; }
                tmem_st_16x256b_x4(a_addr, f);
                if constexpr (EXACT) {
                    // the chunk's mins and row constants: what used their places belongs to products that are done, and to chunks whose sums are read (the wait above)
                    if constexpr (X::MINS) {
                        uint32_t mn[4];
                        X::mins(chunk, lane, mn);
                        tmem_st_16x256b_x1(tmem + (uint32_t(32 * q + 16 * m) << 16) + AMINS + 8 * group, mn);
                    }
                    if (lane < 16) {
                        const float2 k = X::consts(chunk, lane);
                        const uint32_t place = ((group + 2 * turn) % CONSTS) * 128 + 32 * q + 16 * m + lane;
                        if constexpr (X::MINS) consts[place] = k;
                        else reinterpret_cast<float *>(consts)[place] = k.x;
                    }
                }
                if constexpr (AHEAD) {
                    if constexpr (T == T_Q4_K) {                        // every lane has read the first unit's constants
                        __syncwarp();
                        P::second_unit(pre, lane, my_scratch);
                        __syncwarp();
                    }
                    first = P::template load<2>(chunk, lane, my_scratch);
                }
                else second = P::template load<1>(chunk, lane, my_scratch);
                P::template step<1>(second, lane, dec_tab, pre, f);
                tmem_st_16x256b_x4(a_addr + A_COLS / 2, f);
                if constexpr (AHEAD) {
                    second = P::template load<3>(chunk, lane, my_scratch);
                } else {
                    unit_done(0);
                    first = P::template load<2>(chunk, lane, my_scratch);
                }
                P::template step<2>(first, lane, dec_tab, pre, f);
                if constexpr (AHEAD) unit_done(0);
                if (!stage_free(1)) { ok = false; break; }
                tmem_st_16x256b_x4(a_addr + A_COLS, f);
                if constexpr (!AHEAD) second = P::template load<3>(chunk, lane, my_scratch);
                P::template step<3>(second, lane, dec_tab, pre, f);
                tmem_st_16x256b_x4(a_addr + A_COLS + A_COLS / 2, f);
                unit_done(1);
                next += 2;
                if (next >= 2 * uint32_t(S)) { next -= 2 * S; phase ^= 1u; }
            }
        }
        if (!ok && lane == 0) give_up();
    } else if (warp == MMA_WARP || (TWO && warp == MMA_WARP1)) {
        // ---- MMA issuers: the whole warp walks the loops, one elected lane issues (a predicate on the instruction, not a branch: in a
        // branch of one lane every operand is moved to the uniform registers first: 43 cycles a product beside busy decoders). What an issue costs decides the pace of
        // narrow items, whose products take the tensor core 16 to 32 cycles each: with its waits, commits and the walk it is 300 to 450 cycles a unit of eight. So those
        // have two issuers, each for the chunks of one group of decoders, in stages, sums and barriers of their own; a gathering launch has the same sums from one. One / two issuers, us a layer: c3 decode 8 66.9 / 65.2, c5 decode 24 309 / 292,
        // c2 509 tokens 323 / 315, c4 600 685 / 666 ----
        const bool lead = elect_one();
        const uint32_t me = TWO && warp == MMA_WARP1 ? 1 : 0;
        const uint32_t b_lo0 = sw128_desc_lo(saddr(b_st)), b_step = uint32_t(p.cap * 128 * PLANES) >> 4;
        uint32_t gu = 0, next = 0, uses0 = 0, uses1 = 0;
        bool ok = true;
#pragma unroll 1
        for (int it = blockIdx.x; it < n_items && ok; it += gridDim.x) {
            const Item im = locate(it, at);
            const bool wide = takes_both(im.nv);
            const uint32_t h = wide ? 0 : next;
            next = wide ? 0 : next ^ 1u;
            const uint32_t npad = uint32_t(max(im.nv, 1) + 15) & ~15u, id = idesc(128, npad * PLANES, 0), d = tmem + h * ACC_COLS;
            if constexpr (!EXACT) {
            if (wide || h == 0) { if (uses0 > 0) ok = warp_wait(acc_empty, (uses0 - 1) & 1u) && ok; ++uses0; }
            if (wide || h == 1) { if (uses1 > 0) ok = warp_wait(acc_empty + 8, (uses1 - 1) & 1u) && ok; ++uses1; }
            fence_after();
            }
            // from the first to the second step of a unit: with b_pair one box holds both; else B stages in turn
            const uint32_t b_unit = !GATHER ? uint32_t(b_class(im.nv) + 1) * (uint32_t(class_rows * 128 * PLANES) >> 4) : b_step;
            // this issuer's chunks of the item
            auto chunks = [&](auto ME) {
                constexpr uint32_t s0 = 2 * decltype(ME)::value;
                const uint32_t c0 = gu >> 1, part_cols = wide ? SPLIT_COLS : QUARTER_COLS, d0 = d + decltype(ME)::value * 2 * part_cols, d1 = wide || im.nv <= QUARTER_COLS ? d0 + part_cols : d0;
                uint32_t acc = 0;
#pragma unroll 1
                for (uint32_t c = c0 + ((c0 ^ decltype(ME)::value) & 1u); c < c0 + uint32_t(nchunks); c += 2) {
                    const uint32_t turn = c >> 1;
                    const int left = ksteps - 4 * int(c - c0);
                    const uint32_t set = c % SETS;
                    if constexpr (EXACT) { if (c >= uint32_t(SETS) && !warp_wait(set_empty + 8 * set, (c / SETS - 1) & 1u)) return false; }
#pragma unroll
                    for (uint32_t u = 0; u < 2; ++u) {
                        const uint32_t s = s0 + u, a = tmem + A_COL0 + s * A_COLS, b = b_lo0 + 2 * s * b_step;
                        if (!warp_wait(a_full + 8 * s, turn & 1u)) return false;
                        fence_after();
                        if constexpr (EXACT) {
                            const uint32_t ds = tmem + set * SET_COLS;
                            mma_step(lead, ds, ds, a, b, id, u, 1);
                            mma_step(lead, ds, ds, a + A_COLS / 2, b + b_unit, id, 1, 1);
                            if constexpr (X::MINS)
                                if (u == 0) mma_f16<SW32_DESC_HI>(lead, ds + MINS_COL, tmem + AMINS + 8 * decltype(ME)::value, sw128_desc_lo(saddr(mins_st) + s * (X_CAP * 32)), idesc(128, npad, 0), 0);
                        } else {
                            if (left > 2 * int(u)) mma_step(lead, d0, d1, a, b, id, acc, acc | uint32_t(d1 == d0));
                            if (left > 2 * int(u) + 1) mma_step(lead, d0, d1, a + A_COLS / 2, b + b_unit, id, 1, 1);
                            acc = 1;
                        }
                        mma_commit(lead, done + 16 * s + 8);
                    }
                    if constexpr (EXACT) mma_commit(lead, set_full + 8 * set);
                }
                if constexpr (!EXACT) mma_commit(lead, acc_full + 8 * h);
                return true;
            };
            auto products = [&](auto PAIR) {
                const bool by_chunk = GATHER && p.by_chunk && im.nv <= SPLIT_COLS;      // (rows in slot order: chunks())
                const uint32_t half = wide ? ACC_COLS : SPLIT_COLS;      // by_chunk: columns from the sums of one group's chunks to those of the other's
                const uint32_t second = im.nv > SPLIT_COLS ? 0 : !by_chunk || wide ? SPLIT_COLS : im.nv <= QUARTER_COLS ? QUARTER_COLS : 0;      // columns from the accumulator of even products to that of odd ones
                const uint32_t b_half = PAIR && !GATHER ? b_unit : b_step;
                uint32_t first = gu % A_STAGES, turn = gu / A_STAGES;
                int left = ksteps, units = 2 * nchunks;
#pragma unroll 1
                while (true) {
#pragma unroll
                    for (uint32_t s = 0; s < A_STAGES; ++s) {
                        if (s < first) continue;                       // an item's units begin at any stage
                        const uint32_t a = tmem + A_COL0 + s * A_COLS, sb = PAIR ? 2 * s : 2 * (s & 1), b = b_lo0 + sb * b_step;
                        if (!warp_wait(a_full + 8 * s, turn & 1u)) return false;
                        if (!PAIR && !warp_wait(b_full + 8 * sb, (2 * turn + (s >> 1)) & 1u)) return false;      // with b_pair a_full stands for the unit's rows too
                        if constexpr (EXACT) {                         // a chunk's units are the stages 0, 1 or 2, 3, its sums a set of their own
                            const uint32_t c = 2 * turn + (s >> 1), set = c % SETS, ds = tmem + set * SET_COLS;
                            if ((s & 1) == 0 && c >= uint32_t(SETS) && !warp_wait(set_empty + 8 * set, (c / SETS - 1) & 1u)) return false;
                            fence_after();
                            mma_step(lead, ds, ds, a, b, id, s & 1, 1);
                            mma_step(lead, ds, ds, a + A_COLS / 2, b + b_half, id, 1, 1);
                            if constexpr (X::MINS)
                                if ((s & 1) == 0)
                                    mma_f16<SW32_DESC_HI>(lead, ds + MINS_COL, tmem + AMINS + 8 * (s >> 1), sw128_desc_lo(saddr(mins_st) + s * (X_CAP * 32)), idesc(128, npad, 0), 0);
                            mma_commit(lead, done + 16 * s + 8);
                            if (s & 1) mma_commit(lead, set_full + 8 * set);
                            if (--units == 0) return true;
                            continue;
                        }
                        fence_after();
                        const uint32_t dh = by_chunk ? d + (s >> 1) * half : d;
                        const uint32_t acc = left != ksteps && !(by_chunk && left == ksteps - 4);      // the first unit of an item, or of either half, overwrites
                        if (left > 0) mma_step(lead, dh, dh + second, a, b, id, acc, acc | (second == 0));
                        if constexpr (!PAIR) {
                            mma_commit(lead, done + 16 * s);
                            if (!warp_wait(b_full + 8 * (sb + 1), (2 * turn + (s >> 1)) & 1u)) return false;
                            fence_after();
                        }
                        if (left > 1) mma_step(lead, dh, dh + second, a + A_COLS / 2, b + b_half, id, 1, 1);
                        mma_commit(lead, done + 16 * s + 8);
                        left -= 2;
                        if (--units == 0) { mma_commit(lead, acc_full + 8 * h); return true; }
                    }
                    first = 0;
                    ++turn;
                }
            };
            if constexpr (TWO) ok = ok && (me ? chunks(std::integral_constant<uint32_t, 1>{}) : chunks(std::integral_constant<uint32_t, 0>{}));
            else if constexpr (EXACT) ok = ok && products(std::true_type{});
            else ok = ok && (p.b_pair ? products(std::true_type{}) : products(std::false_type{}));
            gu += 2 * nchunks;
        }
        if (!ok && lane == 0) give_up();
        // nothing may be in flight when the tensor memory is freed (after a clean run the epilogue has waited for all of it)
        const uint32_t mine = me ? done : drain;                       // (no step that is the first of a unit has a barrier where there are two issuers)
        mma_commit(lead, mine);
        warp_wait(mine, 0);
    } else if (warp == RAW_WARP) {
        // ---- raw blocks ----
        constexpr int PARTS = chunk_parts<T>();
        constexpr uint32_t BYTES = 8 * CB;
        // Launches of narrow items, and the exact form at every density (first_out_policy); with items of 128 and 256 tokens it costs (c5 prefill 2751 -> 2795 us)
        constexpr bool FIRST_OUT = NARROW || EXACT;
        [[maybe_unused]] const uint64_t policy = FIRST_OUT ? first_out_policy() : 0;
        uint32_t issued = 0, slot = 0, phase = 1;                      // phase: of the empty barrier's wait (none in the first round)
        bool ok = true;
#pragma unroll 1
        for (int it = blockIdx.x; it < n_items && ok && !*abort_flag; it += gridDim.x) {
            const Item im = locate(it, at);
            const CUtensorMap * map = maps.w + (im.e == p.experts ? 2 : 0);
            const int rt = (im.e == p.experts ? 0 : im.e * row_tiles) + im.rb * ITEM_TILES;        // rows past the matrix: the next expert's, never used
#pragma unroll 1
            for (int c = 0; c < nchunks; ++c) {
                if (issued >= uint32_t(S) && !warp_wait(raw_empty + 8 * slot, phase)) { ok = false; break; }
                if (elect_one()) {
                    const uint32_t bar = raw_full + 8 * (issued % (2 * uint32_t(S))), dst = saddr(raw) + slot * BYTES;
                    bar_expect_tx(bar, BYTES);
                    if constexpr (FIRST_OUT) {
                        tma_load_3d_first_out(dst, map, 0, c * PARTS, rt, bar, policy);
                        if (MODE == 0) tma_load_3d_first_out(dst + BYTES / 2, map + 1, 0, c * PARTS, rt, bar, policy);
                    } else {
                        tma_load_3d(dst, map, 0, c * PARTS, rt, bar);
                        if (MODE == 0) tma_load_3d(dst + BYTES / 2, map + 1, 0, c * PARTS, rt, bar);
                    }
                }
                __syncwarp();
                ++issued;
                if (++slot == uint32_t(S)) { slot = 0; phase ^= 1u; }
            }
        }
        if (!ok && lane == 0) give_up();
        // before leaving, every copy must have landed (after a clean run these waits return at once)
#pragma unroll 1
        for (uint32_t i = issued > uint32_t(S) ? issued - S : 0; i < issued; ++i) bar_wait(raw_full + 8 * (i % (2 * uint32_t(S))), (i / (2 * uint32_t(S))) & 1u);
    } else {
        // ---- B loader: warp 2 brings a step's (or a unit's) rows with one box; a gathering launch: lane l of loader w brings rows
        // 4 (6 l + w) .. + 3. Issuing sets the pace of a gather (90 to 120 cycles per four rows and warp), so it takes
        // all the threads that a block may have, with 64 registers. With two loaders / with six / from slot order, us: NVFP4 of 2048 columns, 10 tokens per
        // expert 260 / 252 / 228, 80: 571 / 375 / 309; IQ4 of 4096 columns, 512: 3680 / 2050 / 1415; Q4_K of 3072 columns, 64: 1050 / 788 / 653 ----
        const int lw = warp - LOAD_WARP0, n0 = 4 * (LOAD_WARPS * lane + lw), group = p.b_pair ? 2 : 1;      // steps that share a barrier
        uint32_t gk = 0, sb = 0;
        bool ok = true;
        grid_wait();                                                   // the rows
#pragma unroll 1
        for (int it = blockIdx.x; it < n_items && ok && !*abort_flag && (lw == 0 || GATHER); it += gridDim.x) {
            const Item im = locate(it, at);
            int row[4] = {0, 0, 0, 0};
            if constexpr (GATHER) {
#pragma unroll
                for (int i = 0; i < 4; ++i) row[i] = n0 < im.nv ? x_row(perm[im.slot0 + min(n0 + i, im.nv - 1)]) : 0;      // past the last token: repeat it (dead columns of D)
            }
            const int cls = b_class(im.nv), quads = (im.nv + 3) >> 2, mine = (quads + LOAD_WARPS - 1 - lw) / LOAD_WARPS;
            const uint32_t box_bytes = uint32_t((cls + 1) * class_rows * group * PLANES) * 128u;
#pragma unroll 1
            for (int ks = 0; ks < 4 * nchunks; ks += group, gk += group) {
                const uint32_t freed = gk + group - 1 - uint32_t(BS);  // the (last) step that used the stage before
                if (gk >= uint32_t(BS) && !warp_wait(done + 8 * (freed % STEP_RING), (freed / STEP_RING) & 1u)) { ok = false; break; }
                const uint32_t bar = p.b_pair ? a_full + 4 * sb : b_full + 8 * sb, dst = saddr(b_st) + sb * uint32_t(p.cap * 128 * PLANES);
                if constexpr (EXACT && !GATHER) {
                    if (elect_one()) {
                        const bool mins = X::MINS && (ks & 2) == 0;    // a chunk's first unit brings the tokens' sub-block sums too
                        bar_expect_tx(bar, box_bytes + (mins ? uint32_t((cls + 1) * 16 * 32) : 0u));
                        tma_load_4d(dst, maps.x + cls, 0, im.slot0, 0, ks, bar);
                        if (mins) tma_load_3d(saddr(mins_st) + (sb >> 1) * (X_CAP * 32), maps.x + 2 + cls, 0, im.slot0, ks >> 2, bar);
                    }
                    __syncwarp();
                } else if constexpr (!GATHER) {
                    if (elect_one()) {
                        bar_expect_tx(bar, box_bytes);
                        tma_load_3d(dst, maps.x + cls, 0, im.slot0, ks, bar);      // steps past K lie outside: zeros
                    }
                    __syncwarp();
                } else {
                    const int real = min(group, ksteps - ks);
                    const bool mins = EXACT && X::MINS && (ks & 2) == 0;
                    if (lane == 0) bar_expect_tx(bar, uint32_t(max(real, 0) * mine) * 512u + (mins ? uint32_t(mine) * 128u : 0u));
                    __syncwarp();
                    if (mins && n0 < im.nv) tma_gather4(saddr(mins_st) + (sb >> 1) * (X_CAP * 32) + n0 * 32, maps.x + 2, ks * 4, row[0], row[1], row[2], row[3], bar);
                    if (n0 < im.nv)
#pragma unroll 1
                        for (int i = 0; i < real; ++i)
                            tma_gather4(dst + i * uint32_t(p.cap * 128) + n0 * 128, maps.x, (ks + i) * G_KS, row[0], row[1], row[2], row[3], bar);
                }
                sb += group;
                if (sb == uint32_t(BS)) sb = 0;
            }
        }
        if (!ok && lane == 0) give_up();
        // before leaving, every copy into the stages must have landed (after a clean run these waits return at once)
        // (b_pair: the products that read the last stages have been waited for by the MMA warp, or the unit's barrier is waited for here)
#pragma unroll 1
        for (uint32_t g = gk > uint32_t(BS) ? gk - BS : 0; g < gk; g += group) bar_wait(p.b_pair ? a_full + 4 * (g % BS) : b_full + 8 * (g % BS), (g / BS) & 1u);
    }
    grid_wait();                                                       // every thread, so that a launch that waits for this one has waited for those before it
    grid_release();
    fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_free(tmem, 512);
}

int gemm_sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms;
}
constexpr size_t GEMM_SMEM_LIMIT = 232448 - 1024;

// shared-memory split of a launch: the widest items wanted first, then narrower ones (their B stages are smaller) until the raw
// ring holds at least three chunks
int g_item_tokens = 0;                      // test hook: 256 = 256-token items whatever the batch
template <uint32_t T> bool gemm_fit(int experts, int cap_wanted, GemmArgs & a) {
    constexpr int opts[4][3] = {{256, 4, 3}, {128, 8, 3}, {64, 8, 3}, {64, 8, 2}};      // tokens per item, B stages, fewest raw slots
    for (const auto & o : opts) {
        if (o[0] > cap_wanted) continue;
        for (int s = RAW_SLOTS; s >= o[2]; --s)
            if (gemm_smem<T>(experts, o[0], o[1], s) <= GEMM_SMEM_LIMIT) {
                a.cap = o[0]; a.cap_log2 = o[0] == 256 ? 8 : o[0] == 128 ? 7 : 6; a.b_stages = o[1]; a.raw_slots = s;
                a.b_pair = o[1] == 2 * A_STAGES;
                a.by_chunk = a.cap <= SPLIT_COLS && ceil_div(a.k, 256) % 2 == 0;
                a.both_above = a.k % 256 ? QUARTER_COLS : SPLIT_COLS;
                return true;
            }
    }
    return false;
}
// `rows` fp16 activation rows of length k as [k / 64][rows][64]: a box is box_rows rows of `steps` 64-column steps, one step after the other
bool rows_map(CUtensorMap & m, const void * xb, int rows, int k, int box_rows, int steps) {
    const cuuint64_t dims[3] = {G_KS, cuuint64_t(rows), cuuint64_t(k / G_KS)}, strides[2] = {cuuint64_t(k) * 2, G_KS * 2};
    const cuuint32_t box[3] = {G_KS, cuuint32_t(box_rows), cuuint32_t(steps)};
    return encode_map(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, xb, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}
// the same rows for tile::gather4
bool gather_map(CUtensorMap & m, const void * xb, int rows, int k) {
    const cuuint64_t dims[2] = {cuuint64_t(k), cuuint64_t(rows)}, strides[1] = {cuuint64_t(k) * 2};
    const cuuint32_t box[2] = {G_KS, 1};
    return encode_map(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, xb, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}
// the exact form's sub-block sums for tile::gather4: rows of k / 16 values, sixteen a chunk
bool gather_mins_map(CUtensorMap & m, const void * mins, int rows, int k) {
    const cuuint64_t dims[2] = {cuuint64_t(k / 16), cuuint64_t(rows)}, strides[1] = {cuuint64_t(k) / 8};
    const cuuint32_t box[2] = {16, 1};
    return encode_map(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, mins, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_32B);
}
// the exact form's rows as [k / 64][TERMS][rows][64], boxes of two steps, and its sub-block sums as [k / 256][rows][16]
bool exact_rows_map(CUtensorMap & m, const void * xb, int rows, int k, int box_rows, int terms) {
    const cuuint64_t dims[4] = {G_KS, cuuint64_t(rows), cuuint64_t(terms), cuuint64_t(k / G_KS)}, strides[3] = {cuuint64_t(k) * 2, cuuint64_t(rows) * k * 2, G_KS * 2};
    const cuuint32_t box[4] = {G_KS, cuuint32_t(box_rows), cuuint32_t(terms), 2};
    return encode_map(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, xb, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}
bool mins_map(CUtensorMap & m, const void * mins, int rows, int k, int box_rows) {
    const cuuint64_t dims[3] = {16, cuuint64_t(rows), cuuint64_t(k / 256)}, strides[2] = {cuuint64_t(k) / 8, 32};
    const cuuint32_t box[3] = {16, cuuint32_t(box_rows), 1};
    return encode_map(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, mins, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_32B);
}
// a bank's tiles as [experts * row tiles][parts of a chunk][8-byte words]: a box is one 256-column chunk of `tiles` consecutive row tiles
template <uint32_t T> bool bank_map(CUtensorMap & m, const b2moe_bank * b, int tiles) {
    constexpr int PW = part_words<T>();
    const cuuint64_t line = cuuint64_t(b->cols / Fmt<T>::KT) * Fmt<T>::TILE;       // bytes of a row tile
    const cuuint64_t dims[3] = {cuuint64_t(PW), line / (PW * 8), cuuint64_t(b->experts) * ((b->rows + 15) / 16)}, strides[2] = {PW * 8, line};
    const cuuint32_t box[3] = {PW, chunk_parts<T>(), cuuint32_t(tiles)};
    return encode_map(m, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, b->data, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}
// From this many slots on, the rows of a batch are converted once per token (two launches), below once per slot (one)
constexpr int TOKEN_WISE_SLOTS = 4096;
template <uint32_t T, int DT>
int32_t convert_rows_dt(const void * xv, int rows_x, int slot_rows, bool slots, int topk, const GemmArgs & a, __half * out, float * inv, int * slot_of, bool plan_ready, cudaStream_t s) {
    const auto * x = static_cast<const typename Elem<DT>::type *>(xv);
    const int * plan = a.plan;
    const dim3 block(256);
    if (!slots) {
        launch_overlapped(rows_to_f16_k<T, DT>, dim3(ceil_div(rows_x, 8)), block, 0, s, x, rows_x, a.k, out, inv);
    } else if (slot_of && topk > 1 && topk < 32 && slot_rows >= TOKEN_WISE_SLOTS) {
        launch_overlapped(slot_of_k, dim3(ceil_div(slot_rows, 256)), block, 0, s, plan, a.experts, slot_of);
        if (int32_t rc = launch_status()) return rc;
        launch_overlapped(tokens_to_slots_k<T, DT>, dim3(ceil_div(rows_x, 8)), block, 0, s, x, plan, slot_of, a.experts, rows_x, topk, int(slot_rows > a.A), a.k, out, inv);
    } else {
        launch_overlapped(rows_to_slots_k<T, DT>, dim3(ceil_div(slot_rows, 8)), block, 0, s, x, plan, a.experts, a.A, topk, a.k, out, inv, !plan_ready);
    }
    return launch_status();
}
// m: the banks (gate, up) or (down, null), then the shared expert's (null: none); x (rows_x rows, in token order when map_topk > 0, in
// assignment order otherwise), live: how many of the a.A assignments are expected to be grouped -> fp16 rows in xb (in slot order: slot_rows of them; slot_of: scratch for MODE 0), then the product
template <uint32_t T, int MODE>
int32_t gemm_launch_t(GemmArgs a, long long live, const b2moe_bank * const * m, const void * x, int dtype, int rows_x, int map_topk, bool slots, int slot_rows, __half * xb, float * inv, int * slot_of,
                      bool plan_ready, cudaStream_t s) {
    const int sms = gemm_sm_count();
    if (sms <= 0) return B2MOE_ERR_CUDA;
    const long long per = live / a.experts;                           // mean tokens per expert
    // The width of the items. Gate/up with items of 64 / 128 / 256 tokens, us: NVFP4 (512 experts) 24 per expert 235 / 235 / 279, 64: 342 / 265 / 315,
    // 112: 488 / 339 / 374, 144: 674 / 553 / 464; IQ4 (128 experts) 24: 317 / 317 / 366, 64: 496 / 388 / 431, 112: 702 / 469 / 486, 144: 998 / 800 / 585; Q4_K (256
    // experts) 24: 651 / 652 / 646, 64: 978 / 711 / 718, 112: 1385 / 908 / 881, 144: 1932 / 1427 / 993. The narrow ones leave room for more raw slots.
    const int cap = g_item_tokens == 256 || per > 128 ? 256 : per > 24 ? 128 : 64;
    if (!gemm_fit<T>(a.experts, cap, a)) return B2MOE_ERR_SHAPE;
    const int rows = slots ? slot_rows : rows_x, topk = map_topk;
    int32_t rc = B2MOE_ERR_SHAPE;
    if (dtype == B2MOE_F32) rc = convert_rows_dt<T, B2MOE_F32>(x, rows_x, slot_rows, slots, topk, a, xb, inv, slot_of, plan_ready, s);
    else if (dtype == B2MOE_F16) rc = convert_rows_dt<T, B2MOE_F16>(x, rows_x, slot_rows, slots, topk, a, xb, inv, slot_of, plan_ready, s);
    else if (dtype == B2MOE_BF16) rc = convert_rows_dt<T, B2MOE_BF16>(x, rows_x, slot_rows, slots, topk, a, xb, inv, slot_of, plan_ready, s);
    if (rc) return rc;
    a.inv_scale = inv;
    GemmMaps maps;
    bool mapped = true;
    if (slots) for (int i = 0; i < a.cap >> box_log2(a.cap); ++i) mapped = mapped && rows_map(maps.x[i], xb, rows, a.k, (i + 1) << box_log2(a.cap), a.b_pair ? 2 : 1);
    else mapped = gather_map(maps.x[0], xb, rows, a.k);
    for (int i = 0; i < 4; ++i)
        if (m[i]) mapped = mapped && bank_map<T>(maps.w[i], m[i], MODE == 0 ? 4 : 8);
    if (!mapped) return B2MOE_ERR_CUDA;
    const size_t smem = gemm_smem<T>(a.experts, a.cap, a.b_stages, a.raw_slots);
    auto kernel = a.by_chunk ? (a.out_dtype == B2MOE_F32 ? gemm_tc_k<T, MODE, true, false, 0, true> : gemm_tc_k<T, MODE, false, false, 0, true>)
                             : a.out_dtype == B2MOE_F32 ? gemm_tc_k<T, MODE, true, false> : gemm_tc_k<T, MODE, false, false>;
    if constexpr (MODE == 0)
        if (!slots) {
            if (a.out_dtype != B2MOE_F32) return B2MOE_ERR_SHAPE;      // calls with 16-bit results bring scratch for the rows in slot order
            kernel = gemm_tc_k<T, MODE, true, true>;
        }
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return B2MOE_ERR_CUDA;
    launch_overlapped(kernel, dim3(sms), dim3(g_threads(!slots)), smem, s, a, maps);
    return launch_status();
}
// The exact form: x (a row per token when topk > 0, per assignment otherwise) -> rows in slot order in `rows` (or, gathered: in their own order), then the product
template <uint32_t T> bool exact_fit(int experts, int terms, GemmArgs & a) {
    a.cap = X_CAP; a.cap_log2 = 5; a.b_stages = 2 * A_STAGES; a.b_pair = 1;
    static_assert(X_CAP == 1 << 5);
    for (a.raw_slots = RAW_SLOTS; a.raw_slots >= 3; --a.raw_slots)
        if (gemm_smem<T>(experts, X_CAP, a.b_stages, a.raw_slots, terms) <= GEMM_SMEM_LIMIT) return true;
    return false;
}
size_t exact_rows_bytes(int slot_rows, int k, int terms) { return align_up(size_t(slot_rows) * (size_t(k) * 2 * terms + k / 8), 256); }
template <uint32_t T, int MODE, int DT>
int32_t exact_launch_t(GemmArgs a, const b2moe_bank * const * m, const void * x, int topk, int slot_rows, bool slots, void * rows, bool plan_ready, cudaStream_t s) {
    constexpr int TERMS = DT == B2MOE_F32 ? 2 : 1;
    const int sms = gemm_sm_count();
    if (sms <= 0) return B2MOE_ERR_CUDA;
    if (!exact_fit<T>(a.experts, TERMS, a)) return B2MOE_ERR_SHAPE;
    __half * xb = static_cast<__half *>(rows), * mins = xb + size_t(slot_rows) * a.k * TERMS;
    float * inv = reinterpret_cast<float *>(static_cast<uint8_t *>(rows) + exact_rows_bytes(slot_rows, a.k, TERMS));
    launch_overlapped(exact_rows_k<T, DT, TERMS>, dim3(ceil_div(slot_rows, 8)), dim3(256), 0, s, static_cast<const typename Elem<DT>::type *>(x), static_cast<const int *>(slots ? a.plan : nullptr), a.experts, slots ? a.A : slot_rows, topk,
                      a.k, xb, size_t(slot_rows) * a.k, mins, inv, !plan_ready);
    if (int32_t rc = launch_status()) return rc;
    a.inv_scale = inv;
    GemmMaps maps;
    bool mapped = true;
    if (!slots) {
        mapped = gather_map(maps.x[0], xb, slot_rows, a.k);
        if (gdec::Exact<T>::MINS) mapped = mapped && gather_mins_map(maps.x[2], mins, slot_rows, a.k);
    } else for (int i = 0; i < 2; ++i) {
        mapped = mapped && exact_rows_map(maps.x[i], xb, slot_rows, a.k, 16 * (i + 1), TERMS);
        if (gdec::Exact<T>::MINS) mapped = mapped && mins_map(maps.x[2 + i], mins, slot_rows, a.k, 16 * (i + 1));
    }
    for (int i = 0; i < 4; ++i)
        if (m[i]) mapped = mapped && bank_map<T>(maps.w[i], m[i], MODE == 0 ? 4 : 8);
    if (!mapped) return B2MOE_ERR_CUDA;
    const size_t smem = gemm_smem<T>(a.experts, a.cap, a.b_stages, a.raw_slots, TERMS);
    auto kernel = a.out_dtype == B2MOE_F32 ? gemm_tc_k<T, MODE, true, false, TERMS> : gemm_tc_k<T, MODE, false, false, TERMS>;
    if (!slots) {
        if constexpr (MODE == 0 && TERMS == 1) {
            if (a.out_dtype != B2MOE_F32) return B2MOE_ERR_SHAPE;
            kernel = gemm_tc_k<T, MODE, true, true, TERMS>;
        } else {
            return B2MOE_ERR_SHAPE;
        }
    }
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return B2MOE_ERR_CUDA;
    launch_overlapped(kernel, dim3(sms), dim3(g_threads(!slots)), smem, s, a, maps);
    return launch_status();
}
template <int MODE>
int32_t exact_launch(uint32_t type, const GemmArgs & a, const b2moe_bank * const * m, const void * x, int dtype, int topk, int slot_rows, bool slots, void * rows, bool plan_ready, cudaStream_t s) {
    if (type == T_Q4_K) return dtype == B2MOE_F32 ? exact_launch_t<T_Q4_K, MODE, B2MOE_F32>(a, m, x, topk, slot_rows, slots, rows, plan_ready, s)
                             : dtype == B2MOE_F16 ? exact_launch_t<T_Q4_K, MODE, B2MOE_F16>(a, m, x, topk, slot_rows, slots, rows, plan_ready, s)
                                                  : exact_launch_t<T_Q4_K, MODE, B2MOE_BF16>(a, m, x, topk, slot_rows, slots, rows, plan_ready, s);
    if (type == T_IQ3S4) return dtype == B2MOE_F32 ? exact_launch_t<T_IQ3S4, MODE, B2MOE_F32>(a, m, x, topk, slot_rows, slots, rows, plan_ready, s)
                              : dtype == B2MOE_F16 ? exact_launch_t<T_IQ3S4, MODE, B2MOE_F16>(a, m, x, topk, slot_rows, slots, rows, plan_ready, s)
                                                   : exact_launch_t<T_IQ3S4, MODE, B2MOE_BF16>(a, m, x, topk, slot_rows, slots, rows, plan_ready, s);
    return B2MOE_ERR_FORMAT;
}
template <int MODE, typename... Args>
int32_t gemm_launch(uint32_t type, const Args &... args) {
    switch (type) {
        case T_Q4_K: return gemm_launch_t<T_Q4_K, MODE>(args...);
        case T_IQ3_S: return gemm_launch_t<T_IQ3_S, MODE>(args...);
        case T_IQ3S4: return gemm_launch_t<T_IQ3S4, MODE>(args...);
        case T_IQ4_XS: return gemm_launch_t<T_IQ4_XS, MODE>(args...);
        case T_IQ4_NL: return gemm_launch_t<T_IQ4_NL, MODE>(args...);
        case T_NVFP4G: return gemm_launch_t<T_NVFP4G, MODE>(args...);
    }
    return B2MOE_ERR_FORMAT;
}
bool gemm_fits(uint32_t type, int experts, int cap, GemmArgs & a) {
    switch (type) {
        case T_Q4_K: return gemm_fit<T_Q4_K>(experts, cap, a);
        case T_IQ3_S: return gemm_fit<T_IQ3_S>(experts, cap, a);
        case T_IQ3S4: return gemm_fit<T_IQ3S4>(experts, cap, a);
        case T_IQ4_XS: return gemm_fit<T_IQ4_XS>(experts, cap, a);
        case T_IQ4_NL: return gemm_fit<T_IQ4_NL>(experts, cap, a);
        case T_NVFP4G: return gemm_fit<T_NVFP4G>(experts, cap, a);
    }
    return false;
}

}  // namespace

void gemm_tc_item_tokens(int tokens) { g_item_tokens = tokens; }
// true when the tensor-core GEMM takes banks of this type with rows of length k
bool gemm_tc_supported(uint32_t type, int k, int experts) {
    GemmArgs a{};
    return k >= G_KS && k % G_KS == 0 && gemm_fits(type, experts, 64, a);
}
// scratch: the scaled fp16 copy of `rows_x` activation rows of length k and one float per row
size_t gemm_tc_workspace_bytes(int rows_x, int k) {
    return align_up(size_t(rows_x) * k * 2, 256) + align_up(size_t(rows_x) * sizeof(float), 256);
}
// the same for rows in slot order that come from token rows: an index per row in addition
size_t gemm_tc_slot_bytes(int slot_rows, int k) { return gemm_tc_workspace_bytes(slot_rows, k) + size_t(slot_rows) * sizeof(int); }

// The exact form takes Q4_K banks and IQ3_S codes; its scratch: the rows in slot order (two terms a value for fp32 rows), their
// sub-block sums and scales. slots = false: gate/up on 16-bit rows with fp32 results from a scratch for the n rows of the tokens
bool gemm_exact_supported(uint32_t type, int k, int experts) {
    GemmArgs a{};
    return k > 0 && k % 256 == 0 && (type == T_Q4_K ? exact_fit<T_Q4_K>(experts, 2, a) : type == T_IQ3S4 && exact_fit<T_IQ3S4>(experts, 2, a));
}
int32_t gemm_tc_fit(uint32_t type, int experts, int item_tokens) {
    GemmArgs a{};
    const bool fits = item_tokens != X_CAP ? gemm_fits(type, experts, item_tokens, a) : type == T_Q4_K ? exact_fit<T_Q4_K>(experts, 2, a) : type == T_IQ3S4 && exact_fit<T_IQ3S4>(experts, 2, a);
    return fits ? 16 * a.cap + a.raw_slots : 0;
}
size_t gemm_exact_bytes(int slot_rows, int k, int dtype) { return exact_rows_bytes(slot_rows, k, dtype == B2MOE_F32 ? 2 : 1) + size_t(slot_rows) * sizeof(float); }
int32_t gemm_exact_gateup(const b2moe_bank * gate, const b2moe_bank * up, const b2moe_bank * sg, const b2moe_bank * su, const void * x, int x_dtype,
                          const int * plan, int n, int topk, int shared_tokens, void * act, int act_dtype, void * rows, bool slots, cudaStream_t s) {
    GemmArgs a{};
    const b2moe_bank * banks[4] = {gate, up, shared_tokens ? sg : nullptr, shared_tokens ? su : nullptr};
    a.plan = const_cast<int *>(plan); a.out = act; a.out_dtype = act_dtype;
    a.rows = gate->rows; a.k = gate->cols; a.experts = gate->experts; a.topk = topk; a.A = n * topk;
    return exact_launch<0>(gate->type, a, banks, x, x_dtype, topk, slots ? n * topk + shared_tokens : n, slots, rows, false, s);
}
int32_t gemm_exact_down(const b2moe_bank * down, const b2moe_bank * sd, const void * x, int x_dtype, bool per_token, const int * plan, int n, int topk,
                        int shared_tokens, void * y, int y_dtype, void * rows, bool plan_ready, cudaStream_t s) {
    GemmArgs a{};
    const b2moe_bank * banks[4] = {down, nullptr, shared_tokens ? sd : nullptr, nullptr};
    a.plan = const_cast<int *>(plan); a.out = y; a.out_dtype = y_dtype;
    a.rows = down->rows; a.k = down->cols; a.experts = down->experts; a.topk = topk; a.A = n * topk;
    return exact_launch<1>(down->type, a, banks, x, x_dtype, per_token ? topk : 0, n * topk + shared_tokens, true, rows, plan_ready, s);
}

// rows_buf: optional scratch for the activation rows in slot order (n * topk + shared_tokens rows of length k, their scales and an index each)
int32_t gemm_tc_gateup(const b2moe_bank * gate, const b2moe_bank * up, const b2moe_bank * sg, const b2moe_bank * su, const void * x,
                       int x_dtype, const int * plan, int n, int topk, int shared_tokens, long long live, void * act, int act_dtype, void * ws,
                       void * rows_buf, size_t rows_buf_bytes, cudaStream_t s) {
    const int k = gate->cols, slot_rows = n * topk + shared_tokens;
    const bool slots = rows_buf && rows_buf_bytes >= gemm_tc_slot_bytes(slot_rows, k);
    int * slot_of = slots ? reinterpret_cast<int *>(static_cast<uint8_t *>(rows_buf) + gemm_tc_workspace_bytes(slot_rows, k)) : nullptr;
    __half * xb = static_cast<__half *>(slots ? rows_buf : ws);
    float * inv = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(xb) + align_up(size_t(slots ? slot_rows : n) * k * 2, 256));
    GemmArgs a{};
    const b2moe_bank * banks[4] = {gate, up, shared_tokens ? sg : nullptr, shared_tokens ? su : nullptr};
    a.aux0 = static_cast<const float *>(gate->aux); a.aux1 = static_cast<const float *>(up->aux);
    if (shared_tokens) { a.saux0 = static_cast<const float *>(sg->aux); a.saux1 = static_cast<const float *>(su->aux); }
    a.plan = const_cast<int *>(plan); a.out = act; a.out_dtype = act_dtype;
    a.rows = gate->rows; a.k = k; a.experts = gate->experts; a.topk = topk; a.A = n * topk;
    return gemm_launch<0>(gate->type, a, live, banks, x, x_dtype, n, topk, slots, slot_rows, xb, inv, slot_of, false, s);
}

// per_token: x has a row per token instead of one per assignment (shared_tokens = 0)
int32_t gemm_tc_down(const b2moe_bank * down, const b2moe_bank * sd, const void * x, int x_dtype, bool per_token, const int * plan, int n, int topk,
                     int shared_tokens, long long live, void * y, int y_dtype, void * ws, bool plan_ready, cudaStream_t s) {
    const int rows_x = n * topk + shared_tokens, k = down->cols;
    __half * xb = static_cast<__half *>(ws);
    float * inv = reinterpret_cast<float *>(static_cast<uint8_t *>(ws) + align_up(size_t(rows_x) * k * 2, 256));
    GemmArgs a{};
    const b2moe_bank * banks[4] = {down, nullptr, shared_tokens ? sd : nullptr, nullptr};
    a.aux0 = static_cast<const float *>(down->aux);
    if (shared_tokens) a.saux0 = static_cast<const float *>(sd->aux);
    a.plan = const_cast<int *>(plan); a.out = y; a.out_dtype = y_dtype;
    a.rows = down->rows; a.k = k; a.experts = down->experts; a.topk = topk; a.A = n * topk;
    return gemm_launch<1>(down->type, a, live, banks, x, x_dtype, per_token ? n : rows_x, per_token ? topk : 0, true, rows_x, xb, inv, static_cast<int *>(nullptr), plan_ready, s);
}

}  // namespace b2
