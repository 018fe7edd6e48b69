// Router logits of many 16-bit rows on the 5th-generation tensor cores (included by route.cu).
//
// logits[t][r] = sum_k W[r][k] x[t][k], W fp32. A block takes 128 router rows (M) x NT tokens (N):
//   A: the router rows split exactly into three bf16 terms (hi + mid + lo: the 24 bits of any fp32 value), written to TENSOR MEMORY. TMA brings 64 fp32 columns of them a step, a
//      thread splits half a row of it;
//   B: the activation rows, 64 columns a step, one TMA box in the 128-byte swizzled form. bf16 rows as they are; fp16 rows are split exactly into two bf16 terms in shared memory by
//      the warps that read the sums, a 16-byte piece a thread and step: the first term takes the place of the piece, so the swizzle stays what it was.
// So every product is exact in fp32: three products of terms for bf16 rows, six for fp16 rows. (fp16 terms of the weights times a power of two per 32 columns would take three there, but lose
// what lies far below the largest of the 32: weights of 1e-6 beside one of 1 whose activation is 0 gave an error of 1e-6.)
//
// Numerics. The tensor core cuts its running sums off, always towards zero: 1.7e-8 of the sum per product that meets it. bf16 rows: the leading products of a part of 512 columns
// are one chain of 32, the others (2^-8 of them and less) have sums of their own; the parts are added in column order. fp16 rows: one chain per half
// step, smallest terms first (two of its twelve products meet a sum of full size); half steps and parts are added in fp32 with the rounding errors carried along.
//
// FINE: the sums of half steps with compensation, as for fp16 rows, for bf16 ones: 7.2e-8 where the chains of a part give 4.7e-7, and 1500 cycles a step of 64 tokens.
//
// What bounds it: the chain from a step's copy over its split to the products, 1650 cycles a step of 128 bf16 tokens, 1080 of 64 (most of it the split by two warps a
// scheduler), where the products alone take 768 and 516; 2000 of 64 fp16 tokens, whose products take twice as long and whose sums are read at every step. Two groups of splitting warps on steps in turn: 34.2 us against 31.9 (4096 x 2048 x 512 bf16; three stages instead of four for it); the
// router rows loaded straight from global memory into fragments, no shared memory: 39.0; one accumulator for all terms: 24.9, at 1.65e-6 (this 4.7e-7).
// Registers: 896 threads leave 72, and the form of large bf16 launches (128 tokens, a block per tile) keeps 32 totals a thread: 292 bytes of spill stores, 456 of loads, once a part of 512 columns.
// A launch with few tiles would leave SMs idle: the blocks of a cluster take parts of a tile's columns each, and
// add them in column order through distributed shared memory, so neither the split nor NT changes a bit.
// Every wait is bounded; where one runs out, the tile's logits are summed in a plain loop.
#pragma once
#include "tc_ptx.cuh"
#include "tensor_map.cuh"

namespace b2 {
namespace {
namespace rtc {
using namespace tc;

constexpr int ROWS = 128, STEP = 64, PART_STEPS = 8, MAX_PARTS = 16;
// Warps: 0 copies, 1 issues, 4 .. 11 split, the others read the sums; roles begin at multiples of four: a TMEM lane quarter each
constexpr int TMA_WARP = 0, MMA_WARP = 1, CONV_WARP0 = 4, EPI_WARP0 = 12, EPI_WARPS = 16, THREADS = (EPI_WARP0 + EPI_WARPS) * 32;
// Tensor memory. bf16: the sums of the leading products, those of the others; fp16: two sets of two (the halves of a step), a step each in turn. Then A, two steps of two
// halves: three terms of 32 columns (16 of tensor memory) each
constexpr int ACC = 128, A_COL0 = 2 * ACC, A_TERM = 16, A_HALF = 3 * A_TERM, A_STAGE = 2 * A_HALF;
constexpr int W_BYTES = ROWS * STEP * 4, GATE_BYTES = STEP * 4;
constexpr int stage_bytes(int nt) { return W_BYTES + nt * STEP * 2; }
constexpr int part_bytes(int nt) { return nt * ROWS * 4; }                       // a tile's sums, [token][row]
// Tiles of sums beside the stages. SPLIT: the first of a block's two parts; else bf16: none (totals in registers), fp16: the parts so far. fp16: behind a tile what its sums lack
template <bool FINE, bool SPLIT> constexpr int part_tiles() { return FINE ? 2 : SPLIT ? 1 : 0; }
template <bool FINE, bool SPLIT> constexpr int stages() { return part_tiles<FINE, SPLIT>() ? 3 : 4; }
// fp16: the second terms of a stage's rows, behind the stages
template <int DT> constexpr int low_bytes(int nt) { return DT == B2MOE_F16 ? nt * STEP * 2 : 0; }
constexpr int N_BARS = 3 * 4 + 2 + 2 + 2 + 1;
template <int DT, bool FINE, bool SPLIT> constexpr size_t smem_bytes(int nt) {
    return 1024 + size_t(stages<FINE, SPLIT>()) * (stage_bytes(nt) + low_bytes<DT>(nt) + GATE_BYTES) + part_tiles<FINE, SPLIT>() * part_bytes(nt) + N_BARS * 8 + 16;
}
static_assert(smem_bytes<B2MOE_BF16, false, false>(128) <= 227 * 1024 && smem_bytes<B2MOE_BF16, false, true>(128) <= 227 * 1024 && smem_bytes<B2MOE_F16, true, true>(64) <= 227 * 1024 &&
              3 * stage_bytes(64) >= 2 * part_bytes(64) && 3 * stage_bytes(128) >= part_bytes(128));

// two fp32 operations in one instruction
__device__ __forceinline__ unsigned long long bits2(float2 v) { return (unsigned long long)(__float_as_uint(v.y)) << 32 | __float_as_uint(v.x); }
__device__ __forceinline__ float2 pair_of(uint32_t x, uint32_t y) { return make_float2(__uint_as_float(x), __uint_as_float(y)); }
__device__ __forceinline__ float2 of_bits2(unsigned long long v) { return pair_of(uint32_t(v), uint32_t(v >> 32)); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { unsigned long long r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits2(a)), "l"(bits2(b))); return of_bits2(r); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { unsigned long long r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits2(a)), "l"(bits2(b))); return of_bits2(r); }

// the two values' bf16 terms, largest first, as a pair of 16-bit values each: by cutting off, 8 bits each (an infinity leaves NaN behind, as rounding would)
template <int N> __device__ __forceinline__ void split_terms(float2 w, uint32_t (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint32_t a = __float_as_uint(w.x), b = __float_as_uint(w.y);
        v[i] = __byte_perm(a, b, 0x7632);
        if (i < N - 1) w = sub2(w, pair_of(a & 0xffff0000u, b & 0xffff0000u));
    }
}
// (v, lack) += (sum, lack_sum), the sums so far: plainly, or with the addition's rounding error put into what the sum lacks
template <bool EXACT> __device__ __forceinline__ void add_part(float & v, float & lack, float sum, float lack_sum) {
    const float t = sum + v;
    if (EXACT) {
        const float z = t - sum;
        lack += ((sum - (t - z)) + (v - z)) + lack_sum;
    }
    v = t;
}
struct Maps { CUtensorMap w, x, gate; };
int g_drop_step = -1;                       // test hook (b2moe_harness_wait_probe): every block leaves out the copies of this step of its own

template <int DT, int NT, bool SPLIT, bool FINE>
__global__ void __launch_bounds__(THREADS, 1) router_tc_k(const float * w, const float * shared, const typename Elem<DT>::type * x, float * logits, int ld, int h, int e, int rows,
                                                          int n, int drop_step, const __grid_constant__ Maps maps) {
    namespace cg = cooperative_groups;
    constexpr bool F16 = DT == B2MOE_F16;
    static_assert(!F16 || FINE);
    constexpr int S = stages<FINE, SPLIT>();
    extern __shared__ uint8_t rtc_raw[];
    uint8_t * smem = rtc_raw + (-saddr(rtc_raw) & 1023u);
    const int ks = gridDim.z, n_part = (h + STEP * PART_STEPS - 1) / (STEP * PART_STEPS);
    auto first_part = [&](int z) { return n_part * z / ks; };
    const int p_lo = first_part(blockIdx.z), np = first_part(blockIdx.z + 1) - p_lo;
    const int s_lo = p_lo * PART_STEPS, steps = min((h + STEP - 1) / STEP, (p_lo + np) * PART_STEPS) - s_lo;      // this block's steps
    // see part_tiles; SPLIT: the last part takes the stages' place
    uint8_t * x_low = smem + S * stage_bytes(NT), * parts = x_low + S * low_bytes<DT>(NT);
    float * gate = reinterpret_cast<float *>(parts + part_tiles<FINE, SPLIT>() * part_bytes(NT));      // [stages][64]: the shared expert's gate, router row e
    const uint32_t full = saddr(gate + S * STEP), done = full + 8 * S, x_full = done + 8 * S, a_full = x_full + 8 * S, acc_full = a_full + 16,
                   acc_empty = acc_full + 16, drain = acc_empty + 16;
    uint32_t * tmem_slot = reinterpret_cast<uint32_t *>(gate + S * STEP) + 2 * N_BARS;
    volatile int * gave_up = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // uniform: as in gemm_tc_k
    const int r0 = blockIdx.y * ROWS, t0 = blockIdx.x * NT;                  // tokens on gridDim.x: any batch size
    const bool has_gate = rows > e && r0 + ROWS > e;                    // the tile holds row e

    if (tid == 0) {
#pragma unroll 1
        for (int i = 0; i < S; ++i) { bar_init(full + 8 * i, 1); bar_init(done + 8 * i, 1); bar_init(x_full + 8 * i, EPI_WARPS); }
#pragma unroll 1
        for (int i = 0; i < 2; ++i) { bar_init(a_full + 8 * i, 8); bar_init(acc_full + 8 * i, 1); bar_init(acc_empty + 8 * i, EPI_WARPS); }
        bar_init(drain, 1);
        *gave_up = 0;
        bar_init_fence();
    }
    if (warp == MMA_WARP) tmem_alloc(saddr(tmem_slot), 512);            // all columns: they begin at column 0
    grid_release();
    grid_wait();                                                       // x may be the output of the launch before this one
    fence_before();
    __syncthreads();
    fence_after();
    constexpr uint32_t tmem = 0;

    if (warp == TMA_WARP) {
        if (elect_one()) {
            bool ok = true;
            int g = 0;
#pragma unroll 1
            for (; g < steps; ++g) {
                if (g >= S && !bar_wait(done + 8 * ((g - S) % S), uint32_t((g - S) / S) & 1u)) { ok = false; break; }
                const uint32_t bar = full + 8 * (g % S), dst = saddr(smem) + (g % S) * stage_bytes(NT);
                const int k0 = (s_lo + g) * STEP;
                if (g == drop_step) continue;                           // test hook
                bar_expect_tx(bar, stage_bytes(NT) + (has_gate ? GATE_BYTES : 0));
                tma_load_2d(dst, &maps.w, k0, r0, bar);                 // what lies outside (rows, columns, tokens) arrives as zeros
                tma_load_2d(dst + W_BYTES / 2, &maps.w, k0 + 32, r0, bar);
                tma_load_2d(dst + W_BYTES, &maps.x, k0, t0, bar);
                if (has_gate) tma_load_2d(saddr(gate) + (g % S) * GATE_BYTES, &maps.gate, k0, 0, bar);
            }
            if (!ok) *gave_up = 1;
            // before leaving, every copy must have landed (after a clean run these waits return at once)
#pragma unroll 1
            for (int i = max(0, g - S); i < g; ++i) if (i != drop_step) bar_wait(full + 8 * (i % S), uint32_t(i / S) & 1u);
        }
        __syncwarp();
    } else if (warp == MMA_WARP) {
        {
            const bool lead = elect_one();
            bool ok = true;
            const uint32_t id = idesc(128, NT, 1);
#pragma unroll 1
            for (int g = 0; g < steps; ++g) {
                const int set = g & 1;
                const uint32_t a = tmem + A_COL0 + set * A_STAGE, b = sw128_desc_lo(saddr(smem) + (g % S) * stage_bytes(NT) + W_BYTES);
                [[maybe_unused]] const uint32_t bl = sw128_desc_lo(saddr(x_low) + (g % S) * low_bytes<DT>(NT));
                // half hf's product number k of the weights' term t with the activations' first term (low: the second)
                auto mma = [&](uint32_t d, int hf, int t, int k, bool acc, bool low = false) { mma_f16(lead, d, a + hf * A_HALF + t * A_TERM + 8 * k, (low ? bl : b) + 4 * hf + 2 * k, id, acc); };
                if (!warp_wait((F16 ? x_full : full) + 8 * (g % S), uint32_t(g / S) & 1u) || !warp_wait(a_full + 8 * set, uint32_t(g >> 1) & 1u)) { ok = false; break; }
                if constexpr (FINE) {
                    if (g > 1 && !warp_wait(acc_empty + 8 * set, uint32_t((g >> 1) - 1) & 1u)) { ok = false; break; }
                    fence_after();
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {                   // a half step has sums of its own
                        const uint32_t d = tmem + set * ACC + hf * NT;
#pragma unroll
                        for (int t = 2; t >= 0; --t) {                 // terms t + 1 of the one and t of the other are about as large: 2^-24, 2^-16, 2^-16, 2^-8, 2^-8, 1
                            if (F16) { mma(d, hf, t, 0, t < 2, true); mma(d, hf, t, 1, true, true); }
                            if (t > 0) { mma(d, hf, t, 0, F16 || t < 2); mma(d, hf, t, 1, true); }
                        }
                        mma(d, hf, 0, 0, true); mma(d, hf, 0, 1, true);
                    }
                    mma_commit(lead, acc_full + 8 * set);
                } else {
                    const int p = g / PART_STEPS;
                    const bool more = g % PART_STEPS > 0;
                    if (!more && p > 0 && !warp_wait(acc_empty, uint32_t(p - 1) & 1u)) { ok = false; break; }
                    fence_after();
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        mma(tmem + ACC, hf, 2, 0, more || hf > 0); mma(tmem + ACC, hf, 1, 0, true); mma(tmem + ACC, hf, 2, 1, true); mma(tmem + ACC, hf, 1, 1, true);
                        mma(tmem, hf, 0, 0, more || hf > 0); mma(tmem, hf, 0, 1, true);
                    }
                    if (g % PART_STEPS == PART_STEPS - 1 || g + 1 == steps) mma_commit(lead, acc_full);
                }
                mma_commit(lead, done + 8 * (g % S));
            }
            if (!ok) *gave_up = 1;
            mma_commit(lead, drain);                                         // nothing may be in flight when the tensor memory is freed
            warp_wait(drain, 0);
        }
        __syncwarp();
    } else if (warp >= CONV_WARP0 && warp < EPI_WARP0) {
        // ---- warps (half, quarter q): rows 32 q .. + 31 of the tile, a lane each; that half of every step ----
        const int q = warp & 3, hf = (warp - CONV_WARP0) >> 2, row = 32 * q + lane;
        const bool is_gate = has_gate && r0 + row == e;
        const uint32_t xr = is_gate ? 0u : uint32_t(row & 7) << 4;      // the 128-byte swizzle of the row's 16-byte pieces
        const uint32_t src0 = is_gate ? saddr(gate) + 128 * hf : saddr(smem) + hf * (W_BYTES / 2) + row * 128, src_step = is_gate ? GATE_BYTES : stage_bytes(NT);
        bool ok = true;
#pragma unroll 1
        for (int g = 0; g < steps; ++g) {
            const int s = g % S;
            const uint32_t to = tmem + (uint32_t(32 * q) << 16) + A_COL0 + (g & 1) * A_STAGE + hf * A_HALF;
            if (!warp_wait(full + 8 * (g % S), uint32_t(g / S) & 1u)) { ok = false; break; }
            float v[32];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[4 * i]), "=f"(v[4 * i + 1]), "=f"(v[4 * i + 2]), "=f"(v[4 * i + 3])
                             : "r"(src0 + s * src_step + (uint32_t(16 * i) ^ xr)) : "memory");
            uint32_t t[3][16];
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                uint32_t u[3];
                split_terms(make_float2(v[2 * c], v[2 * c + 1]), u);
                t[0][c] = u[0]; t[1][c] = u[1]; t[2][c] = u[2];
            }
            if (g > 1 && !warp_wait(done + 8 * ((g - 2) % S), uint32_t((g - 2) / S) & 1u)) { ok = false; break; }      // the products of the step that had the place
            fence_after();
#pragma unroll
            for (int c = 0; c < 3; ++c) tmem_st16(to + c * A_TERM, t[c]);
            tmem_st_wait();
            fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(a_full + 8 * (g & 1));
        }
        if (!ok && lane == 0) *gave_up = 1;
    } else if (warp >= EPI_WARP0) {
        // ---- warps q, q + 4, ..: the sums of rows 32 q .. + 31, a lane each; a share of the tokens ----
        constexpr int TOK = NT / (EPI_WARPS / 4);
        const int q = warp & 3, tk0 = TOK * ((warp - EPI_WARP0) >> 2), row = 32 * q + lane;
        const uint32_t from = tmem + (uint32_t(32 * q) << 16) + tk0;
        float * const so_far = reinterpret_cast<float *>(parts) + tk0 * ROWS + row, * const last = reinterpret_cast<float *>(smem) + tk0 * ROWS + row;
        const bool in = r0 + row < rows;
        [[maybe_unused]] float tot[TOK];
        // fp16: step g's activations as two terms, a piece of eight a thread. What a stage's second terms replace was read by products that were done when the stage was filled again
        static_assert(!F16 || NT * STEP == EPI_WARPS * 32 * 8);
        auto split_x = [&](int g) {
            if (!warp_wait(full + 8 * (g % S), uint32_t(g / S) & 1u)) return false;
            const uint32_t piece = 16 * ((warp - EPI_WARP0) * 32 + lane), at = saddr(smem) + (g % S) * stage_bytes(NT) + W_BYTES + piece;
            uint32_t v[4], u0[4], u1[4];
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(at) : "memory");
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t u[2];
                split_terms(__half22float2(*reinterpret_cast<const __half2 *>(&v[i])), u);
                u0[i] = u[0]; u1[i] = u[1];
            }
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(u0[0]), "r"(u0[1]), "r"(u0[2]), "r"(u0[3]) : "memory");
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(saddr(x_low) + (g % S) * low_bytes<DT>(NT) + piece), "r"(u1[0]), "r"(u1[1]), "r"(u1[2]), "r"(u1[3]) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(x_full + 8 * (g % S));
            return true;
        };
        bool ok = true;
        if constexpr (F16)
            for (int g = 0; g < min(2, steps) && ok; ++g) ok = split_x(g);
#pragma unroll 1
        for (int p = 0; p < np && ok; ++p) {
            const bool is_last = p + 1 == np;
            // the finished sum of the part's i-th token (and what it lacks): SPLIT: put away; else added to those before it
            auto put = [&](int i, float v, float lack = 0.f) {
                if (SPLIT) {
                    (is_last ? last : so_far)[i * ROWS] = v;
                    if (FINE) (is_last ? last : so_far)[(NT + i) * ROWS] = lack;
                    return;
                }
                if (FINE) {
                    if (p > 0) add_part<true>(v, lack, so_far[i * ROWS], so_far[(NT + i) * ROWS]);
                    if (!is_last) { so_far[i * ROWS] = v; so_far[(NT + i) * ROWS] = lack; }
                } else {
                    if (p > 0) v = tot[i] + v;
                    tot[i] = v;
                }
                const int tok = t0 + tk0 + i;
                if (is_last && in && tok < n) logits[size_t(tok) * ld + r0 + row] = checked_logit<DT>(FINE ? v + lack : v, w, shared, x, r0 + row, tok, e, h);
            };
            if constexpr (FINE) {
                // The steps' sums are added with their rounding errors carried along (Kahan; lost: what the sum lacks): the plain additions of a part would be the largest error
                float2 sum[TOK / 2], lost[TOK / 2];
#pragma unroll
                for (int i = 0; i < TOK / 2; ++i) sum[i] = lost[i] = make_float2(0.f, 0.f);
                const int g_hi = min(steps, (p + 1) * PART_STEPS);
#pragma unroll 1
                for (int g = p * PART_STEPS; g < g_hi; ++g) {
                    const int set = g & 1;
                    // two steps ahead: the stage is filled once the products of step g - 1 are done
                    if (F16 && g + 2 < steps && !split_x(g + 2)) { ok = false; break; }
                    if (!warp_wait(acc_full + 8 * set, uint32_t(g >> 1) & 1u)) { ok = false; break; }
                    fence_after();
#pragma unroll
                    for (int c = 0; c < TOK; c += 8) {
                        uint32_t v0[8], v1[8];
                        tmem_ld8(from + set * ACC + c, v0);
                        tmem_ld8(from + set * ACC + NT + c, v1);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float2 & s2 = sum[c / 2 + i], & l2 = lost[c / 2 + i];
                            const float2 y = add2(pair_of(v0[2 * i], v0[2 * i + 1]), add2(pair_of(v1[2 * i], v1[2 * i + 1]), l2)), t = add2(s2, y);
                            l2 = sub2(y, sub2(t, s2));
                            s2 = t;
                        }
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0) bar_arrive(acc_empty + 8 * set);
                }
                if (!ok) break;
#pragma unroll
                for (int i = 0; i < TOK; ++i) put(i, i & 1 ? sum[i / 2].y : sum[i / 2].x, i & 1 ? lost[i / 2].y : lost[i / 2].x);
            } else {
                if (!warp_wait(acc_full, uint32_t(p) & 1u)) { ok = false; break; }
                fence_after();
#pragma unroll
                for (int c = 0; c < TOK; c += 8) {
                    uint32_t v0[8], v1[8];
                    tmem_ld8(from + c, v0);
                    tmem_ld8(from + ACC + c, v1);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; ++i) put(c + i, __uint_as_float(v0[i]) + __uint_as_float(v1[i]));
                }
                fence_before();
                __syncwarp();
                if (lane == 0) bar_arrive(acc_empty);
            }
        }
        if (!ok) {
            if (lane == 0) *gave_up = 1;
            if (!SPLIT)
#pragma unroll 1
                for (int i = 0; i < TOK; ++i)
                    if (in && t0 + tk0 + i < n) logits[size_t(t0 + tk0 + i) * ld + r0 + row] = checked_logit<DT>(0.f, w, shared, x, r0 + row, t0 + tk0 + i, e, h, true);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == MMA_WARP) tmem_free(tmem, 512);
    if constexpr (SPLIT) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        // every block of the cluster finishes a share of the tile's tokens; where the parts lie in the cluster's shared memory comes from a table
        __shared__ uint32_t place[MAX_PARTS];
        __shared__ int bad;
        if (tid == 0) bad = 0;
        __syncthreads();
        if (tid < n_part) {
            int z = 0;
            while (first_part(z + 1) <= tid) ++z;
            const int i = tid - first_part(z), last = first_part(z + 1) - first_part(z) - 1;
            const uint32_t local = i < last ? saddr(parts) : saddr(smem);
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(place[tid]) : "r"(local), "r"(z));
            uint32_t flag;
            int v;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(flag) : "r"(saddr(const_cast<const int *>(gave_up))), "r"(z));
            asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(flag) : "memory");
            if (v) bad = 1;
        }
        __syncthreads();
        const int lo = NT * int(blockIdx.z) / ks, hi = NT * (int(blockIdx.z) + 1) / ks;
#pragma unroll 1
        for (int i = tid; i < (hi - lo) * ROWS; i += THREADS) {
            const int tk = lo + i / ROWS, r = i % ROWS;
            if (t0 + tk >= n || r0 + r >= rows) continue;
            const uint32_t off = uint32_t(tk * ROWS + r) * 4u;
            float sum = 0.f, lack = 0.f;
#pragma unroll 1
            for (int q = 0; q < n_part; q += 4) {
                float v[4], l[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] = l[j] = 0.f;
                    if (q + j < n_part) {
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[j]) : "r"(place[q + j] + off) : "memory");
                        if (FINE) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(l[j]) : "r"(place[q + j] + off + part_bytes(NT)) : "memory");
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (q + j < n_part) {
                        if (q + j > 0) add_part<FINE>(v[j], l[j], sum, lack);
                        sum = v[j];
                        lack = l[j];
                    }
            }
            logits[size_t(t0 + tk) * ld + r0 + r] = checked_logit<DT>(FINE ? sum + lack : sum, w, shared, x, r0 + r, t0 + tk, e, h, bad != 0);
        }
        cluster.sync();                                                // the blocks' tiles stay alive until every block has read them
    }
}

// The shape of a launch: tokens a block and blocks a tile's columns are split over, the pair with the fewest cycles. Clusters of such blocks that a B200 holds at once, by size
// (cudaOccupancyMaxActiveClusters; a cluster stays inside a GPC): 16 clusters of 8 take two rounds. With 148 blocks of any cluster: bf16 4096 x 128, 1024 tokens 21.7 us, 12.7; fp16 1536 x 256, 3000 42, 29
constexpr int CLUSTERS[9] = {0, ROUTER_SMS, 74, 45, 33, 26, 22, 15, 15};
struct Shape { int nt, ks; long long cycles; };
template <int DT, bool FINE> Shape shape_of(int rows, int n, int h) {
    const int parts = ceil_div(h, STEP * PART_STEPS);
    Shape best{0, 1, 0};
    for (int nt = FINE ? 64 : 128; nt >= 64; nt -= 64) {
        const long long tiles = (long long)ceil_div(rows, ROWS) * ceil_div(n, nt);
        for (int share = parts; share >= 1; --share) {
            const int ks = ceil_div(parts, share);
            if (ks > 8 || (ks > 1 && (share > 2 || parts > MAX_PARTS))) continue;
            // cycles of a step (measured), of a block's start and end, and of the meeting in a cluster
            const int step = DT == B2MOE_F16 ? 2000 : FINE ? 1500 : nt == 128 ? 1650 : 1080;
            const long long cost = (tiles + CLUSTERS[ks] - 1) / CLUSTERS[ks] * (share * PART_STEPS * step + 6000) + (ks > 1 ? 2000 : 0);
            if (best.nt == 0 || cost < best.cycles) best = Shape{nt, ks, cost};
        }
    }
    return best;
}
template <int DT, int NT, bool FINE> int32_t launch_nt(const Shape & p, const float * w, const float * shared, const typename Elem<DT>::type * x, float * logits, int ld, int h, int e,
                                            int rows, int n, cudaStream_t s) {
    Maps maps;
    const cuuint64_t xd[2] = {cuuint64_t(h), cuuint64_t(n)}, wd[2] = {cuuint64_t(h), cuuint64_t(e)}, gd[2] = {cuuint64_t(h), 1}, xs[1] = {cuuint64_t(h) * 2}, ws[1] = {cuuint64_t(h) * 4};
    const cuuint32_t xb[2] = {STEP, NT}, wb[2] = {STEP / 2, ROWS}, gb[2] = {STEP, 1};
    if (!encode_map(maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, xd, xs, xb, CU_TENSOR_MAP_SWIZZLE_128B) ||       // (copied as they are: bf16 is as good)
        !encode_map(maps.w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, w, wd, ws, wb, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_map(maps.gate, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, shared ? shared : w, gd, ws, gb, CU_TENSOR_MAP_SWIZZLE_NONE)) return B2MOE_ERR_CUDA;
    const size_t smem = p.ks > 1 ? smem_bytes<DT, FINE, true>(NT) : smem_bytes<DT, FINE, false>(NT);
    const auto kernel = p.ks > 1 ? router_tc_k<DT, NT, true, FINE> : router_tc_k<DT, NT, false, FINE>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return B2MOE_ERR_CUDA;
    return launch_cluster_z(kernel, dim3(ceil_div(n, NT), ceil_div(rows, ROWS), p.ks), THREADS, smem, s, w, shared, x, logits, ld, h, e, rows, n, g_drop_step, maps);
}
// 16-bit rows; h a multiple of 8 (strides of the maps)
template <int DT, bool FINE> int32_t launch(const float * w, const float * shared, const typename Elem<DT>::type * x, float * logits, int ld, int h, int e, int rows, int n, cudaStream_t s) {
    const Shape p = shape_of<DT, FINE>(rows, n, h);
    if constexpr (!FINE)
        if (p.nt == 128) return launch_nt<DT, 128, FINE>(p, w, shared, x, logits, ld, h, e, rows, n, s);
    return launch_nt<DT, 64, FINE>(p, w, shared, x, logits, ld, h, e, rows, n, s);
}

}  // namespace rtc
}  // namespace
}  // namespace b2
