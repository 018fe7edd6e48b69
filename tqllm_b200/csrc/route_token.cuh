// Routing of one token by one warp, its keys in registers: used by the routing launches (route.cu) and by the gate/up launch that routes for itself (expert_dec4.cu).
#pragma once
#include <math_constants.h>

#include "common.cuh"

namespace b2 {

// ---- register-resident routing of one token by one warp (experts <= 32 R) ----
// Lane l keeps experts l, l + 32, ... in registers. What bounds it is a chain of instructions that a few warps of an SM run once per launch. Cycles for top-10 of 512, code in the instruction cache, one warp /
// 16 in the block: softmax 2880 / 3490 and ten rounds 3810 / 12000 when every probability was divided in a branch of its own and every round looked through all keys and fetched the
// selected probability from among them; now softmax 1130 / 1960 and the selection 1280 / 2310. Layers, us: c3 8 tokens 57.9 -> 56.7, c2 509 tokens 298.7 -> 293.9, 64 tokens x 4 636 -> 631.
// (As long as weight streams pushed the code out of the L2, fetching the longer code took back what it saves.)
__device__ __forceinline__ uint32_t ordered_bits(float v) {          // monotonic float -> uint (taken entries use 0)
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// a / b to the bit with r = 1 / b rounded to nearest, where not all of b's mantissa bits are set and no residual underflows. Sixteen of them side by side take what one division with its special cases takes.
// Mantissas in [1, 2), u = 2^-24. A first quotient within one ulp has a residual of at most 24 bits: it is exact, and corrects the quotient to the correctly rounded one (P. Markstein, Computation of
// elementary functions on the IBM RISC System/6000 processor, 1990). The first quotient can be further off where a < b: by 1/2 ulp for its own rounding and a / 2 for r's; with a <= b - 2u <= 2 - 6u that
// is at most 1.5 - 3u. Its residual takes 25 bits, whose rounding moves the corrected value by at most 1 / b's mantissa as a whole number (u to 2u) ulp, r's error by 1.5u: to be rounded the wrong way, a / b would have to lie
// that near to the middle between two floats. Such an a / b, more than one ulp from the first quotient, is 1.5 ulp away but for as much, which takes a and b next to 2, where the two add up to less than 3u: it cannot be.
__device__ __forceinline__ float quotient(float a, float b, float r) {
    const float q = a * r;
    return fmaf(fmaf(-q, b, a), r, q);
}
// what a warp needs of shared memory for one token: 8 bytes for each of up to 32 keys, no more than there are experts
struct Picked { uint32_t key; int idx; };

template <int GATING, int R>
__device__ __forceinline__ void route_token_regs(const float * logits, int ld, const float * __restrict__ bias,
                                                 int * __restrict__ ids, float * __restrict__ weights, float * __restrict__ shared_weights,
                                                 int e, int k, int norm, float scale, int token, int lane, Picked * list) {
    const float * x = logits + size_t(token) * ld;
    uint32_t key[R];
    {
        float p[R];
#pragma unroll
        for (int r = 0; r < R; ++r) p[r] = lane + 32 * r < e ? x[lane + 32 * r] : -CUDART_INF_F;
        if (GATING == B2MOE_SOFTMAX) {
            float m = -CUDART_INF_F, low = CUDART_INF_F;
#pragma unroll
            for (int r = 0; r < R; ++r) { m = fmaxf(m, p[r]); low = fminf(low, lane + 32 * r < e ? p[r] : CUDART_INF_F); }
            for (int d = 16; d; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
            float sum = 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r) { p[r] = expf(p[r] - m); sum += p[r]; }      // no expert: 0 (where m is infinite the others make the sum a NaN)
            for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
            // every probability above 2^-100 (the residual does not underflow: exp(-69) = 1.1e-30), a sum (at least 1) whose mantissa is not all ones
            if (__all_sync(0xffffffffu, low - m > -69.f && sum < 0x1p20f && (__float_as_uint(sum) & 0x7fffffu) != 0x7fffffu)) {
                const float inv = 1.f / sum;
#pragma unroll
                for (int r = 0; r < R; ++r) p[r] = quotient(p[r], sum, inv);
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) p[r] = p[r] / sum;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) key[r] = lane + 32 * r < e ? ordered_bits(p[r]) : 0u;
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float v = __frcp_rn(1.f + expf(-p[r]));
                key[r] = lane + 32 * r < e ? ordered_bits(bias ? v + bias[lane + 32 * r] : v) : 0u;
            }
        }
    }
    // The selection: larger keys first, the lower index among equal ones. The k-th largest of the lanes' largest keys is a line that at least k keys reach; those that do are a few more than k,
    // and when they are no more than 32, a lane takes each (in the order of their indices) and counts the ones before it.
    uint32_t best = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) best = max(best, key[r]);
    int above = 0;
#pragma unroll
    for (int i = 0; i < 32; ++i) above += __shfl_sync(0xffffffffu, best, i) > best;
    const uint32_t line = __reduce_min_sync(0xffffffffu, above < k ? best : 0xffffffffu);
    int count = 0, my_idx = 0, rank = 32;
    uint32_t my_key = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool is = key[r] >= line;
        const unsigned m = __ballot_sync(0xffffffffu, is);
        const int at = count + __popc(m & ((1u << lane) - 1u));
        if (is && at < 32 && line != 0u) list[at] = Picked{key[r], lane + 32 * r};
        count += __popc(m);
    }
    __syncwarp();
    if (line != 0u && count <= 32) {
        if (lane < count) {
            const Picked mine = list[lane];
            my_key = mine.key;
            my_idx = mine.idx;
            rank = 0;
#pragma unroll 4
            for (int i = 0; i < count; ++i) {
                const uint32_t o = list[i].key;
                rank += o > my_key || (o == my_key && i < lane);
            }
        }
    } else {                                                            // many equal keys, or fewer than k that count: round by round
        my_key = 0;
        my_idx = 0;
        rank = lane;
#pragma unroll 1
        for (int q = 0; q < k; ++q) {
            uint32_t top = 0;
            int at = 0;
#pragma unroll
            for (int r = 0; r < R; ++r) if (key[r] > top) { top = key[r]; at = r; }      // ascending r: the lowest index keeps a tie
            const uint32_t all = __reduce_max_sync(0xffffffffu, top);
            const int idx = int(__reduce_min_sync(0xffffffffu, (top == all && top != 0u) ? uint32_t(lane + 32 * at) : 0x7fffffffu));
            const int own = (idx & 31) == lane ? idx >> 5 : -1;
#pragma unroll
            for (int r = 0; r < R; ++r) key[r] = r == own ? 0u : key[r];
            if (lane == q && all != 0u) { my_idx = idx; my_key = all; }
        }
    }
    // the probabilities of the selected: out of the key where it is their image (that of no number below zero: a NaN), else from the logit again (the same expression, the same bits)
    float my_p = 0.f;
    if (rank < k && my_key != 0u)
        my_p = GATING == B2MOE_SOFTMAX ? __uint_as_float(my_key & 0x80000000u ? my_key & 0x7fffffffu : 0x7fffffffu) : __frcp_rn(1.f + expf(-x[my_idx]));
    if (norm) {
        float * by_rank = reinterpret_cast<float *>(list);
        __syncwarp();
        if (rank < k) by_rank[rank] = my_p;
        __syncwarp();
        float sum = 0.f;                                                // in the order of the selection
#pragma unroll 4
        for (int q = 0; q < k; ++q) sum += by_rank[q];
        my_p = my_p / fmaxf(sum, 6.103515625e-5f);
        __syncwarp();                                                   // the list is free for the warp's next token
    }
    if (rank < k) {
        if (scale != 0.f && scale != 1.f) my_p *= scale;
        ids[size_t(token) * k + rank] = my_idx;
        weights[size_t(token) * k + rank] = my_p;
    }
    if (lane == 0 && shared_weights) shared_weights[token] = 1.f / (1.f + expf(-x[e]));
}

}  // namespace b2
