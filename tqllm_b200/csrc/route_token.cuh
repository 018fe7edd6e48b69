// Routing of one token by one warp, its keys in registers: used by the routing launches (route.cu) and by the gate/up launch that routes for itself (expert_dec4.cu).
#pragma once
#include <math_constants.h>

#include "common.cuh"

namespace b2 {

// ---- register-resident routing of one token by one warp (experts <= 32 R) ----
// Lane l keeps experts l, l + 32, ... in registers; a round is a local scan, one warp-wide max of an order-preserving
// integer image of the key and one warp-wide min over the indices that hold it (ties -> lowest index), so the ten
// rounds of a top-10 are ten short chains of register operations instead of shared-memory scans and shuffle ladders.
__device__ __forceinline__ uint32_t ordered_bits(float v) {          // monotonic float -> uint (taken entries use 0)
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
template <int GATING, int R>
__device__ __forceinline__ void route_token_regs(const float * logits, int ld, const float * __restrict__ bias,
                                                 int * __restrict__ ids, float * __restrict__ weights, float * __restrict__ shared_weights,
                                                 int e, int k, int norm, float scale, int token, int lane) {
    const float * x = logits + size_t(token) * ld;
    float p[R];
    uint32_t key[R];
#pragma unroll
    for (int r = 0; r < R; ++r) p[r] = lane + 32 * r < e ? x[lane + 32 * r] : -CUDART_INF_F;
    if (GATING == B2MOE_SOFTMAX) {
        float m = -CUDART_INF_F;
#pragma unroll
        for (int r = 0; r < R; ++r) m = fmaxf(m, p[r]);
        for (int d = 16; d; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
        float sum = 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r) if (lane + 32 * r < e) { p[r] = expf(p[r] - m); sum += p[r]; }
        for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
#pragma unroll
        for (int r = 0; r < R; ++r) { p[r] = p[r] / sum; key[r] = lane + 32 * r < e ? ordered_bits(p[r]) : 0u; }
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool in = lane + 32 * r < e;
            p[r] = 1.f / (1.f + expf(-p[r]));
            key[r] = in ? ordered_bits(bias ? p[r] + bias[lane + 32 * r] : p[r]) : 0u;
        }
    }
    // lane q keeps the q-th selection (k <= 32 on this path): one coalesced store of ids and weights at the end instead of a
    // store per round and a read-modify-write pass of lane 0 over global memory
    float sel_sum = 0.f, my_p = 0.f;
    int my_idx = 0;
    for (int q = 0; q < k; ++q) {
        uint32_t best = 0;
        int br = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) if (key[r] > best) { best = key[r]; br = r; }     // ascending r: the lowest index keeps a tie
        const uint32_t top = __reduce_max_sync(0xffffffffu, best);
        const int idx = int(__reduce_min_sync(0xffffffffu, (best == top && best != 0u) ? uint32_t(lane + 32 * br) : 0x7fffffffu));
        const int owner = idx & 31, orow = idx >> 5;
        float pv = 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r) if (r == orow) { pv = p[r]; if (lane == owner) key[r] = 0u; }
        pv = __shfl_sync(0xffffffffu, pv, owner);
        if (lane == q) { my_idx = idx == 0x7fffffff ? 0 : idx; my_p = pv; }
        sel_sum += pv;
    }
    if (lane < k) {
        float w = my_p;
        if (norm) w = w / fmaxf(sel_sum, 6.103515625e-5f);
        if (scale != 0.f && scale != 1.f) w *= scale;
        ids[size_t(token) * k + lane] = my_idx;
        weights[size_t(token) * k + lane] = w;
    }
    if (lane == 0 && shared_weights) shared_weights[token] = 1.f / (1.f + expf(-x[e]));
}

}  // namespace b2
