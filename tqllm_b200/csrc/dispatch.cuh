// Device code of the token -> expert dispatch shared by the stand-alone kernels (dispatch.cu) and the fused
// top-k + dispatch kernel (route.cu). See dispatch.cu for the method.
#pragma once
#include "common.cuh"

namespace b2 {

__device__ __forceinline__ int valid_id(const int * ids, int a, int A, int e) {
    if (a >= A) return -1;
    const int v = ids[a];
    return (v >= 0 && v < e) ? v : -1;
}

// the lanes whose id equals this lane's (meaningless where id < 0): a vote per bit of the ids. For kernels of many steps:
// __match_any_sync queues behind the other warps of the SM (32 warps of dispatch_small_k, 5,090 ids: 18 us with it, 13.5 with the
// votes); in the routing launch, of two steps a warp, the shorter code wins (15.4 against 16.5 us).
__device__ __forceinline__ unsigned same_id(int id, int bits) {
    unsigned peers = __ballot_sync(0xffffffffu, id >= 0);
#pragma unroll 4
    for (int b = 0; b < bits; ++b) {
        const unsigned m = __ballot_sync(0xffffffffu, (id >> b) & 1);
        peers &= (id >> b) & 1 ? m : ~m;
    }
    return peers;
}

// One warp walks the assignments [a0, a1) in order, 32 per step, and calls step(assignment, expert or -1, lanes with the same
// expert): the ids of eight steps are loaded together, so that a walk waits for memory once per 256 assignments and not at
// every step.
template <bool VOTES, class F>
__device__ __forceinline__ void walk_ids(const int * ids, int a0, int a1, int e, int lane, F step) {
    const int bits = 32 - __clz(e - 1);
#pragma unroll 1
    for (int b = a0; b < a1; b += 256) {
        int id[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) id[j] = valid_id(ids, b + 32 * j + lane, a1, e);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (b + 32 * j >= a1) break;
            step(b + 32 * j + lane, id[j], VOTES ? same_id(id[j], bits) : __match_any_sync(0xffffffffu, id[j]));
            __syncwarp();             // a step's counter updates are in place before the next step's leaders read them
        }
    }
}

// the `n` counters at h, `stride` apart -> their exclusive prefix sums; returns the total. Eight at a time: the loads of a batch do
// not wait for its stores (one load per store would, since both go to the same array).
template <class C>
__device__ __forceinline__ int prefix_counters(C * h, int n, int stride) {
    int run = 0;
    for (int c0 = 0; c0 < n; c0 += 8) {
        int v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = c0 + i < n ? h[size_t(c0 + i) * stride] : 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c0 + i < n) { h[size_t(c0 + i) * stride] = C(run); run += v[i]; }
    }
    return run;
}

// exclusive prefix sums of (a, b) over the threads of a block of whole warps, and their totals; w: 32 entries of shared memory
__device__ __forceinline__ int2 block_scan(int a, int b, int2 * w, int2 & total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int pa = a, pb = b;
    for (int d = 1; d < 32; d <<= 1) {
        const int oa = __shfl_up_sync(0xffffffffu, pa, d), ob = __shfl_up_sync(0xffffffffu, pb, d);
        if (lane >= d) { pa += oa; pb += ob; }
    }
    if (lane == 31) w[warp] = make_int2(pa, pb);
    __syncthreads();
    const int2 own = lane < nw ? w[lane] : make_int2(0, 0);
    int wa = own.x, wb = own.y;
    for (int d = 1; d < 32; d <<= 1) {
        const int oa = __shfl_up_sync(0xffffffffu, wa, d), ob = __shfl_up_sync(0xffffffffu, wb, d);
        if (lane >= d) { wa += oa; wb += ob; }
    }
    total = make_int2(__shfl_sync(0xffffffffu, wa, 31), __shfl_sync(0xffffffffu, wb, 31));
    const int la = __shfl_sync(0xffffffffu, wa - own.x, warp), lb = __shfl_sync(0xffffffffu, wb - own.y, warp);
    return make_int2(la + pa - a, lb + pb - b);
}

// counts cs[0..e1) -> offsets[0..e1], active list, pass list and the header words, by all threads of the block, each with a
// contiguous span of the experts (one warp for all of them was a chain of e1 / 32 dependent steps, three times over: 2 us of dispatch_place_k at 512 experts).
// cs, os and as are shared-memory copies; with `write` every result also goes to the plan in global memory. The caller
// synchronises before (cs) and after (os).
__device__ inline void finish_plan(int * plan, const int * cs, int * os, int * as, int * offsets, int * active, int * passes, int e1, bool write) {
    __shared__ int2 wsum[2][32];
    const int nt = blockDim.x, span = (e1 + nt - 1) / nt, lo = min(e1, int(threadIdx.x) * span), hi = min(e1, lo + span);
    int sum = 0, act = 0;
    for (int i = lo; i < hi; ++i) { sum += cs[i]; act += cs[i] > 0; }
    int2 total, at = block_scan(sum, act, wsum[0], total);
    for (int i = lo; i < hi; ++i) {
        const int c = cs[i];
        os[i] = at.x;
        if (write) offsets[i] = at.x;
        if (c > 0) {
            as[at.y] = i;
            if (write) active[at.y] = i;
            ++at.y;
        }
        at.x += c;
    }
    if (!write) return;
    if (threadIdx.x == 0) { offsets[e1] = total.x; os[e1] = total.x; plan[PLAN_NGROUPED] = total.x; plan[PLAN_NACTIVE] = total.y; plan[PLAN_STATUS] = 0; }
    __syncthreads();
    // pass list: active experts from the last (the shared expert, the heaviest) to the first, cut into passes of
    // PASS_TOKENS tokens; passes[i] = number of passes before the i-th expert of that order
    const int na = total.y, sp = (na + nt - 1) / nt, l2 = min(na, int(threadIdx.x) * sp), h2 = min(na, l2 + sp);
    int mine = 0;
    for (int i = l2; i < h2; ++i) mine += (cs[as[na - 1 - i]] + PASS_TOKENS - 1) / PASS_TOKENS;
    int rp = block_scan(mine, 0, wsum[1], total).x;
    for (int i = l2; i < h2; ++i) { passes[i] = rp; rp += (cs[as[na - 1 - i]] + PASS_TOKENS - 1) / PASS_TOKENS; }
    if (threadIdx.x == 0) { passes[na] = total.x; plan[PLAN_NPASS] = total.x; }
}

// shared memory of dispatch_small_body for a block of `warps` warps: hist [warps][e] (16-bit) + three int arrays of e + 2
__host__ __device__ inline size_t dispatch_small_smem(int warps, int e) { return (size_t(warps) * e * 2 + 15) / 16 * 16 + size_t(3) * (e + 2) * 4; }

// ---- single block (up to 32 warps): every phase in shared memory (decode-sized batches); hist = [warps][e] ----
template <bool VOTES>
__device__ __forceinline__ void dispatch_small_body(const int * ids, int A, int e, int shared_first, int shared_tokens,
                                                    int * __restrict__ plan, unsigned short * hist) {
    const int e1 = e + 1;
    int * counts = plan + PLAN_HDR, * offsets = counts + e1, * active = offsets + e1 + 1, * perm = active + e1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int * cs = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(hist) + (size_t(nw) * e * 2 + 15) / 16 * 16), * os = cs + e + 2, * as = os + e + 2;
    const int chunk = ((A + nw - 1) / nw + 31) / 32 * 32;   // per warp, a multiple of 32
    for (int i = threadIdx.x; i < nw * e; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int a0 = warp * chunk;
    const int a1 = min(A, a0 + chunk);
    unsigned short * h = hist + warp * e;
    walk_ids<VOTES>(ids, a0, a1, e, lane, [&](int, int id, unsigned peers) {
        if (id >= 0 && lane == __ffs(peers) - 1) h[id] += (unsigned short)__popc(peers);
    });
    __syncthreads();
    for (int x = threadIdx.x; x < e; x += blockDim.x) counts[x] = cs[x] = prefix_counters(hist + x, nw, e);
    if (threadIdx.x == 0) { counts[e] = shared_tokens; cs[e] = shared_tokens; }
    __syncthreads();
    finish_plan(plan, cs, os, as, offsets, active, perm + A + shared_tokens, e1, true);
    __syncthreads();
    walk_ids<VOTES>(ids, a0, a1, e, lane, [&](int a, int id, unsigned peers) {
        if (id >= 0) perm[os[id] + h[id] + __popc(peers & ((1u << lane) - 1u))] = a;
        __syncwarp();
        if (id >= 0 && lane == __ffs(peers) - 1) h[id] += (unsigned short)__popc(peers);
    });
    for (int t = threadIdx.x; t < shared_tokens; t += blockDim.x) perm[os[e] + t] = A + shared_first + t;
}


inline bool dispatch_small_path(int e, int A) { return A <= 32 * 2048 / 8 && dispatch_small_smem(32, e) <= 46 * 1024; }

}  // namespace b2
