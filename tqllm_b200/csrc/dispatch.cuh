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

// exclusive prefix sums of (x, y, z) over the threads of a block's first `used` warps, and their totals, for those warps; w: 32
// entries of shared memory; one barrier for the whole block
__device__ __forceinline__ int3 block_scan(int3 v, int used, int3 * w, int3 & total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int3 p = v;
    if (warp < used) {
#pragma unroll 1
        for (int d = 1; d < 32; d <<= 1) {
            const int ox = __shfl_up_sync(0xffffffffu, p.x, d), oy = __shfl_up_sync(0xffffffffu, p.y, d), oz = __shfl_up_sync(0xffffffffu, p.z, d);
            if (lane >= d) { p.x += ox; p.y += oy; p.z += oz; }
        }
        if (lane == 31) w[warp] = p;
    }
    __syncthreads();
    if (warp >= used) return p;
    const int3 own = lane < used ? w[lane] : make_int3(0, 0, 0);
    int3 q = own;
#pragma unroll 1
    for (int d = 1; d < 32; d <<= 1) {
        const int ox = __shfl_up_sync(0xffffffffu, q.x, d), oy = __shfl_up_sync(0xffffffffu, q.y, d), oz = __shfl_up_sync(0xffffffffu, q.z, d);
        if (lane >= d) { q.x += ox; q.y += oy; q.z += oz; }
    }
    total = make_int3(__shfl_sync(0xffffffffu, q.x, 31), __shfl_sync(0xffffffffu, q.y, 31), __shfl_sync(0xffffffffu, q.z, 31));
    return make_int3(__shfl_sync(0xffffffffu, q.x - own.x, warp) + p.x - v.x, __shfl_sync(0xffffffffu, q.y - own.y, warp) + p.y - v.y,
                     __shfl_sync(0xffffffffu, q.z - own.z, warp) + p.z - v.z);
}

// counts cs[0..e1) -> offsets os[0..e1] and, with `write`, the plan's offsets, active list, pass list and header words, by the threads of
// the block, each with a contiguous span of the experts (one warp for all of them was a chain of e1 / 32 dependent steps, three times
// over: 2 us of dispatch_place_k at 512 experts). The pass list runs over the active experts from the last (the shared expert, the heaviest) to the
// first, cut into passes of PASS_TOKENS tokens: passes[i] = passes before the i-th expert of that order = all of them but those up to
// that expert, so tokens, experts and passes take one scan and one barrier together. (Two scans, the second behind
// the list that it read, took 3.6 to 8 thousand cycles of a routing launch. The loops are rolled: the code runs once a launch, and with unrolled ones its fetch
// took longer than the scan: 2.4 to 3 us against 1.3 at 8 to 64 tokens.) cs and os are shared-memory copies, or the plan's own arrays.
// The caller synchronises before (cs) and after (os).
__device__ inline void finish_plan(int * plan, const int * cs, int * os, int * offsets, int * active, int * passes, int e1, bool write) {
    __shared__ int3 wsum[32];
    const int nt = blockDim.x, span = (e1 + nt - 1) / nt, lo = min(e1, int(threadIdx.x) * span), hi = min(e1, lo + span);
    const int used = ((e1 + span - 1) / span + 31) >> 5;
    int3 v = make_int3(0, 0, 0), total;
    for (int i = lo; i < hi; ++i) { const int c = cs[i]; v.x += c; v.y += c > 0; v.z += (c + PASS_TOKENS - 1) / PASS_TOKENS; }
    int3 at = block_scan(v, used, wsum, total);
    for (int i = lo; i < hi; ++i) {
        const int c = cs[i];
        os[i] = at.x;
        if (write) offsets[i] = at.x;
        at.x += c;
        if (c > 0) {
            at.z += (c + PASS_TOKENS - 1) / PASS_TOKENS;
            if (write) { active[at.y] = i; passes[total.y - 1 - at.y] = total.z - at.z; }
            ++at.y;
        }
    }
    if (write && threadIdx.x == 0) {
        offsets[e1] = total.x; os[e1] = total.x; passes[total.y] = total.z;
        plan[PLAN_NGROUPED] = total.x; plan[PLAN_NACTIVE] = total.y; plan[PLAN_NPASS] = total.z; plan[PLAN_STATUS] = 0;
    }
}

// shared memory of dispatch_small_body for a block of `warps` warps: hist [warps][e] (16-bit) + counts and offsets, e + 2 ints each
__host__ __device__ inline size_t dispatch_small_smem(int warps, int e) { return (size_t(warps) * e * 2 + 15) / 16 * 16 + size_t(2) * (e + 2) * 4; }

// ---- single block (up to 32 warps): every phase in shared memory (decode-sized batches); hist = [warps][e] ----
template <bool VOTES>
__device__ __forceinline__ void dispatch_small_body(const int * ids, int A, int e, int shared_first, int shared_tokens,
                                                    int * __restrict__ plan, unsigned short * hist) {
    const int e1 = e + 1;
    int * counts = plan + PLAN_HDR, * offsets = counts + e1, * active = offsets + e1 + 1, * perm = active + e1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int * cs = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(hist) + (size_t(nw) * e * 2 + 15) / 16 * 16), * os = cs + e + 2;
    const int chunk = ((A + nw - 1) / nw + 31) / 32 * 32;   // per warp, a multiple of 32
    const int used = (A + chunk - 1) / chunk;               // warps that have assignments: a decode step's ids fill a few of them
    const int a0 = warp * chunk;
    const int a1 = min(A, a0 + chunk);
    unsigned short * h = hist + warp * e;
    // one step a warp: its id and the lanes that share it stay in registers for the second walk
    int id1 = -1;
    unsigned peers1 = 0;
    const bool one = chunk == 32;
    if (one && warp < used) id1 = valid_id(ids, a0 + lane, a1, e);          // asked for before the counters are cleared
    if (warp < used) for (int i = lane; i < e; i += 32) h[i] = 0;
    __syncwarp();
    if (one) {
        if (warp < used) {
            peers1 = VOTES ? same_id(id1, 32 - __clz(e - 1)) : __match_any_sync(0xffffffffu, id1);
            if (id1 >= 0 && lane == __ffs(peers1) - 1) h[id1] = (unsigned short)__popc(peers1);
        }
    } else if (warp < used) {
        walk_ids<VOTES>(ids, a0, a1, e, lane, [&](int, int id, unsigned peers) {
            if (id >= 0 && lane == __ffs(peers) - 1) h[id] += (unsigned short)__popc(peers);
        });
    }
    __syncthreads();
    for (int x = threadIdx.x; x < e; x += blockDim.x) counts[x] = cs[x] = prefix_counters(hist + x, used, e);
    if (threadIdx.x == 0) { counts[e] = shared_tokens; cs[e] = shared_tokens; }
    __syncthreads();
    finish_plan(plan, cs, os, offsets, active, perm + A + shared_tokens, e1, true);
    __syncthreads();
    if (one) {
        if (id1 >= 0) perm[os[id1] + h[id1] + __popc(peers1 & ((1u << lane) - 1u))] = a0 + lane;
    } else if (warp < used) {
        walk_ids<VOTES>(ids, a0, a1, e, lane, [&](int a, int id, unsigned peers) {
            if (id >= 0) perm[os[id] + h[id] + __popc(peers & ((1u << lane) - 1u))] = a;
            __syncwarp();
            if (id >= 0 && lane == __ffs(peers) - 1) h[id] += (unsigned short)__popc(peers);
        });
    }
    for (int t = threadIdx.x; t < shared_tokens; t += blockDim.x) perm[os[e] + t] = A + shared_first + t;
}

// One block while its counters fit a block's ordinary shared memory: up to 654 experts. Beyond 4,096 ids two launches over many blocks are the
// faster form (640 experts: 640 ids 4.8 us in one block and 10.5 in two launches, 4,000 ids 10.7 and 11.0, 8,000 ids 15.7 and 11.2). Up to 619 experts
// the line stays at 8,192 ids: callers have sized their scratch by it, and two launches need some.
inline bool dispatch_small_path(int e, int A) { return A <= (e <= 619 ? 8192 : 4096) && dispatch_small_smem(32, e) <= 46 * 1024; }

}  // namespace b2
