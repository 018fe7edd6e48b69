// Token -> expert dispatch on the device: per-expert histogram, exclusive prefix sum, stable permutation.
// The permutation lists, expert by expert, the assignment indices in ascending order: the order the reference's
// host builder fill_pass_lists (src/models/qwen/qwen4exp/prefill_plan.hpp:62-76) and its single-block
// dedup_maps_k (src/experts/moe.cu:453-483) produce, without the O(A^2) walk of the latter or the atomics of group_k
// (src/experts/moe.cu:168-176), whose list order is not deterministic.
//
// Method: the assignments are cut into chunks that one warp walks 32 at a time. A vote per bit of the ids finds the lanes
// holding the same expert, so each distinct expert of a step has one leader lane that bumps the chunk's private
// counter by the group size (no atomics); an exclusive scan over (expert, chunk) turns the counters into each
// chunk's first output slot per expert; a second walk in the same order hands every assignment
// base + (number of lower lanes with the same expert), which keeps ascending order inside an expert.
#include <algorithm>

#include "common.cuh"
#include "dispatch.cuh"

namespace b2 {
namespace {

constexpr int CHUNK = 256;   // assignments per warp-chunk on the multi-block path with counters in global memory
constexpr int WALK_WARPS = 8, WALK_THREADS = WALK_WARPS * 32, WALK_MAX_BLOCKS = 148;

__global__ void dispatch_small_k(const int * ids, int A, int e, int shared_first, int shared_tokens, int * __restrict__ plan) {
    extern __shared__ unsigned short hist[];       // [32 warps][e]
    grid_release();
    grid_wait();
    dispatch_small_body<true>(ids, A, e, shared_first, shared_tokens, plan, hist);
}

// ---- multi-block path: two launches. Every block counts its segment of the assignments in shared memory, a private row of
// counters per warp, and leaves the sums as its row of `rows` [blocks][e]; then every block adds up the rows (all of them: the
// experts' totals and offsets; those below its own: its first slot per expert), counts its segment again and places it. Nothing
// is cleared, no block waits for another, and the sums over the rows are a few batches of independent loads. Bound by latency:
// the launch, one load of the ids, the batches of rows, the plan's header and pass list in
// block 0. Measured on the device: 41,000 ids on 512 experts 41 us + a memset -> 20 us, 65,536 on 128 experts 15 us.
struct WalkArgs { const int * ids; int A, e, seg, shared_first, shared_tokens; int * rows, * plan; };
__host__ __device__ inline int row_parts(int e) { return e >= WALK_THREADS ? 1 : WALK_THREADS / e; }
// hist [warps][e], totals and lower sums [row_parts][e], counts and offsets of e + 2 each
inline size_t walk_smem(int e) { return (size_t(WALK_WARPS) * e + size_t(2) * row_parts(e) * e + size_t(2) * (e + 2)) * sizeof(int); }

__device__ __forceinline__ void count_segment(const WalkArgs & p, int a0, int a1, int * hist, int lane, int warp) {
    for (int i = threadIdx.x; i < WALK_WARPS * p.e; i += WALK_THREADS) hist[i] = 0;
    __syncthreads();
    walk_ids<true>(p.ids, a0, a1, p.e, lane, [&](int, int id, unsigned peers) {
        if (id >= 0 && lane == __ffs(peers) - 1) hist[warp * p.e + id] += __popc(peers);
    });
    __syncthreads();
}
__global__ void __launch_bounds__(WALK_THREADS) dispatch_count_k(const WalkArgs p) {
    extern __shared__ int walk_mem[];
    grid_release();
    grid_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int a0 = blockIdx.x * p.seg * WALK_WARPS + warp * p.seg;
    count_segment(p, a0, min(p.A, a0 + p.seg), walk_mem, lane, warp);
    for (int x = threadIdx.x; x < p.e; x += WALK_THREADS) {
        int sum = 0;
#pragma unroll
        for (int w = 0; w < WALK_WARPS; ++w) sum += walk_mem[w * p.e + x];
        p.rows[size_t(blockIdx.x) * p.e + x] = sum;
    }
}
__global__ void __launch_bounds__(WALK_THREADS) dispatch_place_k(const WalkArgs p) {
    extern __shared__ int walk_mem[];
    grid_release();
    grid_wait();
    const int e = p.e, e1 = e + 1, parts = row_parts(e), blocks = gridDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int * hist = walk_mem, * total = hist + WALK_WARPS * e, * lower = total + parts * e, * cs = lower + parts * e, * os = cs + e + 2;
    int * counts = p.plan + PLAN_HDR, * offsets = counts + e1, * active = offsets + e1 + 1, * perm = active + e1;
    for (int i = threadIdx.x; i < parts * e; i += WALK_THREADS) {
        const int x = i % e, part = i / e, per = (blocks + parts - 1) / parts, r1 = min(blocks, (part + 1) * per);
        int sum = 0, below = 0;
        for (int r = part * per; r < r1; r += 16) {
            int v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = r + j < r1 ? p.rows[size_t(r + j) * e + x] : 0;
#pragma unroll
            for (int j = 0; j < 16; ++j) { sum += v[j]; below += r + j < int(blockIdx.x) ? v[j] : 0; }
        }
        total[i] = sum;
        lower[i] = below;
    }
    const int a0 = blockIdx.x * p.seg * WALK_WARPS + warp * p.seg, a1 = min(p.A, a0 + p.seg);
    count_segment(p, a0, a1, hist, lane, warp);
    for (int x = threadIdx.x; x < e; x += WALK_THREADS) {
        int sum = 0, below = 0;
        for (int q = 0; q < parts; ++q) { sum += total[q * e + x]; below += lower[q * e + x]; }
        cs[x] = sum;
        lower[x] = below;
        prefix_counters(hist + x, WALK_WARPS, e);
        if (blockIdx.x == 0) counts[x] = sum;
    }
    if (threadIdx.x == 0) {
        cs[e] = p.shared_tokens;
        if (blockIdx.x == 0) counts[e] = p.shared_tokens;
    }
    __syncthreads();
    finish_plan(p.plan, cs, os, offsets, active, perm + p.A + p.shared_tokens, e1, blockIdx.x == 0);
    __syncthreads();
    int * h = hist + warp * e;
    walk_ids<true>(p.ids, a0, a1, e, lane, [&](int a, int id, unsigned peers) {
        if (id >= 0) perm[os[id] + lower[id] + h[id] + __popc(peers & ((1u << lane) - 1u))] = a;
        __syncwarp();
        if (id >= 0 && lane == __ffs(peers) - 1) h[id] += __popc(peers);
    });
    for (int t = blockIdx.x * WALK_THREADS + threadIdx.x; t < p.shared_tokens; t += blocks * WALK_THREADS) perm[os[e] + t] = p.A + p.shared_first + t;
}
// Assignments per warp: 128 (four steps; a block of eight warps takes 1,024) while that makes at most a block per SM, and
// beyond that what a block per SM leaves, since every block reads every row.
inline int walk_seg(int A) { return std::max(128, (ceil_div(A, WALK_MAX_BLOCKS * WALK_WARPS) + 31) / 32 * 32); }
inline int walk_blocks(int A) { return ceil_div(A, walk_seg(A) * WALK_WARPS); }         // at most WALK_MAX_BLOCKS
// the counters have to fit a block's ordinary shared memory: up to 981 experts
inline bool walk_path(int e) { return walk_smem(e) <= 46 * 1024; }

// ---- more experts than that: chunk counters in global scratch [chunks][e] ----
__global__ void dispatch_hist_k(const int * __restrict__ ids, int A, int e, int * __restrict__ hist) {
    const int lane = threadIdx.x & 31, chunk = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int a0 = chunk * CHUNK;
    if (a0 >= A) return;
    int * h = hist + size_t(chunk) * e;
    for (int a = a0 + lane; a - lane < min(A, a0 + CHUNK); a += 32) {
        const int id = valid_id(ids, a, A, e);
        const unsigned peers = __match_any_sync(0xffffffffu, id);
        if (id >= 0 && lane == __ffs(peers) - 1) h[id] += __popc(peers);
        __syncwarp();
    }
}
__global__ void dispatch_scan_k(int * __restrict__ hist, int chunks, int e, int A, int shared_tokens, int * __restrict__ plan) {
    const int e1 = e + 1;
    int * counts = plan + PLAN_HDR, * offsets = counts + e1, * active = offsets + e1 + 1;
    for (int x = threadIdx.x; x < e; x += blockDim.x)
        counts[x] = prefix_counters(hist + x, chunks, e);
    if (threadIdx.x == 0) counts[e] = shared_tokens;
    __syncthreads();
    finish_plan(plan, counts, offsets, offsets, active, active + e1 + A + shared_tokens, e1, true);
}
__global__ void dispatch_scatter_k(const int * __restrict__ ids, int A, int e, int shared_first, int shared_tokens, int * __restrict__ hist,
                                   int * __restrict__ plan) {
    const int e1 = e + 1;
    const int * offsets = plan + PLAN_HDR + e1;
    int * perm = plan + PLAN_HDR + e1 + e1 + 1 + e1;
    const int lane = threadIdx.x & 31, chunk = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int a0 = chunk * CHUNK;
    if (blockIdx.x == 0)
        for (int t = threadIdx.x; t < shared_tokens; t += blockDim.x) perm[offsets[e] + t] = A + shared_first + t;
    if (a0 >= A) return;
    int * h = hist + size_t(chunk) * e;
    for (int a = a0 + lane; a - lane < min(A, a0 + CHUNK); a += 32) {
        const int id = valid_id(ids, a, A, e);
        const unsigned peers = __match_any_sync(0xffffffffu, id);
        if (id >= 0) perm[offsets[id] + h[id] + __popc(peers & ((1u << lane) - 1u))] = a;
        __syncwarp();
        if (id >= 0 && lane == __ffs(peers) - 1) h[id] += __popc(peers);
        __syncwarp();
    }
}

__global__ void plan_to_groups_k(const int * __restrict__ plan, int n, int e, int * __restrict__ counts, int * __restrict__ groups) {
    const int e1 = e + 1;
    const int * pc = plan + PLAN_HDR, * offsets = pc + e1, * perm = offsets + e1 + 1 + e1;
    const int x = blockIdx.x;
    if (threadIdx.x == 0) counts[x] = pc[x];
    for (int j = threadIdx.x; j < pc[x]; j += blockDim.x) groups[size_t(x) * n + j] = perm[offsets[x] + j];
}

inline bool small_path(int e, int A) { return dispatch_small_path(e, A); }

}  // namespace
}  // namespace b2

using namespace b2;

extern "C" B2MOE_API int64_t b2moe_plan_ints(int32_t experts, int32_t assignments, int32_t shared_tokens) {
    if (experts <= 0 || assignments < 0 || shared_tokens < 0) return 0;
    const int64_t e1 = int64_t(experts) + 1;
    return PLAN_HDR + e1 + (e1 + 1) + e1 + assignments + shared_tokens + (e1 + 1);
}
extern "C" B2MOE_API void b2moe_plan_view_of(int32_t experts, int32_t assignments, int32_t shared_tokens, b2moe_plan_view * v) {
    const int64_t e1 = int64_t(experts) + 1;
    v->counts = PLAN_HDR;
    v->offsets = v->counts + e1;
    v->active = v->offsets + e1 + 1;
    v->perm = v->active + e1;
    v->passes = v->perm + assignments + shared_tokens;
    v->total = v->passes + e1 + 1;
}
extern "C" B2MOE_API size_t b2moe_dispatch_workspace_bytes(int32_t experts, int32_t assignments) {
    if (experts <= 0 || assignments < 0) return 0;
    if (small_path(experts, assignments)) return 16;
    // a size that grows with the assignments, so that scratch for the largest batch serves every smaller one: the number of blocks does
    // not (151,552 ids take 148 blocks, one more 119)
    const int rows = walk_path(experts) ? std::min(ceil_div(assignments, 128 * WALK_WARPS), WALK_MAX_BLOCKS) : ceil_div(assignments, CHUNK);
    return align_up(size_t(rows) * experts * sizeof(int), 16);
}

extern "C" B2MOE_API int32_t b2moe_dispatch_range(const int32_t * ids, int32_t n, int32_t topk, int32_t experts, int32_t shared_first,
                                        int32_t shared_count, int32_t * plan, void * workspace, size_t workspace_bytes,
                                        b2moe_stream stream) {
    if (n <= 0 || topk <= 0 || experts <= 0 || shared_first < 0 || shared_count < 0 || shared_first + shared_count > n) return B2MOE_ERR_SHAPE;
    if ((long long)n * topk > 0x3fffffffLL) return B2MOE_ERR_SHAPE;
    if (!ids || !plan) return B2MOE_ERR_NULL;
    const int A = n * topk;
    cudaStream_t s = as_stream(stream);
    if (small_path(experts, A)) {
        launch_overlapped(dispatch_small_k, dim3(1), dim3(1024), dispatch_small_smem(32, experts), s, ids, A, experts, shared_first, shared_count, plan);
        return launch_status();
    }
    const size_t need = b2moe_dispatch_workspace_bytes(experts, A);
    if (!workspace) return B2MOE_ERR_NULL;
    if (workspace_bytes < need) return B2MOE_ERR_WORKSPACE;
    int * hist = static_cast<int *>(workspace);
    if (walk_path(experts)) {
        const WalkArgs w{ids, A, experts, walk_seg(A), shared_first, shared_count, hist, plan};
        launch_overlapped(dispatch_count_k, dim3(walk_blocks(A)), dim3(WALK_THREADS), walk_smem(experts), s, w);
        launch_overlapped(dispatch_place_k, dim3(walk_blocks(A)), dim3(WALK_THREADS), walk_smem(experts), s, w);
        return launch_status();
    }
    const int chunks = ceil_div(A, CHUNK);
    if (cudaMemsetAsync(hist, 0, size_t(chunks) * experts * sizeof(int), s) != cudaSuccess) return B2MOE_ERR_CUDA;
    dispatch_hist_k<<<ceil_div(chunks, 8), 256, 0, s>>>(ids, A, experts, hist);
    dispatch_scan_k<<<1, 1024, 0, s>>>(hist, chunks, experts, A, shared_count, plan);
    dispatch_scatter_k<<<ceil_div(chunks, 8), 256, 0, s>>>(ids, A, experts, shared_first, shared_count, hist, plan);
    return launch_status();
}

extern "C" B2MOE_API int32_t b2moe_dispatch(const int32_t * ids, int32_t n, int32_t topk, int32_t experts, int32_t shared_tokens,
                                  int32_t * plan, void * workspace, size_t workspace_bytes, b2moe_stream stream) {
    if (shared_tokens != 0 && shared_tokens != n) return B2MOE_ERR_SHAPE;
    return b2moe_dispatch_range(ids, n, topk, experts, 0, shared_tokens, plan, workspace, workspace_bytes, stream);
}

extern "C" B2MOE_API int32_t b2moe_plan_to_groups(const int32_t * plan, int32_t n, int32_t topk, int32_t experts, int32_t * counts,
                                        int32_t * groups, b2moe_stream stream) {
    if (n <= 0 || topk <= 0 || experts <= 0) return B2MOE_ERR_SHAPE;
    if (!plan || !counts || !groups) return B2MOE_ERR_NULL;
    plan_to_groups_k<<<experts, 128, 0, as_stream(stream)>>>(plan, n, experts, counts, groups);
    return launch_status();
}
