// Routing kernels: the top-k router and the deterministic expert sort that turns
// m_indices[T, k] into per-expert row ranges and a stable permutation.
//
// The sort replaces cub::DeviceHistogram + cub::DeviceScan + the atomic-slot
// GetGroupIndex kernel of the reference (csrc/moe_kernels.h:108-127, 452-471).
// It is a counting sort in three small launches (per-chunk histograms, one scan
// block, per-chunk scatter with warp-level match ranks) or a single launch when
// the rows fit one chunk; no atomics decide the order, so the result is the
// stable order torch.where produces (test/util.py:80).
#include <mutex>

#include "common.cuh"

namespace dq {
namespace route {

constexpr int kChunk = 2048;    // rows per sort block
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kRowsPerWarp = kChunk / kSortWarps;  // 256: eight passes of 32 consecutive rows
constexpr int kMaxExperts = 1024;

__device__ __forceinline__ int bucket_of(int id, int E) { return (id >= 0 && id < E) ? id : E; }

// ---------------------------------------------------------------- pass 1: chunk histograms
__global__ void __launch_bounds__(kSortThreads) sort_hist_kernel(const int* ids, int n, int E,
                                                                 int* chunk_hist /*[chunks][E+1]*/) {
    pdl_enter();
    extern __shared__ int s_hist[];  // E+1
    for (int i = threadIdx.x; i <= E; i += kSortThreads) s_hist[i] = 0;
    __syncthreads();
    const int base = blockIdx.x * kChunk + threadIdx.x;
    int id[kChunk / kSortThreads];  // all of a thread's loads before the first use
#pragma unroll
    for (int i = 0; i < kChunk / kSortThreads; ++i) id[i] = base + i * kSortThreads < n ? ids[base + i * kSortThreads] : 0;
#pragma unroll
    for (int i = 0; i < kChunk / kSortThreads; ++i)
        if (base + i * kSortThreads < n) atomicAdd(&s_hist[bucket_of(id[i], E)], 1);  // integer counts: order-independent
    __syncthreads();
    for (int i = threadIdx.x; i <= E; i += kSortThreads) chunk_hist[size_t(blockIdx.x) * (E + 1) + i] = s_hist[i];
}

// block-wide exclusive scan of s_val[0..len) in place (len <= kMaxExperts + 1), returns the total in s_val[len]
__device__ void block_exclusive_scan(int* s_val, int len, int* s_warp_tot) {
    // each thread owns a contiguous run so that the scan is one pass
    const int nthreads = blockDim.x;
    const int per = (len + nthreads - 1) / nthreads;
    const int lo = min(threadIdx.x * per, len);
    const int hi = min(lo + per, len);
    int sum = 0;
    for (int i = lo; i < hi; ++i) sum += s_val[i];
    // exclusive scan of per-thread sums across the block
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int nw = nthreads >> 5;
        int w = lane < nw ? s_warp_tot[lane] : 0;
        int wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += v;
        }
        if (lane < nw) s_warp_tot[lane] = wi - w;
        if (lane == nw - 1) s_warp_tot[32] = wi;
    }
    __syncthreads();
    int run = s_warp_tot[warp] + incl - sum;
    for (int i = lo; i < hi; ++i) {
        const int v = s_val[i];
        s_val[i] = run;
        run += v;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_val[len] = s_warp_tot[32];
    __syncthreads();
}

// ---------------------------------------------------------------- pass 2: scan
// chunk_hist becomes, per chunk and bucket, the first destination row of that chunk's rows.
// kStaged: the whole table fits shared memory and is scanned there (coalesced in, coalesced out; walking the table
// bucket by bucket in global memory is a chain of strided round trips: 15.7 us at 64 chunks x 129 buckets).
template <bool kStaged>
__global__ void __launch_bounds__(1024) sort_scan_kernel(int* chunk_hist, int chunks, int E, int* counts,
                                                         int* offsets, int* mtile_prefix) {
    pdl_enter();
    extern __shared__ int s_hist[];  // kStaged: [chunks][E + 1]
    __shared__ int s_tot[kMaxExperts + 2];
    __shared__ int s_tiles[kMaxExperts + 2];
    __shared__ int s_warp_tot[33];
    const int total = chunks * (E + 1);
    int* tab = kStaged ? s_hist : chunk_hist;
    if constexpr (kStaged) {
        for (int i = threadIdx.x; i < total; i += blockDim.x) s_hist[i] = chunk_hist[i];
        __syncthreads();
    }
    // one warp per bucket, lanes over chunks: the chunk counters of a bucket are scanned 32 at a time
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    for (int b = warp; b <= E; b += nwarps) {
        int run = 0;
        for (int c0 = 0; c0 < chunks; c0 += 32) {
            const int c = c0 + lane;
            const int v = c < chunks ? tab[size_t(c) * (E + 1) + b] : 0;
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            if (c < chunks) tab[size_t(c) * (E + 1) + b] = run + incl - v;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) {
            s_tot[b] = run;
            s_tiles[b] = b < E ? (run + 127) / 128 : 0;
            if (b < E && counts != nullptr) counts[b] = run;
        }
    }
    __syncthreads();
    block_exclusive_scan(s_tot, E + 1, s_warp_tot);
    block_exclusive_scan(s_tiles, E + 1, s_warp_tot);
    for (int b = threadIdx.x; b <= E; b += blockDim.x) {
        offsets[b] = s_tot[b];  // offsets[E] = number of kept rows
        if (mtile_prefix != nullptr) mtile_prefix[b] = s_tiles[b];
    }
    for (int i = threadIdx.x; i < total; i += blockDim.x) chunk_hist[i] = tab[i] + s_tot[i % (E + 1)];
}

// ---------------------------------------------------------------- pass 3: scatter
// kSingle: the whole problem is one chunk; histogram, scan and scatter in one block.
template <bool kSingle>
__global__ void __launch_bounds__(kSortThreads) sort_scatter_kernel(const int* ids, int n, int E,
                                                                    const int* chunk_base, int* counts, int* offsets,
                                                                    int* mtile_prefix, int* dest_to_src,
                                                                    int* src_to_dest) {
    pdl_enter();
    extern __shared__ int s_mem[];
    // s_warp_hist[w][E+1]: rows of bucket b seen so far by warp w, then exclusive prefix over warps
    int* s_warp_hist = s_mem;
    int* s_base = s_mem + kSortWarps * (E + 1);  // [E+2] destination of the chunk's first row per bucket
    int* s_tiles = s_base + (E + 2);             // [E+2] (kSingle only)
    __shared__ int s_warp_tot[33];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kSortWarps * (E + 1); i += kSortThreads) s_warp_hist[i] = 0;
    __syncthreads();

    const int base = blockIdx.x * kChunk + warp * kRowsPerWarp;
    int* my_hist = s_warp_hist + warp * (E + 1);
    int bucket[kRowsPerWarp / 32];
    int rank[kRowsPerWarp / 32];
#pragma unroll
    for (int it = 0; it < kRowsPerWarp / 32; ++it)  // all loads before the first use
        bucket[it] = base + it * 32 + lane < n ? bucket_of(ids[base + it * 32 + lane], E) : -1;
#pragma unroll
    for (int it = 0; it < kRowsPerWarp / 32; ++it) {
        const bool live = base + it * 32 + lane < n;
        const int b = bucket[it];
        // lanes holding the same bucket, in row order
        const unsigned peers = __match_any_sync(0xffffffffu, b);
        const int before = __popc(peers & ((1u << lane) - 1u));
        int seen = 0;
        if (live) seen = my_hist[b];
        __syncwarp();
        if (live && before == 0) my_hist[b] = seen + __popc(peers);
        __syncwarp();
        rank[it] = seen + before;
    }
    __syncthreads();
    // exclusive prefix over the warps of this block, per bucket
    for (int b = threadIdx.x; b <= E; b += kSortThreads) {
        int run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const int v = s_warp_hist[w * (E + 1) + b];
            s_warp_hist[w * (E + 1) + b] = run;
            run += v;
        }
        if constexpr (kSingle) {
            s_base[b] = run;
            s_tiles[b] = b < E ? (run + 127) / 128 : 0;
            if (b < E && counts != nullptr) counts[b] = run;
        } else {
            s_base[b] = chunk_base[size_t(blockIdx.x) * (E + 1) + b];
        }
    }
    __syncthreads();
    if constexpr (kSingle) {
        block_exclusive_scan(s_base, E + 1, s_warp_tot);
        block_exclusive_scan(s_tiles, E + 1, s_warp_tot);
        for (int b = threadIdx.x; b <= E; b += kSortThreads) {
            offsets[b] = s_base[b];
            if (mtile_prefix != nullptr) mtile_prefix[b] = s_tiles[b];
        }
    }
#pragma unroll
    for (int it = 0; it < kRowsPerWarp / 32; ++it) {
        const int r = base + it * 32 + lane;
        if (r < n) {
            const int b = bucket[it];
            const int dest = s_base[b] + my_hist[b] + rank[it];
            if (b < E) {
                dest_to_src[dest] = r;
                if (src_to_dest != nullptr) src_to_dest[r] = dest;
            } else {
                dest_to_src[dest] = -1;  // dropped rows sort behind every expert
                if (src_to_dest != nullptr) src_to_dest[r] = -1;
            }
        }
    }
}

__global__ void mtile_prefix_kernel(const int* __restrict__ offsets, int E, int* __restrict__ mtile_prefix) {
    __shared__ int s_tiles[kMaxExperts + 2];
    __shared__ int s_warp_tot[33];
    for (int b = threadIdx.x; b <= E; b += blockDim.x) s_tiles[b] = b < E ? (offsets[b + 1] - offsets[b] + 127) / 128 : 0;
    __syncthreads();
    block_exclusive_scan(s_tiles, E + 1, s_warp_tot);
    for (int b = threadIdx.x; b <= E; b += blockDim.x) mtile_prefix[b] = s_tiles[b];
}

// out[r] = values[s] for the rows r of segment s, segments laid out back to back with
// counts[s] rows each (S <= kMaxExperts). Every block rebuilds the small prefix in shared memory.
__global__ void __launch_bounds__(256) segment_ids_kernel(const int* __restrict__ counts,
                                                          const int* __restrict__ values, int S,
                                                          int* __restrict__ out, int n) {
    __shared__ int s_pref[kMaxExperts + 2];
    __shared__ int s_warp_tot[33];
    for (int i = threadIdx.x; i < S; i += blockDim.x) s_pref[i] = counts[i];
    __syncthreads();
    block_exclusive_scan(s_pref, S, s_warp_tot);  // s_pref[S] = total
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        int lo = 0, hi = S;  // last segment whose start is <= r and which is not empty before r
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (s_pref[mid] <= r) lo = mid; else hi = mid;
        }
        out[r] = r < s_pref[S] ? values[lo] : -1;
    }
}

size_t sort_workspace_bytes(int n, int E) {
    const int chunks = ceil_div(n > 0 ? n : 1, kChunk);
    return align_up(size_t(chunks) * (E + 1) * sizeof(int), 256);
}

int route_sort(const int* ids, int n, int E, int* counts, int* offsets, int* mtile_prefix, int* dest_to_src,
               int* src_to_dest, void* ws, size_t ws_bytes, cudaStream_t stream) {
    DQ_CHECK(n >= 0 && E > 0 && E <= kMaxExperts);
    DQ_CHECK(offsets != nullptr);
    if (n == 0) {
        DQ_CUDA(cudaMemsetAsync(offsets, 0, (E + 1) * sizeof(int), stream));
        if (counts != nullptr) DQ_CUDA(cudaMemsetAsync(counts, 0, E * sizeof(int), stream));
        if (mtile_prefix != nullptr) DQ_CUDA(cudaMemsetAsync(mtile_prefix, 0, (E + 1) * sizeof(int), stream));
        return DQMOE_OK;
    }
    DQ_CHECK(ids != nullptr && dest_to_src != nullptr);
    const int chunks = ceil_div(n, kChunk);
    const size_t smem_scatter = (size_t(kSortWarps) * (E + 1) + 2 * (E + 2)) * sizeof(int);
    // shared-memory opt-ins are per function and per device
    constexpr int kScanSmemMax = 160 * 1024;
    static std::mutex mu;
    static bool configured[64] = {};
    int dev = 0;
    DQ_CUDA(cudaGetDevice(&dev));
    DQ_CHECK(dev >= 0 && dev < 64);
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!configured[dev]) {
            DQ_CUDA(cudaFuncSetAttribute(sort_scatter_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
            DQ_CUDA(cudaFuncSetAttribute(sort_scatter_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
            DQ_CUDA(cudaFuncSetAttribute(sort_scan_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kScanSmemMax));
            configured[dev] = true;
        }
    }
    if (chunks == 1) {
        DQ_RC(launch_pdl(sort_scatter_kernel<true>, dim3(1), kSortThreads, smem_scatter, stream, ids, n, E, nullptr, counts,
                         offsets, mtile_prefix, dest_to_src, src_to_dest));
        return DQMOE_OK;
    }
    if (ws == nullptr || ws_bytes < sort_workspace_bytes(n, E) || !is_aligned(ws, 16))
        return fail(DQMOE_ERR_WORKSPACE, __FILE__, __LINE__, "ws_bytes >= sort_workspace_bytes(n, E)",
                    "sort workspace %zu bytes, need %zu", ws_bytes, sort_workspace_bytes(n, E));
    int* chunk_hist = static_cast<int*>(ws);
    DQ_RC(launch_pdl(sort_hist_kernel, dim3(chunks), kSortThreads, (E + 1) * sizeof(int), stream, ids, n, E, chunk_hist));
    const size_t smem_scan = size_t(chunks) * (E + 1) * sizeof(int);
    if (smem_scan <= size_t(kScanSmemMax))
        DQ_RC(launch_pdl(sort_scan_kernel<true>, dim3(1), 1024, smem_scan, stream, chunk_hist, chunks, E, counts, offsets,
                         mtile_prefix));
    else
        DQ_RC(launch_pdl(sort_scan_kernel<false>, dim3(1), 1024, 0, stream, chunk_hist, chunks, E, counts, offsets,
                         mtile_prefix));
    DQ_RC(launch_pdl(sort_scatter_kernel<false>, dim3(chunks), kSortThreads, smem_scatter, stream, ids, n, E, chunk_hist,
                     counts, offsets, mtile_prefix, dest_to_src, src_to_dest));
    return DQMOE_OK;
}

// ---------------------------------------------------------------- top-k router
// One warp per token. Ranking is by logit (both scoring functions are monotonic),
// value descending then expert id ascending; weights are the selected scores
// normalised to sum 1. Output rows have `slots` >= k entries: entries k.. name the shared
// experts E, E+1, ... (every token, weight 1), which the layer then treats like routed ones.
template <int kPerLane>
__device__ __forceinline__ void topk_of_token(const float* row, int E, int k, int slots, int scoring, int lane, int* indices,
                                              float* weights) {
    float x[kPerLane];
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
        const int e = i * 32 + lane;
        x[i] = e < E ? row[e] : -INFINITY;
        m = fmaxf(m, x[i]);
    }
    m = warp_max(m);
    float sel_score = 0.0f;  // lane j keeps the j-th selected score
    int sel_idx = 0;
    float denom = 0.0f;
    uint32_t taken = 0;      // bit i: this lane's i-th expert has been selected (an expert is chosen at most once,
                             // also when fewer than k logits are above -inf)
    for (int j = 0; j < k; ++j) {
        float bv = -INFINITY;
        int bi = 0x7fffffff;
#pragma unroll
        for (int i = 0; i < kPerLane; ++i) {
            const int e = i * 32 + lane;
            if (e < E && ((taken >> i) & 1u) == 0u && (x[i] > bv || (x[i] == bv && e < bi))) {
                bv = x[i];
                bi = e;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) {
                bv = ov;
                bi = oi;
            }
        }
        // remove the winner from its owner lane
#pragma unroll
        for (int i = 0; i < kPerLane; ++i)
            if (i * 32 + lane == bi) taken |= 1u << i;
        const float score = scoring == DQMOE_SCORE_SIGMOID ? 1.0f / (1.0f + expf(-bv)) : expf(bv - m);
        denom += score;
        if (lane == j) {
            sel_score = score;
            sel_idx = bi;
        }
    }
    if (lane < k) {
        indices[lane] = sel_idx;
        weights[lane] = sel_score / denom;
    } else if (lane < slots) {
        indices[lane] = E + (lane - k);
        weights[lane] = 1.0f;
    }
}

template <int kPerLane>
__global__ void __launch_bounds__(256) route_topk_kernel(const float* logits, int T, int E, int k, int slots,
                                                         int scoring, int* indices, float* weights) {
    pdl_enter();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= T) return;
    topk_of_token<kPerLane>(logits + size_t(warp) * E, E, k, slots, scoring, threadIdx.x & 31, indices + size_t(warp) * slots,
                            weights + size_t(warp) * slots);
}

// Router and expert sort of a small call in one block: 32 warps take a token each in turn, then sort the rows they have just
// named (32 at a time, in row order; the same stable order as the kernels above).
constexpr int kRouteSortThreads = 1024;
constexpr int kRouteSortWarps = kRouteSortThreads / 32;
template <int kPerLane>
__global__ void __launch_bounds__(kRouteSortThreads) route_sort_small_kernel(const float* logits, int T, int E, int k, int slots,
                                                                             int scoring, int* indices, float* weights, int* counts,
                                                                             int* offsets, int* mtile_prefix, int* dest_to_src,
                                                                             int* src_to_dest) {
    pdl_enter();
    extern __shared__ int s_mem[];
    const int E_all = E + slots - k, n = T * slots;
    int* s_warp_hist = s_mem;                                   // [warp][E_all + 1]: rows of a bucket in the warps before
    int* s_base = s_warp_hist + kRouteSortWarps * (E_all + 1);  // [E_all + 2]
    int* s_tiles = s_base + E_all + 2;                          // [E_all + 2]
    __shared__ int s_warp_tot[33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kRouteSortWarps * (E_all + 1); i += kRouteSortThreads) s_warp_hist[i] = 0;
    for (int t = warp; t < T; t += kRouteSortWarps)
        topk_of_token<kPerLane>(logits + size_t(t) * E, E, k, slots, scoring, lane, indices + size_t(t) * slots, weights + size_t(t) * slots);
    __syncthreads();  // the block's own stores to `indices` are visible to it
    // consecutive rows per warp, 32 at a time
    const int per_warp = (n + kRouteSortThreads - 1) / kRouteSortThreads * 32;
    const int base = warp * per_warp;
    int* my_hist = s_warp_hist + warp * (E_all + 1);
    constexpr int kPasses = kChunk / kRouteSortThreads;
    int bucket[kPasses], rank[kPasses];
#pragma unroll
    for (int it = 0; it < kPasses; ++it) {
        const int r = base + it * 32 + lane;
        const bool live = it * 32 < per_warp && r < n;
        const int b = live ? bucket_of(indices[r], E_all) : -1;  // a row without a choice (NaN logits) sorts behind every expert
        const unsigned peers = __match_any_sync(0xffffffffu, b);
        const int before = __popc(peers & ((1u << lane) - 1u));
        int seen = 0;
        if (live) seen = my_hist[b];
        __syncwarp();
        if (live && before == 0) my_hist[b] = seen + __popc(peers);
        __syncwarp();
        bucket[it] = b;
        rank[it] = seen + before;
    }
    __syncthreads();
    for (int b = threadIdx.x; b <= E_all; b += kRouteSortThreads) {
        int run = 0;
        for (int w = 0; w < kRouteSortWarps; ++w) {
            const int v = s_warp_hist[w * (E_all + 1) + b];
            s_warp_hist[w * (E_all + 1) + b] = run;
            run += v;
        }
        s_base[b] = run;
        s_tiles[b] = b < E_all ? (run + 127) / 128 : 0;
        if (b < E_all) counts[b] = run;
    }
    __syncthreads();
    block_exclusive_scan(s_base, E_all + 1, s_warp_tot);
    block_exclusive_scan(s_tiles, E_all + 1, s_warp_tot);
    for (int b = threadIdx.x; b <= E_all; b += kRouteSortThreads) {
        offsets[b] = s_base[b];
        mtile_prefix[b] = s_tiles[b];
    }
#pragma unroll
    for (int it = 0; it < kPasses; ++it) {
        if (bucket[it] < 0) continue;
        const int r = base + it * 32 + lane;
        const int dest = s_base[bucket[it]] + my_hist[bucket[it]] + rank[it];
        dest_to_src[dest] = bucket[it] < E_all ? r : -1;
        src_to_dest[r] = bucket[it] < E_all ? dest : -1;
    }
}

static int check_topk(const float* logits, int T, int E, int k, int n_shared, int scoring, const int* indices, const float* weights) {
    DQ_CHECK(T >= 0 && E > 0 && E <= kMaxExperts && k > 0 && k <= 32 && k <= E);
    DQ_CHECK_FMT(n_shared >= 0 && k + n_shared <= 32 && E + n_shared <= kMaxExperts, "n_shared=%d", n_shared);
    DQ_CHECK(scoring == DQMOE_SCORE_SOFTMAX || scoring == DQMOE_SCORE_SIGMOID);
    if (T > 0) DQ_CHECK(logits != nullptr && indices != nullptr && weights != nullptr);
    return DQMOE_OK;
}

int route_topk(const float* logits, int T, int E, int k, int n_shared, int scoring, int* indices, float* weights,
               cudaStream_t stream) {
    DQ_RC(check_topk(logits, T, E, k, n_shared, scoring, indices, weights));
    const int slots = k + n_shared;
    if (T == 0) return DQMOE_OK;
    const int blocks = ceil_div(T, 8);
    if (E <= 32) DQ_RC(launch_pdl(route_topk_kernel<1>, dim3(blocks), 256, 0, stream, logits, T, E, k, slots, scoring,
                                  indices, weights));
    else if (E <= 64) DQ_RC(launch_pdl(route_topk_kernel<2>, dim3(blocks), 256, 0, stream, logits, T, E, k, slots, scoring,
                                       indices, weights));
    else if (E <= 128) DQ_RC(launch_pdl(route_topk_kernel<4>, dim3(blocks), 256, 0, stream, logits, T, E, k, slots, scoring,
                                        indices, weights));
    else if (E <= 256) DQ_RC(launch_pdl(route_topk_kernel<8>, dim3(blocks), 256, 0, stream, logits, T, E, k, slots, scoring,
                                        indices, weights));
    else if (E <= 512) DQ_RC(launch_pdl(route_topk_kernel<16>, dim3(blocks), 256, 0, stream, logits, T, E, k, slots, scoring,
                                        indices, weights));
    else DQ_RC(launch_pdl(route_topk_kernel<32>, dim3(blocks), 256, 0, stream, logits, T, E, k, slots, scoring, indices,
                          weights));
    return DQMOE_OK;
}

// Router, then the expert sort of the rows it names (E routed experts, n_shared shared ones behind them).
// In one launch while a warp has at most two tokens, and up to 192 choices (T k): it saves a launch, but a warp takes its T / 32 tokens one
// choice after the other. Two kernels / one, us per MoE block: 10 choices (H 1024, I 2048, E 8, k 2) 30.4 / 29.6, 64 tokens 30.9 / 27.9,
// 96 30.8 / 30.1, 128 30.7 / 32.5; H 2048, I 3072, E 3, k 1 64 tokens 31.1 / 31.1, 96 33.7 / 35.7, 192 42.1 / 46.3; H 2048, I 1408, E 64,
// k 6 32 tokens 105.7 / 105.7, 43 105.6 / 108.3; 768 choices (H 7168, I 2048, E 33) 277 / 285.
constexpr int kRouteSortTokens = 64, kRouteSortChoices = 192;
int route_and_sort(const float* logits, int T, int E, int k, int n_shared, int scoring, int* indices, float* weights, int* counts,
                   int* offsets, int* mtile_prefix, int* dest_to_src, int* src_to_dest, void* ws, size_t ws_bytes, cudaStream_t stream) {
    const int slots = k + n_shared, E_all = E + n_shared;
    const size_t smem = (size_t(kRouteSortWarps) * (E_all + 1) + 2 * (E_all + 2)) * sizeof(int);
    if (T == 0 || T > kRouteSortTokens || int64_t(T) * k > kRouteSortChoices || int64_t(T) * slots > kChunk || E > 256 || smem > 48 * 1024) {
        DQ_RC(route_topk(logits, T, E, k, n_shared, scoring, indices, weights, stream));
        return route_sort(indices, T * slots, E_all, counts, offsets, mtile_prefix, dest_to_src, src_to_dest, ws, ws_bytes, stream);
    }
    DQ_RC(check_topk(logits, T, E, k, n_shared, scoring, indices, weights));
    auto kern = E <= 32 ? route_sort_small_kernel<1> : E <= 64 ? route_sort_small_kernel<2> : E <= 128 ? route_sort_small_kernel<4>
                                                                                                       : route_sort_small_kernel<8>;
    DQ_RC(launch_pdl(kern, dim3(1), kRouteSortThreads, smem, stream, logits, T, E, k, slots, scoring, indices, weights, counts, offsets,
                     mtile_prefix, dest_to_src, src_to_dest));
    return DQMOE_OK;
}

}  // namespace route
}  // namespace dq

extern "C" {

size_t dqmoe_route_sort_workspace_bytes(int n, int E) { return dq::route::sort_workspace_bytes(n, E); }

int dqmoe_route_sort(const int32_t* expert_ids, int n, int E, int32_t* counts, int32_t* offsets,
                     int32_t* dest_to_src, int32_t* src_to_dest, void* workspace, size_t workspace_bytes,
                     dqmoe_stream_t stream) {
    return dq::route::route_sort(expert_ids, n, E, counts, offsets, nullptr, dest_to_src, src_to_dest, workspace,
                                 workspace_bytes, static_cast<cudaStream_t>(stream));
}

int dqmoe_mtile_prefix(const int32_t* offsets, int E, int32_t* mtile_prefix, dqmoe_stream_t stream) {
    DQ_CHECK(E > 0 && E <= dq::route::kMaxExperts && offsets != nullptr && mtile_prefix != nullptr);
    dq::route::mtile_prefix_kernel<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(offsets, E, mtile_prefix);
    DQ_LAUNCH_CHECK();
    return DQMOE_OK;
}

int dqmoe_segment_ids(const int32_t* counts, const int32_t* values, int S, int32_t* out, int n,
                      dqmoe_stream_t stream) {
    DQ_CHECK(S > 0 && S <= dq::route::kMaxExperts && n >= 0);
    if (n == 0) return DQMOE_OK;
    DQ_CHECK(counts != nullptr && values != nullptr && out != nullptr);
    const int blocks = dq::ceil_div(n, 256) < dq::sm_count() * 4 ? dq::ceil_div(n, 256) : dq::sm_count() * 4;
    dq::route::segment_ids_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(counts, values, S, out, n);
    DQ_LAUNCH_CHECK();
    return DQMOE_OK;
}

int dqmoe_route_topk(const float* logits, int T, int E, int k, int scoring, int32_t* indices, float* weights,
                     dqmoe_stream_t stream) {
    return dq::route::route_topk(logits, T, E, k, 0, scoring, indices, weights, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
