// Streaming row kernels around the grouped GEMM: activations and their scales
// into expert order (by token in the layer, by sorted row as stand-alone
// operators), also fused with 1x128 FP8 quantisation, the scatter back to slot
// order and the weighted combine over the k slots of a token. All are HBM-bound:
// one warp per row or strip of a row, 16-byte accesses, a grid that is a
// multiple of the SM count.
//
// Replaces expandInputRowsGatherKernel, expandInputScale{,Block}GatherKernel and
// finalizeScatterKernel of the reference (csrc/moe_kernels.h:487-620).
#include "common.cuh"

namespace dq {
namespace permute {

constexpr int kThreads = 256;
constexpr int kWarpsPerBlock = kThreads / 32;

static int grid_for_rows(int64_t rows) {
    const int64_t want = (rows + kWarpsPerBlock - 1) / kWarpsPerBlock;
    const int64_t cap = int64_t(sm_count()) * 8;
    return int(want < cap ? (want > 0 ? want : 1) : cap);
}

__device__ __forceinline__ void copy_row16(const uint8_t* src, uint8_t* dst, int vecs,
                                           int lane) {
    int i = lane;
    for (; i + 96 < vecs; i += 128) {
        const Vec16 a = ld_stream16(src + size_t(i) * 16);
        const Vec16 b = ld_stream16(src + size_t(i + 32) * 16);
        const Vec16 c = ld_stream16(src + size_t(i + 64) * 16);
        const Vec16 d = ld_stream16(src + size_t(i + 96) * 16);
        st16(dst + size_t(i) * 16, a);
        st16(dst + size_t(i + 32) * 16, b);
        st16(dst + size_t(i + 64) * 16, c);
        st16(dst + size_t(i + 96) * 16, d);
    }
    for (; i < vecs; i += 32) st16(dst + size_t(i) * 16, ld_stream16(src + size_t(i) * 16));
}

// dst[r] = src[map[r] / k]  (kGather)   or   dst[map[r]] = src[r]  (!kGather)
template <bool kGather>
__global__ void __launch_bounds__(kThreads) row_move_kernel(const uint8_t* src, uint8_t* dst, const int* map, int n,
                                                            int k, int row_vecs, const float* src_scale,
                                                            float* dst_scale, int scale_cols) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * kWarpsPerBlock;
    for (int r = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); r < n; r += warps) {
        const int m = map[r];
        if (m < 0) continue;
        const size_t s_row = kGather ? size_t(m / k) : size_t(r);
        const size_t d_row = kGather ? size_t(r) : size_t(m);
        copy_row16(src + s_row * row_vecs * 16, dst + d_row * row_vecs * 16, row_vecs, lane);
        if (scale_cols > 0) {
            for (int c = lane; c < scale_cols; c += 32) dst_scale[d_row * scale_cols + c] = src_scale[s_row * scale_cols + c];
        }
    }
}

// out[t, :] = sum_j w[t, j] * d[t, j, :]; one warp per (token, 256-column strip). HBM-bound; the slots of a token are
// fetched kSlotBatch at a time before the first is used, so that a lane has that many 16-byte loads in flight (T = 8192,
// k = 8, H = 7168: one slot after the other 246 us, batches of eight 194 us = 5.4 TB/s). The batch is k itself, at most 8: the
// registers of empty slots cost occupancy (T = 2049, k = 2, H = 4096: in batches of eight 25.9 us, of two 13.1; T = 4096, k = 5,
// H = 2048: one after the other 22.7, in batches of eight 25.6, of five 16.6). Three slots take the batch of four
// (T = 4096, H = 2880: 16.6 us, in a batch of three 17.1).
template <int kSlotBatch>
__global__ void __launch_bounds__(kThreads) finalize_weighted_kernel(const uint8_t* d, const float* w, uint8_t* out,
                                                                     int T, int k, int row_vecs) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int strips = (row_vecs + 31) / 32;
    const int64_t items = int64_t(T) * strips;
    const int64_t warps = int64_t(gridDim.x) * kWarpsPerBlock;
    for (int64_t it = int64_t(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5); it < items; it += warps) {
        const int t = int(it / strips);
        const int v = int(it % strips) * 32 + lane;
        if (v >= row_vecs) continue;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int j0 = 0; j0 < k; j0 += kSlotBatch) {
            float wj[kSlotBatch];
            Vec16 x[kSlotBatch];
#pragma unroll
            for (int u = 0; u < kSlotBatch; ++u) wj[u] = j0 + u < k ? w[size_t(t) * k + j0 + u] : 0.0f;
#pragma unroll
            for (int u = 0; u < kSlotBatch; ++u)
                if (wj[u] != 0.0f) x[u] = ld_stream16(d + ((size_t(t) * k + j0 + u) * row_vecs + v) * 16);
#pragma unroll
            for (int u = 0; u < kSlotBatch; ++u) {
                if (wj[u] == 0.0f) continue;  // a dropped slot's row is never written
                acc[0] = fmaf(wj[u], bf16_lo(x[u].x), acc[0]);
                acc[1] = fmaf(wj[u], bf16_hi(x[u].x), acc[1]);
                acc[2] = fmaf(wj[u], bf16_lo(x[u].y), acc[2]);
                acc[3] = fmaf(wj[u], bf16_hi(x[u].y), acc[3]);
                acc[4] = fmaf(wj[u], bf16_lo(x[u].z), acc[4]);
                acc[5] = fmaf(wj[u], bf16_hi(x[u].z), acc[5]);
                acc[6] = fmaf(wj[u], bf16_lo(x[u].w), acc[6]);
                acc[7] = fmaf(wj[u], bf16_hi(x[u].w), acc[7]);
            }
        }
        Vec16 o{pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                pack_bf16x2(acc[6], acc[7])};
        st16(out + (size_t(t) * row_vecs + v) * 16, o);
    }
}

// The layer's way into expert order: token t's row goes to rows src_to_dest[t*k + j] of the sorted matrix (negative: a
// dropped slot). One warp per (token, strip of 128 16-byte vectors); a token is read - and in the quantising form
// converted - once for its k copies, where the gathers above and below read it k times (HBM-bound: k + 1 rows of traffic
// per token, the k writes dominating. It also clears the amax words fc1 collects into, one per row or one in all, which
// saves a memset between two kernels. 8192 tokens of 7168, k = 8, quantising: gather 353 us, scatter 111 us = 5.3 TB/s;
// 16384 bf16 rows of 2880, k = 3: 102 / 62 us; 16384 e4m3 rows of 2048, k = 8: 82 / 50 us).
__device__ __forceinline__ int slot_dest(const int* src_to_dest, int t, int k, int j0, int lane) {
    if (src_to_dest == nullptr) return t;  // rows stay where they are (k = 1)
    return j0 + lane < k ? src_to_dest[size_t(t) * k + j0 + lane] : -1;
}

__global__ void __launch_bounds__(kThreads) scatter_rows_kernel(const uint8_t* src, uint8_t* dst,
                                                                const int* src_to_dest, int T, int k, int row_vecs,
                                                                const float* src_scale, float* dst_scale,
                                                                int scale_cols, float* scale_t, int n_pad, float* amax,
                                                                int amax_per_row) {
    pdl_wait();
    pdl_launch();  // after the wait: the grouped GEMM behind relies on the sort before this kernel being complete
    const int lane = threadIdx.x & 31;
    if (amax != nullptr && !amax_per_row && blockIdx.x == 0 && threadIdx.x == 0) amax[0] = 0.0f;
    const int strips = (row_vecs + 127) / 128;
    const int64_t items = int64_t(T) * strips;
    const int64_t warps = int64_t(gridDim.x) * kWarpsPerBlock;
    for (int64_t it = int64_t(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5); it < items; it += warps) {
        const int t = int(it / strips);
        const int strip = int(it % strips);
        const int v0 = strip * 128 + lane;
        Vec16 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v0 + 32 * u < row_vecs) x[u] = ld_stream16(src + (size_t(t) * row_vecs + v0 + 32 * u) * 16);
        for (int j0 = 0; j0 < k; j0 += 32) {
            const int mine = slot_dest(src_to_dest, t, k, j0, lane);
            const int jn = min(32, k - j0);
            for (int j = 0; j < jn; ++j) {
                const int r = __shfl_sync(0xffffffffu, mine, j);
                if (r < 0) continue;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (v0 + 32 * u < row_vecs) st16(dst + (size_t(r) * row_vecs + v0 + 32 * u) * 16, x[u]);
                if (amax_per_row && strip == 0 && lane == 0) amax[r] = 0.0f;
                if (strip == 0)
                    for (int c = lane; c < scale_cols; c += 32) {
                        const float sf = src_scale[size_t(t) * scale_cols + c];
                        dst_scale[size_t(r) * scale_cols + c] = sf;
                        if (scale_t != nullptr) scale_t[size_t(c) * n_pad + r] = sf;
                    }
            }
        }
    }
}

// The same with 1x128 FP8 quantisation of the bf16 row on the way: a lane owns 16 consecutive columns per step, so a
// 128-column group is 8 lanes; two steps of 512 columns per strip. cols is a multiple of 16.
__global__ void __launch_bounds__(kThreads) scatter_quant_1x128_kernel(const uint8_t* x, int T, int k, int cols,
                                                                       const int* src_to_dest, uint8_t* q, float* scale,
                                                                       float* scale_t, int n_pad) {
    pdl_wait();
    pdl_launch();  // after the wait: the grouped GEMM behind relies on the sort before this kernel being complete
    const int lane = threadIdx.x & 31;
    const int groups = (cols + 127) / 128;
    const int strips = (cols + 1023) / 1024;
    const int64_t items = int64_t(T) * strips;
    const int64_t warps = int64_t(gridDim.x) * kWarpsPerBlock;
    for (int64_t it = int64_t(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5); it < items; it += warps) {
        const int t = int(it / strips);
        const int c0 = int(it % strips) * 1024 + lane * 16;
        Vec16 raw[2][2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const uint8_t* xr = x + (size_t(t) * cols + c0 + 512 * s) * 2;
#pragma unroll
            for (int u = 0; u < 2; ++u) raw[s][u] = c0 + 512 * s < cols ? ld_stream16(xr + 16 * u) : Vec16{0, 0, 0, 0};
        }
        Vec16 o[2];
        float sf[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const uint32_t w[8] = {raw[s][0].x, raw[s][0].y, raw[s][0].z, raw[s][0].w,
                                   raw[s][1].x, raw[s][1].y, raw[s][1].z, raw[s][1].w};
            float amax = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fmaxf(fabsf(bf16_lo(w[i])), fabsf(bf16_hi(w[i]))));
#pragma unroll
            for (int d = 4; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
            sf[s] = scale_from_amax(amax);
            const float inv = inv_scale(sf[s]);
            uint32_t b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                b[i] = f2e4m3x4(bf16_lo(w[2 * i]) * inv, bf16_hi(w[2 * i]) * inv, bf16_lo(w[2 * i + 1]) * inv, bf16_hi(w[2 * i + 1]) * inv);
            o[s] = Vec16{b[0], b[1], b[2], b[3]};
        }
        for (int j0 = 0; j0 < k; j0 += 32) {
            const int mine = slot_dest(src_to_dest, t, k, j0, lane);
            const int jn = min(32, k - j0);
            for (int j = 0; j < jn; ++j) {
                const int r = __shfl_sync(0xffffffffu, mine, j);
                if (r < 0) continue;
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int c = c0 + 512 * s;
                    if (c < cols) {
                        st16(q + size_t(r) * cols + c, o[s]);
                        if ((lane & 7) == 0) {
                            scale[size_t(r) * groups + (c >> 7)] = sf[s];
                            if (scale_t != nullptr) scale_t[size_t(c >> 7) * n_pad + r] = sf[s];
                        }
                    }
                }
            }
        }
    }
}

// q[r, :], scale[r, :] = 1x128 FP8 quantisation of bf16 row map[r] / k (map == nullptr: row r).
// One warp per row; a lane owns 8 consecutive columns, so a 128-column group is 16 lanes.
__global__ void __launch_bounds__(kThreads) quant_1x128_kernel(const uint8_t* x, int64_t rows, int cols, int k,
                                                               const int* map, uint8_t* q, float* scale) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int groups = (cols + 127) / 128;
    const int64_t warps = int64_t(gridDim.x) * kWarpsPerBlock;
    for (int64_t r = int64_t(blockIdx.x) * kWarpsPerBlock + (threadIdx.x >> 5); r < rows; r += warps) {
        int64_t s_row = r;
        if (map != nullptr) {
            const int m = map[r];
            if (m < 0) continue;
            s_row = m / k;
        }
        const uint8_t* xr = x + size_t(s_row) * cols * 2;
        uint8_t* qr = q + size_t(r) * cols;
        for (int c0 = 0; c0 < cols; c0 += 256) {
            const int c = c0 + lane * 8;
            float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (c < cols) {
                const Vec16 raw = ld_stream16(xr + size_t(c) * 2);
                v[0] = bf16_lo(raw.x); v[1] = bf16_hi(raw.x); v[2] = bf16_lo(raw.y); v[3] = bf16_hi(raw.y);
                v[4] = bf16_lo(raw.z); v[5] = bf16_hi(raw.z); v[6] = bf16_lo(raw.w); v[7] = bf16_hi(raw.w);
            }
            float amax = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
            // reduce over the 16 lanes of this 128-column group
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            const float sf = scale_from_amax(amax);
            const float inv = inv_scale(sf);
            if (c < cols) {
                uint2 o;
                o.x = f2e4m3x4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv);
                o.y = f2e4m3x4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv);
                *reinterpret_cast<uint2*>(qr + c) = o;
                if ((lane & 15) == 0) scale[size_t(r) * groups + (c >> 7)] = sf;
            }
        }
    }
}

// Block scales a second time by tile, for the grouped GEMM, which then fetches the 128 scales of a row tile and K block in
// one piece: out[tile][c][r] = scale[first row of the tile + r][c], every expert starting a new 128-row tile. One block per
// tile and 32 columns, transposed through shared memory. (Written by the scatter itself, four bytes at a time, the same
// matrix cost 56 us at 65536 rows x 56 columns; here ~15 us.)
__global__ void __launch_bounds__(kThreads) scale_tiles_kernel(const float* scale, int cols, const int* offsets,
                                                               const int* mtile_prefix, int E, float* out) {
    pdl_enter();
    __shared__ float s[128][33];
    const int chunks = (cols + 31) / 32;
    const int total = mtile_prefix[E] * chunks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int it = blockIdx.x; it < total; it += gridDim.x) {
        const int tile = it / chunks, c0 = (it % chunks) * 32;
        int lo = 0, hi = E;  // expert of the tile: last e with mtile_prefix[e] <= tile
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (mtile_prefix[mid] <= tile) lo = mid; else hi = mid;
        }
        const int row0 = offsets[lo] + (tile - mtile_prefix[lo]) * 128;
        const int rows = min(128, offsets[lo + 1] - row0);
#pragma unroll 4
        for (int r = warp; r < 128; r += kWarpsPerBlock)
            s[r][lane] = r < rows && c0 + lane < cols ? scale[size_t(row0 + r) * cols + c0 + lane] : 0.0f;
        __syncthreads();
        const int r = threadIdx.x & 127;
#pragma unroll 4
        for (int c = threadIdx.x >> 7; c < 32; c += kThreads / 128)
            if (c0 + c < cols) out[(size_t(tile) * cols + c0 + c) * 128 + r] = s[r][c];
        __syncthreads();
    }
}

// Arguments have been checked by the layer (layer.cu).
int scale_tiles(const float* scale, int n, int cols, const int* offsets, const int* mtile_prefix, int E, float* out,
                cudaStream_t stream) {
    const int64_t blocks = (int64_t(ceil_div(n, 128)) + (E < n ? E : n)) * ceil_div(cols, 32);
    const int64_t cap = int64_t(sm_count()) * 8;
    DQ_RC(launch_pdl(scale_tiles_kernel, dim3(unsigned(blocks < cap ? blocks : cap)), kThreads, 0, stream, scale, cols, offsets,
                     mtile_prefix, E, out));
    return DQMOE_OK;
}
int scatter_rows(const void* src, size_t row_bytes, int T, int k, const int* src_to_dest, void* dst, const float* src_scale,
                 int scale_cols, float* dst_scale, float* scale_t, int n_pad, float* amax, int amax_per_row, cudaStream_t stream) {
    const int row_vecs = int(row_bytes / 16);
    DQ_CHECK(is_aligned(src, 16) && is_aligned(dst, 16));
    DQ_RC(launch_pdl(scatter_rows_kernel, dim3(grid_for_rows(int64_t(T) * ceil_div(row_vecs, 128))), kThreads, 0, stream,
                     static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), src_to_dest, T, k, row_vecs, src_scale,
                     dst_scale, scale_cols, scale_t, n_pad, amax, amax_per_row));
    return DQMOE_OK;
}
int scatter_quant_1x128(const void* x_bf16, int T, int k, int H, const int* src_to_dest, void* q, float* scale, float* scale_t, int n_pad,
                        cudaStream_t stream) {
    DQ_CHECK(is_aligned(x_bf16, 16) && is_aligned(q, 16) && H % 16 == 0);
    DQ_RC(launch_pdl(scatter_quant_1x128_kernel, dim3(grid_for_rows(int64_t(T) * ceil_div(H, 1024))), kThreads, 0, stream,
                     static_cast<const uint8_t*>(x_bf16), T, k, H, src_to_dest, static_cast<uint8_t*>(q), scale, scale_t, n_pad));
    return DQMOE_OK;
}

}  // namespace permute
}  // namespace dq

using namespace dq;

extern "C" {

int dqmoe_permute_rows(const void* src, size_t row_bytes, int k, const int32_t* dest_to_src, int n, void* dst,
                       const float* src_scale, int scale_cols, float* dst_scale, dqmoe_stream_t stream) {
    DQ_CHECK(n >= 0 && k > 0 && scale_cols >= 0);
    if (n == 0) return DQMOE_OK;
    DQ_CHECK(src != nullptr && dst != nullptr && dest_to_src != nullptr);
    DQ_CHECK_FMT(row_bytes % 16 == 0 && row_bytes > 0, "row_bytes=%zu must be a multiple of 16", row_bytes);
    DQ_CHECK(is_aligned(src, 16) && is_aligned(dst, 16));
    if (scale_cols > 0) DQ_CHECK(src_scale != nullptr && dst_scale != nullptr);
    DQ_RC(launch_pdl(permute::row_move_kernel<true>, dim3(permute::grid_for_rows(n)), permute::kThreads, 0,
                     static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst),
                     dest_to_src, n, k, int(row_bytes / 16), src_scale, dst_scale, scale_cols));
    return DQMOE_OK;
}

int dqmoe_finalize_scatter(const void* rows, size_t row_bytes, const int32_t* dest_to_src, int n, void* d,
                           dqmoe_stream_t stream) {
    DQ_CHECK(n >= 0);
    if (n == 0) return DQMOE_OK;
    DQ_CHECK(rows != nullptr && d != nullptr && dest_to_src != nullptr);
    DQ_CHECK_FMT(row_bytes % 16 == 0 && row_bytes > 0, "row_bytes=%zu must be a multiple of 16", row_bytes);
    DQ_CHECK(is_aligned(rows, 16) && is_aligned(d, 16));
    DQ_RC(launch_pdl(permute::row_move_kernel<false>, dim3(permute::grid_for_rows(n)), permute::kThreads, 0,
                     static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(rows), static_cast<uint8_t*>(d),
                     dest_to_src, n, 1, int(row_bytes / 16), nullptr, nullptr, 0));
    return DQMOE_OK;
}

int dqmoe_finalize_weighted(const void* d_bf16, const float* weights, void* out_bf16, int T, int k, int H,
                            dqmoe_stream_t stream) {
    DQ_CHECK(T >= 0 && k > 0 && H > 0);
    if (T == 0) return DQMOE_OK;
    DQ_CHECK(d_bf16 != nullptr && weights != nullptr && out_bf16 != nullptr);
    DQ_CHECK_FMT(H % 8 == 0, "H=%d must be a multiple of 8", H);
    DQ_CHECK(is_aligned(d_bf16, 16) && is_aligned(out_bf16, 16));
    const int row_vecs = H / 8;
    const int64_t items = int64_t(T) * ((row_vecs + 31) / 32);
    using Kernel = void (*)(const uint8_t*, const float*, uint8_t*, int, int, int);
    static const Kernel kernels[8] = {permute::finalize_weighted_kernel<1>, permute::finalize_weighted_kernel<2>,
                                      permute::finalize_weighted_kernel<4>, permute::finalize_weighted_kernel<4>,
                                      permute::finalize_weighted_kernel<5>, permute::finalize_weighted_kernel<6>,
                                      permute::finalize_weighted_kernel<7>, permute::finalize_weighted_kernel<8>};
    const Kernel kern = kernels[(k < 8 ? k : 8) - 1];
    DQ_RC(launch_pdl(kern, dim3(permute::grid_for_rows(items)), permute::kThreads, 0, static_cast<cudaStream_t>(stream),
                     static_cast<const uint8_t*>(d_bf16), weights, static_cast<uint8_t*>(out_bf16), T, k, row_vecs));
    return DQMOE_OK;
}

int dqmoe_quant_fp8_block_1x128(const void* x_bf16, int64_t rows, int cols, void* q, float* scale,
                                dqmoe_stream_t stream) {
    DQ_CHECK(rows >= 0 && cols > 0);
    if (rows == 0) return DQMOE_OK;
    DQ_CHECK(x_bf16 != nullptr && q != nullptr && scale != nullptr);
    DQ_CHECK_FMT(cols % 8 == 0, "cols=%d must be a multiple of 8", cols);
    DQ_CHECK(is_aligned(x_bf16, 16) && is_aligned(q, 8));
    // Strips of a row with 16 columns per lane where rows and output allow it: more loads in flight than a warp per row has
    // (row form / strips, us: 4096 x 4096 15.0 / 9.8, 100000 x 1024 81 / 54, 100000 x 528 54 / 42). Up to 512 columns half a
    // strip stays empty or more, and the row form is as fast or faster (100000 rows of 512 41.5 / 39.9, 20000 rows of 512
    // 8.3 / 8.6, 100000 rows of 256 20.9 / 36.1).
    if (cols > 512 && cols % 16 == 0 && is_aligned(q, 16) && rows < (int64_t(1) << 31))
        return permute::scatter_quant_1x128(x_bf16, int(rows), 1, cols, nullptr, q, scale, nullptr, 0, static_cast<cudaStream_t>(stream));
    DQ_RC(launch_pdl(permute::quant_1x128_kernel, dim3(permute::grid_for_rows(rows)), permute::kThreads, 0,
                     static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(x_bf16), rows, cols, 1, nullptr,
                     static_cast<uint8_t*>(q), scale));
    return DQMOE_OK;
}

int dqmoe_permute_quant_block_1x128(const void* x_bf16, int H, int k, const int32_t* dest_to_src, int n, void* q,
                                    float* scale, dqmoe_stream_t stream) {
    DQ_CHECK(n >= 0 && k > 0 && H > 0);
    if (n == 0) return DQMOE_OK;
    DQ_CHECK(x_bf16 != nullptr && q != nullptr && scale != nullptr && dest_to_src != nullptr);
    DQ_CHECK_FMT(H % 8 == 0, "H=%d must be a multiple of 8", H);
    DQ_CHECK(is_aligned(x_bf16, 16) && is_aligned(q, 8));
    DQ_RC(launch_pdl(permute::quant_1x128_kernel, dim3(permute::grid_for_rows(n)), permute::kThreads, 0,
                     static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(x_bf16), n, H, k, dest_to_src,
                     static_cast<uint8_t*>(q), scale));
    return DQMOE_OK;
}

}  // extern "C"
