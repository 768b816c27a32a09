// Dynamic FP8 E4M3 quantisers over bf16 data, bit-exact to the reference's torch
// expressions (test/util.py:18-68): sf = max(amax, 1e-4) / 448 and
// q = e4m3_rne(x * (1 / sf)), both divisions IEEE round-to-nearest. (This file
// must not be compiled with fast-math; the reference's own CUDA quantisers are,
// csrc/moe_kernels.h:136-398 with setup.py:37, and so differ from torch.)
//   rowwise       one scale per row           per_token_cast_to_fp8 / per_channel_cast_to_fp8
//   128x128       one scale per weight block  per_block_cast_to_fp8
//   tensor        one scale per tensor/expert (the reference has it for the intermediate only)
//   requant       second pass for the intermediate when stage 1 collected the amax
#include <mutex>

#include "common.cuh"
#include "ptx_sm100.cuh"

namespace dq {
namespace quant {

constexpr int kThreads = 256;

__device__ __forceinline__ void unpack8(const Vec16& raw, float (&v)[8]) {
    v[0] = bf16_lo(raw.x); v[1] = bf16_hi(raw.x); v[2] = bf16_lo(raw.y); v[3] = bf16_hi(raw.y);
    v[4] = bf16_lo(raw.z); v[5] = bf16_hi(raw.z); v[6] = bf16_lo(raw.w); v[7] = bf16_hi(raw.w);
}
__device__ __forceinline__ float amax8(const float (&v)[8], float m) {
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v[i]));
    return m;
}
__device__ __forceinline__ uint2 quant8(const float (&v)[8], float inv) {
    uint2 o;
    o.x = f2e4m3x4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv);
    o.y = f2e4m3x4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv);
    return o;
}

__device__ __forceinline__ float block_max(float v, float* s_red) {
    v = warp_max(v);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
    __syncthreads();
    float m = 0.0f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) m = fmaxf(m, s_red[w]);
    __syncthreads();
    return m;
}

// One block per row (grid-stride): amax pass, then quantise pass (second read hits L1/L2).
__global__ void __launch_bounds__(kThreads) rowwise_kernel(const uint8_t* x, int64_t rows, int cols, uint8_t* q,
                                                           float* scale) {
    pdl_enter();
    __shared__ float s_red[kThreads / 32];
    const int vecs = cols / 8;
    for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
        const uint8_t* xr = x + size_t(r) * cols * 2;
        float m = 0.0f;
        for (int i = threadIdx.x; i < vecs; i += kThreads) {
            float v[8];
            unpack8(ld_stream16(xr + size_t(i) * 16), v);
            m = amax8(v, m);
        }
        const float amax = block_max(m, s_red);
        const float sf = scale_from_amax(amax);
        const float inv = inv_scale(sf);
        if (threadIdx.x == 0) scale[r] = sf;
        uint8_t* qr = q + size_t(r) * cols;
        for (int i = threadIdx.x; i < vecs; i += kThreads) {
            float v[8];
            unpack8(ld_stream16(xr + size_t(i) * 16), v);
            *reinterpret_cast<uint2*>(qr + size_t(i) * 8) = quant8(v, inv);
        }
    }
}

// Short rows (up to 2048 columns): one warp per row, the row's vectors (at most eight per lane) fetched together and kept
// in registers between the amax and the conversion. Above, a warp would have to read the row twice and the block form,
// whose 256 threads hold the row's loads in flight, is the better one. (16384 x 2048: block form 30.2 us, warp form 17.6 us.)
constexpr int kShortRowVecs = 256;
__global__ void __launch_bounds__(kThreads) rowwise_short_kernel(const uint8_t* x, int64_t rows, int cols, uint8_t* q,
                                                                 float* scale) {
    pdl_enter();
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = int64_t(gridDim.x) * (kThreads / 32);
    const int vecs = cols / 8;
    for (int64_t r = (int64_t(blockIdx.x) * kThreads + threadIdx.x) >> 5; r < rows; r += nwarps) {
        const uint8_t* xr = x + size_t(r) * cols * 2;
        Vec16 raw[kShortRowVecs / 32];
#pragma unroll
        for (int i = 0; i < kShortRowVecs / 32; ++i)
            raw[i] = lane + 32 * i < vecs ? ld_stream16(xr + size_t(lane + 32 * i) * 16) : Vec16{0, 0, 0, 0};
        float m = 0.0f;
#pragma unroll
        for (int i = 0; i < kShortRowVecs / 32; ++i) {
            float v[8];
            unpack8(raw[i], v);
            m = amax8(v, m);
        }
        const float sf = scale_from_amax(warp_max(m));
        const float inv = inv_scale(sf);
        if (lane == 0) scale[r] = sf;
        uint8_t* qr = q + size_t(r) * cols;
#pragma unroll
        for (int i = 0; i < kShortRowVecs / 32; ++i) {
            if (lane + 32 * i < vecs) {
                float v[8];
                unpack8(raw[i], v);
                *reinterpret_cast<uint2*>(qr + size_t(lane + 32 * i) * 8) = quant8(v, inv);
            }
        }
    }
}

// Second pass over the bf16 intermediate when stage 1 already produced the amax: one warp per (row, strip of 128 16-byte
// vectors), four vectors per lane in flight. A warp per whole row left most of the chip idle when there are few long rows
// (32 rows of 14336: 13.4 us; in strips 2.7 us).
__global__ void __launch_bounds__(kThreads) requant_rows_kernel(const uint8_t* x, int64_t rows, int cols, uint8_t* q,
                                                                float* scale, const float* amax_in, int amax_per_row,
                                                                const int* rows_dev) {
    pdl_enter();
    if (rows_dev != nullptr) rows = rows < *rows_dev ? rows : *rows_dev;  // row count known only on the device
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * kThreads + threadIdx.x) >> 5;
    const int64_t nwarps = int64_t(gridDim.x) * (kThreads / 32);
    const int vecs = cols / 8;
    const int strips = (vecs + 127) / 128;
    for (int64_t it = warp; it < rows * strips; it += nwarps) {
        const int64_t r = it / strips;
        const int strip = int(it - r * strips);
        const int i0 = strip * 128 + lane;
        const uint8_t* xr = x + size_t(r) * cols * 2;
        uint8_t* qr = q + size_t(r) * cols;
        Vec16 raw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i0 + 32 * j < vecs) raw[j] = ld_stream16(xr + size_t(i0 + 32 * j) * 16);
        const float sf = scale_from_amax(amax_in[amax_per_row ? r : 0]);
        const float inv = inv_scale(sf);
        if (lane == 0 && strip == 0 && (amax_per_row || r == 0)) scale[amax_per_row ? r : 0] = sf;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (i0 + 32 * j < vecs) {
                float v[8];
                unpack8(raw[j], v);
                *reinterpret_cast<uint2*>(qr + size_t(i0 + 32 * j) * 8) = quant8(v, inv);
            }
        }
    }
}

// kWide neighbouring 128x128 weight blocks per thread block: 16 row lanes x kWide x 16 column vectors. A thread's eight 16-byte
// vectors are fetched together and stay in registers between the amax and the conversion, and the next blocks' are on their way
// while these are reduced and written (HBM-bound: 3 B per element; 8 x 4096 x 14336: fetched one by one and read a second
// time for the conversion 417 us, in one pass 284 us, with the next block's loads ahead 269 us = 5.2 TB/s, two blocks side by side
// 225 us = 6.3 TB/s: rows are then read in pieces of 512 bytes by one warp each and written in pieces of 256). One thread block of
// 512 per SM: with two the loads ahead spill (512 us); four blocks wide leave 64 registers per thread.
template <int kWide>
__global__ void __launch_bounds__(kThreads * kWide) block128_kernel(const uint8_t* w, int e, int rows, int cols, uint8_t* q,
                                                                    float* scale) {
    pdl_enter();
    __shared__ float s_red[2][16 * kWide];
    const int bc = (cols + 127) / 128, br = (rows + 127) / 128, gc = (bc + kWide - 1) / kWide;
    const int64_t groups = int64_t(e) * br * gc;
    const int half_warp = threadIdx.x >> 4;  // 16 lanes: one row's 128 columns
    const int tx = threadIdx.x & 15, cb = half_warp % kWide, ty = half_warp / kWide;
    struct Place {
        size_t first;   // this thread's first element
        int rows_left;  // rows of the matrix from it on, 0 beyond the last column
    };
    auto place = [&](int64_t g) {
        const int ei = int(g / (int64_t(br) * gc));
        const int r0 = int((g / gc) % br) * 128 + ty, c = (int(g % gc) * kWide + cb) * 128 + tx * 8;
        return Place{(size_t(ei) * rows + r0) * cols + c, c < cols ? max(0, rows - r0) : 0};
    };
    auto fetch = [&](const Place& pl, Vec16 (&raw)[8]) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            raw[i] = 16 * i < pl.rows_left ? ld_stream16(w + (pl.first + size_t(16 * i) * cols) * 2) : Vec16{0, 0, 0, 0};
    };
    Vec16 raw[8];
    int64_t g = blockIdx.x;
    if (g >= groups) return;
    Place pl = place(g);
    fetch(pl, raw);
    for (int parity = 0;; parity ^= 1) {
        float m = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float v[8];
            unpack8(raw[i], v);
            m = amax8(v, m);
        }
        const int64_t next = g + gridDim.x;
        const bool more = next < groups;
        Place pn{0, 0};
        Vec16 ahead[8];
        if (more) {
            pn = place(next);
            fetch(pn, ahead);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (tx == 0) s_red[parity][half_warp] = m;
        __syncthreads();  // one per round: the other buffer was last read before the round in between
        float amax = 0.0f;
#pragma unroll
        for (int r = 0; r < 16; ++r) amax = fmaxf(amax, s_red[parity][r * kWide + cb]);
        const float sf = scale_from_amax(amax);
        const float inv = inv_scale(sf);
        const int col_block = int(g % gc) * kWide + cb;
        if (tx == 0 && ty == 0 && col_block < bc) scale[(g / gc) * bc + col_block] = sf;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (16 * i < pl.rows_left) {
                float v[8];
                unpack8(raw[i], v);
                *reinterpret_cast<uint2*>(q + pl.first + size_t(16 * i) * cols) = quant8(v, inv);
            }
        }
        if (!more) break;
        g = next;
        pl = pn;
#pragma unroll
        for (int i = 0; i < 8; ++i) raw[i] = ahead[i];
    }
}

// per-tensor pass 1: amax of each of e slices into amax[e] (zeroed before)
__global__ void __launch_bounds__(kThreads) tensor_amax_kernel(const uint8_t* x, int64_t vecs_per, float* amax) {
    pdl_enter();
    __shared__ float s_red[kThreads / 32];
    const int ei = blockIdx.y;
    const uint8_t* xe = x + size_t(ei) * vecs_per * 16;
    float m = 0.0f;
    for (int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x; i < vecs_per; i += int64_t(gridDim.x) * kThreads) {
        float v[8];
        unpack8(ld_stream16(xe + size_t(i) * 16), v);
        m = amax8(v, m);
    }
    m = block_max(m, s_red);
    if (threadIdx.x == 0) atomic_max_nonneg(amax + ei, m);
}
// per-tensor pass 2
__global__ void __launch_bounds__(kThreads) tensor_quant_kernel(const uint8_t* x, int64_t vecs_per, const float* amax,
                                                                uint8_t* q, float* scale) {
    pdl_enter();
    const int ei = blockIdx.y;
    const float sf = scale_from_amax(amax[ei]);
    const float inv = inv_scale(sf);
    if (blockIdx.x == 0 && threadIdx.x == 0) scale[ei] = sf;
    const uint8_t* xe = x + size_t(ei) * vecs_per * 16;
    uint8_t* qe = q + size_t(ei) * vecs_per * 8;
    for (int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x; i < vecs_per; i += int64_t(gridDim.x) * kThreads) {
        float v[8];
        unpack8(ld_stream16(xe + size_t(i) * 16), v);
        *reinterpret_cast<uint2*>(qe + size_t(i) * 8) = quant8(v, inv);
    }
}

// Slices that eight blocks hold in registers (up to 8 x 1024 threads x 8 vectors = 524288 elements): one cluster per slice
// takes the amax through distributed shared memory and converts what it holds, one launch in place of a memset and two
// passes. Latency-bound at these sizes (16 x 4096: 14 us from the first operation to the end of the last, now 5.3).
constexpr int kSmallBlocks = 8, kSmallThreads = 1024, kSmallVecs = 8;
__global__ void __launch_bounds__(kSmallThreads, 1) tensor_small_kernel(const uint8_t* x, int64_t vecs_per,
                                                                        uint8_t* q, float* scale, float* amax) {
    pdl_enter();
    __shared__ float s_red[kSmallThreads / 32];
    __shared__ float s_block;
    const int ei = blockIdx.y;
    const uint32_t rank = ptx::cluster_ctarank();
    const uint8_t* xe = x + size_t(ei) * vecs_per * 16;
    Vec16 raw[kSmallVecs];
    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < kSmallVecs; ++j) {
        const int64_t i = int64_t(j) * (kSmallBlocks * kSmallThreads) + rank * kSmallThreads + threadIdx.x;
        raw[j] = i < vecs_per ? ld_stream16(xe + size_t(i) * 16) : Vec16{0, 0, 0, 0};
    }
#pragma unroll
    for (int j = 0; j < kSmallVecs; ++j) {
        float v[8];
        unpack8(raw[j], v);
        m = amax8(v, m);
    }
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = warp_max(s_red[threadIdx.x]);
        if (threadIdx.x == 0) s_block = m;
    }
    ptx::cluster_sync();
    m = 0.0f;
#pragma unroll
    for (int b = 0; b < kSmallBlocks; ++b) {
        float other;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(other) : "r"(ptx::map_to_cta(&s_block, uint32_t(b))) : "memory");
        m = fmaxf(m, other);
    }
    const float sf = scale_from_amax(m);
    const float inv = inv_scale(sf);
    if (rank == 0 && threadIdx.x == 0) {
        scale[ei] = sf;
        if (amax != nullptr) amax[ei] = m;  // as the general form leaves it
    }
    uint8_t* qe = q + size_t(ei) * vecs_per * 8;
#pragma unroll
    for (int j = 0; j < kSmallVecs; ++j) {
        const int64_t i = int64_t(j) * (kSmallBlocks * kSmallThreads) + rank * kSmallThreads + threadIdx.x;
        if (i < vecs_per) {
            float v[8];
            unpack8(raw[j], v);
            *reinterpret_cast<uint2*>(qe + size_t(i) * 8) = quant8(v, inv);
        }
    }
    ptx::cluster_sync();  // no block leaves while another may still read its word
}

static int tensor_small(const void* x, int e, int64_t vecs, void* q, float* scale, float* amax, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSmallBlocks, unsigned(e), 1);
    cfg.blockDim = dim3(kSmallThreads, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kSmallBlocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    DQ_CUDA(cudaLaunchKernelEx(&cfg, tensor_small_kernel, static_cast<const uint8_t*>(x), vecs, static_cast<uint8_t*>(q), scale,
                               amax));
    return DQMOE_OK;
}
// Only as many slices as run at once, one block per SM: every slice, however short, costs a cluster of eight blocks, and from
// the second wave on the general form is the faster one (general / cluster, us: 1 slice of 65536 11.1 / 7.9, 18 slices of 64
// 11.3 / 8.9, of 524288 18.5 / 12.5; 32 of 65536 11.2 / 14.1, 256 of 8192 11.5 / 76.6, 1024 of 131072 175 / 329).
static bool tensor_small_fits(int e, int64_t vecs) {
    return vecs <= int64_t(kSmallBlocks) * kSmallThreads * kSmallVecs && int64_t(e) * kSmallBlocks <= sm_count();
}

// Scratch of dqmoe_quant_fp8_tensor_static: lives in the library image of every GPU that
// loads it (4 KiB per device) so that the call needs no caller- or library-made allocation.
constexpr int kStaticMaxSlices = 1024;
static __device__ __align__(256) float g_static_amax[kStaticMaxSlices];

// Device address of g_static_amax on the current device. In host code the array's name is
// only a handle for the runtime, not an address a kernel may use, so the address is looked
// up once per device (with that device current) and cached.
static int static_amax_address(float** out) {
    constexpr int kMaxDevices = 64;
    static float* cached[kMaxDevices] = {nullptr};
    static std::mutex mu;  // two host threads may make their first call on a device at once
    int dev = 0;
    DQ_CUDA(cudaGetDevice(&dev));
    DQ_CHECK(dev >= 0 && dev < kMaxDevices);
    std::lock_guard<std::mutex> lk(mu);
    if (cached[dev] == nullptr) {
        float* p = nullptr;
        DQ_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_static_amax));
        DQ_CHECK(p != nullptr);
        cached[dev] = p;
    }
    *out = cached[dev];
    return DQMOE_OK;
}

static int grid_cap(int64_t want, int per_sm) {
    const int64_t cap = int64_t(sm_count()) * per_sm;
    return int(want < cap ? (want > 0 ? want : 1) : cap);
}

}  // namespace quant
}  // namespace dq

using namespace dq;

extern "C" {

int dqmoe_quant_fp8_rowwise(const void* x_bf16, int64_t rows, int cols, void* q, float* scale,
                            dqmoe_stream_t stream) {
    DQ_CHECK(rows >= 0 && cols > 0);
    if (rows == 0) return DQMOE_OK;
    DQ_CHECK(x_bf16 != nullptr && q != nullptr && scale != nullptr);
    DQ_CHECK_FMT(cols % 8 == 0, "cols=%d must be a multiple of 8", cols);
    DQ_CHECK(is_aligned(x_bf16, 16) && is_aligned(q, 8));
    if (cols / 8 <= quant::kShortRowVecs) {
        DQ_RC(launch_pdl(quant::rowwise_short_kernel, dim3(quant::grid_cap((rows + 7) / 8, 8)), quant::kThreads, 0,
                         static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(x_bf16), rows, cols,
                         static_cast<uint8_t*>(q), scale));
        return DQMOE_OK;
    }
    DQ_RC(launch_pdl(quant::rowwise_kernel, dim3(quant::grid_cap(rows, 16)), quant::kThreads, 0,
                     static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(x_bf16), rows, cols,
                     static_cast<uint8_t*>(q), scale));
    return DQMOE_OK;
}

int dqmoe_requant_from_amax_dev(const void* act_bf16, int64_t n_max, int I, const float* amax, int per_row, void* q,
                                float* scale, const int32_t* n_rows_device, dqmoe_stream_t stream) {
    DQ_CHECK(n_max >= 0 && I > 0);
    if (n_max == 0) return DQMOE_OK;
    DQ_CHECK(act_bf16 != nullptr && q != nullptr && scale != nullptr && amax != nullptr);
    DQ_CHECK_FMT(I % 8 == 0, "I=%d must be a multiple of 8", I);
    DQ_CHECK(is_aligned(act_bf16, 16) && is_aligned(q, 8));
    DQ_RC(launch_pdl(quant::requant_rows_kernel, dim3(quant::grid_cap((n_max * ((I / 8 + 127) / 128) + 7) / 8, 8)),
                     quant::kThreads, 0, static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(act_bf16), n_max, I,
                     static_cast<uint8_t*>(q), scale, amax, per_row ? 1 : 0, n_rows_device));
    return DQMOE_OK;
}

int dqmoe_requant_from_amax(const void* act_bf16, int64_t n, int I, const float* amax, int per_row, void* q,
                            float* scale, dqmoe_stream_t stream) {
    return dqmoe_requant_from_amax_dev(act_bf16, n, I, amax, per_row, q, scale, nullptr, stream);
}

int dqmoe_quant_fp8_block_128x128(const void* w_bf16, int e, int rows, int cols, void* q, float* scale,
                                  dqmoe_stream_t stream) {
    DQ_CHECK(e >= 0 && rows > 0 && cols > 0);
    if (e == 0) return DQMOE_OK;
    DQ_CHECK(w_bf16 != nullptr && q != nullptr && scale != nullptr);
    DQ_CHECK_FMT(cols % 8 == 0, "cols=%d must be a multiple of 8", cols);
    DQ_CHECK(is_aligned(w_bf16, 16) && is_aligned(q, 8));
    // Two wide everywhere: one / two wide, us: 4096 x 4096 18.2 / 17.8, 3 x 1000 x 5000 15.8 / 15.4, 16 x 600 x 512 15.6 / 15.4,
    // 5 x 2000 x 7000 42.1 / 38.6, 8 x 4096 x 14336 269 / 225.
    constexpr int kWide = 2;
    const int64_t groups = int64_t(e) * ((rows + 127) / 128) * ((cols + 128 * kWide - 1) / (128 * kWide));
    DQ_RC(launch_pdl(quant::block128_kernel<kWide>, dim3(quant::grid_cap(groups, 1)), quant::kThreads * kWide, 0,
                     static_cast<cudaStream_t>(stream), static_cast<const uint8_t*>(w_bf16), e, rows, cols,
                     static_cast<uint8_t*>(q), scale));
    return DQMOE_OK;
}

int dqmoe_quant_fp8_tensor(const void* x_bf16, int e, int64_t numel_per, void* q, float* scale, float* amax_scratch,
                           dqmoe_stream_t stream) {
    DQ_CHECK(e >= 0 && numel_per >= 0 && e <= 65535);
    if (e == 0 || numel_per == 0) return DQMOE_OK;
    DQ_CHECK(x_bf16 != nullptr && q != nullptr && scale != nullptr && amax_scratch != nullptr);
    DQ_CHECK_FMT(numel_per % 8 == 0, "numel_per=%lld must be a multiple of 8", (long long) numel_per);
    DQ_CHECK(is_aligned(x_bf16, 16) && is_aligned(q, 8));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (quant::tensor_small_fits(e, numel_per / 8)) return quant::tensor_small(x_bf16, e, numel_per / 8, q, scale, amax_scratch, s);
    DQ_CUDA(cudaMemsetAsync(amax_scratch, 0, size_t(e) * sizeof(float), s));
    const int64_t vecs = numel_per / 8;
    const int gx = quant::grid_cap((vecs + quant::kThreads - 1) / quant::kThreads, e >= 8 ? 2 : 8);
    dim3 grid(gx, e);
    DQ_RC(launch_pdl(quant::tensor_amax_kernel, dim3(grid), quant::kThreads, 0, s, static_cast<const uint8_t*>(x_bf16), vecs,
                     amax_scratch));
    DQ_RC(launch_pdl(quant::tensor_quant_kernel, dim3(grid), quant::kThreads, 0, s, static_cast<const uint8_t*>(x_bf16), vecs,
                     amax_scratch, static_cast<uint8_t*>(q), scale));
    return DQMOE_OK;
}

// Per-tensor / per-expert FP8 quantiser for callers that cannot allocate device memory and
// have no spare buffer to lend: the amax scratch is the library's own static device array.
// Same kernels and results as dqmoe_quant_fp8_tensor. Limits and rules:
//   * at most 1024 slices (e <= 1024); larger e is rejected with an error;
//   * the first call on each device looks up the array's device address (a host-side runtime
//     query, no allocation) - make that first call outside any stream capture;
//   * all calls on one device share the array: it is cleared at the start of every call, and
//     two calls whose kernels overlap on the GPU (different streams) race on it.
int dqmoe_quant_fp8_tensor_static(const void* x_bf16, int e, int64_t numel_per, void* q, float* scale,
                                  dqmoe_stream_t stream) {
    DQ_CHECK(e >= 0 && numel_per >= 0);
    DQ_CHECK_FMT(e <= quant::kStaticMaxSlices, "e=%d exceeds the %d slices the static scratch holds", e,
                 quant::kStaticMaxSlices);
    if (e == 0 || numel_per == 0) return DQMOE_OK;
    DQ_CHECK(x_bf16 != nullptr && q != nullptr && scale != nullptr);
    DQ_CHECK_FMT(numel_per % 8 == 0, "numel_per=%lld must be a multiple of 8", (long long) numel_per);
    DQ_CHECK(is_aligned(x_bf16, 16) && is_aligned(q, 8));
    if (quant::tensor_small_fits(e, numel_per / 8))
        return quant::tensor_small(x_bf16, e, numel_per / 8, q, scale, nullptr, static_cast<cudaStream_t>(stream));
    float* amax = nullptr;
    const int rc = quant::static_amax_address(&amax);
    if (rc != DQMOE_OK) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // the array keeps the previous call's maxima: the reduction must start from zero
    DQ_CUDA(cudaMemsetAsync(amax, 0, size_t(e) * sizeof(float), s));
    const int64_t vecs = numel_per / 8;
    const int gx = quant::grid_cap((vecs + quant::kThreads - 1) / quant::kThreads, e >= 8 ? 2 : 8);
    dim3 grid(gx, e);
    DQ_RC(launch_pdl(quant::tensor_amax_kernel, dim3(grid), quant::kThreads, 0, s, static_cast<const uint8_t*>(x_bf16), vecs,
                     amax));
    DQ_RC(launch_pdl(quant::tensor_quant_kernel, dim3(grid), quant::kThreads, 0, s, static_cast<const uint8_t*>(x_bf16), vecs,
                     amax, static_cast<uint8_t*>(q), scale));
    return DQMOE_OK;
}

}  // extern "C"
