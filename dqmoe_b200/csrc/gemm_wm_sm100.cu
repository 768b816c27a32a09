// Host side and kernels of the grouped GEMM with the weights on M (gemm_wm.cuh).
#include <mutex>

#include "common.cuh"
#include "gemm_tile.cuh"
#include "gemm_wm.cuh"

namespace dq {
namespace gemm {
int grouped_gemm_by_counts(const gemm_wm::Form& wm, const float* a_scale, const void* w, const int* mtile_prefix, int K, int gated,
                           int line, cudaStream_t stream);
}  // namespace gemm

namespace gemm_wm {

constexpr int kMaxDevices = 64;

template <bool kFp8, int kMode, bool kGated, bool kPair>
__global__ void __launch_bounds__(kThreads, 1)
moe_GemmGrouped_GemmUniversal_tcgen05_wm(const __grid_constant__ Maps maps, const __grid_constant__ Params p) {
    weights_on_m<kFp8, kMode, kGated, kPair>(maps, p);
}

template <bool kFp8, int kMode, bool kGated, bool kPair>
static int launch(const Maps& maps, const Params& p, cudaStream_t stream) {
    auto kern = moe_GemmGrouped_GemmUniversal_tcgen05_wm<kFp8, kMode, kGated, kPair>;
    // the shared-memory opt-in is per function and per device
    static std::mutex mu;
    static bool configured[kMaxDevices] = {};
    int dev = 0;
    DQ_CUDA(cudaGetDevice(&dev));
    DQ_CHECK(dev >= 0 && dev < kMaxDevices);
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!configured[dev]) {
            DQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_bytes<kMode == kBlock>())));
            configured[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(kPair ? sm_count() & ~1 : sm_count()), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = smem_bytes<kMode == kBlock>();
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = p.n_rows <= kPdlGemmRows ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;  // pairs: clusters of two CTAs on neighbouring SMs; an even grid
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = kPair ? 2 : 1;
    DQ_CUDA(cudaLaunchKernelEx(&cfg, kern, maps, p));
    return DQMOE_OK;
}

// Weights as fc1's tiles read them: eight gate rows and the eight value rows of the same columns in turn.
static int make_weight_map(CUtensorMap* map, const void* w, int esz, int E, int N, int K, bool gated) {
    gemm::EncodeTiledFn fn = gemm::encode_fn();
    if (fn == nullptr) return fail(DQMOE_ERR_CUDA, __FILE__, __LINE__, "cuTensorMapEncodeTiled", "driver entry point not found");
    const cuuint64_t row = cuuint64_t(K) * esz;
    const CUtensorMapDataType dt = esz == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const cuuint32_t box_k = cuuint32_t(kKBytes / esz);
    cuuint32_t one[5] = {1, 1, 1, 1, 1};
    CUresult r;
    if (gated) {
        cuuint64_t dim[5] = {cuuint64_t(K), 8, 2, cuuint64_t(N / 8), cuuint64_t(E)};
        cuuint64_t stride[4] = {row, row * N, row * 8, row * 2 * N};
        cuuint32_t box[5] = {box_k, 8, 2, kWRows / 16, 1};
        r = fn(map, dt, 5, const_cast<void*>(w), dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        cuuint64_t dim[3] = {cuuint64_t(K), cuuint64_t(N), cuuint64_t(E)};
        cuuint64_t stride[2] = {row, row * N};
        cuuint32_t box[3] = {box_k, kWRows, 1};
        r = fn(map, dt, 3, const_cast<void*>(w), dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r != CUDA_SUCCESS)
        return fail(DQMOE_ERR_CUDA, __FILE__, __LINE__, "cuTensorMapEncodeTiled", "CUresult %d (E %d N %d K %d)", int(r), E, N, K);
    return DQMOE_OK;
}

static int form(const void* a, const float* a_scale, const void* w, const float* w_scale, const int* offsets, int n, int N, int K, int E,
                int quant_mode, int gated, void* out, float* amax, const int* dest_to_src, const float* bias, float* out_scale,
                float* out_scale_t, int n_pad, bool row_tiles_too, Form* f) {
    const bool block = quant_mode == DQMOE_QUANT_FP8_BLOCK;
    DQ_CHECK(quant_mode == DQMOE_QUANT_NONE || quant_mode == DQMOE_QUANT_FP8_TENSOR || quant_mode == DQMOE_QUANT_FP8_CHANNEL || block);
    DQ_CHECK(n > 0 && N > 0 && K > 0 && E > 0 && E <= kMaxExperts);
    const bool fp8 = quant_mode != DQMOE_QUANT_NONE;
    const int esz = fp8 ? 1 : 2;
    DQ_CHECK_FMT((size_t(K) * esz) % 16 == 0, "K=%d: rows must be a multiple of 16 bytes", K);
    DQ_CHECK_FMT(N % (gated && block ? 16 : 8) == 0, "N=%d: output rows must be 16-byte vectors", N);
    DQ_CHECK(is_aligned(a, 16) && is_aligned(w, 16) && is_aligned(out, 16));
    DQ_CHECK(a != nullptr && w != nullptr && out != nullptr && offsets != nullptr && (gated || dest_to_src != nullptr));
    if (fp8) DQ_CHECK(a_scale != nullptr && w_scale != nullptr && (block || !gated || amax != nullptr));
    // a tile's scales are read four rows at a time, up to its rows rounded up to 16
    if (block) DQ_CHECK(n_pad % 4 == 0 && n_pad >= n + 15 && is_aligned(a_scale, 16) && (!gated || (out_scale != nullptr && out_scale_t != nullptr)));

    // A pair shares each row between two CTAs, half the bytes through L2 for wide tiles, and computes rows in steps of 32 instead of
    // 16. Pairs / singles, us per layer call. Even routing, rows per expert on average: 20 (H 2048, I 1408, E 64, k 6, per-tensor) 120 /
    // 111; 30 (H 2048, I 768, E 128, k 8) per-tensor 145 / 141, per-channel 139 / 138, bf16 224 / 227; 30 (H 7168, I 2048, E 32) 246 / 243;
    // 47 (E 128, per-channel) 146 / 142, bf16 235 / 235; 100 (E 32) 280 / 290; 125 (H 4096, I 14336, E 8) 285 / 295; 250 (E 32, bf16)
    // 701 / 793. Skewed routing (Zipf 1.1), where a few experts have several hundred rows: 30 (E 128) per-tensor 125 / 134, per-channel
    // 123 / 132, bf16 183 / 199; 30 (H 2880, I 2880, E 64, k 3, bf16) 352 / 381; 47 (E 128) 138 / 148, 137 / 145, 206 / 223. So from 30
    // rows on, but from 48 where a tile per expert does not fill the chip and the singles' smaller ones spread further (H 2048, I 3072,
    // E 3, k 1, bf16: 30 rows 38 / 35, 47 rows 39 / 35). Block mode hands its accumulators over every few K blocks, which across two SMs
    // takes twice as long.
    const int cta_cols = gated ? kWRows / 2 : kWRows;
    const bool fills = 2 * int64_t(E) * ceil_div(N, 2 * cta_cols) >= sm_count();
    const bool pair = !block && n / E >= (fills ? 30 : 48);
    f->pair = pair;
    Params& p = f->p;
    p.n_rows = n;
    p.N = N;
    p.E = E;
    p.w_rows = gated ? 2 * N : N;
    p.w_tiles = ceil_div(N, pair || (block && gated) ? 2 * cta_cols : cta_cols);
    p.kb_count = ceil_div(K * esz, kKBytes);
    p.offsets = offsets;
    p.sa = a_scale;
    p.sb = w_scale;
    p.out = out;
    p.amax = amax;
    p.out_scale = out_scale;
    p.out_scale_t = out_scale_t;
    p.n_pad = n_pad;
    p.bias = bias;
    p.dest_to_src = dest_to_src;
    p.status = device_status_word();
    if (p.status == nullptr) return DQMOE_ERR_CUDA;

    // Only the boxes that a tile of this call can need (each CTA of a pair loads half of one): encoding a map takes 0.5 us (MoE block
    // of 5 tokens: C++ 23.3 -> 20.3 us).
    const int unit = pair ? 32 : 16;
    const int limit = block ? kBlockTok : kMaxTok;
    const int most = (n < limit ? ceil_div(n, unit) * unit : limit) / (pair ? 2 : 1);
    f->maps = {};
    DQ_RC(make_weight_map(&f->maps.w, w, esz, E, N, K, gated != 0));
    for (int i = 0; i < 4 && (row_tiles_too || (16 << i) <= most); ++i) DQ_RC(gemm::make_map(&f->maps.rows[i], a, esz, uint64_t(n), uint64_t(K), 16 << i));
    return DQMOE_OK;
}

// Arguments as gemm::grouped_gemm takes them; bf16, per-tensor / per-channel FP8 and block FP8 operands, the last with the activation
// scales by column (a_scale) and, where a line > 0 lets the kernel take row tiles instead, by row (a_scale_rows).
int grouped_gemm(const void* a, const float* a_scale, const void* w, const float* w_scale, const int* offsets, int n, int N, int K,
                 int E, int quant_mode, int gated, void* out, float* amax, const int* dest_to_src, const float* bias,
                 float* out_scale, float* out_scale_t, int n_pad, int line, const float* a_scale_rows, const int* mtile_prefix,
                 cudaStream_t stream) {
    DQ_CHECK(n >= 0);
    if (n == 0) return DQMOE_OK;
    Form f;
    DQ_RC(form(a, a_scale, w, w_scale, offsets, n, N, K, E, quant_mode, gated, out, amax, dest_to_src, bias, out_scale, out_scale_t, n_pad,
               line > 0, &f));
    if (line > 0) return gemm::grouped_gemm_by_counts(f, a_scale_rows, w, mtile_prefix, K, gated, line, stream);

#define DQ_WM_LAUNCH(FP8, MODE)                                                                                             \
    (gated ? (f.pair ? launch<FP8, MODE, true, true>(f.maps, f.p, stream) : launch<FP8, MODE, true, false>(f.maps, f.p, stream))  \
           : (f.pair ? launch<FP8, MODE, false, true>(f.maps, f.p, stream) : launch<FP8, MODE, false, false>(f.maps, f.p, stream)))
    switch (quant_mode) {
        case DQMOE_QUANT_NONE: return DQ_WM_LAUNCH(false, kNone);
        case DQMOE_QUANT_FP8_TENSOR: return DQ_WM_LAUNCH(true, kTensor);
        case DQMOE_QUANT_FP8_CHANNEL: return DQ_WM_LAUNCH(true, kChannel);
        default:
            return gated ? launch<true, kBlock, true, false>(f.maps, f.p, stream) : launch<true, kBlock, false, false>(f.maps, f.p, stream);
    }
#undef DQ_WM_LAUNCH
}

}  // namespace gemm_wm
}  // namespace dq
