// Shared host/device helpers of the dqmoe_b200 library: error reporting for the
// C ABI, the host-mapped device status word, and small device utilities.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>
#include <string>

#include "../../include/dqmoe.h"

namespace dq {

// ---------------------------------------------------------------- host errors

// Message of the last failure on this thread (returned by dqmoe_last_error()).
std::string& last_error();

int fail(int code, const char* file, int line, const char* cond, const char* fmt = nullptr, ...);

// Argument check in the reference's CPU_CHECK form (csrc/util.h:173-195): the
// C ABI returns DQMOE_ERR_INVALID and the Python layer raises RuntimeError with
// the "[ASSERT FAILED] ..." text.
#define DQ_CHECK(cond)                                                              \
    do {                                                                            \
        if (!(cond)) return ::dq::fail(DQMOE_ERR_INVALID, __FILE__, __LINE__, #cond); \
    } while (0)
#define DQ_CHECK_FMT(cond, ...)                                                                  \
    do {                                                                                         \
        if (!(cond)) return ::dq::fail(DQMOE_ERR_INVALID, __FILE__, __LINE__, #cond, __VA_ARGS__); \
    } while (0)
// CUDA failures become error returns; the reference's CUDA_CHECK calls exit()
// (csrc/util.h:61-80).
#define DQ_CUDA(expr)                                                                   \
    do {                                                                                \
        cudaError_t e_ = (expr);                                                        \
        if (e_ != cudaSuccess)                                                          \
            return ::dq::fail(DQMOE_ERR_CUDA, __FILE__, __LINE__, #expr, "%s",          \
                              cudaGetErrorString(e_));                                  \
    } while (0)
#define DQ_LAUNCH_CHECK() DQ_CUDA(cudaGetLastError())
#define DQ_RC(expr)                         \
    do {                                    \
        const int rc_ = (expr);             \
        if (rc_ != DQMOE_OK) return rc_;    \
    } while (0)

// Host-mapped status word of the current device (allocated once per device in
// pinned host memory; kernels write a non-zero code when a bounded wait gives up).
// Returns the device-side pointer, or nullptr with last_error() set.
int* device_status_word();
// Host view of the same word for the current device.
volatile int* host_status_word();

int sm_count();

namespace decode {
constexpr int kAmaxParts = 4096;  // floats the layer workspace holds for the per-block amax values of the decode path's fc1
}

// Programmatic dependent launch. A kernel launched through launch_pdl calls pdl_launch() and pdl_wait() first thing (the grouped
// GEMMs set up their barriers and TMEM in between): the next kernel's blocks may become resident while this one runs, and no thread
// touches global memory before all earlier kernels of the stream have completed. What such a kernel reads may therefore still be
// written while it is resident: its pointers are not __restrict__ and its loads are plain ones (ld_stream16).
// Early GEMMs are the exception: the weights-on-M form on single CTAs, block mode by counts, and the block-scaled GEMM as the layer
// launches it. Before their wait they read the expert sort's table, past L1 (ld_relaxed_gpu), and their weights with the weights'
// tiled scales. That is sound because they start only when the sort and all before it are complete: the kernels that may stand right
// behind the sort (both row scatters, the MXFP8 quantiser, the scale tiling) and the early GEMMs themselves call pdl_launch() after
// their wait. The re-quantisation pass and fc1's row tiles call it first, but start behind one of those.
// Between the short kernels of the layer the gap shrinks from ~2 us to below 1 us (MoE block of 5 tokens, H 1024,
// I 2048: 45.8 -> 34.6 us).
// The grouped GEMMs are launched this way up to kPdlGemmRows rows only. Their blocks, one per SM, otherwise take the SMs in the
// order in which the kernel before leaves them instead of in the launch order, which spreads the blocks that share a weight
// tile over both dies: 4096 tokens x 2, block FP8 1886 -> 1959 us, 8192 x 8 5312 -> 6088 us. Up to some 2000 rows little is shared
// and the gap counts (layer calls, without / with: H 1024, I 2048, E 4, 512 rows 31 / 27 us, 2048 rows 41 / 36; H 4096, I 14336,
// E 8, 864 rows 276 / 272, 2048 rows 456 / 453; H 7168, I 2048, E 32, 2048 rows 292 / 289). In between it goes either way: with
// 128 small experts (H 2048, I 768) 2048 rows cost 141 / 147 in MXFP8, 157 / 159 in block FP8 and 153 / 152 per-channel, 4096 rows of
// the large models 974 / 981 in block FP8 and 804 / 795 per-channel.
constexpr int kPdlGemmRows = 2048;
template <class... KArgs, class... Args>
static inline int launch_pdl(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(unsigned(threads), 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    DQ_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...));
    return DQMOE_OK;
}
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
    pdl_launch();
    pdl_wait();
}

static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
static inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
static inline bool is_aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// ---------------------------------------------------------------- device utils

// 16-byte vector used by all streaming kernels (coalesced 128-bit accesses).
struct __align__(16) Vec16 {
    uint32_t x, y, z, w;
};

// For data that nobody writes as long as the kernel is resident: in kernels that start only after their predecessors' end.
__device__ __forceinline__ Vec16 ld_nc16(const void* p) {
    Vec16 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
// The same as a plain load, for kernels launched through launch_pdl. They are resident while their predecessors still write
// what they read after pdl_wait, which the non-coherent path (ld.global.nc, __ldg, a const __restrict__ argument) does not
// allow for. Volatile, so that it stays behind the wait.
__device__ __forceinline__ Vec16 ld_stream16(const void* p) {
    Vec16 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
// For the few words that a programmatic dependent reads before its own pdl_wait, written by a kernel that is known to be over by
// then. Its end makes them visible at gpu scope, but only the wait covers what this SM's L1 may still hold of an earlier call
// that used the same workspace: a relaxed load at gpu scope is served from L2. Volatile, like the others.
__device__ __forceinline__ int ld_relaxed_gpu(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st16(void* p, const Vec16& v) {
    asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// round-to-nearest-even fp32 -> bf16 bits (matches torch's .to(bfloat16))
__device__ __forceinline__ uint32_t f2bf_bits(float f) {
    return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(f)));
}
// fp32 rounded to the nearest bf16 value (ties to even), returned as fp32. Done as a 16-bit Veltkamp split on the fp32 pipe
// (c = 65537 x; x_hi = c - (c - x), every step rounded), used by the decode kernels. Equal to the conversion for all normal
// inputs with |x| < 2^111 (checked exhaustively on random and tie patterns); subnormal results may differ in the last bit.
__device__ __forceinline__ float bf_round(float f) {
    const float c = __fmul_rn(f, 65537.0f);
    return __fsub_rn(c, __fsub_rn(c, f));
}
// the same through the conversion instruction, for all inputs
__device__ __forceinline__ float bf_round_cvt(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }
// two fp32 -> packed bf16x2 with one conversion instruction
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// silu(g) = g / (1 + exp(-g)) with exp(-g) = 2^(-g log2 e). The PTX ISA gives ex2.approx 2 ulp and rcp.approx 1 ulp; the rounding
// of -g log2 e moves the power by up to |g| 2^-23 relative. So the result is within (|g| + 8) 2^-23 of silu(g), 2^-16 at g = -87:
// far inside the rounding to bf16 that follows (2^-9). With .ftz a power below 2^-126 counts as 0 (the sum is 1 either way), and
// so does a reciprocal below 2^-126, that is a silu of less than 1e-36 at g < -87.3. Infinities and NaN as in IEEE arithmetic.
// Tested for every bf16 gate.
__device__ __forceinline__ float silu_approx(float g) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return g * r;
}
// SwiGLU of two columns with the torch oracle's rounding points: gate, value, silu(gate) and the product to bf16. Two
// columns per conversion: cvt.rn.bf16x2 takes 2 cycles of a sub-partition for a warp's 64 values, a single-value cvt
// followed by a shift 16 for the same 64; and the product of two bf16 values rounded to bf16 is one mul.bf16x2.
// fc1 before / after: per-channel FP8 (H 2048, I 768, 16384 tokens x 8) 371 / 320 us, block FP8 (H 4096, I 14336,
// 4096 tokens x 2) 1100 / 1065 us, bf16 (2880 x 2880, 16384 x 3) 1278 / 1251 us.
__device__ __forceinline__ uint32_t swiglu_bf16x2(float g0, float g1, float v0, float v1) {
    const uint32_t g2 = pack_bf16x2(g0, g1);
    const uint32_t s2 = pack_bf16x2(silu_approx(bf16_lo(g2)), silu_approx(bf16_hi(g2)));
    const uint32_t v2 = pack_bf16x2(v0, v1);
    const __nv_bfloat162 r = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&s2), *reinterpret_cast<const __nv_bfloat162*>(&v2));
    return *reinterpret_cast<const uint32_t*>(&r);
}
// running maximum of |x| over packed bf16 pairs, and its value (NaN counts for nothing, as with fmaxf)
__device__ __forceinline__ void amax_bf16x2(uint32_t& m2, uint32_t x2) {
    x2 &= 0x7fff7fffu;
    const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&m2), *reinterpret_cast<const __nv_bfloat162*>(&x2));
    m2 = *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ float amax_bf16x2_value(uint32_t m2) { return fmaxf(bf16_lo(m2), bf16_hi(m2)); }

// two fp32 -> two e4m3 bytes (round-to-nearest-even, saturating to +-448), lo in bits 0..7
__device__ __forceinline__ uint32_t f2e4m3x2(float lo, float hi) {
    uint16_t r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t f2e4m3x4(float a, float b, float c, float d) {
    return f2e4m3x2(a, b) | (f2e4m3x2(c, d) << 16);
}

// The reference's torch quantisers: sf = clamp(amax, 1e-4) / 448 ; inv = 1 / sf
// (test/util.py:21-23). Both divisions are IEEE round-to-nearest.
__device__ __forceinline__ float scale_from_amax(float amax) { return __fdiv_rn(fmaxf(amax, 1e-4f), 448.0f); }
__device__ __forceinline__ float inv_scale(float sf) { return __fdiv_rn(1.0f, sf); }

// one e4m3 byte -> fp32 (exact)
__device__ __forceinline__ float e4m3_to_float(uint32_t byte) {
    const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(byte & 0xffu), __NV_E4M3);
    return __half2float(*reinterpret_cast<const __half*>(&h));
}
// eight floats -> eight e2m1 nibbles (round to nearest even, saturating at 6), element i in nibble i
__device__ __forceinline__ uint32_t f2e2m1x8(const float (&x)[8]) {
    uint32_t out;
    asm("{\n\t"
        ".reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t"
        "}"
        : "=r"(out)
        : "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7]));
    return out;
}
// NVFP4 scale of a 16-value block: the e4m3 byte nearest to (amax / 6) / g (saturating at 448), g = the tensor's
// global scale; *inv = 1 / (value of that byte * g), or 0 for an all-zero block. A value x of the block is stored
// as e2m1(x * inv).
__device__ __forceinline__ uint32_t nvfp4_scale_byte(float amax, float g, float* inv) {
    const uint32_t byte = f2e4m3x2(__fdiv_rn(__fdiv_rn(amax, 6.0f), g), 0.0f) & 0xffu;
    const float d = e4m3_to_float(byte) * g;
    *inv = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    return byte;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// non-negative floats order like their bit patterns
__device__ __forceinline__ void atomic_max_nonneg(float* addr, float v) {
    atomicMax(reinterpret_cast<int*>(addr), __float_as_int(v));
}

}  // namespace dq
