// Grouped GEMM with the weights on the M side of the tensor core: D[weight row][token] = W A^T. A tile is 128 weight
// rows per CTA (64 gate and 64 value rows in fc1) by up to 256 rows of one expert, in steps of 16 (32 on a CTA pair), so
// an expert of 300 rows computes 304 or 320 of them, where tiles with the rows on M compute 384 or 512. Used by the layer
// for bf16 and per-tensor / per-channel FP8 operands; gemm_sm100.cu has the form with the rows on M.
//
// What bounds it: for many rows per expert the tensor pipe under the power limit, for few rows the weights from HBM.
// Everything else is meant to stay out of their way:
//   - an expert's rows are split evenly over ceil(rows / 256) tiles, so no tile is nearly empty;
//   - shared memory is cut into as many stages as the launch's largest tile allows (4 of 48 KiB at 256 rows, 10 of 18 KiB
//     at 16), so that a few rows leave the memory to weights in flight;
//   - the accumulator is read as 16 x 256-bit fragments, in which a thread holds rows r and r + 8 of a token pair. fc1's
//     weight rows are interleaved by eight (one TMA box of a five-dimensional view), so r and r + 8 are gate and value of
//     the same column and SwiGLU stays in the thread; stmatrix.trans then turns the fragment into token rows.
//
// Replaces the same reference kernels as gemm_sm100.cu (csrc/moe_gemm_template.h:72-1039, csrc/moe_kernels.h:301-444, 581-620).
#include <mutex>

#include "common.cuh"
#include "gemm_tile.cuh"
#include "ptx_sm100.cuh"

namespace dq {
namespace gemm_wm {

constexpr int kWRows = 128;                       // weight rows per CTA = lanes of TMEM
constexpr int kMaxTok = 256;                      // rows of an expert per tile
constexpr int kKBytes = 128;                      // K bytes per stage: one 128-byte swizzle row
constexpr int kUmmaKBytes = 32;                   // K bytes per tcgen05.mma
constexpr int kABytes = kWRows * kKBytes;         // 16 KiB
constexpr int kStageArea = 4 * (kABytes + kMaxTok * kKBytes);
constexpr int kMaxStages = 10;
constexpr int kThreads = 384;                     // warp 0 TMA, warp 1 MMA, warps 2-3 idle, warps 4..11 epilogue
constexpr int kEpiWarps = 8;
constexpr int kMaxExperts = 1024;
constexpr int kMaxDevices = 64;
constexpr int kTmemCols = 512;                    // two accumulator buffers of up to 256 tokens
constexpr int kSub = 16;                          // tokens per pass through the store buffers
constexpr long long kWaitLimit = 1000000000LL;    // clock cycles before a wait gives up (~0.5 s)

enum Mode : int { kNone = 0, kTensor = 1, kChannel = 2 };

struct Params {
    int n_rows;               // rows of A (expanded rows n)
    int N;                    // output columns (fc1: I, fc2: H)
    int E;
    int w_rows;               // weight rows per expert (fc1: 2I, fc2: H)
    int w_tiles;              // tiles per expert along the output columns
    int kb_count;             // ceil(K bytes / 128)
    const int* offsets;       // [E+1] first row of each expert
    const float* sa;          // activation scales: tensor [1], channel [n]
    const float* sb;          // weight scales: tensor [E], channel [E, w_rows]
    void* out;
    float* amax;              // fc1: channel [n], tensor [1]
    const float* bias;        // [E, w_rows] fp32 added to the dequantised product, or nullptr
    const int* dest_to_src;   // fc2: output row of each row
    int* status;              // host-mapped status word
};

struct Maps {
    CUtensorMap w;            // weights: fc1 [E][I/8][gate, value][8][K], fc2 [E][H][K]
    CUtensorMap rows[4];      // activation rows, boxes of 16, 32, 64 and 128 rows
};

struct SharedTail {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t tmem_full[2];
    uint64_t tmem_empty[2];
    uint32_t tmem_base;
    int abort_flag;
    int max_tok;                                  // tokens of the largest tile
    unsigned long long dst[2][kMaxTok];           // output row of each token of the tile, 0 = none
    float sa[2][kMaxTok];                         // its activation scale (channel mode)
    alignas(16) uint4 stage[2][2][kSub * 16];     // per epilogue warpgroup: two buffers of 16 tokens x (64 or 128 columns)
    int tprefix[kMaxExperts + 1];                 // cumulative token tiles
    int offsets[kMaxExperts + 1];
};

constexpr size_t kSmemBytes = 1024 + size_t(kStageArea) + sizeof(SharedTail);
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");

__host__ __device__ constexpr int round_up(int x, int m) { return (x + m - 1) / m * m; }

// Rows of one expert per tile when its `count` rows go to ceil(count / 256) tiles.
template <bool kPair>
__device__ __forceinline__ int tile_tokens(int count, int tiles) {
    return round_up((count + tiles - 1) / tiles, kPair ? 32 : 16);
}

struct Tile {
    int e, wt, row0, rows, tok;  // expert, tile along the output columns, first row, rows, tokens computed (rows rounded up)
};

// Tiles are numbered expert-major; inside an expert the token tile runs fastest, so that concurrently running CTAs share
// one weight tile.
template <bool kPair>
__device__ __forceinline__ Tile decode_tile(int t, int& e_cursor, const SharedTail& st, int w_tiles) {
    while (t >= st.tprefix[e_cursor + 1] * w_tiles) ++e_cursor;
    const int local = t - st.tprefix[e_cursor] * w_tiles;
    const int tiles = st.tprefix[e_cursor + 1] - st.tprefix[e_cursor];
    const int count = st.offsets[e_cursor + 1] - st.offsets[e_cursor];
    const int nt = tile_tokens<kPair>(count, tiles);
    Tile tl;
    tl.e = e_cursor;
    tl.wt = local / tiles;
    const int j = local - tl.wt * tiles;
    tl.row0 = st.offsets[e_cursor] + j * nt;
    tl.rows = min(nt, count - j * nt);
    tl.tok = round_up(tl.rows, kPair ? 32 : 16);
    return tl;
}

__device__ __forceinline__ void group_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <bool kFp8, int kMode, bool kGated, bool kPair>
__global__ void __launch_bounds__(kThreads, 1)
moe_GemmGrouped_GemmUniversal_tcgen05_wm(const __grid_constant__ Maps maps, const Params p) {
    pdl_launch();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    SharedTail& st = *reinterpret_cast<SharedTail*>(smem + kStageArea);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    constexpr int kKElems = kFp8 ? kKBytes : kKBytes / 2;
    constexpr int kKind = kFp8 ? 0 : 1;               // kind::f8f6f4, kind::f16
    constexpr int kCtaCols = kGated ? kWRows / 2 : kWRows;   // output columns per CTA
    // In a pair, CTA 0 (the leader) issues the MMAs for both and owns the barriers they wait on.
    const int cta_rank = kPair ? int(ptx::cluster_ctarank()) : 0;
    const bool leader = cta_rank == 0;
    const int tile_first = kPair ? int(blockIdx.x >> 1) : int(blockIdx.x);
    const int tile_step = kPair ? int(gridDim.x >> 1) : int(gridDim.x);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            ptx::mbar_init(&st.full[s], 1);
            ptx::mbar_init(&st.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(&st.tmem_full[b], 1);
            ptx::mbar_init(&st.tmem_empty[b], kPair ? 2 * kEpiWarps : kEpiWarps);  // both CTAs' epilogue warps
        }
        st.abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async();
    }
    if constexpr (kPair) ptx::cluster_sync();  // the peer's barriers exist before anything signals them
    if (warp == 1) {
        if constexpr (kPair) {
            ptx::tmem_alloc_pair(&st.tmem_base, kTmemCols);
            ptx::tmem_relinquish_pair();
        } else {
            ptx::tmem_alloc(&st.tmem_base, kTmemCols);
            ptx::tmem_relinquish();
        }
    }
    pdl_wait();  // from here on global memory is read
    for (int i = threadIdx.x; i <= p.E; i += kThreads) st.offsets[i] = p.offsets[i];
    __syncthreads();
    if (warp == 2) {  // token tiles per expert, cumulative, and the largest
        int run = 0, largest = 0;
        for (int e0 = 0; e0 < p.E; e0 += 32) {
            const int e = e0 + lane;
            const int count = e < p.E ? st.offsets[e + 1] - st.offsets[e] : 0;
            const int tiles = (count + kMaxTok - 1) / kMaxTok;
            if (tiles > 0) largest = max(largest, tile_tokens<kPair>(count, tiles));
            int sum = tiles;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += up;
            }
            if (e < p.E) st.tprefix[e + 1] = run + sum;
            run += __shfl_sync(0xffffffffu, sum, 31);
        }
        largest = __reduce_max_sync(0xffffffffu, largest);
        if (lane == 0) {
            st.tprefix[0] = 0;
            st.max_tok = largest;
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    if constexpr (kPair) ptx::cluster_sync();  // both CTAs hold their TMEM before the first pair MMA
    ptx::tc_fence_after();

    const uint32_t tmem_base = st.tmem_base;
    const int total_tiles = st.tprefix[p.E] * p.w_tiles;
    volatile int* abort_flag = &st.abort_flag;
    const int kb_count = p.kb_count;
    const uint32_t stage_bytes = kABytes + uint32_t(st.max_tok) * (kPair ? kKBytes / 2 : kKBytes);
    const int stages = min(kMaxStages, int(kStageArea / stage_bytes));

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (ptx::elect_one()) {
            ptx::prefetch_tensormap(&maps.w);
            for (int i = 0; i < 4; ++i) ptx::prefetch_tensormap(&maps.rows[i]);
            int s = 0;
            uint32_t ph = 0;
            int e_cursor = 0;
            bool ok = true;
            for (int t = tile_first; ok && t < total_tiles; t += tile_step) {
                const Tile tl = decode_tile<kPair>(t, e_cursor, st, p.w_tiles);
                const int unit = tl.wt * (kPair ? 2 : 1) + cta_rank;        // this CTA's 64 or 128 output columns
                const int rows_here = kPair ? tl.tok / 2 : tl.tok;          // each CTA of a pair loads half of the tokens
                const int row_first = tl.row0 + (kPair ? cta_rank * rows_here : 0);
                const uint32_t bytes = kABytes + uint32_t(rows_here) * kKBytes;
                for (int kb = 0; kb < kb_count; ++kb) {
                    if (!ptx::mbar_wait(&st.empty[s], ph ^ 1u, abort_flag, kWaitLimit)) {
                        ok = false;
                        break;
                    }
                    uint8_t* sw = smem + size_t(s) * stage_bytes;
                    uint8_t* sr = sw + kABytes;
                    const int k0 = kb * kKElems;
                    // all bytes of a pair are credited to the leader's barrier
                    uint32_t bar;
                    if constexpr (kPair) {
                        bar = ptx::map_to_cta(&st.full[s], 0);
                        if (leader) ptx::mbar_arrive_expect_tx(&st.full[s], 2 * bytes);
                    } else {
                        bar = ptx::smem_u32(&st.full[s]);
                        ptx::mbar_arrive_expect_tx(&st.full[s], bytes);
                    }
                    if constexpr (kGated)
                        ptx::tma_load_5d<kPair>(sw, &maps.w, k0, 0, 0, unit * (kCtaCols / 8), tl.e, bar);
                    else
                        ptx::tma_load_3d<kPair>(sw, &maps.w, k0, unit * kCtaCols, tl.e, bar);
                    int r = row_first;
                    auto rows_box = [&](int i) {
                        ptx::tma_load_2d_any<kPair>(sr, &maps.rows[i], k0, r, bar);
                        sr += (kKBytes * 16) << i;
                        r += 16 << i;
                    };
                    for (int left = rows_here >> 7; left > 0; --left) rows_box(3);
                    if (rows_here & 64) rows_box(2);
                    if (rows_here & 32) rows_box(1);
                    if (rows_here & 16) rows_box(0);
                    if (++s == stages) s = 0, ph ^= 1u;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (leader && ptx::elect_one()) {
            // operand format code: e4m3 = 0 (kind::f8f6f4); bf16 = 1 (kind::f16)
            constexpr uint32_t idesc0 = ptx::make_idesc(kFp8 ? 0u : 1u, kPair ? 2 * kWRows : kWRows, 0);
            const uint64_t desc0 = ptx::smem_desc_sw128(ptx::smem_u32(smem));
            // completion of everything issued so far -> one barrier (of both CTAs in a pair)
            auto commit = [&](uint64_t* bar) {
                if constexpr (kPair) {
                    ptx::umma_commit_pair(ptx::map_to_cta(bar, 0));
                    ptx::umma_commit_pair(ptx::map_to_cta(bar, 1));
                } else {
                    ptx::umma_commit(bar);
                }
            };
            int s = 0;
            uint32_t ph = 0;
            uint32_t acc_it = 0;
            int e_cursor = 0;
            bool ok = true;
            for (int t = tile_first; ok && t < total_tiles; t += tile_step, ++acc_it) {
                const Tile tl = decode_tile<kPair>(t, e_cursor, st, p.w_tiles);
                const uint32_t idesc = idesc0 | (uint32_t(tl.tok) >> 3) << 17;
                const uint32_t buf = acc_it & 1u;
                if (!ptx::mbar_wait(&st.tmem_empty[buf], ((acc_it >> 1) & 1u) ^ 1u, abort_flag, kWaitLimit)) break;
                ptx::tc_fence_after();
                const uint32_t d_tmem = tmem_base + buf * kMaxTok;
                for (int kb = 0; kb < kb_count; ++kb) {
                    if (!ptx::mbar_wait(&st.full[s], ph, abort_flag, kWaitLimit)) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint64_t dw = ptx::smem_desc_advance(desc0, uint32_t(s) * stage_bytes);
                    const uint64_t dr = ptx::smem_desc_advance(dw, kABytes);
#pragma unroll
                    for (int k = 0; k < kKBytes / kUmmaKBytes; ++k) {
                        const uint32_t accumulate = kb == 0 && k == 0 ? 0u : 1u;
                        if constexpr (kPair)
                            ptx::umma_pair<kKind>(d_tmem, ptx::smem_desc_advance(dw, k * kUmmaKBytes),
                                                  ptx::smem_desc_advance(dr, k * kUmmaKBytes), idesc, accumulate);
                        else
                            ptx::umma<kKind>(d_tmem, ptx::smem_desc_advance(dw, k * kUmmaKBytes),
                                             ptx::smem_desc_advance(dr, k * kUmmaKBytes), idesc, accumulate);
                    }
                    commit(&st.empty[s]);
                    if (++s == stages) s = 0, ph ^= 1u;
                }
                if (!ok) break;
                commit(&st.tmem_full[buf]);
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        // ------------------------------------------------------------ epilogue warps
        // Two warpgroups share a tile: each takes every other 32 tokens, 16 at a time through its store buffers. A
        // warpgroup's warps meet at named barriers; a warp whose wait gave up goes on to all of them without storing.
        const int q = warp & 3;            // TMEM lane quarter this warp may read
        const int h = (warp - 4) >> 2;     // warpgroup
        const int wg_thread = threadIdx.x & 127;
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
        uint32_t acc_it = 0;
        uint32_t sub_it = 0;
        uint32_t amax2 = 0;                // tensor mode: running maximum of |act|, bf16 pairs
        int e_cursor = 0;
        bool ok = true;
        auto release_tmem = [&](uint32_t b) {  // one arrival per warp, after all of its lanes are done with the buffer
            __syncwarp();
            if (lane != 0) return;
            if constexpr (kPair)
                ptx::mbar_arrive_cluster(ptx::map_to_cta(&st.tmem_empty[b], 0));
            else
                ptx::mbar_arrive(&st.tmem_empty[b]);
        };

        for (int t = tile_first; t < total_tiles; t += tile_step, ++acc_it) {
            const Tile tl = decode_tile<kPair>(t, e_cursor, st, p.w_tiles);
            const uint32_t buf = acc_it & 1u;
            const int col_cta = (tl.wt * (kPair ? 2 : 1) + cta_rank) * kCtaCols;
            {   // where the tile's tokens go, and their scales: one token per thread
                const int tok = threadIdx.x - 4 * 32;
                unsigned long long dst = 0;
                if (tok < tl.rows) {
                    const int row = tl.row0 + tok;
                    const int out_row = kGated ? row : p.dest_to_src[row];
                    if (out_row >= 0) dst = reinterpret_cast<unsigned long long>(p.out) + size_t(out_row) * p.N * 2;
                    if constexpr (kMode == kChannel) st.sa[buf][tok] = p.sa[row];
                }
                st.dst[buf][tok] = dst;
            }
            // this thread's weight rows r and r + 8 of the warp's two 16-row groups: scale and bias
            const bool has_bias = p.bias != nullptr;
            float sw[2][2], bw[2][2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    int wr;
                    if constexpr (kGated)
                        wr = min(col_cta + q * 16 + i * 8 + (lane >> 2), p.N - 1) + v * p.N;
                    else
                        wr = min(col_cta + q * 32 + i * 16 + v * 8 + (lane >> 2), p.N - 1);
                    sw[i][v] = 1.0f;
                    if constexpr (kMode == kChannel) sw[i][v] = p.sb[size_t(tl.e) * p.w_rows + wr];
                    if constexpr (kMode == kTensor) sw[i][v] = p.sa[0] * p.sb[tl.e];
                    bw[i][v] = has_bias ? p.bias[size_t(tl.e) * p.w_rows + wr] : 0.0f;
                }
            group_sync(3, kEpiWarps * 32);
            if (ok) ok = ptx::mbar_wait_warp(&st.tmem_full[buf], (acc_it >> 1) & 1u, abort_flag, kWaitLimit);
            ptx::tc_fence_after();
            const uint32_t t_buf = t_lane + buf * kMaxTok;
            if (h * 32 >= tl.tok) {
                ptx::tc_fence_before();
                release_tmem(buf);
            }
            for (int c = h * 32; c < tl.tok; c += 64) {
                // fragment registers 4g .. 4g+3: tokens c + 8g + 2 (lane % 4) + {0, 1} of row lane / 4, then of row lane / 4 + 8
                uint32_t f[2][16];
                ptx::tmem_ld_16x256b_x4(t_buf + c, f[0]);
                ptx::tmem_ld_16x256b_x4(t_buf + (16u << 16) + c, f[1]);
                ptx::tmem_wait_ld16(f[0], f[1]);
                if (c + 64 >= tl.tok) {
                    ptx::tc_fence_before();
                    release_tmem(buf);
                }
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                    const int c0 = c + sub * kSub;
                    if (c0 >= tl.rows) break;
                    uint4* stage = st.stage[h][sub_it & 1u];
                    ++sub_it;
                    uint32_t o[2][2][2];  // [16-row group][row, row + 8 (plain only)][8 tokens]
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        float s0 = 1.0f, s1 = 1.0f;
                        if constexpr (kMode == kChannel) {
                            const float2 s = *reinterpret_cast<const float2*>(&st.sa[buf][c0 + g * 8 + 2 * (lane & 3)]);
                            s0 = s.x, s1 = s.y;
                        }
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t* x = &f[i][(sub * 2 + g) * 4];
                            float y[2][2];
#pragma unroll
                            for (int v = 0; v < 2; ++v) {
                                y[v][0] = __uint_as_float(x[2 * v]) * (s0 * sw[i][v]) + bw[i][v];
                                y[v][1] = __uint_as_float(x[2 * v + 1]) * (s1 * sw[i][v]) + bw[i][v];
                            }
                            if constexpr (kGated) {
                                o[i][0][g] = swiglu_bf16x2(y[0][0], y[0][1], y[1][0], y[1][1]);
                            } else {
                                o[i][0][g] = pack_bf16x2(y[0][0], y[0][1]);
                                o[i][1][g] = pack_bf16x2(y[1][0], y[1][1]);
                            }
                        }
                    }
                    // fragments -> token rows of kCtaCols columns; 16-byte pieces are XOR-swizzled against bank conflicts
                    constexpr int kPieces = kCtaCols / 8;
                    const int tok_st = ((lane >> 3) & 1) * 8 + (lane & 7);
                    if constexpr (kGated) {
                        const int piece = q * 2 + (lane >> 4);
                        ptx::stmatrix_x4_trans(&stage[tok_st * kPieces + (piece ^ (tok_st & 7))], o[0][0][0], o[0][0][1], o[1][0][0],
                                               o[1][0][1]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int piece = q * 4 + i * 2 + (lane >> 4);
                            ptx::stmatrix_x4_trans(&stage[tok_st * kPieces + (piece ^ (tok_st & 7))], o[i][0][0], o[i][0][1],
                                                   o[i][1][0], o[i][1][1]);
                        }
                    }
                    group_sync(1 + h, 128);
#pragma unroll
                    for (int u = 0; u < kSub * kPieces / 128; ++u) {
                        const int at = u * 128 + wg_thread;
                        const int tok = at / kPieces, piece = at % kPieces;
                        const uint4 v = stage[tok * kPieces + (piece ^ (tok & 7))];
                        const unsigned long long dst = st.dst[buf][c0 + tok];
                        const int col = col_cta + piece * 8;
                        const bool store = ok && dst != 0 && col < p.N;  // N is a multiple of 8
                        if (store) st16(reinterpret_cast<uint8_t*>(dst) + size_t(col) * 2, Vec16{v.x, v.y, v.z, v.w});
                        if constexpr (kGated && kMode != kNone) {
                            uint32_t m2 = kMode == kTensor ? amax2 : 0u;
                            if (store) {
                                amax_bf16x2(m2, v.x);
                                amax_bf16x2(m2, v.y);
                                amax_bf16x2(m2, v.z);
                                amax_bf16x2(m2, v.w);
                            }
                            if constexpr (kMode == kTensor) {
                                amax2 = m2;
                            } else {  // eight lanes hold a token's columns
#pragma unroll
                                for (int d = 1; d < 8; d <<= 1) amax_bf16x2(m2, __shfl_xor_sync(0xffffffffu, m2, d));
                                if (store && piece == 0) atomic_max_nonneg(p.amax + tl.row0 + c0 + tok, amax_bf16x2_value(m2));
                            }
                        }
                    }
                }
            }
        }
        if constexpr (kGated && kMode == kTensor) {
            const float m = warp_max(amax_bf16x2_value(amax2));
            if (lane == 0 && m > 0.0f) atomic_max_nonneg(p.amax, m);
        }
    }

    // ---------------------------------------------------------------- teardown
    if (*abort_flag != 0) {
        // a wait gave up: report instead of trapping, let copies in flight land, then free TMEM
        if (threadIdx.x == 0 && p.status != nullptr) {
            *reinterpret_cast<volatile int*>(p.status) = 160 + (kGated ? 0 : 10) + kMode;
            __threadfence_system();
        }
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before();
    __syncthreads();
    if constexpr (kPair) ptx::cluster_sync();  // the peer has stopped using this CTA's barriers and TMEM
    if (warp == 1) {
        ptx::tc_fence_after();
        if constexpr (kPair)
            ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
        else
            ptx::tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ---------------------------------------------------------------- host side

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
            DQ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemBytes)));
            configured[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(kPair ? sm_count() & ~1 : sm_count()), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = kSmemBytes;
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

// Arguments as gemm::grouped_gemm takes them; bf16 and per-tensor / per-channel FP8 operands.
int grouped_gemm(const void* a, const float* a_scale, const void* w, const float* w_scale, const int* offsets, int n, int N, int K,
                 int E, int quant_mode, int gated, void* out, float* amax, const int* dest_to_src, const float* bias,
                 cudaStream_t stream) {
    DQ_CHECK(quant_mode == DQMOE_QUANT_NONE || quant_mode == DQMOE_QUANT_FP8_TENSOR || quant_mode == DQMOE_QUANT_FP8_CHANNEL);
    DQ_CHECK(n >= 0 && N > 0 && K > 0 && E > 0 && E <= kMaxExperts);
    if (n == 0) return DQMOE_OK;
    const bool fp8 = quant_mode != DQMOE_QUANT_NONE;
    const int esz = fp8 ? 1 : 2;
    DQ_CHECK_FMT((size_t(K) * esz) % 16 == 0, "K=%d: rows must be a multiple of 16 bytes", K);
    DQ_CHECK_FMT(N % 8 == 0, "N=%d: output rows must be 16-byte vectors", N);
    DQ_CHECK(is_aligned(a, 16) && is_aligned(w, 16) && is_aligned(out, 16));
    DQ_CHECK(a != nullptr && w != nullptr && out != nullptr && offsets != nullptr && (gated || dest_to_src != nullptr));
    if (fp8) DQ_CHECK(a_scale != nullptr && w_scale != nullptr && (!gated || amax != nullptr));

    const bool pair = n / E >= 24;
    const int cta_cols = gated ? kWRows / 2 : kWRows;
    Params p;
    p.n_rows = n;
    p.N = N;
    p.E = E;
    p.w_rows = gated ? 2 * N : N;
    p.w_tiles = ceil_div(N, pair ? 2 * cta_cols : cta_cols);
    p.kb_count = ceil_div(K * esz, kKBytes);
    p.offsets = offsets;
    p.sa = a_scale;
    p.sb = w_scale;
    p.out = out;
    p.amax = amax;
    p.bias = bias;
    p.dest_to_src = dest_to_src;
    p.status = device_status_word();
    if (p.status == nullptr) return DQMOE_ERR_CUDA;

    Maps maps;
    DQ_RC(make_weight_map(&maps.w, w, esz, E, N, K, gated != 0));
    for (int i = 0; i < 4; ++i) DQ_RC(gemm::make_map(&maps.rows[i], a, esz, uint64_t(n), uint64_t(K), 16 << i));

#define DQ_WM_LAUNCH(FP8, MODE)                                                                                         \
    (gated ? (pair ? launch<FP8, MODE, true, true>(maps, p, stream) : launch<FP8, MODE, true, false>(maps, p, stream))  \
           : (pair ? launch<FP8, MODE, false, true>(maps, p, stream) : launch<FP8, MODE, false, false>(maps, p, stream)))
    switch (quant_mode) {
        case DQMOE_QUANT_NONE: return DQ_WM_LAUNCH(false, kNone);
        case DQMOE_QUANT_FP8_TENSOR: return DQ_WM_LAUNCH(true, kTensor);
        default: return DQ_WM_LAUNCH(true, kChannel);
    }
#undef DQ_WM_LAUNCH
}

}  // namespace gemm_wm
}  // namespace dq
