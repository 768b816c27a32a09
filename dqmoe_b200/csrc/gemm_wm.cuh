// Grouped GEMM with the weights on the M side of the tensor core: D[weight row][token] = W A^T. A tile is 128 weight
// rows per CTA (64 gate and 64 value rows in fc1) by up to 256 rows of one expert, in steps of 16 (32 on a CTA pair), so
// an expert of 300 rows computes 304 or 320 of them, where tiles with the rows on M compute 384 or 512. Used by the layer
// for bf16 and per-tensor / per-channel FP8 operands, and in block mode (tiles of up to 64 rows) for few rows per expert; gemm_sm100.cu
// has the form with the rows on M.
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
// Row tiles (gemm_sm100.cu) / this form, us per layer call: per-tensor FP8 at the Mixtral shape (H 4096, I 14336, E 8, k 2) 16 tokens
// 261 / 240, 777 with biases 427 / 380; per-channel 16384 x 8 (H 2048, I 768, E 128) 919 / 852; bf16 16384 x 3 (2880 x 2880, E 64)
// 2523 / 2303. Tiles of 128 instead of 256 tokens cost bf16's fc1 1545 instead of 1207 us: operands through L2 and their energy count,
// the chip runs these launches at 1.3-1.6 GHz under its power limit.
//
// Replaces the same reference kernels as gemm_sm100.cu (csrc/moe_gemm_template.h:72-1039, csrc/moe_kernels.h:301-444, 581-620).
#pragma once

#include <type_traits>

#include "common.cuh"
#include "gemm_tile.cuh"
#include "ptx_sm100.cuh"

namespace dq {
namespace gemm_wm {

constexpr int kWRows = 128;                       // weight rows per CTA = lanes of TMEM
constexpr int kMaxTok = 256;                      // rows of an expert per tile
constexpr int kBlockTok = 64;                     // the same in block mode
constexpr int kKBytes = 128;                      // K bytes per stage: one 128-byte swizzle row
constexpr int kUmmaKBytes = 32;                   // K bytes per tcgen05.mma
constexpr int kABytes = kWRows * kKBytes;         // 16 KiB
// Bytes of the stages: four 256-token tiles of a single CTA or six of a pair; in block mode, which needs room for scales and the
// re-quantisation, seven of 64 tokens, ten of 16.
constexpr int stage_area(bool block) { return block ? 180 * 1024 : 4 * (kABytes + kMaxTok * kKBytes); }
constexpr int kMaxStages = 10;
constexpr int kThreads = 384;                     // warp 0 TMA, warp 1 MMA, warp 2 scale products (block mode), warp 3 idle, warps 4..11 epilogue
constexpr int kEpiWarps = 8;
constexpr int kMaxExperts = 1024;
constexpr int kTmemCols = 512;                    // two accumulator buffers of up to 256 tokens
constexpr int kSub = 16;                          // tokens per pass through the store buffers
constexpr long long kWaitLimit = 1000000000LL;    // clock cycles before a wait gives up (~0.5 s)

enum Mode : int { kNone = 0, kTensor = 1, kChannel = 2, kBlock = 3 };

struct Params {
    int n_rows;               // rows of A (expanded rows n)
    int N;                    // output columns (fc1: I, fc2: H)
    int E;
    int w_rows;               // weight rows per expert (fc1: 2I, fc2: H)
    int w_tiles;              // tiles per expert along the output columns
    int kb_count;             // ceil(K bytes / 128)
    const int* offsets;       // [E+1] first row of each expert
    const float* sa;          // activation scales: tensor [1], channel [n], block [ceil(K/128)][n_pad]
    const float* sb;          // weight scales: tensor [E], channel [E, w_rows], block [E, ceil(w_rows/128), ceil(K/128)]
    void* out;
    float* amax;              // fc1: channel [n], tensor [1]
    float* out_scale;         // fc1, block mode: [n, ceil(I/128)]
    float* out_scale_t;       // the same by column, [ceil(I/128)][n_pad]
    int n_pad;                // rows of the scale matrices by column
    const float* bias;        // [E, w_rows] fp32 added to the dequantised product, or nullptr
    const int* dest_to_src;   // fc2: output row of each row
    int* status;              // host-mapped status word
};

struct Maps {
    CUtensorMap w;            // weights: fc1 [E][I/8][gate, value][8][K], fc2 [E][H][K]
    CUtensorMap rows[4];      // activation rows, boxes of 16, 32, 64 and 128 rows
};

// What a launch needs, made by form() (gemm_wm_sm100.cu).
struct Form {
    Maps maps;
    Params p;
    bool pair;
};

constexpr int kProdTok = kTmemCols;               // scale products: one token per accumulator column
constexpr int kAccBufs = 4;                       // accumulator buffers of block mode, of two or four K blocks each

struct BlockTail {
    uint64_t prod_empty[kAccBufs];                // the epilogue warps are done with the products of an accumulator buffer
    // fc1: per pair of tokens the products of their scales with that of the gate rows (x, y) and of the value rows (z, w); the
    // second array with the value rows' second scale block, where there is one. fc2: one product per token, packed.
    alignas(16) float prod[2][kProdTok * 2];
    float amax[2][kBlockTok], inv[kBlockTok];     // fc1: of each token's columns in the tile's first and second half
};
struct RowScaleTail {
    float sa[2][kMaxTok];                         // channel mode: the activation scale of each token of the tile
};

template <bool kBlockMode>
struct SharedTail : std::conditional_t<kBlockMode, BlockTail, RowScaleTail> {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t tmem_full[kAccBufs];
    uint64_t tmem_empty[kAccBufs];
    uint32_t tmem_base;
    int abort_flag;
    int max_tok;                                  // tokens of the largest tile
    unsigned long long dst[2][kMaxTok];           // output row of each token of the tile, 0 = none
    alignas(16) uint4 stage[2][2][kSub * 16];     // per epilogue warpgroup: two buffers of 16 tokens x (64 or 128 columns)
    int tprefix[kMaxExperts + 1];                 // cumulative token tiles
    int offsets[kMaxExperts + 1];
};

template <bool kBlockMode>
constexpr size_t smem_bytes() { return 1024 + size_t(stage_area(kBlockMode)) + sizeof(SharedTail<kBlockMode>); }
static_assert(smem_bytes<false>() <= 227 * 1024 && smem_bytes<true>() <= 227 * 1024, "shared memory of one CTA");

// An expert's rows in units of 16 (32 on a pair) are spread over its tiles as evenly as whole units allow: the first tiles take one
// more than the others. With tiles of one size, rounded up, 780 rows on pairs were 4 x 224 = 896, now 224 + 3 x 192 = 800.
template <bool kPair>
constexpr int kUnit = kPair ? 32 : 16;
template <bool kPair>
__device__ __forceinline__ int largest_tile(int count, int tiles) {
    const int units = (count + kUnit<kPair> - 1) / kUnit<kPair>;
    return (units + tiles - 1) / tiles * kUnit<kPair>;
}

// Block mode starts an expert's first tile at a multiple of four rows, so that the scales of four rows are one aligned vector;
// the rows before the expert's own are computed and dropped.
template <bool kBlockMode>
__device__ __forceinline__ int expert_base(int offset) { return kBlockMode ? offset & ~3 : offset; }
template <bool kBlockMode>
__device__ __forceinline__ int expert_rows(int offset, int end) { return end > offset ? end - expert_base<kBlockMode>(offset) : 0; }

struct Tile {
    int e, wt, row0, rows, tok;  // expert, tile along the output columns, first row, rows, tokens computed (rows rounded up)
};

// Tiles are numbered expert-major; inside an expert the token tile runs fastest, so that concurrently running CTAs share
// one weight tile.
template <bool kPair, bool kBlockMode>
__device__ __forceinline__ Tile decode_tile(int t, int& e_cursor, const SharedTail<kBlockMode>& st, int w_tiles) {
    while (t >= st.tprefix[e_cursor + 1] * w_tiles) ++e_cursor;
    const int local = t - st.tprefix[e_cursor] * w_tiles;
    const int tiles = st.tprefix[e_cursor + 1] - st.tprefix[e_cursor];
    const int count = expert_rows<kBlockMode>(st.offsets[e_cursor], st.offsets[e_cursor + 1]);
    const int units = (count + kUnit<kPair> - 1) / kUnit<kPair>;
    const int each = units / tiles, more = units - each * tiles;
    Tile tl;
    tl.e = e_cursor;
    tl.wt = local / tiles;
    const int j = local - tl.wt * tiles;
    const int first = (j * each + min(j, more)) * kUnit<kPair>;
    tl.row0 = expert_base<kBlockMode>(st.offsets[e_cursor]) + first;
    tl.tok = (each + (j < more ? 1 : 0)) * kUnit<kPair>;
    tl.rows = min(tl.tok, count - first);
    return tl;
}

// two fp32 FMAs in one instruction (packed fp32 of sm_100): a += x * s
__device__ __forceinline__ void ffma2(float& a0, float& a1, uint32_t x0, uint32_t x1, float s0, float s1) {
    const float2 r = __ffma2_rn(make_float2(__uint_as_float(x0), __uint_as_float(x1)), make_float2(s0, s1), make_float2(a0, a1));
    a0 = r.x;
    a1 = r.y;
}

// Block mode: accumulator columns of one K block of a tile, and K blocks per 128-column buffer. Few tokens put several K blocks
// in one buffer, so that the hand-over between tensor core and epilogue (some 1000 cycles for a warp's wait, loads, products and
// release, however few tokens there are) is made once for up to four of them.
__device__ __forceinline__ int block_cols(int tok) { return tok > 32 ? 64 : 32; }

__device__ __forceinline__ void group_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <bool kFp8, int kMode, bool kGated, bool kPair>
__device__ __forceinline__ void weights_on_m(const Maps& maps, const Params& p) {
    constexpr bool kEarly = !kPair;  // see below
    if constexpr (!kEarly) pdl_launch();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr bool kBlockMode = kMode == kBlock;
    constexpr int kStageArea = stage_area(kBlockMode);
    SharedTail<kBlockMode>& st = *reinterpret_cast<SharedTail<kBlockMode>*>(smem + kStageArea);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    constexpr int kKElems = kFp8 ? kKBytes : kKBytes / 2;
    constexpr int kKind = kFp8 ? 0 : 1;               // kind::f8f6f4, kind::f16
    constexpr int kCtaCols = kGated ? kWRows / 2 : kWRows;   // output columns per CTA and pass
    static_assert(!kBlockMode || (kFp8 && !kPair), "block mode: e4m3, single CTAs");
    constexpr int kBufs = kBlockMode ? kAccBufs : 2;  // accumulator buffers
    constexpr int kBufCols = kTmemCols / kBufs;
    // fc1 in block mode re-quantises groups of 128 columns, two passes of a CTA over the same tokens
    constexpr int kPassMax = kBlockMode && kGated ? 2 : 1;
    constexpr int kTileCols = kCtaCols * kPassMax * (kPair ? 2 : 1);
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
        for (int b = 0; b < kBufs; ++b) {
            ptx::mbar_init(&st.tmem_full[b], kBlockMode ? 2 : 1);                  // block mode: and the warp of the scale products
            ptx::mbar_init(&st.tmem_empty[b], kPair ? 2 * kEpiWarps : kEpiWarps);  // both CTAs' epilogue warps
            if constexpr (kBlockMode) ptx::mbar_init(&st.prod_empty[b], kEpiWarps);
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
    // kEarly: launched as a dependent, this kernel starts while the one before it still runs, but not before the expert sort and all
    // that came before it are complete, since the kernels in between (the row scatter, fc1) let their dependents start only after
    // their own wait (the re-quantisation pass between fc1 and fc2 before it, but it starts only after fc1's). So the row counts are
    // there, and are read past L1, and so are the weights: the first stages' weights are fetched before the wait, by TMA and so from
    // L2 on, and every role that touches what the kernel before reads or writes waits for itself. Without / with, us per call: per-tensor
    // 9 tokens at the Mixtral shape 235.5 / 227.0, bf16 438 / 421, MoE block of 5 tokens (H 1024, I 2048) 30.4 / 27.7, 96 tokens
    // (H 7168, I 2048, E 33) 278 / 278. Not on pairs: 777 tokens 389 / 396, the weights then contend with the re-quantisation pass.
    if constexpr (!kEarly) pdl_wait();
    for (int i = threadIdx.x; i <= p.E; i += kThreads) st.offsets[i] = ld_relaxed_gpu(p.offsets + i);
    __syncthreads();
    if (warp == 2) {  // token tiles per expert, cumulative, and the largest
        int run = 0, largest = 0;
        for (int e0 = 0; e0 < p.E; e0 += 32) {
            const int e = e0 + lane;
            const int count = e < p.E ? expert_rows<kBlockMode>(st.offsets[e], st.offsets[e + 1]) : 0;
            constexpr int kLimit = kBlockMode ? kBlockTok : kMaxTok;
            const int tiles = (count + kLimit - 1) / kLimit;
            if (tiles > 0) largest = max(largest, largest_tile<kPair>(count, tiles));
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
    // passes of the tile at column tile wt
    auto passes = [&](int wt) { return kPassMax == 2 && wt * kTileCols + kCtaCols < p.N ? 2 : 1; };

    if (warp < 4) {

      if (warp == 0) {
          // ------------------------------------------------------------ TMA producer
          if (ptx::elect_one()) {
              ptx::prefetch_tensormap(&maps.w);
              // announces a stage's bytes (all those of a pair to the leader's barrier) and fetches its weights
              auto load_weights = [&](const Tile& tl, int pass, int kb, int s) {
                  const int col = tl.wt * kTileCols + (pass + cta_rank) * kCtaCols;  // this CTA's 64 or 128 output columns
                  const uint32_t bytes = kABytes + uint32_t(kPair ? tl.tok / 2 : tl.tok) * kKBytes;
                  uint8_t* sw = smem + size_t(s) * stage_bytes;
                  uint32_t bar;
                  if constexpr (kPair) {
                      bar = ptx::map_to_cta(&st.full[s], 0);
                      if (leader) ptx::mbar_arrive_expect_tx(&st.full[s], 2 * bytes);
                  } else {
                      bar = ptx::smem_u32(&st.full[s]);
                      ptx::mbar_arrive_expect_tx(&st.full[s], bytes);
                  }
                  if constexpr (kGated)
                      ptx::tma_load_5d<kPair>(sw, &maps.w, kb * kKElems, 0, 0, col / 8, tl.e, bar);
                  else
                      ptx::tma_load_3d<kPair>(sw, &maps.w, kb * kKElems, col, tl.e, bar);
              };
              int ahead = 0;  // stages whose weights are on their way before the wait
              for (int t = tile_first, cursor = 0; kEarly && ahead < stages && t < total_tiles; t += tile_step) {
                  const Tile tl = decode_tile<kPair, kBlockMode>(t, cursor, st, p.w_tiles);
                  for (int pass = 0; pass < passes(tl.wt); ++pass)
                      for (int kb = 0; ahead < stages && kb < kb_count; ++kb, ++ahead) load_weights(tl, pass, kb, ahead);
              }
              pdl_wait();
              int s = 0;
              uint32_t ph = 0;
              int e_cursor = 0;
              bool ok = true;
              for (int t = tile_first; ok && t < total_tiles; t += tile_step) {
                  const Tile tl = decode_tile<kPair, kBlockMode>(t, e_cursor, st, p.w_tiles);
                  const int rows_here = kPair ? tl.tok / 2 : tl.tok;          // each CTA of a pair loads half of the tokens
                  const int row_first = tl.row0 + (kPair ? cta_rank * rows_here : 0);
                  for (int pass = 0; ok && pass < passes(tl.wt); ++pass) {
                      for (int kb = 0; kb < kb_count; ++kb) {
                          if (ahead > 0) {
                              --ahead;
                          } else {
                              if (!ptx::mbar_wait(&st.empty[s], ph ^ 1u, abort_flag, kWaitLimit)) {
                                  ok = false;
                                  break;
                              }
                              load_weights(tl, pass, kb, s);
                          }
                          uint8_t* sr = smem + size_t(s) * stage_bytes + kABytes;
                          const int k0 = kb * kKElems;
                          uint32_t bar;
                          if constexpr (kPair)
                              bar = ptx::map_to_cta(&st.full[s], 0);
                          else
                              bar = ptx::smem_u32(&st.full[s]);
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
          }
          __syncwarp();
      } else if (warp == 1) {
          // ------------------------------------------------------------ MMA issuer
          if (leader && ptx::elect_one()) {
              pdl_wait();  // no rows come before it, and the limit of the waits below is for this kernel's own time
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
              auto mma_stage = [&](uint32_t d_tmem, int s, uint32_t idesc, bool first) {
                  const uint64_t dw = ptx::smem_desc_advance(desc0, uint32_t(s) * stage_bytes);
                  const uint64_t dr = ptx::smem_desc_advance(dw, kABytes);
#pragma unroll
                  for (int k = 0; k < kKBytes / kUmmaKBytes; ++k) {
                      const uint32_t accumulate = first && k == 0 ? 0u : 1u;
                      if constexpr (kPair)
                          ptx::umma_pair<kKind>(d_tmem, ptx::smem_desc_advance(dw, k * kUmmaKBytes),
                                                ptx::smem_desc_advance(dr, k * kUmmaKBytes), idesc, accumulate);
                      else
                          ptx::umma<kKind>(d_tmem, ptx::smem_desc_advance(dw, k * kUmmaKBytes),
                                           ptx::smem_desc_advance(dr, k * kUmmaKBytes), idesc, accumulate);
                  }
              };
              int s = 0, buf = 0;
              uint32_t ph = 0, buf_ph = 0;
              auto next_buf = [&] {
                  if (++buf == kBufs) buf = 0, buf_ph ^= 1u;
              };
              int e_cursor = 0;
              bool ok = true;
              for (int t = tile_first; ok && t < total_tiles; t += tile_step) {
                  const Tile tl = decode_tile<kPair, kMode == kBlock>(t, e_cursor, st, p.w_tiles);
                  const uint32_t idesc = idesc0 | (uint32_t(tl.tok) >> 3) << 17;
                  if constexpr (!kBlockMode) {
                      if (!ptx::mbar_wait(&st.tmem_empty[buf], buf_ph ^ 1u, abort_flag, kWaitLimit)) break;
                      ptx::tc_fence_after();
                  }
                  const int cols = block_cols(tl.tok);
                  for (int pass = 0; ok && pass < passes(tl.wt); ++pass) {
                      for (int kb = 0, col = 0; kb < kb_count; ++kb) {
                          // block mode: the stage first - its barrier is long over - so that the MMAs follow the buffer's at once
                          if (!ptx::mbar_wait(&st.full[s], ph, abort_flag, kWaitLimit) ||
                              (kBlockMode && col == 0 && !ptx::mbar_wait(&st.tmem_empty[buf], buf_ph ^ 1u, abort_flag, kWaitLimit))) {
                              ok = false;
                              break;
                          }
                          ptx::tc_fence_after();
                          mma_stage(tmem_base + uint32_t(buf * kBufCols + col), s, idesc, kBlockMode || kb == 0);
                          commit(&st.empty[s]);
                          if (++s == stages) s = 0, ph ^= 1u;
                          if constexpr (kBlockMode) {
                              col += cols;
                              if (col == kBufCols || kb + 1 == kb_count) {
                                  commit(&st.tmem_full[buf]);
                                  next_buf();
                                  col = 0;
                              }
                          }
                      }
                  }
                  if constexpr (!kBlockMode) {
                      if (!ok) break;
                      commit(&st.tmem_full[buf]);
                      next_buf();
                  }
              }
          }
          __syncwarp();
      } else if (warp == 2) {
          // ------------------------------------------------------------ scale products (block mode)
          // Four tokens of one of a buffer's K blocks per lane: their activation scales, fetched four buffers ahead, times the
          // scales of this CTA's weight rows. The epilogue warps then read finished products, two tokens at a time, where each of them would
          // multiply the same pairs again. They find them behind the accumulator buffer's barrier, on which these warps arrive too.
          if constexpr (kBlockMode) {
              pdl_wait();
              const int KB = kb_count, NB = (p.w_rows + 127) / 128;
              const int at_buf = lane * 4;  // place in a buffer's products
              int buf = 0;
              uint32_t buf_ph = 0;
              int e_cursor = 0;
              bool ok = true;
              for (int t = tile_first; ok && t < total_tiles; t += tile_step) {
                  const Tile tl = decode_tile<kPair, kBlockMode>(t, e_cursor, st, p.w_tiles);
                  const int cols = block_cols(tl.tok), group = kBufCols / cols;
                  const int kb_mine = at_buf / cols, tok = at_buf % cols;
                  const bool mine = tok < tl.tok;
                  const float* sa = p.sa + tl.row0 + tok;
                  const float* sb = p.sb + size_t(tl.e) * NB * KB;
                  const int v0 = p.N + tl.wt * 128;  // fc1: first value row of the tile
                  const float* sb0 = sb + size_t(min(tl.wt, NB - 1)) * KB;
                  const float* sb1 = sb + size_t(min(v0 >> 7, NB - 1)) * KB;
                  const float* sb2 = sb + size_t(min((v0 >> 7) + 1, NB - 1)) * KB;
                  const bool split = kGated && (v0 & 127) != 0;
                  for (int pass = 0; ok && pass < passes(tl.wt); ++pass) {
                      auto load_sa = [&](int kb) {
                          return mine && kb < KB ? *reinterpret_cast<const float4*>(sa + size_t(kb) * p.n_pad) : make_float4(0.f, 0.f, 0.f, 0.f);
                      };
                      float4 ahead[4];
#pragma unroll
                      for (int u = 0; u < 4; ++u) ahead[u] = load_sa(u * group + kb_mine);
                      float w0 = 0.f, w1 = 0.f, w2 = 0.f, n0 = 0.f, n1 = 0.f, n2 = 0.f;  // weight scales of 32 K blocks, one per lane; the next 32
                      auto load_sb = [&](int kb) {
                          if (kb >= KB) return;
                          n0 = sb0[kb];
                          if constexpr (kGated) n1 = sb1[kb];
                          if (split) n2 = sb2[kb];
                      };
                      load_sb(lane);
                      for (int kb0 = 0; ok && kb0 < KB;) {
#pragma unroll
                          for (int u = 0; u < 4; ++u) {
                              if (kb0 >= KB) break;
                              if ((kb0 & 31) == 0) {
                                  w0 = n0, w1 = n1, w2 = n2;
                                  load_sb(kb0 + 32 + lane);
                              }
                              const float4 a = ahead[u];
                              ahead[u] = load_sa(kb0 + 4 * group + kb_mine);
                              const int from = (kb0 + kb_mine) & 31;
                              const float f0 = __shfl_sync(0xffffffffu, w0, from);
                              const float f1 = kGated ? __shfl_sync(0xffffffffu, w1, from) : 0.f;
                              const float f2 = split ? __shfl_sync(0xffffffffu, w2, from) : 0.f;
                              ok = ptx::mbar_wait_warp(&st.prod_empty[buf], buf_ph ^ 1u, abort_flag, kWaitLimit);
                              if (!ok) break;
                              if (mine) {
                                  const int at = buf * kBufCols + at_buf;
                                  if constexpr (kGated) {
                                      float4* d0 = reinterpret_cast<float4*>(st.prod[0] + at * 2);
                                      d0[0] = make_float4(a.x * f0, a.y * f0, a.x * f1, a.y * f1);
                                      d0[1] = make_float4(a.z * f0, a.w * f0, a.z * f1, a.w * f1);
                                      if (split) {
                                          float4* d1 = reinterpret_cast<float4*>(st.prod[1] + at * 2);
                                          d1[0] = make_float4(a.x * f0, a.y * f0, a.x * f2, a.y * f2);
                                          d1[1] = make_float4(a.z * f0, a.w * f0, a.z * f2, a.w * f2);
                                      }
                                  } else {
                                      *reinterpret_cast<float4*>(st.prod[0] + at) = make_float4(a.x * f0, a.y * f0, a.z * f0, a.w * f0);
                                  }
                              }
                              __syncwarp();
                              if (lane == 0) ptx::mbar_arrive(&st.tmem_full[buf]);
                              if (++buf == kBufs) buf = 0, buf_ph ^= 1u;
                              kb0 += group;
                          }
                      }
                  }
              }
          }
      }
    } else if constexpr (kBlockMode) {
        pdl_wait();
        if constexpr (kEarly) pdl_launch();  // after the wait: see above
        // ------------------------------------------------------------ epilogue warps, block mode
        // The first warpgroup has the first half of the tile's tokens, the second the other: up to 64 sums per thread.
        const int q = warp & 3;
        const int h = (warp - 4) >> 2;
        const int wg_thread = threadIdx.x & 127;
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
        constexpr int kPieces = kCtaCols / 8;
        const int tok_st = ((lane >> 3) & 1) * 8 + (lane & 7);                  // token of 16 and 16-byte piece that this thread
        const int tok_ld = wg_thread / kPieces, piece_ld = wg_thread % kPieces;  // writes to and reads from the store buffers
        int buf = 0;
        uint32_t buf_ph = 0;
        uint32_t sub_it = 0, tile_it = 0;
        int e_cursor = 0;
        bool ok = true;
        // one arrival per warp, after all of its lanes are done: the accumulator buffer to the MMA thread, its products to their warps
        auto release = [&](uint64_t* bar) {
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(bar);
        };

        for (int t = tile_first; t < total_tiles; t += tile_step, ++tile_it) {
            int count, tok0, group, n_pass, out_row = -1;  // out_row: fc2: where this thread's token of the tile goes; used after the K loop
            int split_at = 128;                     // fc1: column of the tile from which the value rows are in their second scale block
            {
                const Tile tl = decode_tile<kPair, kBlockMode>(t, e_cursor, st, p.w_tiles);
                const int first = (tl.tok / kSub + 1) / 2 * kSub;
                tok0 = h == 0 ? 0 : first;
                count = h == 0 ? first : tl.tok - first;
                group = kBufCols / block_cols(tl.tok);
                n_pass = passes(tl.wt);
                if constexpr (kGated) {
                    split_at = 128 - ((p.N + tl.wt * 128) & 127);
                } else {
                    const int tok = int(threadIdx.x) - 128, row = tl.row0 + tok;
                    if (tok < tl.rows && row >= st.offsets[tl.e] && row < st.offsets[tl.e + 1]) out_row = p.dest_to_src[row];
                }
            }

            // kUnits: 16-token units of this warpgroup; kGroup: K blocks per buffer
            auto tile_work = [&](auto units_tag, auto group_tag) {
                constexpr int kUnits = decltype(units_tag)::value, kGroup = decltype(group_tag)::value;
                constexpr int kCols = kBufCols / kGroup;
                [[maybe_unused]] uint4 act[kPassMax][kUnits];  // fc1: eight columns of a token per unit, bf16
#pragma unroll
                for (int pass = 0; pass < kPassMax; ++pass) {
                    if (pass >= n_pass) break;
                    const float* prod = st.prod[kGated && pass * kCtaCols + q * 16 >= split_at ? 1 : 0];
                    // acc[u][i][4g ..]: as the fragment registers, group i of 16 weight rows
                    float acc[kUnits][2][8];
#pragma unroll
                    for (int u = 0; u < kUnits; ++u)
#pragma unroll
                        for (int i = 0; i < 2; ++i)
#pragma unroll
                            for (int r = 0; r < 8; ++r) acc[u][i][r] = 0.0f;
                    bool ready = false;
                    for (int kb = 0; kb < kb_count; kb += kGroup) {
                        if (ok && !ready) ok = ptx::mbar_wait_warp(&st.tmem_full[buf], buf_ph, abort_flag, kWaitLimit);
                        ptx::tc_fence_after();
                        const int this_buf = buf;
                        uint32_t x[kGroup * kUnits][2][8];
                        const uint32_t t_buf = t_lane + uint32_t(this_buf * kBufCols + tok0);
#pragma unroll
                        for (int u = 0; u < kGroup * kUnits; ++u) {  // columns of K blocks past the last hold old sums, not used
                            const uint32_t at = t_buf + (u / kUnits) * kCols + (u % kUnits) * kSub;
                            ptx::tmem_ld_16x256b_x2(at, x[u][0]);
                            ptx::tmem_ld_16x256b_x2(at + (16u << 16), x[u][1]);
                        }
                        ptx::tmem_wait_ld_units(x);
                        ptx::tc_fence_before();
                        release(&st.tmem_empty[this_buf]);
                        if (++buf == kBufs) buf = 0, buf_ph ^= 1u;
                        // ask for the next buffer now: the answers arrive under the FMAs, and the lanes agree on one
                        const bool over = ptx::mbar_test_wait(&st.tmem_full[buf], buf_ph);
                        const float* prod_buf = prod + (this_buf * kBufCols + tok0 + 2 * (lane & 3)) * (kGated ? 2 : 1);
#pragma unroll
                        for (int b = 0; b < kGroup; ++b) {
                            if (b > 0 && kb + b >= kb_count) break;
#pragma unroll
                            for (int u = 0; u < kUnits; ++u)
#pragma unroll
                                for (int g = 0; g < 2; ++g) {
                                    float4 f;
                                    if constexpr (kGated) {
                                        f = *reinterpret_cast<const float4*>(prod_buf + (b * kCols + u * kSub + 8 * g) * 2);
                                    } else {
                                        const float2 f2 = *reinterpret_cast<const float2*>(prod_buf + b * kCols + u * kSub + 8 * g);
                                        f = make_float4(f2.x, f2.y, f2.x, f2.y);
                                    }
#pragma unroll
                                    for (int i = 0; i < 2; ++i) {
                                        const uint32_t* y = &x[b * kUnits + u][i][4 * g];
                                        ffma2(acc[u][i][4 * g], acc[u][i][4 * g + 1], y[0], y[1], f.x, f.y);
                                        ffma2(acc[u][i][4 * g + 2], acc[u][i][4 * g + 3], y[2], y[3], f.z, f.w);
                                    }
                                }
                        }
                        ready = __all_sync(0xffffffffu, over);
                        release(&st.prod_empty[this_buf]);
                    }

                    // ---- the sums of the pass are complete. What follows needs the tile again: in the K loop the registers are sums.
                    const Tile tl = decode_tile<kPair, kBlockMode>(t, e_cursor, st, p.w_tiles);
                    const int col_cta = tl.wt * kTileCols + pass * kCtaCols;
                    if constexpr (!kGated) {
                        st.dst[tile_it & 1u][threadIdx.x - 128] =
                            out_row >= 0 ? reinterpret_cast<unsigned long long>(p.out) + size_t(out_row) * p.N * 2 : 0ull;
                        group_sync(3, kEpiWarps * 32);
                    }
                    float bw[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
                    if (p.bias != nullptr) {
#pragma unroll
                        for (int i = 0; i < 2; ++i)
#pragma unroll
                            for (int v = 0; v < 2; ++v) {
                                const int wr = kGated ? min(col_cta + q * 16 + i * 8 + (lane >> 2), p.N - 1) + v * p.N
                                                      : min(col_cta + q * 32 + i * 16 + v * 8 + (lane >> 2), p.N - 1);
                                bw[i][v] = p.bias[size_t(tl.e) * p.w_rows + wr];
                            }
                    }
#pragma unroll
                    for (int sub = 0; sub < kUnits; ++sub) {
                        uint4* stage = st.stage[h][sub_it & 1u];
                        ++sub_it;
                        uint32_t o[2][2][2];
#pragma unroll
                        for (int g = 0; g < 2; ++g)
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const float* y = &acc[sub][i][g * 4];
                                if constexpr (kGated) {
                                    o[i][0][g] = swiglu_bf16x2(y[0] + bw[i][0], y[1] + bw[i][0], y[2] + bw[i][1], y[3] + bw[i][1]);
                                } else {
                                    o[i][0][g] = pack_bf16x2(y[0] + bw[i][0], y[1] + bw[i][0]);
                                    o[i][1][g] = pack_bf16x2(y[2] + bw[i][1], y[3] + bw[i][1]);
                                }
                            }
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
                        if constexpr (kGated) {
                            act[pass][sub] = stage[tok_ld * kPieces + (piece_ld ^ (tok_ld & 7))];
                            uint32_t m2 = 0;
                            if (col_cta + piece_ld * 8 < p.N) {
                                amax_bf16x2(m2, act[pass][sub].x);
                                amax_bf16x2(m2, act[pass][sub].y);
                                amax_bf16x2(m2, act[pass][sub].z);
                                amax_bf16x2(m2, act[pass][sub].w);
                            }
#pragma unroll
                            for (int d = 1; d < 8; d <<= 1) amax_bf16x2(m2, __shfl_xor_sync(0xffffffffu, m2, d));
                            if (piece_ld == 0) st.amax[pass][tok0 + sub * kSub + tok_ld] = amax_bf16x2_value(m2);
                        } else {
#pragma unroll
                            for (int u = 0; u < kSub * kPieces / 128; ++u) {
                                const int tok = u * (128 / kPieces) + tok_ld;
                                const uint4 v = stage[tok * kPieces + (piece_ld ^ (tok & 7))];
                                const unsigned long long dst = st.dst[tile_it & 1u][tok0 + sub * kSub + tok];
                                const int col = col_cta + piece_ld * 8;
                                if (ok && dst != 0 && col < p.N)
                                    st16(reinterpret_cast<uint8_t*>(dst) + size_t(col) * 2, Vec16{v.x, v.y, v.z, v.w});
                            }
                        }
                    }
                }
                if constexpr (kGated) {  // scale of each token's 128 columns, one token per thread; then the quantised rows
                    const Tile tl = decode_tile<kPair, kBlockMode>(t, e_cursor, st, p.w_tiles);
                    const int row_lo = st.offsets[tl.e], row_hi = st.offsets[tl.e + 1];
                    group_sync(1 + h, 128);
                    if (wg_thread < count) {
                        const int tok = tok0 + wg_thread, row = tl.row0 + tok;
                        const float sf = scale_from_amax(n_pass == 2 ? fmaxf(st.amax[0][tok], st.amax[1][tok]) : st.amax[0][tok]);
                        st.inv[tok] = inv_scale(sf);
                        if (ok && row >= row_lo && row < row_hi && tok < tl.rows) {
                            p.out_scale[size_t(row) * ((p.N + 127) / 128) + tl.wt] = sf;
                            p.out_scale_t[size_t(tl.wt) * p.n_pad + row] = sf;
                        }
                    }
                    group_sync(1 + h, 128);
#pragma unroll
                    for (int sub = 0; sub < kUnits; ++sub) {
                        const int tok = tok0 + sub * kSub + tok_ld, row = tl.row0 + tok;
                        const float inv = st.inv[tok];
#pragma unroll
                        for (int pass = 0; pass < 2; ++pass) {
                            const int col = tl.wt * kTileCols + pass * kCtaCols + piece_ld * 8;
                            const uint4 a = act[pass][sub];
                            if (ok && row >= row_lo && row < row_hi && tok < tl.rows && col < p.N)
                                *reinterpret_cast<uint2*>(static_cast<uint8_t*>(p.out) + size_t(row) * p.N + col) =
                                    make_uint2(f2e4m3x4(bf16_lo(a.x) * inv, bf16_hi(a.x) * inv, bf16_lo(a.y) * inv, bf16_hi(a.y) * inv),
                                               f2e4m3x4(bf16_lo(a.z) * inv, bf16_hi(a.z) * inv, bf16_lo(a.w) * inv, bf16_hi(a.w) * inv));
                        }
                    }
                }
            };
            const auto one = std::integral_constant<int, 1>{};
            const auto two = std::integral_constant<int, 2>{};
            const auto four = std::integral_constant<int, 4>{};
            const int units = count / kSub;
            if (units == 0) {  // 16 tokens: none for this warpgroup, which hands the buffers on
                for (int trip = 0; trip < (kb_count + group - 1) / group * n_pass; ++trip) {
                    if (ok) ok = ptx::mbar_wait_warp(&st.tmem_full[buf], buf_ph, abort_flag, kWaitLimit);
                    release(&st.tmem_empty[buf]);
                    release(&st.prod_empty[buf]);
                    if (++buf == kBufs) buf = 0, buf_ph ^= 1u;
                }
                if constexpr (!kGated) {
                    st.dst[tile_it & 1u][threadIdx.x - 128] =
                        out_row >= 0 ? reinterpret_cast<unsigned long long>(p.out) + size_t(out_row) * p.N * 2 : 0ull;
                    group_sync(3, kEpiWarps * 32);
                }
            } else if (group == 4) {
                tile_work(one, four);
            } else if (units == 1) {
                tile_work(one, two);
            } else {
                tile_work(two, two);
            }
        }
    } else {
        pdl_wait();
        if constexpr (kEarly) pdl_launch();  // after the wait: see above
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

        // What the epilogue of a tile reads from global memory, fetched while the tile before is worked on: where this thread's
        // token goes and its scale, scale and bias of this thread's weight rows r and r + 8 of the warp's two 16-row groups.
        struct TileData {
            Tile tl;
            int col_cta, out_row;
            float sa, sw[2][2], bw[2][2];
        };
        const int tok_mine = threadIdx.x - 4 * 32;
        auto fetch = [&](int t, TileData& d) {
            d.tl = decode_tile<kPair, kMode == kBlock>(t, e_cursor, st, p.w_tiles);
            d.col_cta = (d.tl.wt * (kPair ? 2 : 1) + cta_rank) * kCtaCols;
            d.out_row = -1;
            if (tok_mine < d.tl.rows) {
                const int row = d.tl.row0 + tok_mine;
                d.out_row = kGated ? row : p.dest_to_src[row];
                if constexpr (kMode == kChannel) d.sa = p.sa[row];
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    int wr;
                    if constexpr (kGated)
                        wr = min(d.col_cta + q * 16 + i * 8 + (lane >> 2), p.N - 1) + v * p.N;
                    else
                        wr = min(d.col_cta + q * 32 + i * 16 + v * 8 + (lane >> 2), p.N - 1);
                    d.sw[i][v] = 1.0f;
                    if constexpr (kMode == kChannel) d.sw[i][v] = p.sb[size_t(d.tl.e) * p.w_rows + wr];
                    if constexpr (kMode == kTensor) d.sw[i][v] = p.sa[0] * p.sb[d.tl.e];
                    d.bw[i][v] = p.bias != nullptr ? p.bias[size_t(d.tl.e) * p.w_rows + wr] : 0.0f;
                }
        };
        TileData next;
        if (tile_first < total_tiles) fetch(tile_first, next);

        for (int t = tile_first; t < total_tiles; t += tile_step, ++acc_it) {
            const TileData td = next;
            const Tile& tl = td.tl;
            const uint32_t buf = acc_it & 1u;
            const int col_cta = td.col_cta;
            st.dst[buf][tok_mine] = td.out_row >= 0 ? reinterpret_cast<unsigned long long>(p.out) + size_t(td.out_row) * p.N * 2 : 0ull;
            if constexpr (kMode == kChannel) st.sa[buf][tok_mine] = td.sa;
            if (t + tile_step < total_tiles) fetch(t + tile_step, next);
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
                                y[v][0] = __uint_as_float(x[2 * v]) * (s0 * td.sw[i][v]) + td.bw[i][v];
                                y[v][1] = __uint_as_float(x[2 * v + 1]) * (s1 * td.sw[i][v]) + td.bw[i][v];
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

}  // namespace gemm_wm
}  // namespace dq
