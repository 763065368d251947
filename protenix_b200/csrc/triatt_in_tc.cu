// Triangle attention, stage 1 on the 5th-generation tensor cores:
//   LN(z) -> q, k [u][h][t][32] (q pre-scaled by log2(e)/sqrt(32)), v transposed [u][h][32][ld] (zero pad columns),
//   in fp16 (projections of standardised rows: far inside its range), bias[h][u][t] = log2(e) * (W_bias LN(z))_h (zero
//   pad columns) and mask_bias[u][t] = log2(e) * inf * (mask - 1) (-inf in the pad columns) in fp32, for the pair
//   element (u, t) = z[u][t] (starting node) or z[t][u] (ending node).
//
// Persistent kernel, one CTA per SM, on the row-tile pipeline of px_rowpipe.cuh (TMA-fed raw rows, LayerNorm folded
// into the resident weights plus one correction K step).  The CTAs
// work in pairs on the same tiles; CTA parity picks two of the four heads.
//
//   warps 0..7    epilogue of q | k: a thread owns one pair element and both heads of q (warps 0..3) or k (4..7):
//                 a warp's 32 rows of a head, 2 KB, are staged (64-byte swizzle) and leave by TMA.  Written by their threads in
//                 pieces of 16 bytes, half a sector each, they took the kernel from 32 to 42 us at N = 384 and from 119 to 144 at N = 768.
//   warps 8..15   epilogue of v | bias: v goes through a [32 d][t] staging tile per head and run and a TMA store (the transpose),
//                 the two bias values of the row are written directly.
//   warps 16..19  (bf16 rows 16..23) statistics, correction row, scale pair, mask bias.
//   then          a TMA producer and the MMA issuers of the two products (N = 128 and N = 80), each into two accumulators in turn.
// Algorithmic HBM traffic per pair element: 256 + 4 read, 3*256 + 16 + 4 written.  Every wait is bounded.
#include <math_constants.h>

#include "px_rowpipe.cuh"

namespace px {

constexpr int kAiH = 4, kAiD = 32;
constexpr int kAiW1Panel = 80 * 128;           // [v 64 | bias 16][64 k]
constexpr int kAiStageOut = 32 * 256;          // per run [32 d][t] fp16: one head
constexpr int ai_threads(bool f16) { return 32 * (16 + tile_stats_warps(f16) + 3); }
// Stages of the row-tile ring: two, or three where shared memory holds them, which is where the rows are standardised ones (they need
// one correction panel).  Which: triatt_in_stages.
// tensor memory: q|k (128) | v|bias (80) | -, twice

template <int kStages>
struct AiBars {
  TileBars<kStages> tile;
  uint64_t acc_full[2][2], acc_free[2][2];   // [product][accumulator]
  uint64_t w_full;
  uint32_t tmem_base;
};
template <bool kF16, int kStages>
struct AiLayout {
  static constexpr int w0 = 0;                                  // [q 64 | k 64][128 k]
  static constexpr int w1 = w0 + kOperandBytes;                 // [v 64 | bias 16][128 k]
  static constexpr int wx0 = w1 + 2 * kAiW1Panel;               // correction panels
  static constexpr int wx1 = wx0 + 128 * 32;
  static constexpr int a = wx1 + 128 * 32;                      // row-tile ring
  static constexpr int ax = a + kStages * kTileBytes;
  static constexpr int out = ax + tile_extras(kStages, kF16) * kTileExtra;   // v staging, per head
  static constexpr int qk = out + 2 * kAiStageOut;              // q, k staging: 8 warps x 2 heads x [32 t][32] fp16
  static constexpr int scale = qk + 8 * 2 * 2048;               // float2 (rstd, rstd or 0 beyond n) per row and slot
  static constexpr int bars = scale + tile_slots(kStages) * 128 * 8;
  static constexpr int total = bars + (int)sizeof(AiBars<kStages>);
};
static_assert(AiLayout<true, 3>::total + 1024 <= 232448 && AiLayout<false, 2>::total + 1024 <= 232448, "shared memory budget");
static_assert(AiLayout<true, 3>::a % 1024 == 0, "tile ring must keep the swizzle alignment");

// The resident weights of a CTA (variant: which pair of heads): q carries the softmax scale, the bias rows log2(e).
template <bool kF16>
struct AiWeights {
  const float *ln_w, *ln_b;
  const bf16 *q, *k, *v, *bias;
  static constexpr int kBytes = AiLayout<kF16, 2>::a;          // the ring lies behind the weights, however many stages it has
  __device__ __forceinline__ void fold(unsigned char* sm, int hpair, int warp, int warps, int lane, int tid, int threads) const {
    unsigned char *w0 = sm + AiLayout<kF16, 2>::w0, *w1 = sm + AiLayout<kF16, 2>::w1, *wx0 = sm + AiLayout<kF16, 2>::wx0, *wx1 = sm + AiLayout<kF16, 2>::wx1;
    const float qscale = kLog2e * rsqrtf((float)kAiD);
    fold_weight_rows<kF16, kF16>(w0, wx0, 0, kPanelBytes, q, 64 * hpair, 64, ln_w, ln_b, qscale, warp, warps, lane);
    fold_weight_rows<kF16, kF16>(w0, wx0, 64, kPanelBytes, k, 64 * hpair, 64, ln_w, ln_b, 1.0f, warp, warps, lane);
    fold_weight_rows<kF16, kF16>(w1, wx1, 0, kAiW1Panel, v, 64 * hpair, 64, ln_w, ln_b, 1.0f, warp, warps, lane);
    fold_weight_rows<kF16, kF16>(w1, wx1, 64, kAiW1Panel, bias, 2 * hpair, 2, ln_w, ln_b, kLog2e, warp, warps, lane);
    // rows 66..79 of the second operand and rows 66..127 of its correction panel are padding
    for (int i = tid; i < 14 * 16; i += threads)
      *reinterpret_cast<uint4*>(w1 + operand_piece_offset(66 + i / 16, i % 16, kAiW1Panel)) = make_uint4(0u, 0u, 0u, 0u);
    for (int i = tid; i < 62 * 2; i += threads) *reinterpret_cast<uint4*>(wx1 + 66 * 32 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
};

// kF16: the rows are the standardised fp16 copy of an fp32 pair tensor (fp16 weights); otherwise bf16 rows of z.
template <bool kF16, int kStages, int kRun, int kSets>
__global__ void __launch_bounds__(ai_threads(kF16), 1)
triatt_in_tc_kernel(const __grid_constant__ CUtensorMap map_z, const __grid_constant__ CUtensorMap map_v,
                    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const float* __restrict__ mask,
                    const AiWeights<kF16> weights, const unsigned char* __restrict__ folded,
                    float* __restrict__ bias_out, float* __restrict__ mb_out, int n_u, int n,
                    int ldm, int swap, float eps, float inf, int runs_t, int n_tiles) {
  typedef AiLayout<kF16, kStages> Layout;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  AiBars<kStages>& bars = *reinterpret_cast<AiBars<kStages>*>(sm + Layout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int hpair = blockIdx.x & 1;                      // this CTA's heads: 2*hpair, 2*hpair + 1
  typedef TileCtx<kStages, kF16, kRun, kSets> Ctx;
  constexpr int kPer = 128 / kRun;                       // runs of a tile
  constexpr int kCtl = 16 + tile_stats_warps(kF16);      // first control warp
  Ctx ctx;
  ctx.tiles = sm + Layout::a;
  ctx.extras = sm + Layout::ax;
  ctx.bars = &bars.tile;
  ctx.first_tile = blockIdx.x >> 1;
  ctx.tile_step = gridDim.x >> 1;
  ctx.n_tiles = n_tiles;
  ctx.runs_t = runs_t;
  ctx.n_u = n_u;
  ctx.n_t = n;
  ctx.swap = swap;

  const bool skip = cta_begin();         // an earlier bounded wait gave up: do not start new work
  if (threadIdx.x == 32) prefetch_maps(map_z, map_v, map_q, map_k);
  if (threadIdx.x == 0) {
    tile_bars_init(ctx, 2);
    mbar_init(&bars.w_full, 1);
    for (int b = 0; b < 4; ++b) {
      mbar_init(&bars.acc_full[b >> 1][b & 1], 1);
      mbar_init(&bars.acc_free[b >> 1][b & 1], 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kCtl) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  if (!cta_ready(skip, warp == kCtl, bars.tmem_base, 512u, [&] {
        if (folded && threadIdx.x == 0)
          folded_load(sm, folded + hpair * AiWeights<kF16>::kBytes, AiWeights<kF16>::kBytes, &bars.w_full);
      }))
    return;
  fold_here(weights, folded, sm, hpair, &bars.w_full);
  const uint32_t tmem_base = bars.tmem_base;

  if (warp >= kCtl) {
    if (warp == kCtl) {
      tile_producer_loop(ctx, &map_z);
    } else if (warp == kCtl + 1) {
      tile_product_loop(ctx, tmem_base, smem_u32(sm + Layout::w0), kPanelBytes, smem_u32(sm + Layout::wx0),
                        umma_idesc_16(128, 128, kF16, kF16), &bars.w_full, bars.acc_full[0], bars.acc_free[0], 2, 256);
    } else {
      tile_product_loop(ctx, tmem_base + 128, smem_u32(sm + Layout::w1), kAiW1Panel, smem_u32(sm + Layout::wx1),
                        umma_idesc_16(128, 80, kF16, kF16), &bars.w_full, bars.acc_full[1], bars.acc_free[1], 2, 256);
    }
  } else if (warp >= 16) {
    // ------------------------------------------------------------------ row statistics (tile_stats_loop) and mask bias
    // The mask bias comes after the hand-over: its load of the mask, up to 2 us from memory, otherwise holds up both the products and
    // the stage of every tile.  bf16, starting node: 40.0 -> 33.5 us at N = 384, 147 -> 120 at 768, 592 -> 465 at 1536; ending node
    // (a sector of the mask serves eight u) 35.9 -> 33.8, 125 -> 123 and 494 -> 479; N = 128 9.4 -> 9.0.
    float2* scale = reinterpret_cast<float2*>(sm + Layout::scale);
    tile_stats_loop(
        ctx, eps, warp - 16, lane,
        [&](int k, int, int t, int r, float rstd, float) { scale[(k % Ctx::kSlots) * 128 + r] = make_float2(rstd, t < n ? rstd : 0.f); },
        TileNothingAhead(),
        [&](int u, int t) {
          if (hpair == 0 && u < n_u) {                   // mask bias, -inf in the pad columns [n, ldm)
            float mv = -CUDART_INF_F;
            if (t < n)
              mv = mask ? (__ldg(mask + (swap ? ((size_t)t * n_u + u) : ((size_t)u * n + t))) - 1.0f) * inf * kLog2e : 0.f;
            mb_out[(size_t)u * ldm + t] = mv;
            // an odd number of runs of 64 leaves 64 columns of the padding to the last one
            if (kRun == 64 && t >= 64 * (runs_t - 1) && t + 64 < ldm) mb_out[(size_t)u * ldm + t + 64] = -CUDART_INF_F;
          }
        });
  } else if (warp < 8) {
    // ------------------------------------------------------------------ epilogue of q | k
    const int which = warp >> 2, qw = warp & 3;          // 0: q, 1: k
    const int row = 32 * qw + lane;
    const uint32_t t_acc = tmem_base + ((uint32_t)(32 * qw) << 16) + 64 * which;
    unsigned char* stage = sm + Layout::qk + warp * 4096;
    int k = 0;
    for (int tile = ctx.first_tile; tile < n_tiles; tile += ctx.tile_step, ++k) {
      const Run run = run_at<kRun>(kPer * tile + 32 * qw / kRun, runs_t);
      const int u = run.u, tw = run.t + 32 * qw % kRun;   // the warp's first row
      const int ab = k & 1, an = k >> 1;
      bool ok = mbar_wait(&bars.acc_full[0][ab], an & 1, 32u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float rstd = reinterpret_cast<const float2*>(sm + Layout::scale)[(k % Ctx::kSlots) * 128 + row].x;
      uint32_t h0[32], h1[32];
      tmem_ld32(t_acc + 256 * ab, h0);
      tmem_ld32(t_acc + 256 * ab + 32, h1);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.acc_free[0][ab]);  // this warp has read its part of the accumulator
      if (lane == 0) tma_store_wait_read<0>();            // the stores of the tile before have read the staging area
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t(&v)[32] = j < 4 ? h0 : h1;
        const int e = 8 * (j & 3);
        *reinterpret_cast<uint4*>(stage + (j >> 2) * 2048 + lane * 64 + (((j & 3) ^ ((lane >> 1) & 3)) << 4)) =
            make_uint4(pack_f16x2(rstd * __uint_as_float(v[e]), rstd * __uint_as_float(v[e + 1])),
                       pack_f16x2(rstd * __uint_as_float(v[e + 2]), rstd * __uint_as_float(v[e + 3])),
                       pack_f16x2(rstd * __uint_as_float(v[e + 4]), rstd * __uint_as_float(v[e + 5])),
                       pack_f16x2(rstd * __uint_as_float(v[e + 6]), rstd * __uint_as_float(v[e + 7])));
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0 && tw < n && u < n_u) {
        for (int e = 0; e < 2; ++e)
          tma_store_3d(which ? &map_k : &map_q, smem_u32(stage + e * 2048), 0, tw, u * kAiH + 2 * hpair + e);
        tma_store_commit();
      }
    }
    if (lane == 0) tma_store_wait_read<0>();
  } else {
    // ------------------------------------------------------------------ epilogue of v | bias
    const int half = (warp >> 2) & 1, qw = warp & 3;
    const int row = 32 * qw + lane;
    const uint32_t t_acc = tmem_base + ((uint32_t)(32 * qw) << 16) + 128 + 32 * half;
    const bool leader = (threadIdx.x & 127) == 0;        // of the four warps of a head
    int k = 0;
    bool ok = true;
    for (int tile = ctx.first_tile; tile < n_tiles && ok; tile += ctx.tile_step, ++k) {
      const Run run = run_at<kRun>(kPer * tile + 32 * qw / kRun, runs_t);
      const int u = run.u, t = run.t + row % kRun;
      const int ab = k & 1, an = k >> 1;
      unsigned char* const area = sm + Layout::out + half * kAiStageOut;
      unsigned char* const stage = area + row / kRun * (kAiStageOut / kPer) + row % kRun * 2;
      ok = mbar_wait(&bars.acc_full[1][ab], an & 1, 64u);
      // the store that last read the staging area (one tile ago) must be through with it
      if (leader) tma_store_wait_read<0>();
      ok = named_barrier_all(1 + half, 128, ok);           // all four warps go on, or none
      if (!ok) break;
      tc_fence_after();
      const float2 sc = reinterpret_cast<const float2*>(sm + Layout::scale)[(k % Ctx::kSlots) * 128 + row];
      uint32_t v[32], b[16];
      tmem_ld32(t_acc + 256 * ab, v);
      if (half == 0) tmem_ld16(tmem_base + ((uint32_t)(32 * qw) << 16) + 256 * ab + 128 + 64, b);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.acc_free[1][ab]);  // this warp has read its part of the accumulator
#pragma unroll
      for (int e = 0; e < 32; ++e)
        *reinterpret_cast<__half*>(stage + e * (2 * kRun)) = __float2half_rn(sc.y * __uint_as_float(v[e]));
      if (half == 0 && u < n_u) {                        // zero in the pad columns [n, ldm)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float* const to = bias_out + ((size_t)(2 * hpair + e) * n_u + u) * ldm + t;
          *to = sc.y * __uint_as_float(b[e]);
          if (kRun == 64 && t >= 64 * (runs_t - 1) && t + 64 < ldm) to[64] = 0.f;     // an odd number of runs
        }
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      named_barrier(1 + half, 128);
      if (leader) {
        for (int h = 0; h < kPer; ++h) {
          const Run r = run_at<kRun>(kPer * tile + h, runs_t);
          if (r.u < n_u) tma_store_3d(&map_v, smem_u32(area) + h * (kAiStageOut / kPer), r.t, r.u * 128 + 64 * hpair + 32 * half, 0);
        }
        tma_store_commit();
      }
    }
    if (leader) tma_store_wait_read<0>();
  }

  tc_fence_before();
  cta_teardown_sync();
  if (warp == kCtl) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

PX_DEFINE_FAMILY_HOOKS(triatt_in)

template <bool kF16, int kStages, int kRun, int kSets>
static int32_t launch_triatt_in_runs(const void* z, const float* mask, const AiWeights<kF16>& weights, const void* folded,
                                px_f16* q, px_f16* k, px_f16* v, float* bias, float* mask_bias, int64_t n_u,
                                int64_t n, int64_t ldm, int32_t ending, float eps, float inf, cudaStream_t st) {
  CUtensorMap mz, mv, mq, mk;
  const CUtensorMapDataType zt = kF16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  // pair element (u, t) is row u*n + t of z, or row t*n_u + u when the two indices are exchanged
  const bool ok = ending ? make_map_3d(&mz, zt, z, 128, (uint64_t)n_u, (uint64_t)n, 256, (uint64_t)n_u * 256, 64, 1,
                                       CU_TENSOR_MAP_SWIZZLE_128B, kRun)
                         : make_map_3d(&mz, zt, z, 128, (uint64_t)n, (uint64_t)n_u, 256, (uint64_t)n * 256, 64, kRun,
                                       CU_TENSOR_MAP_SWIZZLE_128B, 1);
  if (!ok) return PX_ERR_LAUNCH;
  // v is [n_u * 128 rows (u, head, d)][ldt]: a store writes [32 rows][a run]
  const uint64_t ldt = (uint64_t)px_ld(n);
  if (!make_map_3d(&mv, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, v, ldt, (uint64_t)n_u * 128, 1, ldt * 2, ldt * 2 * n_u * 128, kRun,
                   32, CU_TENSOR_MAP_SWIZZLE_NONE, 1))
    return PX_ERR_LAUNCH;
  // q, k: [n_u * 4][n][32], a store writes [32 t][32]
  for (int i = 0; i < 2; ++i)
    if (!make_map_3d(i ? &mk : &mq, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, i ? k : q, kAiD, (uint64_t)n, (uint64_t)n_u * kAiH, kAiD * 2,
                     (uint64_t)n * kAiD * 2, kAiD, 32, CU_TENSOR_MAP_SWIZZLE_64B))
      return PX_ERR_LAUNCH;
  const size_t smem = AiLayout<kF16, kStages>::total + 1024;
  static SmemLimit limit;
  if (!limit.set(triatt_in_tc_kernel<kF16, kStages, kRun, kSets>, smem)) return PX_ERR_LAUNCH;
  const int64_t n_tiles = tiles_of(n_u, n, kRun);
  if (n_tiles > 0x7fffffff) return PX_ERR_UNSUPPORTED;
  // Whole tiles of bf16 rows take little longer than ragged ones (their statistics are the same work), and an even number serves them 2 to 4 %
  // better from 132 to 230 tokens (N = 160 13.5 us against 14.0), 1 to 2 % worse at 430 and 450; standardised rows gain 3 to 8 % there.
  const int pairs = even_grid(n_tiles, sm_count() / 2, kF16 ? tile_period(n_u, n, kRun) : 1);
  return launch_pdl(triatt_in_tc_kernel<kF16, kStages, kRun, kSets>, dim3(2 * pairs), ai_threads(kF16), smem, st, mz, mv, mq, mk, mask, weights,
                    (const unsigned char*)folded, bias, mask_bias, (int)n_u, (int)n, (int)ldm, (int)ending, eps, inf, (int)runs_of(n, kRun),
                    (int)n_tiles)
             ? PX_OK
             : PX_ERR_LAUNCH;
}

template <bool kF16, int kStages>
static int32_t launch_triatt_in(const void* z, const float* mask, const AiWeights<kF16>& weights, const void* folded,
                                px_f16* q, px_f16* k, px_f16* v, float* bias, float* mask_bias, int64_t n_u,
                                int64_t n, int64_t ldm, int32_t ending, float eps, float inf, cudaStream_t st) {
  const bool two_runs = two_runs_pay(n_u, n);
  // Two sets of statistics warps for bf16 rows where a CTA has 2 to 12 tiles: a single tile is measured faster by eight warps than by four, and
  // from more tiles on the time is that of the memory, which tiles measured ahead of their turn only crowd.  The starting node keeps two
  // with ragged tiles, which have less to write and the same to measure.  One set | two, us, starting node: N = 64 11.3 | 11.5, 100 12.8 | 12.5,
  // 200 20.5 | 19.5, 300 32.3 | 31.5, 512 64.8 | 64.9, 768 139 | 141, ragged 437 53.1 | 52.3, 776 156 | 151, 1096 287 | 282; ending node 64
  // 11.2 | 11.6, 200 20.6 | 19.5, 300 32.4 | 31.9, 384 42.3 | 43.3, 448 54.7 | 56.2, 768 138 | 146, 1024 231 | 245; 96 rows of 768 24.5 | 22.8.
  const int64_t room = sm_count() / 2, rounds = (tiles_of(n_u, n, two_runs ? 64 : 128) + room - 1) / room;
  constexpr int kTwo = kF16 ? 1 : 2;
  const auto run = rounds > 1 && (rounds <= 12 || (!ending && n % 64))
                       ? (two_runs ? launch_triatt_in_runs<kF16, kStages, 64, kTwo> : launch_triatt_in_runs<kF16, kStages, 128, kTwo>)
                       : (two_runs ? launch_triatt_in_runs<kF16, kStages, 64, 1> : launch_triatt_in_runs<kF16, kStages, 128, 1>);
  return run(z, mask, weights, folded, q, k, v, bias, mask_bias, n_u, n, ldm, ending, eps, inf, st);
}

// Stages for the standardised rows of an fp32 pair tensor.  Three let the two CTAs of a pair drift apart, and once the rows are larger than
// L2 the second one finds its tile gone: N = 1024, starting node, 390 MB read from memory where two stages read 273.
// Two | three, us: starting node N = 437 39.8 | 39.2, 576 64.3 | 63.7, 640 74.9 | 77.2, 704 95.5 | 95.7, 768 107 | 114, 1024 187 | 213,
// 1536 425 | 512; ending node, whose tiles take 256 bytes from each of 128 places, 512 52.4 | 48.4, 704 103 | 89, 768 117 | 116,
// 832 143 | 130, 896 156 | 162, 1024 207 | 224, 1536 468 | 568.  L2 holds the rows of 704 tokens, two thirds of those of 862.
// (One instantiation each: a count known at run time only cost 0.1 us a launch.)
static int triatt_in_stages(int64_t n_u, int64_t n, int32_t ending) {
  return n_u * n * (2 * kC) > (ending ? l2_bytes() * 3 / 2 : l2_bytes()) ? 2 : 3;
}
static bool triatt_in_args_ok(const void* z, const void* q, const void* k, const void* v, const float* bias, const float* mask_bias,
                              int64_t n_u, int64_t n_t, int64_t ldm) {
  return z && q && k && v && bias && mask_bias && n_u > 0 && n_t > 0 && n_u <= 32768 && n_t <= 32768 && ldm == px_ld_mask(n_t) &&
         !(((uintptr_t)z | (uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15);
}
template <bool kF16>
static AiWeights<kF16> ai_weights(const float* ln_w, const float* ln_b, const px_w16* q, const px_w16* k, const px_w16* v,
                                  const px_w16* bias) {
  return {ln_w, ln_b, (const bf16*)q, (const bf16*)k, (const bf16*)v, (const bf16*)bias};
}
static bool ai_weights_ok(const float* ln_w, const float* ln_b, const px_w16* q, const px_w16* k, const px_w16* v, const px_w16* bias) {
  return ln_w && ln_b && q && k && v && bias &&
         !(((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)bias | (uintptr_t)ln_w | (uintptr_t)ln_b) & 15);
}

}  // namespace px

using namespace px;

extern "C" int64_t px_triatt_in_folded_bytes(void) { return 2 * AiWeights<true>::kBytes; }

extern "C" int32_t px_triatt_in_fold(const float* ln_w, const float* ln_b, const px_w16* w_q, const px_w16* w_k, const px_w16* w_v,
                                     const px_w16* w_bias, int32_t rows_dtype, void* folded, void* stream) {
  if (!ai_weights_ok(ln_w, ln_b, w_q, w_k, w_v, w_bias) || !folded || ((uintptr_t)folded & 15)) return PX_ERR_BAD_ARG;
  if (rows_dtype != PX_F16 && rows_dtype != PX_BF16) return PX_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  return (rows_dtype == PX_F16 ? launch_fold(ai_weights<true>(ln_w, ln_b, w_q, w_k, w_v, w_bias), 2, folded, st)
                               : launch_fold(ai_weights<false>(ln_w, ln_b, w_q, w_k, w_v, w_bias), 2, folded, st))
             ? PX_OK
             : PX_ERR_LAUNCH;
}

extern "C" int32_t px_triatt_in_proj_folded(const void* z, int32_t z_dtype, const float* mask, const void* folded, px_f16* q,
                                            px_f16* k, px_f16* v, float* bias, float* mask_bias, int64_t n_u, int64_t n_t,
                                            int64_t ldm, int32_t ending, float eps, float inf, void* stream) {
  if (!triatt_in_args_ok(z, q, k, v, bias, mask_bias, n_u, n_t, ldm) || !folded || ((uintptr_t)folded & 15)) return PX_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (z_dtype == PX_F16)
    return (triatt_in_stages(n_u, n_t, ending) == 2 ? launch_triatt_in<true, 2> : launch_triatt_in<true, 3>)(
        z, mask, AiWeights<true>{}, folded, q, k, v, bias, mask_bias, n_u, n_t, ldm, ending, eps, inf, st);
  if (z_dtype == PX_BF16)
    return launch_triatt_in<false, 2>(z, mask, AiWeights<false>{}, folded, q, k, v, bias, mask_bias, n_u, n_t, ldm, ending, eps, inf, st);
  return PX_ERR_UNSUPPORTED;
}

extern "C" int32_t px_triatt_in_proj(const void* z, int32_t z_dtype, const float* mask, const float* ln_w,
                                     const float* ln_b, const px_bf16* w_q, const px_bf16* w_k, const px_bf16* w_v,
                                     const px_bf16* w_bias, px_f16* q, px_f16* k, px_f16* v, float* bias,
                                     float* mask_bias, int64_t n_u, int64_t n_t, int64_t ldm, int32_t ending,
                                     float eps, float inf, void* stream) {
  if (!triatt_in_args_ok(z, q, k, v, bias, mask_bias, n_u, n_t, ldm) || !ai_weights_ok(ln_w, ln_b, w_q, w_k, w_v, w_bias))
    return PX_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (z_dtype == PX_F16)   // standardised rows of an fp32 pair tensor (px_standardise_rows)
    return (triatt_in_stages(n_u, n_t, ending) == 2 ? launch_triatt_in<true, 2> : launch_triatt_in<true, 3>)(
        z, mask, ai_weights<true>(ln_w, ln_b, w_q, w_k, w_v, w_bias), nullptr, q, k, v, bias, mask_bias, n_u, n_t, ldm, ending, eps, inf, st);
  if (z_dtype == PX_BF16)
    return launch_triatt_in<false, 2>(z, mask, ai_weights<false>(ln_w, ln_b, w_q, w_k, w_v, w_bias), nullptr, q, k, v, bias, mask_bias, n_u,
                                      n_t, ldm, ending, eps, inf, st);
  return PX_ERR_UNSUPPORTED;
}
