// Triangle multiplication, stage 1 on the 5th-generation tensor cores:
//   a[c][u][t] = mask * (W_ap LN(z))_c * sigmoid((W_ag LN(z))_c),  b likewise, for the pair element (u, t),
//   stored channel-major in fp16 with the contraction index t contiguous.  (a and b are products of a bounded gate
//   and a projection of a standardised row: far inside the fp16 range, and fp16 keeps three more bits than bf16.)
//
// Persistent kernel, one CTA per SM.  A tile is 128 pair elements (128 t, or two runs of 64); the CTAs work in
// pairs on the same sequence of tiles, each CTA producing 64 of the 128 channels of a and of b (the second read of
// a tile comes from L2).  Halving the weights a CTA keeps resident leaves shared memory for output staging
// (px_rowpipe.cuh has the parts shared with the other row kernels):
//   * The weights stay in shared memory for the whole kernel with gamma and the 1/2 of the sigmoid folded in;
//     LayerNorm's mean and beta terms enter the product as one extra K step (see px_rowpipe.cuh).
//   * The gated outputs are staged as [channel][t] in shared memory (two-byte stores, conflict-free) and leave
//     through TMA stores, 256 or 128 bytes per channel.  Four warps share a staging area of 32 channels.
//
//   warps 0..7    epilogue of output a: a thread owns one pair element (accumulator lane) and 32 of the CTA's 64
//                 channels; warps 8..15 do the same for output b, concurrently.
//   warps 16..19  (bf16 rows 16..23) statistics, correction row, the row's scale pair.
//   then          a TMA producer of the row tiles (bf16 rows of z, or standardised fp16 rows), three-stage ring, and
//                 the MMA issuers of outputs a and b, each 8 MMAs M=128 (t) N=128 (projection | gate) K=16 plus the
//                 correction step, into two accumulators in turn.
// Algorithmic HBM traffic per pair element: 256 + 4 read, 512 written.  Every mbarrier wait is bounded.
#include "px_rowpipe.cuh"

namespace px {

constexpr int kTiStages = 3, kTiSets = 2;     // sets of statistics warps for bf16 rows
constexpr int kTiWExtra = 128 * 32;            // [128 rows][16 k] weight-side correction panel
constexpr int kTiStageOut = 32 * 256;          // per run [32 channels][t] fp16
constexpr int ti_threads(bool f16) { return 32 * (16 + tile_stats_warps(f16) + 3); }
// tensor memory: out a | out b, twice

struct TiBars {
  TileBars<kTiStages, tile_fulls(kTiStages, kTiSets)> tile;
  uint64_t acc_full[2][2], acc_free[2][2];   // [output][accumulator]
  uint64_t w_full;
  uint32_t tmem_base;
};
struct TiLayout {
  static constexpr int w = 0;                                   // per output: [projection 64 | gate 64][128 k]
  static constexpr int wx = w + 2 * kOperandBytes;              // per output: correction panel
  static constexpr int a = wx + 2 * kTiWExtra;                  // row-tile ring
  static constexpr int ax = a + kTiStages * kTileBytes;       // row-tile correction panels
  static constexpr int out = ax + tile_slots(kTiStages) * kTileExtra;   // output staging, per output and half of its channels
  static constexpr int scale = out + 4 * kTiStageOut;           // float2 (rstd, rstd*mask/2) per row and slot
  static constexpr int bars = scale + tile_slots(kTiStages) * 128 * 8;
  static constexpr int total = bars + (int)sizeof(TiBars);
};
static_assert(TiLayout::total + 1024 <= 232448, "shared memory budget");

// The resident weights of a CTA (variant: which 64 channels), [projection 64 | gate 64] per output with the correction panels
// behind; the gate rows carry the 1/2 of sigmoid(x) = 1/2 + 1/2 tanh(x/2).
template <bool kF16>
struct TiWeights {
  const float *ln_w, *ln_b;
  const bf16 *ap, *ag, *bp, *bg;
  static constexpr int kBytes = TiLayout::a;
  __device__ __forceinline__ void fold(unsigned char* sm, int variant, int warp, int warps, int lane, int, int) const {
    const int chan0 = 64 * variant;
    unsigned char *w0 = sm + TiLayout::w, *x0 = sm + TiLayout::wx;
    fold_weight_rows<kF16, kF16>(w0, x0, 0, kPanelBytes, ap, chan0, 64, ln_w, ln_b, 1.0f, warp, warps, lane);
    fold_weight_rows<kF16, kF16>(w0, x0, 64, kPanelBytes, ag, chan0, 64, ln_w, ln_b, 0.5f, warp, warps, lane);
    fold_weight_rows<kF16, kF16>(w0 + kOperandBytes, x0 + kTiWExtra, 0, kPanelBytes, bp, chan0, 64, ln_w, ln_b, 1.0f, warp, warps, lane);
    fold_weight_rows<kF16, kF16>(w0 + kOperandBytes, x0 + kTiWExtra, 64, kPanelBytes, bg, chan0, 64, ln_w, ln_b, 0.5f, warp, warps, lane);
  }
};

// kF16: the rows are the standardised fp16 copy of an fp32 pair tensor (fp16 weights); otherwise bf16 rows of z.
template <bool kF16, int kRun>
__global__ void __launch_bounds__(ti_threads(kF16), 1)
trimul_in_tc_kernel(const __grid_constant__ CUtensorMap map_z, const __grid_constant__ CUtensorMap map_a,
                    const __grid_constant__ CUtensorMap map_b, const float* __restrict__ mask,
                    const TiWeights<kF16> weights, const unsigned char* __restrict__ folded, int n_u, int n_t, int swap, float eps, int runs_t, int n_tiles) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  TiBars& bars = *reinterpret_cast<TiBars*>(sm + TiLayout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  constexpr int kCtl = 16 + tile_stats_warps(kF16);      // first control warp
  const int chan0 = 64 * (blockIdx.x & 1);               // this CTA's channels of a and b
  typedef TileCtx<kTiStages, kF16, kRun, kTiSets> Ctx;
  constexpr int kPer = 128 / kRun;                       // runs of a tile
  Ctx ctx;
  ctx.tiles = sm + TiLayout::a;
  ctx.extras = sm + TiLayout::ax;
  ctx.bars = &bars.tile;
  ctx.first_tile = blockIdx.x >> 1;
  ctx.tile_step = gridDim.x >> 1;
  ctx.n_tiles = n_tiles;
  ctx.runs_t = runs_t;
  ctx.n_u = n_u;
  ctx.n_t = n_t;
  ctx.swap = swap;

  const bool skip = cta_begin();         // an earlier bounded wait gave up: do not start new work
  if (threadIdx.x == 32) prefetch_maps(map_z, map_a, map_b);
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
          folded_load(sm, folded + (blockIdx.x & 1) * TiWeights<kF16>::kBytes, TiWeights<kF16>::kBytes, &bars.w_full);
      }))
    return;
  fold_here(weights, folded, sm, blockIdx.x & 1, &bars.w_full);
  const uint32_t tmem_base = bars.tmem_base;

  if (warp >= kCtl) {
    if (warp == kCtl) {
      tile_producer_loop(ctx, &map_z);
    } else {
      const int ph = warp - kCtl - 1;                            // MMA issuer of output ph
      tile_product_loop(ctx, tmem_base + 128 * ph, smem_u32(sm + TiLayout::w) + ph * kOperandBytes, kPanelBytes,
                        smem_u32(sm + TiLayout::wx) + ph * kTiWExtra, umma_idesc_16(128, 128, kF16, kF16), &bars.w_full, bars.acc_full[ph],
                        bars.acc_free[ph], 2, 256);
    }
  } else if (warp >= 16) {
    // ------------------------------------------------------------------ row statistics (bf16 rows: two lanes a row)
    float2* scale = reinterpret_cast<float2*>(sm + TiLayout::scale);
    tile_stats_loop(
        ctx, eps, warp - 16, lane,
        [&](int k, int, int, int r, float rstd, float mk) { scale[(k % Ctx::kSlots) * 128 + r] = make_float2(rstd, 0.5f * rstd * mk); },
        [&](int u, int t) {
          return t >= n_t || u >= n_u ? 0.f : mask ? __ldg(mask + (swap ? ((size_t)t * n_u + u) : ((size_t)u * n_t + t))) : 1.f;
        });
  } else {
    // ------------------------------------------------------------------ epilogue of output ph
    const int ph = warp >> 3, half = (warp >> 2) & 1, qw = warp & 3;
    const int row = 32 * qw + lane;                      // this thread's pair element = accumulator lane
    const uint32_t t_acc = tmem_base + ((uint32_t)(32 * qw) << 16) + 128 * ph + 32 * half;
    const int group = 2 * ph + half;                     // four warps that share a staging area
    const bool leader = (threadIdx.x & 127) == 0;
    const CUtensorMap* map_out = ph ? &map_b : &map_a;
    int k = 0;
    bool ok = true;
    for (int tile = ctx.first_tile; tile < n_tiles && ok; tile += ctx.tile_step, ++k) {
      const int ab = k & 1;
      const uint32_t t_buf = t_acc + 256 * ab;
      unsigned char* const area = sm + TiLayout::out + group * kTiStageOut;
      unsigned char* const stage = area + row / kRun * (kTiStageOut / kPer) + row % kRun * 2;
      ok = mbar_wait(&bars.acc_full[ph][ab], (k >> 1) & 1, 32u);
      // the store that last read the staging area (one tile ago) must be through with it
      if (leader) tma_store_wait_read<0>();
      ok = named_barrier_all(1 + group, 128, ok);          // all four warps go on, or none
      if (!ok) break;
      tc_fence_after();
      const float2 sc = reinterpret_cast<const float2*>(sm + TiLayout::scale)[(k % Ctx::kSlots) * 128 + row];
      // mask * p * sigmoid(g) = h + h * tanh(g / 2) with h = mask * p / 2 (the halves are folded in)
      auto emit = [&](const uint32_t(&p)[16], const uint32_t(&g)[16], int hh) {
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float h = sc.y * __uint_as_float(p[e]);
          const float v = fmaf(h, tanh_fast(sc.x * __uint_as_float(g[e])), h);
          *reinterpret_cast<__half*>(stage + (16 * hh + e) * (2 * kRun)) = __float2half_rn(v);
        }
      };
      uint32_t p0[16], g0[16], p1[16], g1[16];
      tmem_ld16(t_buf, p0);
      tmem_ld16(t_buf + 64, g0);
      tmem_ld16(t_buf + 16, p1);
      tmem_ld16(t_buf + 64 + 16, g1);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.acc_free[ph][ab]);  // this warp has read its part of the accumulator
      emit(p0, g0, 0);
      emit(p1, g1, 1);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      named_barrier(1 + group, 128);
      if (leader) {
        for (int h = 0; h < kPer; ++h) {
          const Run r = run_at<kRun>(kPer * tile + h, runs_t);
          if (r.u < n_u) tma_store_3d(map_out, smem_u32(area) + h * (kTiStageOut / kPer), r.t, r.u, chan0 + 32 * half);
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

PX_DEFINE_FAMILY_HOOKS(trimul_in)

template <bool kF16, int kRun>
static int32_t launch_trimul_in_runs(const void* z, const float* mask, const TiWeights<kF16>& weights, const void* folded, px_f16* a,
                                px_f16* b, int64_t n_u, int64_t n_t, int64_t ld, int32_t incoming, float eps, cudaStream_t st) {
  CUtensorMap mz, ma, mb;
  const CUtensorMapDataType zt = kF16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  // pair element (u, t) is row u*n_t + t of z, or row t*n_u + u when the two indices are exchanged
  const bool ok = incoming ? make_map_3d(&mz, zt, z, 128, (uint64_t)n_u, (uint64_t)n_t, 256, (uint64_t)n_u * 256, 64, 1,
                                         CU_TENSOR_MAP_SWIZZLE_128B, kRun)
                           : make_map_3d(&mz, zt, z, 128, (uint64_t)n_t, (uint64_t)n_u, 256, (uint64_t)n_t * 256, 64, kRun,
                                         CU_TENSOR_MAP_SWIZZLE_128B, 1);
  if (!ok) return PX_ERR_LAUNCH;
  // outputs [128 channels][n_u][ld]: a store writes [32 channels][one u][a run]
  if (!make_map_3d(&ma, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a, (uint64_t)ld, (uint64_t)n_u, 128, (uint64_t)ld * 2,
                   (uint64_t)n_u * ld * 2, kRun, 1, CU_TENSOR_MAP_SWIZZLE_NONE, 32) ||
      !make_map_3d(&mb, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, b, (uint64_t)ld, (uint64_t)n_u, 128, (uint64_t)ld * 2,
                   (uint64_t)n_u * ld * 2, kRun, 1, CU_TENSOR_MAP_SWIZZLE_NONE, 32))
    return PX_ERR_LAUNCH;
  const size_t smem = TiLayout::total + 1024;
  static SmemLimit limit;
  if (!limit.set(trimul_in_tc_kernel<kF16, kRun>, smem)) return PX_ERR_LAUNCH;
  const int64_t n_tiles = tiles_of(n_u, n_t, kRun);     // (runs cover the pad columns)
  if (n_tiles > 0x7fffffff) return PX_ERR_UNSUPPORTED;
  const int pairs = even_grid(n_tiles, sm_count() / 2, tile_period(n_u, n_t, kRun));
  return launch_pdl(trimul_in_tc_kernel<kF16, kRun>, dim3(2 * pairs), ti_threads(kF16), smem, st, mz, ma, mb, mask, weights,
                    (const unsigned char*)folded, (int)n_u, (int)n_t, (int)incoming, eps, (int)runs_of(n_t, kRun), (int)n_tiles)
             ? PX_OK
             : PX_ERR_LAUNCH;
}

template <bool kF16>
static int32_t launch_trimul_in(const void* z, const float* mask, const TiWeights<kF16>& weights, const void* folded, px_f16* a,
                                px_f16* b, int64_t n_u, int64_t n_t, int64_t ld, int32_t incoming, float eps, cudaStream_t st) {
  if (!incoming && ld == n_t && one_row_pays(n_u, n_t)) n_t *= n_u, ld = n_t, n_u = 1;
  return (two_runs_pay(n_u, n_t) ? launch_trimul_in_runs<kF16, 64> : launch_trimul_in_runs<kF16, 128>)(z, mask, weights, folded, a, b, n_u, n_t,
                                                                                                ld, incoming, eps, st);
}

static bool trimul_in_shapes_ok(const void* z, const px_f16* a, const px_f16* b, int64_t n_u, int64_t n_t, int64_t ld) {
  return z && a && b && n_u > 0 && n_t > 0 && n_u <= 32768 && n_t <= 32768 && ld == px_ld(n_t) &&
         !(((uintptr_t)z | (uintptr_t)a | (uintptr_t)b) & 15);
}
template <bool kF16>
static TiWeights<kF16> ti_weights(const float* ln_w, const float* ln_b, const px_w16* ap, const px_w16* ag, const px_w16* bp,
                                  const px_w16* bg) {
  return {ln_w, ln_b, (const bf16*)ap, (const bf16*)ag, (const bf16*)bp, (const bf16*)bg};
}
static bool ti_weights_ok(const float* ln_w, const float* ln_b, const px_w16* ap, const px_w16* ag, const px_w16* bp,
                          const px_w16* bg) {
  return ln_w && ln_b && ap && ag && bp && bg &&
         !(((uintptr_t)ap | (uintptr_t)ag | (uintptr_t)bp | (uintptr_t)bg | (uintptr_t)ln_w | (uintptr_t)ln_b) & 15);
}

}  // namespace px

using namespace px;

extern "C" int64_t px_trimul_in_folded_bytes(void) { return 2 * TiWeights<true>::kBytes; }

extern "C" int32_t px_trimul_in_fold(const float* ln_w, const float* ln_b, const px_w16* w_ap, const px_w16* w_ag,
                                     const px_w16* w_bp, const px_w16* w_bg, int32_t rows_dtype, void* folded, void* stream) {
  if (!ti_weights_ok(ln_w, ln_b, w_ap, w_ag, w_bp, w_bg) || !folded || ((uintptr_t)folded & 15)) return PX_ERR_BAD_ARG;
  if (rows_dtype != PX_F16 && rows_dtype != PX_BF16) return PX_ERR_UNSUPPORTED;
  return (rows_dtype == PX_F16 ? launch_fold(ti_weights<true>(ln_w, ln_b, w_ap, w_ag, w_bp, w_bg), 2, folded, (cudaStream_t)stream)
                               : launch_fold(ti_weights<false>(ln_w, ln_b, w_ap, w_ag, w_bp, w_bg), 2, folded, (cudaStream_t)stream))
             ? PX_OK
             : PX_ERR_LAUNCH;
}

extern "C" int32_t px_trimul_in_proj_folded(const void* z, int32_t z_dtype, const float* mask, const void* folded, px_f16* a,
                                            px_f16* b, int64_t n_u, int64_t n_t, int64_t ld, int32_t incoming, float eps,
                                            void* stream) {
  if (!trimul_in_shapes_ok(z, a, b, n_u, n_t, ld) || !folded || ((uintptr_t)folded & 15)) return PX_ERR_BAD_ARG;
  if (z_dtype == PX_F16)
    return launch_trimul_in<true>(z, mask, TiWeights<true>{}, folded, a, b, n_u, n_t, ld, incoming, eps, (cudaStream_t)stream);
  if (z_dtype == PX_BF16)
    return launch_trimul_in<false>(z, mask, TiWeights<false>{}, folded, a, b, n_u, n_t, ld, incoming, eps, (cudaStream_t)stream);
  return PX_ERR_UNSUPPORTED;
}

extern "C" int32_t px_trimul_in_proj(const void* z, int32_t z_dtype, const float* mask, const float* ln_w,
                                     const float* ln_b, const px_w16* w_ap, const px_w16* w_ag,
                                     const px_w16* w_bp, const px_w16* w_bg, px_f16* a, px_f16* b, int64_t n_u,
                                     int64_t n_t, int64_t ld, int32_t incoming, float eps, void* stream) {
  if (!trimul_in_shapes_ok(z, a, b, n_u, n_t, ld) || !ti_weights_ok(ln_w, ln_b, w_ap, w_ag, w_bp, w_bg)) return PX_ERR_BAD_ARG;
  if (z_dtype == PX_F16)   // standardised rows of an fp32 pair tensor (px_standardise_rows)
    return launch_trimul_in<true>(z, mask, ti_weights<true>(ln_w, ln_b, w_ap, w_ag, w_bp, w_bg), nullptr, a, b, n_u, n_t, ld,
                                  incoming, eps, (cudaStream_t)stream);
  if (z_dtype == PX_BF16)
    return launch_trimul_in<false>(z, mask, ti_weights<false>(ln_w, ln_b, w_ap, w_ag, w_bp, w_bg), nullptr, a, b, n_u, n_t, ld,
                                   incoming, eps, (cudaStream_t)stream);
  return PX_ERR_UNSUPPORTED;
}
