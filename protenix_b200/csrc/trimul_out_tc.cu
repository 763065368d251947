// Triangle multiplication, stage 3 on the 5th-generation tensor cores:
//   z_out[i][j] = [z_in[i][j] +] (W_z LN_out(x[:, i, j])) * sigmoid(W_g LN_in(z_in[i][j])),
//   x [128 channels][n_i][ld] fp16, channel-major and scaled by PX_TRIMUL_X_SCALE as the contraction leaves it
//   (LN_out runs with eps * scale^2, which gives exactly LN_out of the unscaled x).
//
// Persistent kernel, one CTA per SM, 128 pair elements (two runs of 64 consecutive j of one i) per tile.  Both LayerNorms are
// folded into the resident weights plus one shared correction K step (px_rowpipe.cuh); nothing is normalised or
// transposed on the way in:
//   * the z tile arrives by TMA as a K-major operand (rows of 128 channels): the bf16 rows of z themselves, or, for an
//     fp32 z, its standardised fp16 copy `zn` (px_standardise_rows), whose statistics are known;
//   * the x tile arrives by TMA exactly as it lies in memory, [128 channels][64 j] a run, and is used as an MN-major
//     operand: the tensor core reads it transposed;
//   * the statistics of both are summed by threads from the tiles in shared memory (Gram products with the sums of squares on their
//     diagonals and rows of ones behind the weights took 600 to 1200 cycles more of the tensor pipe a tile, and the statistics of a
//     tile as long to come: bf16 N = 200 15.3 -> 14.5 us, 437 45.0 -> 42.7, 768 109 -> 105, 1536 435 -> 420; fp32 N = 128 8.5 -> 8.2,
//     200 15.0 -> 14.5, 640 98.5 -> 96.5, from 768 on level).
//
//   warps 0..15   epilogue: a thread owns one pair element and 32 channels: p * sigmoid(g) + residual (the raw z
//                 tile in shared memory), packed to bf16 over the z tile in place, which leaves through a TMA store.
//                 fp32 rows are staged the same way and stored or added by TMA; where the residual lies in another tensor, it
//                 is read and the rows are written with plain accesses.
//   warps 16..    statistics of 16 rows a warp at a time (8 warps, or 4 where the z side has none): correction rows, scales.
//   then          TMA producer (z and x tiles); MMA issuers of the gate and of the projection product.
// Tensor memory: one or two sets of gate accumulator (128) | projection accumulator (128).
// Algorithmic HBM traffic per pair element: 256 + 128*sizeof(Tz) read, 128*sizeof(Tz) written.  Every wait is bounded.
#include <cstring>

#include "px_rowpipe.cuh"

namespace px {

__host__ __device__ constexpr int to_stats_warps(bool standardised) { return standardised ? 4 : 8; }
__host__ __device__ constexpr int to_threads(bool standardised) { return 32 * (16 + to_stats_warps(standardised) + 3); }
constexpr int kToWBytes = 2 * kPanelBytes;     // [128 weight rows][128 k]
constexpr int kToWExtra = 128 * 32;
constexpr int kToStages = 2;
constexpr int kToSlots = kToStages + 1;
constexpr uint32_t kToColG = 0, kToColP = 128, kToColSet = 256;

// a_ready, the correction rows and the scales of a stage are written anew for the tile two later, whose load waits for a_empty, which the
// epilogue hands back when it has used them all.
struct ToBars {
  uint64_t raw_full[kToStages], a_ready[kToStages], a_empty[kToStages];
  uint64_t acc_full[2], acc_free[2], w_full;
  uint32_t tmem_base;
};
struct ToLayout {
  static constexpr int wg = 0;                                  // gate weights
  static constexpr int wz = wg + kToWBytes;                     // projection weights
  static constexpr int wxg = wz + kToWBytes;                    // correction panels (k 0..7: z, k 8..15: x)
  static constexpr int wxz = wxg + kToWExtra;
  static constexpr int zt = wxz + kToWExtra;                    // z tiles (later the output rows)
  static constexpr int xt = zt + kToStages * kOperandBytes;     // x tiles, [128 c][64 j] per j block
  static constexpr int ax = xt + kToStages * kOperandBytes;     // tile-side correction panels
  static constexpr int scale = ax + kToStages * 128 * 32;       // float2 (rstd_z, rstd_x) per row and slot
  static constexpr int bars = scale + kToSlots * 128 * 8;
  static constexpr int total = bars + (int)sizeof(ToBars);
};
static_assert(ToLayout::zt % 1024 == 0 && ToLayout::xt % 1024 == 0, "tiles must keep the swizzle alignment");
static_assert(ToLayout::total + 1024 <= 232448, "shared memory budget");

// The resident weights: gate | projection, and their correction panels.  The gate rows carry
// the 1/2 of sigmoid(x) = 1/2 + 1/2 tanh(x/2); the z statistics use k 0..7 of the correction step, the x statistics k 8..15.
template <bool kF16>
struct ToWeights {
  const float *ln_in_w, *ln_in_b, *ln_out_w, *ln_out_b;
  const bf16 *w_z, *w_g;
  static constexpr int kBytes = ToLayout::zt;
  static_assert(kBytes == 2 * (kToWBytes + kToWExtra), "no padding in the image");
  __device__ __forceinline__ void fold(unsigned char* sm, int, int warp, int warps, int lane, int, int) const {
    fold_weight_rows<kF16, kF16>(sm + ToLayout::wg, sm + ToLayout::wxg, 0, kPanelBytes, w_g, 0, 128, ln_in_w, ln_in_b, 0.5f, warp, warps,
                                 lane, 0);
    fold_weight_rows<true, true>(sm + ToLayout::wz, sm + ToLayout::wxz, 0, kPanelBytes, w_z, 0, 128, ln_out_w, ln_out_b, 1.0f, warp, warps,
                                 lane, 1);
  }
};

template <typename Tz, bool kBulk, int kRun>
__global__ void __launch_bounds__(to_threads(sizeof(Tz) != 2), 1)
trimul_out_tc_kernel(const __grid_constant__ CUtensorMap map_z, const __grid_constant__ CUtensorMap map_x,
                     const __grid_constant__ CUtensorMap map_out, const Tz* __restrict__ z_in, Tz* __restrict__ z_out,
                     const ToWeights<sizeof(Tz) != 2> weights, const unsigned char* __restrict__ folded,
                     int n_i, int n, int add_residual, float eps, int runs_j, int n_tiles) {
  constexpr int kPer = 128 / kRun;                     // runs of a tile
  constexpr bool kTma = sizeof(Tz) == 2;               // bf16: residual from the z tile, output through TMA
  constexpr bool kF16 = !kTma;                           // operand format of the z side; the x side is always fp16
  constexpr int kStats = to_stats_warps(kF16), kThreads = to_threads(kF16), kLoad = 16 + kStats;   // kLoad: the producer's warp
  constexpr int kSets = kTma ? 2 : 1;                    // sets of accumulators (two made no difference to fp32 rows)
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  ToBars& bars = *reinterpret_cast<ToBars*>(sm + ToLayout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;

  const bool skip = cta_begin();         // an earlier bounded wait gave up: do not start new work
  if (threadIdx.x == 32) {
    prefetch_maps(map_z, map_x);
    if (kTma || kBulk) prefetch_maps(map_out);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kToStages; ++s) {
      mbar_init(&bars.raw_full[s], 1);
      mbar_init(&bars.a_ready[s], kStats);
      mbar_init(&bars.a_empty[s], 1);                      // the epilogue, which waits for everything else that reads the stage
    }
    mbar_init(&bars.w_full, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars.acc_full[b], 2);
      mbar_init(&bars.acc_free[b], 16);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kLoad) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (kF16)                                                // standardised rows: known statistics of the z side, (0, 1)
    for (int i = threadIdx.x; i < kToSlots * 128; i += kThreads) {
      if (i < kToStages * 128) write_correction_row(sm + ToLayout::ax + (i >> 7) * 128 * 32, i & 127, 0.f, 1.f, false, 0, false);
      reinterpret_cast<float2*>(sm + ToLayout::scale)[i].x = 1.f;
    }
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  if (!cta_ready(skip, warp == kLoad, bars.tmem_base, 512u, [&] {
        if (folded && threadIdx.x == 0) folded_load(sm, folded, ToWeights<kF16>::kBytes, &bars.w_full);
      }))
    return;
  fold_here(weights, folded, sm, 0, &bars.w_full);
  const uint32_t tmem_base = bars.tmem_base;
  const int first_tile = blockIdx.x, tile_step = gridDim.x;

  if (warp >= kLoad) {
    if (warp == kLoad) {
      // ---------------------------------------------------------------- tile producer: z (bf16 rows) and x
      int k = 0;
      for (int tile = first_tile; tile < n_tiles; tile += tile_step, ++k) {
        const int s = k % kToStages, m = k / kToStages;
        if (!mbar_wait_warp(&bars.a_empty[s], (m & 1) ^ 1, 1u)) break;
        // Where rows are added in L2, a tile is asked for once the one before has arrived and been measured: loads that queue
        // further ahead delay the additions (asked for with the stage: 553 -> 568 us at N = 1536, 247 -> 256 at 1024; below 500 level).
        if (kBulk && add_residual && k && !mbar_wait_warp(&bars.a_ready[(k - 1) % kToStages], ((k - 1) / kToStages) & 1, 1u)) break;
        if (elect_lane()) {
          mbar_expect_tx(&bars.raw_full[s], 2 * kOperandBytes);
          const uint32_t zdst = smem_u32(sm + ToLayout::zt + s * kOperandBytes), xdst = smem_u32(sm + ToLayout::xt + s * kOperandBytes);
          for (int h = 0; h < kPer; ++h) {
            const Run r = run_at<kRun>(kPer * tile + h, runs_j);
            for (int p = 0; p < 2; ++p)
              tma_load_3d(zdst + p * kPanelBytes + h * (kRun * 128), &map_z, &bars.raw_full[s], 64 * p, r.t, r.u);
            for (int p = 0; p < kRun / 64; ++p) tma_load_3d(xdst + (h + p) * kPanelBytes, &map_x, &bars.raw_full[s], r.t + 64 * p, r.u, 0);
          }
          // The tile that takes this stage next is asked of L2 (a stage is held until its rows have left, so only two tiles are on
          // their way): bf16 N = 768 122 -> 107 us, fp32 without a residual N = 1024 230 -> 203.  Not where rows are added in L2,
          // which is then what is waited for: 552 -> 610 at N = 1536, 140 -> 151 at N = 768.
          const int next = tile + 2 * tile_step;
          if ((kTma || (kBulk && !add_residual)) && next < n_tiles) {
            for (int h = 0; h < kPer; ++h) {
              const Run r = run_at<kRun>(kPer * next + h, runs_j);
              for (int p = 0; p < 2; ++p) tma_prefetch_3d(&map_z, 64 * p, r.t, r.u);
              for (int p = 0; p < kRun / 64; ++p) tma_prefetch_3d(&map_x, r.t + 64 * p, r.u, 0);
            }
          }
        }
        __syncwarp();
      }
    } else {
      // ---------------------------------------------------------------- gate / projection product
      const bool proj = warp == kLoad + 2;
      const uint32_t idesc = proj ? umma_idesc_f16(128, 128, true, false) : umma_idesc_16(128, 128, kF16, kF16);
      const uint32_t d_tmem = tmem_base + (proj ? kToColP : kToColG);
      const uint32_t w_addr = smem_u32(sm + (proj ? ToLayout::wz : ToLayout::wg));
      const uint64_t wx_desc = umma_desc_sw32(smem_u32(sm + (proj ? ToLayout::wxz : ToLayout::wxg)));
      int k = 0;
      const bool have_w = mbar_wait_warp(&bars.w_full, 0, 4u);   // the resident weights
      for (int tile = first_tile; tile < n_tiles && have_w; tile += tile_step, ++k) {
        const int s = k % kToStages, m = k / kToStages, b = k % kSets;
        const uint32_t d = d_tmem + b * kToColSet;
        if (!mbar_wait_warp(&bars.raw_full[s], m & 1, 4u) || !mbar_wait_warp(&bars.acc_free[b], ((k / kSets) & 1) ^ 1, 8u)) break;
        tc_fence_after();
        if (elect_lane()) {
          const uint32_t a_addr = smem_u32(sm + (proj ? ToLayout::xt : ToLayout::zt) + s * kOperandBytes);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            const uint64_t a_desc = proj ? umma_desc_mn_sw128(a_addr + ks * 2048, kPanelBytes, 1024)
                                         : umma_desc_sw128(a_addr + (ks >> 2) * kPanelBytes) + 2 * (ks & 3);
            umma_bf16(d, a_desc, umma_desc_sw128(w_addr + (ks >> 2) * kPanelBytes) + 2 * (ks & 3), idesc, ks ? 1u : 0u);
          }
        }
        __syncwarp();
        if (!mbar_wait_warp(&bars.a_ready[s], m & 1, 4u)) break;   // the correction step needs the statistics
        tc_fence_after();
        if (elect_lane()) {
          umma_bf16(d, umma_desc_sw32(smem_u32(sm + ToLayout::ax + s * 128 * 32)), wx_desc, umma_idesc_bf16(128, 128, false, false),
                    1u);
          umma_commit(&bars.acc_full[b]);
        }
        __syncwarp();
      }
    }
  } else if (warp >= 16) {
    // ------------------------------------------------------------------ row statistics
    // z: two lanes a row.  x, whose rows lie across the tile ([128 c][64 j] a panel): a lane sums two neighbouring j over the
    // channels 8 i + 2 (lane / 8) and the one behind, so that a warp's load meets every bank once, and four lanes add up.
    const int sw = warp - 16;
    float* scale = reinterpret_cast<float*>(sm + ToLayout::scale);
    int k = 0;
    for (int tile = first_tile; tile < n_tiles; tile += tile_step, ++k) {
      const int s = k % kToStages;
      if (!mbar_wait_warp(&bars.raw_full[s], (k / kToStages) & 1, 16u)) break;
      unsigned char* ax = sm + ToLayout::ax + s * 128 * 32;
      float* sc = scale + (k % kToSlots) * 256;
      if (!kF16) {
        const int r = 16 * sw + (lane >> 1), half = lane & 1;
        float mean, var;
        bf16_row_stats(sm + ToLayout::zt + s * kOperandBytes, r, half, mean, var);
        // rstd * (W'x - mean * s + std * t): the row side of the correction step holds (-mean, std)
        if (half == 0) {
          write_correction_row(ax, r, -mean, sqrtf(var + eps), false, 0, false);
          sc[2 * r] = rsqrtf(var + eps);
        }
      }
#pragma unroll 1
      for (int r0 = 16 * sw; r0 < 128; r0 += 16 * kStats) {
        const unsigned char* x = sm + ToLayout::xt + s * kOperandBytes + (r0 >> 6) * kPanelBytes + (lane & 3) * 4;
        const int piece = ((r0 & 63) >> 3) + ((lane >> 2) & 1), c0 = 2 * (lane >> 3);
        const auto pair = [&](int c) { return unpack_f16x2(*reinterpret_cast<const uint32_t*>(x + c * 128 + ((piece ^ (c & 7)) << 4))); };
        const float2 x0 = pair(0);                         // about one of its values, nothing cancels
        float s0 = 0.f, s1 = 0.f, q0 = 0.f, q1 = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          float2 d = pair(8 * (i >> 1) + c0 + (i & 1));
          add2(d.x, d.y, -x0.x, -x0.y);
          add2(s0, s1, d.x, d.y);
          fma2(q0, q1, d.x, d.y, d.x, d.y, q0, q1);
        }
#pragma unroll
        for (int o = 8; o < 32; o *= 2) {
          add2(s0, s1, __shfl_xor_sync(0xffffffffu, s0, o), __shfl_xor_sync(0xffffffffu, s1, o));
          add2(q0, q1, __shfl_xor_sync(0xffffffffu, q0, o), __shfl_xor_sync(0xffffffffu, q1, o));
        }
        if (lane < 16) {
          const bool odd = lane >= 8;
          const int r = r0 + 2 * (lane & 7) + odd;
          const float m = (odd ? s1 : s0) * (1.0f / kC), var = fmaxf((odd ? q1 : q0) * (1.0f / kC) - m * m, 0.f);
          const float e = eps * (PX_TRIMUL_X_SCALE * PX_TRIMUL_X_SCALE);   // x arrives scaled
          write_correction_row(ax, r, -((odd ? x0.y : x0.x) + m), sqrtf(var + e), false, 1, false);
          sc[2 * r + 1] = rsqrtf(var + e);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.a_ready[s]);
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int part = warp >> 2, qw = warp & 3;
    const int row = 32 * qw + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * qw) << 16);
    const bool leader = threadIdx.x == 0;
    int k = 0;
    bool ok = true;
    for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step, ++k) {
      const int s = k % kToStages;
      const Run run = run_at<kRun>(kPer * tile + 32 * qw / kRun, runs_j);
      const int i = run.u, jw = run.t + 32 * qw % kRun;     // the warp's first element
      const int valid = i >= n_i || jw >= n ? 0 : n - jw < 32 ? n - jw : 32;
      RowsOutReq rq;
      if (!kTma && !kBulk) {                               // the residual values are requested before the wait
        rows_out_request(rq, reinterpret_cast<const float*>(z_in), (long long)i * n + jw, 1, valid, 32 * part, lane, add_residual != 0);
        // the residual lines of the next tile are asked of L2 now: a tile later they are a hit, not a trip to HBM
        const int nt = tile + tile_step;
        if (add_residual && nt < n_tiles) {
          const Run r2 = run_at<kRun>(kPer * nt + 32 * qw / kRun, runs_j);
          const int i2 = r2.u, j2 = r2.t + 32 * qw % kRun + lane;
          if (j2 < n && i2 < n_i)
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(reinterpret_cast<const float*>(z_in) + ((size_t)i2 * n + j2) * kC + 32 * part));
        }
      }
      const int b = k % kSets;
      ok = mbar_wait(&bars.acc_full[b], (k / kSets) & 1, 32u);
      ok = named_barrier_all(1, 512, ok);                  // all sixteen warps go on, or none
      if (!ok) break;
      tc_fence_after();
      const float2 sc = reinterpret_cast<const float2*>(sm + ToLayout::scale)[(k % kToSlots) * 128 + row];
      unsigned char* ztile = sm + ToLayout::zt + s * kOperandBytes;
      uint32_t g[32], p[32];
      tmem_ld32(lane_addr + b * kToColSet + kToColG + 32 * part, g);
      tmem_ld32(lane_addr + b * kToColSet + kToColP + 32 * part, p);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.acc_free[b]);          // this warp has read its part of the accumulators
      float v[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        // p * sigmoid(g) = h + h * tanh(g / 2) with h = p / 2 (the half of g is folded into the weights)
        const float h = 0.5f * sc.y * __uint_as_float(p[e]);
        v[e] = fmaf(h, tanh_fast(sc.x * __uint_as_float(g[e])), h);
      }
      if (kTma) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          unsigned char* piece = ztile + operand_piece_offset(row, 4 * part + q);
          uint32_t w[4];
          if (add_residual) {
            const uint4 zv = *reinterpret_cast<const uint4*>(piece);
            const uint32_t zw[4] = {zv.x, zv.y, zv.z, zv.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 r2 = unpack_bf16x2(zw[e]);
              w[e] = pack_bf16x2_int(v[8 * q + 2 * e] + r2.x, v[8 * q + 2 * e + 1] + r2.y);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = pack_bf16x2_int(v[8 * q + 2 * e], v[8 * q + 2 * e + 1]);
          }
          *reinterpret_cast<uint4*>(piece) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        named_barrier(1, 512);
        if (leader) {
          for (int h = 0; h < kPer; ++h) {
            const Run r = run_at<kRun>(kPer * tile + h, runs_j);
            for (int pnl = 0; pnl < 2 && r.u < n_i; ++pnl)
              tma_store_3d(&map_out, smem_u32(ztile + pnl * kPanelBytes) + h * (kRun * 128), 64 * pnl, r.t, r.u);
          }
          tma_store_commit();
          tma_store_wait_read<0>();                          // the store has read the stage: hand it back
          mbar_arrive(&bars.a_empty[s]);
        }
      } else if (kBulk) {
        // fp32 rows: staged inside the stage's tiles, which the tensor core has finished reading (16 warps x 4 KB)
        unsigned char* stg = sm + (warp < 8 ? ToLayout::zt : ToLayout::xt) + s * kOperandBytes + (warp & 7) * 4096;
        rows_bulk_out(stg, v, &map_out, add_residual != 0, 32 * part, jw, i, valid > 0, lane);
        if (lane == 0) tma_store_wait_read<0>();
        named_barrier(1, 512);
        if (leader) mbar_arrive(&bars.a_empty[s]);
      } else {
        // fp32 rows: coalesced through a warp-private staging area inside the stage's tiles, which the tensor core
        // has finished reading (16 warps x 4 KB = the z tile and the x tile)
        unsigned char* stg = sm + (warp < 8 ? ToLayout::zt : ToLayout::xt) + s * kOperandBytes + (warp & 7) * 4096;
        rows_out_store(stg, v, rq, reinterpret_cast<float*>(z_out), (long long)i * n + jw, 1, valid, 32 * part, lane);
        named_barrier(1, 512);
        if (leader) mbar_arrive(&bars.a_empty[s]);
      }
    }
    if (kTma ? leader : kBulk && lane == 0) tma_store_wait_read<0>();
  }

  tc_fence_before();
  cta_teardown_sync();
  if (warp == kLoad) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

PX_DEFINE_FAMILY_HOOKS(trimul_out)

// kBulk (fp32 z): the output goes through TMA, which covers everything but a residual from another tensor.
template <typename Tz, bool kBulk, int kRun>
static int32_t launch_trimul_out_runs(const px_f16* x, const void* z_in, const px_f16* zn, void* z_out,
                                 const ToWeights<sizeof(Tz) != 2>& weights, const void* folded,
                                 int64_t n_i, int64_t n, int64_t ld, int32_t add_residual, float eps, cudaStream_t st) {
  CUtensorMap mz, mx, mout;
  // operand rows: bf16 z itself, or the standardised fp16 copy of an fp32 z
  if (!make_map_3d(&mz, sizeof(Tz) == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                   sizeof(Tz) == 2 ? z_in : (const void*)zn, 128, (uint64_t)n, (uint64_t)n_i, 256, (uint64_t)n * 256, 64, kRun,
                   CU_TENSOR_MAP_SWIZZLE_128B, 1))
    return PX_ERR_LAUNCH;
  if (sizeof(Tz) == 2) {
    if (!make_map_3d(&mout, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, z_out, 128, (uint64_t)n, (uint64_t)n_i, 256, (uint64_t)n * 256,
                     64, kRun, CU_TENSOR_MAP_SWIZZLE_128B, 1))
      return PX_ERR_LAUNCH;
  } else if (kBulk) {
    if (!make_map_3d(&mout, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, z_out, 128, (uint64_t)n, (uint64_t)n_i, 512, (uint64_t)n * 512, 32, 32,
                     CU_TENSOR_MAP_SWIZZLE_128B, 1))
      return PX_ERR_LAUNCH;
  } else {
    memset(&mout, 0, sizeof(mout));
  }
  // x [128 channels][n_i][ld]: a load brings [128 channels][one i][64 j]
  if (!make_map_3d(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, (uint64_t)ld, (uint64_t)n_i, 128, (uint64_t)ld * 2,
                   (uint64_t)n_i * ld * 2, 64, 1, CU_TENSOR_MAP_SWIZZLE_128B, 128))
    return PX_ERR_LAUNCH;
  const size_t smem = ToLayout::total + 1024;
  static SmemLimit limit;
  if (!limit.set(trimul_out_tc_kernel<Tz, kBulk, kRun>, smem)) return PX_ERR_LAUNCH;
  const int64_t n_tiles = tiles_of(n_i, n, kRun);
  if (n_tiles > 0x7fffffff) return PX_ERR_UNSUPPORTED;
  const int grid = even_grid(n_tiles, sm_count(), tile_period(n_i, n, kRun));
  return launch_pdl(trimul_out_tc_kernel<Tz, kBulk, kRun>, dim3(grid), to_threads(sizeof(Tz) != 2), smem, st, mz, mx, mout, (const Tz*)z_in, (Tz*)z_out, weights,
                    (const unsigned char*)folded, (int)n_i, (int)n, (int)add_residual, eps, (int)runs_of(n, kRun), (int)n_tiles)
             ? PX_OK
             : PX_ERR_LAUNCH;
}

template <typename Tz, bool kBulk>
static int32_t launch_trimul_out(const px_f16* x, const void* z_in, const px_f16* zn, void* z_out,
                                 const ToWeights<sizeof(Tz) != 2>& weights, const void* folded,
                                 int64_t n_i, int64_t n, int64_t ld, int32_t add_residual, float eps, cudaStream_t st) {
  const Cut cut = output_cut(n_i, n, ld == n, sizeof(Tz) == 4 ? 18 : 0);
  if (cut == Cut::kOneRow) n *= n_i, ld = n, n_i = 1;
  return (cut == Cut::kRuns ? launch_trimul_out_runs<Tz, kBulk, 64> : launch_trimul_out_runs<Tz, kBulk, 128>)(
      x, z_in, zn, z_out, weights, folded, n_i, n, ld, add_residual, eps, st);
}

static bool trimul_out_args_ok(const px_f16* x, const void* z_in, const px_f16* zn, const void* z_out, int32_t z_dtype, int64_t n_i,
                               int64_t n_j, int64_t ld) {
  return x && z_in && z_out && !(z_dtype == PX_F32 && (!zn || ((uintptr_t)zn & 15))) && n_i > 0 && n_j > 0 && n_i <= 32768 &&
         n_j <= 32768 && ld == px_ld(n_j) && !(((uintptr_t)x | (uintptr_t)z_in | (uintptr_t)z_out) & 15);
}
template <bool kF16>
static ToWeights<kF16> to_weights(const float* ln_in_w, const float* ln_in_b, const float* ln_out_w, const float* ln_out_b,
                                  const px_f16* w_z, const px_w16* w_g) {
  return {ln_in_w, ln_in_b, ln_out_w, ln_out_b, (const bf16*)w_z, (const bf16*)w_g};
}
static bool to_weights_ok(const float* ln_in_w, const float* ln_in_b, const float* ln_out_w, const float* ln_out_b,
                          const px_f16* w_z, const px_w16* w_g) {
  return ln_in_w && ln_in_b && ln_out_w && ln_out_b && w_z && w_g &&
         !(((uintptr_t)w_z | (uintptr_t)w_g | (uintptr_t)ln_in_w | (uintptr_t)ln_in_b | (uintptr_t)ln_out_w | (uintptr_t)ln_out_b) & 15);
}

}  // namespace px

using namespace px;

extern "C" int64_t px_trimul_out_folded_bytes(void) { return ToWeights<true>::kBytes; }

extern "C" int32_t px_trimul_out_fold(const float* ln_in_w, const float* ln_in_b, const float* ln_out_w, const float* ln_out_b,
                                      const px_f16* w_z, const px_w16* w_g, int32_t rows_dtype, void* folded, void* stream) {
  if (!to_weights_ok(ln_in_w, ln_in_b, ln_out_w, ln_out_b, w_z, w_g) || !folded || ((uintptr_t)folded & 15)) return PX_ERR_BAD_ARG;
  if (rows_dtype != PX_F16 && rows_dtype != PX_BF16) return PX_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  return (rows_dtype == PX_F16 ? launch_fold(to_weights<true>(ln_in_w, ln_in_b, ln_out_w, ln_out_b, w_z, w_g), 1, folded, st)
                               : launch_fold(to_weights<false>(ln_in_w, ln_in_b, ln_out_w, ln_out_b, w_z, w_g), 1, folded, st))
             ? PX_OK
             : PX_ERR_LAUNCH;
}

extern "C" int32_t px_trimul_out_folded(const px_f16* x, const void* z_in, const px_f16* zn, void* z_out, int32_t z_dtype,
                                        const void* folded, int64_t n_i, int64_t n_j, int64_t ld, int32_t add_residual, float eps,
                                        void* stream) {
  if (!trimul_out_args_ok(x, z_in, zn, z_out, z_dtype, n_i, n_j, ld) || !folded || ((uintptr_t)folded & 15)) return PX_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (z_dtype == PX_F32)
    return (add_residual && z_in != z_out ? launch_trimul_out<float, false> : launch_trimul_out<float, true>)(x, z_in, zn, z_out, ToWeights<true>{}, folded, n_i, n_j, ld, add_residual, eps, st);
  if (z_dtype == PX_BF16)
    return launch_trimul_out<bf16, false>(x, z_in, nullptr, z_out, ToWeights<false>{}, folded, n_i, n_j, ld, add_residual, eps, st);
  return PX_ERR_UNSUPPORTED;
}

extern "C" int32_t px_trimul_out(const px_f16* x, const void* z_in, const px_f16* zn, void* z_out, int32_t z_dtype,
                                 const float* ln_in_w, const float* ln_in_b, const float* ln_out_w,
                                 const float* ln_out_b, const px_f16* w_z, const px_w16* w_g, int64_t n_i,
                                 int64_t n_j, int64_t ld, int32_t add_residual, float eps, void* stream) {
  if (!to_weights_ok(ln_in_w, ln_in_b, ln_out_w, ln_out_b, w_z, w_g) || !trimul_out_args_ok(x, z_in, zn, z_out, z_dtype, n_i, n_j, ld))
    return PX_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (z_dtype == PX_F32)
    return (add_residual && z_in != z_out ? launch_trimul_out<float, false> : launch_trimul_out<float, true>)(x, z_in, zn, z_out, to_weights<true>(ln_in_w, ln_in_b, ln_out_w, ln_out_b, w_z, w_g), nullptr, n_i,
                                    n_j, ld, add_residual, eps, st);
  if (z_dtype == PX_BF16)
    return launch_trimul_out<bf16, false>(x, z_in, nullptr, z_out, to_weights<false>(ln_in_w, ln_in_b, ln_out_w, ln_out_b, w_z, w_g), nullptr,
                                   n_i, n_j, ld, add_residual, eps, st);
  return PX_ERR_UNSUPPORTED;
}
