// SwiGLU transition for 128-channel rows on the 5th-generation tensor cores:
//   x_out = [x +] W_o( silu(W_a LN(x)) * (W_b LN(x)) ),  hidden width 512, the [rows][512] intermediates never
//   leave the SM (tensor memory -> registers -> tensor memory).  Both products take fp16 operands, whatever the
//   storage type of x: the rows pass through registers for the LayerNorm anyway, a normalised row and the weights
//   lie far inside the fp16 range, and fp16 keeps three more bits than bf16 (h saturates at +-65504).
//
// Persistent kernel, one CTA per SM, 128 rows per tile, three tiles in flight: while the tensor core works through
// the eight 64-wide hidden chunks of one tile, the next tile is being normalised and the previous one written out.
//
//   warps 0..7    SwiGLU, two groups of four warps that take the hidden chunks in turn, each with its own H buffer: a thread
//                 owns one row, pulls a|b out of tensor memory in steps of 16, forms h = silu(a) * b, and writes h (fp16)
//                 over a values it has read, as the A operand of the second product.  No thread needs another's values, so
//                 the groups meet at no barrier and one group's chain of waits runs beside the other's arithmetic (all
//                 eight warps on one chunk, two barriers each: 67 us against 61 at N = 384, 476..525 against 416..438 at N = 1024).
//   warps 8..11   LayerNorm: eight lanes a row, eight rows in flight per warp; the normalised rows
//                 are written as the K-major, 128-byte-swizzled A operand of the first product (two buffers).
//   warps 12..15  output: accumulator -> shared staging (where the residual waits) -> TMA store or addition (two accumulators).
//   warp 16       TMA producer of the weight chunks: rows 64c..64c+63 of W_a and W_b and columns 64c..64c+63 of
//                 W_o, 48 KB, 3-stage ring (the weights are re-read from L2 for every tile: 384 KB per 128 rows).
//   warps 17, 18  MMA issuers: H = A [W_a;W_b]_c^T (M=128, N=128, K=128) and OUT += h W_o,c^T (M=128, N=128, K=64, h
//                 as the TMEM-resident A operand).  One warp for both, each first product right behind the second one that frees
//                 its buffer, was slower (64.7 us against 61 at N = 384).
// What bounds it: above some 700 tokens the power limit (1.6 GHz at N = 768; without the weight loads, the tanh, the
// LayerNorm or the products it takes 90 to 100 % of its time), below it the chain p_ready -> second product (256 cycles of
// the tensor pipe) -> first product (512) -> h, of which two run side by side.
// Tensor memory: H_0 | H_1 | OUT_0 | OUT_1, 128 columns each.  Every mbarrier wait is bounded.
#include "px_rowpipe.cuh"

namespace px {

constexpr int kTrStages = 3;
constexpr int kTrABytes = 2 * 128 * 128;            // one tile: two k panels of [128 rows][64 k] fp16
constexpr int kTrW1Bytes = 2 * 128 * 128;           // [W_a chunk; W_b chunk]: two k panels of [128 rows][64 k]
constexpr int kTrW2Bytes = 128 * 128;               // W_o chunk: [128 out rows][64 hidden]
constexpr int kTrStageBytes = kTrW1Bytes + kTrW2Bytes;
constexpr int kTrChunks = 8;                        // 512 hidden / 64
constexpr int kTrWarps = 20;
constexpr int kTrThreads = 32 * kTrWarps;

struct TransBars {
  uint64_t a_full[2], a_free[2], w_full[kTrStages], w_empty[kTrStages], h_full[2], h_free[2], p_ready[2], out_full[2],
      out_free[2], res_full[4];
  uint32_t tmem_base;
};
struct TransLayout {
  static constexpr int a = 0;                                  // two normalised tiles
  static constexpr int w = a + 2 * kTrABytes;                  // weight ring
  static constexpr int stg = w + kTrStages * kTrStageBytes;    // output staging: [128 rows][32 fp32]
  static constexpr int affine = stg + 128 * 128;               // gamma / 2 and beta / 2
  static constexpr int bars = affine + 2 * kC * 4;
  static constexpr int total = bars + (int)sizeof(TransBars);
};

// Sixteen channels of a row as they are stored: lane p of the row's eight holds 8p..8p+7 and 64+8p..64+8p+7, whatever the type, so
// that both types are summed in one order.
template <typename Tz>
struct Raw16;
template <>
struct Raw16<bf16> {
  uint4 v[2];
  __device__ __forceinline__ void load(const bf16* row, int p) {
#pragma unroll
    for (int i = 0; i < 2; ++i) v[i] = *reinterpret_cast<const uint4*>(row + 64 * i + 8 * p);
  }
  __device__ __forceinline__ void zero() { v[0] = v[1] = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ void get(float (&x)[16]) const {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = unpack_bf16x2(w[e]);
        x[8 * i + 2 * e] = f.x, x[8 * i + 2 * e + 1] = f.y;
      }
    }
  }
};
template <>
struct Raw16<float> {
  float4 v[4];
  __device__ __forceinline__ void load(const float* row, int p) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4*>(row + 64 * (i >> 1) + 8 * p + 4 * (i & 1));
  }
  __device__ __forceinline__ void zero() { v[0] = v[1] = v[2] = v[3] = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void get(float (&x)[16]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) x[4 * i] = v[i].x, x[4 * i + 1] = v[i].y, x[4 * i + 2] = v[i].z, x[4 * i + 3] = v[i].w;
  }
};

template <typename Tz>
__global__ void __launch_bounds__(kTrThreads, 1)
transition_tc_kernel(const __grid_constant__ CUtensorMap map_wa, const __grid_constant__ CUtensorMap map_wb,
                     const __grid_constant__ CUtensorMap map_wo, const __grid_constant__ CUtensorMap map_out,
                     const __grid_constant__ CUtensorMap map_res, const Tz* __restrict__ x_in,
                     const float* __restrict__ ln_w, const float* __restrict__ ln_b, long long rows, int n_tiles,
                     int add_residual, int apart, float eps) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  TransBars& bars = *reinterpret_cast<TransBars*>(sm + TransLayout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int first_tile = blockIdx.x, tile_step = gridDim.x;

  const bool skip = cta_begin();         // an earlier bounded wait gave up: do not start new work
  if (threadIdx.x == 32) prefetch_maps(map_wa, map_wb, map_wo, map_out, map_res);
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars.a_full[b], 4);
      mbar_init(&bars.a_free[b], 1);
      mbar_init(&bars.h_full[b], 1);
      mbar_init(&bars.h_free[b], 1);
      mbar_init(&bars.p_ready[b], 4);
      mbar_init(&bars.out_full[b], 1);
      mbar_init(&bars.out_free[b], 4);
    }
    for (int q = 0; q < 4; ++q) mbar_init(&bars.res_full[q], 1);
    for (int s = 0; s < kTrStages; ++s) {
      mbar_init(&bars.w_full[s], 1);
      mbar_init(&bars.w_empty[s], 2);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (!cta_ready(skip, warp == 16, bars.tmem_base, 512u)) return;
  const uint32_t tmem_base = bars.tmem_base;

  if (warp >= 16) {
    if (warp == 16) {
      // ---------------------------------------------------------------- weight producer
      int j = 0;                                      // chunk counter over all tiles of this CTA
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
        for (int c = 0; c < kTrChunks && ok; ++c, ++j) {
          const int s = j % kTrStages;
          ok = mbar_wait_warp(&bars.w_empty[s], ((j / kTrStages) & 1) ^ 1, 1u);
          if (!ok) break;
          if (elect_lane()) {
            mbar_expect_tx(&bars.w_full[s], kTrStageBytes);
            const uint32_t base = smem_u32(sm + TransLayout::w + s * kTrStageBytes);
            for (int p = 0; p < 2; ++p) {  // k panel p: rows 0..63 from W_a, rows 64..127 from W_b
              tma_load_3d(base + p * 16384, &map_wa, &bars.w_full[s], 64 * p, 64 * c, 0);
              tma_load_3d(base + p * 16384 + 8192, &map_wb, &bars.w_full[s], 64 * p, 64 * c, 0);
            }
            tma_load_3d(base + kTrW1Bytes, &map_wo, &bars.w_full[s], 64 * c, 0, 0);
          }
          __syncwarp();
        }
      }
    } else if (warp == 17) {
      // ---------------------------------------------------------------- first product: H = A [W_a;W_b]_c^T
      constexpr uint32_t idesc = umma_idesc_f16(128, 128);
      int j = 0, k = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step, ++k) {
        const int ab = k & 1;
        ok = mbar_wait_warp(&bars.a_full[ab], (k >> 1) & 1, 2u);
        const uint32_t a_addr = smem_u32(sm + TransLayout::a + ab * kTrABytes);
        for (int c = 0; c < kTrChunks && ok; ++c, ++j) {
          const int s = j % kTrStages, hb = j & 1;
          ok = mbar_wait_warp(&bars.w_full[s], (j / kTrStages) & 1, 4u) && mbar_wait_warp(&bars.h_free[hb], ((j >> 1) & 1) ^ 1, 4u);
          if (!ok) break;
          tc_fence_after();
          if (elect_lane()) {
            const uint32_t wbase = smem_u32(sm + TransLayout::w + s * kTrStageBytes);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
              umma_bf16(tmem_base + 128 * hb, umma_desc_sw128(a_addr + (ks >> 2) * 16384) + 2 * (ks & 3),
                        umma_desc_sw128(wbase + (ks >> 2) * 16384) + 2 * (ks & 3), idesc, ks ? 1u : 0u);
            umma_commit(&bars.h_full[hb]);
            umma_commit(&bars.w_empty[s]);              // this warp's share of the reads of the stage
            if (c == kTrChunks - 1) umma_commit(&bars.a_free[ab]);   // the tile has been read for the last time
          }
          __syncwarp();
        }
      }
    } else if (warp == 18) {
      // ---------------------------------------------------------------- second product: OUT += h W_o,c^T
      constexpr uint32_t idesc = umma_idesc_f16(128, 128);
      int j = 0, k = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step, ++k) {
        const int ob = k & 1;
        ok = mbar_wait_warp(&bars.out_free[ob], ((k >> 1) & 1) ^ 1, 8u);
        for (int c = 0; c < kTrChunks && ok; ++c, ++j) {
          const int s = j % kTrStages, hb = j & 1;
          ok = mbar_wait_warp(&bars.w_full[s], (j / kTrStages) & 1, 4u) && mbar_wait_warp(&bars.p_ready[hb], (j >> 1) & 1, 8u);
          if (!ok) break;
          tc_fence_after();
          if (elect_lane()) {
            const uint64_t dwo = umma_desc_sw128(smem_u32(sm + TransLayout::w + s * kTrStageBytes) + kTrW1Bytes);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_bf16_ts(tmem_base + 256 + 128 * ob, tmem_base + 128 * hb + 8 * ks, dwo + 2 * ks, idesc, (c | ks) ? 1u : 0u);
            umma_commit(&bars.h_free[hb]);
            umma_commit(&bars.w_empty[s]);
            if (c == kTrChunks - 1) umma_commit(&bars.out_full[ob]);
          }
          __syncwarp();
        }
      }
    }
  } else if (warp >= 12) {
    // ------------------------------------------------------------------ output rows
    // Blocks of 128 bytes a row (32 fp32 or 64 bf16 channels) pass through a warp's staging area, 128-byte swizzle, and leave
    // by TMA: stored, or for fp32 rows whose residual is the output itself added in L2.  Any other residual comes the same way:
    // its block is fetched (`apart`) into the staging area as soon as the block before has left it, and the thread that owns a row adds
    // to it in place.  With loads, additions and stores of the warps' own: fp32 316 us against 273 at N = 768, bf16 278 against 255.
    const int qw = warp - 12;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * qw) << 16) + 256;
    unsigned char* const stg = sm + TransLayout::stg + qw * 4096;
    unsigned char* const row = stg + lane * 128;
    uint64_t* const res_full = &bars.res_full[qw];
    constexpr int kBlocks = sizeof(Tz);                    // blocks of a tile: 2 bf16, 4 fp32
    const bool fetch = add_residual && apart, add = add_residual && !apart;
    auto request = [&](int tile, int q) {
      if (fetch && lane == 0) {
        mbar_expect_tx(res_full, 4096);
        tma_load_3d(smem_u32(stg), &map_res, res_full, (128 / kBlocks) * q, tile * 128 + 32 * qw, 0);
      }
    };
    if (first_tile < n_tiles) request(first_tile, 0);
    int k = 0;
    uint32_t block = 0;
    bool ok = true;
    for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step, ++k) {
      const int ob = k & 1, first = tile * 128 + 32 * qw;
      ok = mbar_wait(&bars.out_full[ob], (k >> 1) & 1, 32u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int q = 0; q < kBlocks; ++q, ++block) {
        uint32_t r[128 / kBlocks];
#pragma unroll
        for (int hh = 0; hh < 4 / kBlocks; ++hh)
          tmem_ld32(lane_addr + 128 * ob + (128 / kBlocks) * q + 32 * hh, *reinterpret_cast<uint32_t(*)[32]>(&r[32 * hh]));
        tmem_wait_ld();
        if (q == kBlocks - 1) {                              // this warp has read its part of the accumulator
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.out_free[ob]);
        }
        if (fetch) {
          ok = mbar_wait(res_full, block & 1, 128u);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        } else {
          if (lane == 0) tma_store_wait_read<0>();           // the block before has left the staging area
          __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4* at = reinterpret_cast<uint4*>(row + ((c ^ (lane & 7)) << 4));
          uint4 old = make_uint4(0u, 0u, 0u, 0u), o;
          if (fetch) old = *at;
          // the second product is of h / 2
          if constexpr (sizeof(Tz) == 4) {
            auto sum = [&](uint32_t x, uint32_t res) { return __float_as_uint(fmaf(2.0f, __uint_as_float(x), __uint_as_float(res))); };
            o = make_uint4(sum(r[4 * c], old.x), sum(r[4 * c + 1], old.y), sum(r[4 * c + 2], old.z), sum(r[4 * c + 3], old.w));
          } else {
            auto sum = [&](int e, uint32_t res) {
              const float2 z = unpack_bf16x2(res);
              return pack_bf16x2(fmaf(2.0f, __uint_as_float(r[e]), z.x), fmaf(2.0f, __uint_as_float(r[e + 1]), z.y));
            };
            o = make_uint4(sum(8 * c, old.x), sum(8 * c + 2, old.y), sum(8 * c + 4, old.z), sum(8 * c + 6, old.w));
          }
          *at = o;
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0 && first < rows) {
          if (add)
            tma_add_3d(&map_out, smem_u32(stg), (128 / kBlocks) * q, first, 0);
          else
            tma_store_3d(&map_out, smem_u32(stg), (128 / kBlocks) * q, first, 0);
          tma_store_commit();
        }
        if (fetch && (q + 1 < kBlocks || tile + tile_step < n_tiles)) {
          if (lane == 0) tma_store_wait_read<0>();
          request(q + 1 < kBlocks ? tile : tile + tile_step, q + 1 < kBlocks ? q + 1 : 0);
        }
      }
    }
    if (lane == 0) tma_store_wait_read<0>();
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ LayerNorm -> swizzled A operand
    const int qw = warp - 8;
    // The normalised rows enter the first product halved: a' = a / 2 is the argument of the gate's tanh, b' = b / 2,
    // and h' = a' b' (1 + tanh a') = silu(a) b / 2 is what the SwiGLU warps write; the output warps double the second
    // product.  Powers of two: nothing changes but two multiplications per hidden element that are no longer needed.
    float* const affine = reinterpret_cast<float*>(sm + TransLayout::affine);     // gamma / 2, then beta / 2
    affine[threadIdx.x - 256] = 0.5f * ln_w[threadIdx.x - 256];
    affine[kC + threadIdx.x - 256] = 0.5f * ln_b[threadIdx.x - 256];
    named_barrier(1, 128);
    // Eight lanes a row and four rows at a time, 16 channels a lane: three exchanges a sum for four rows.  With 32 lanes a row the exchanges were a third of the instructions of
    // these four warps, and they were late: 61 us against 58 at N = 384, 15.2 against 13.6 for one tile, 434 against 399 at N = 1024.
    const int piece = lane & 7, r0 = lane >> 3;
    int k = 0;
    for (int tile = first_tile; tile < n_tiles; tile += tile_step, ++k) {
      const int ab = k & 1;
      const long long row0 = (long long)tile * 128 + 32 * qw + r0;
      bool ok = mbar_wait(&bars.a_free[ab], ((k >> 1) & 1) ^ 1, 16u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      unsigned char* sa = sm + TransLayout::a + ab * kTrABytes;
      // eight rows per batch; the next batch is requested (as stored) before this one is reduced
      Raw16<Tz> raw[2];
      auto request = [&](int rb) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const long long grow = row0 + rb + 4 * j;
          if (grow < rows) {
            raw[j].load(x_in + (size_t)grow * kC, piece);
          } else {
            raw[j].zero();
          }
        }
      };
      request(0);
#pragma unroll 1
      for (int rb = 0; rb < 32; rb += 8) {
        float x[2][16], sum[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) raw[j].get(x[j]);
        if (rb + 8 < 32) request(rb + 8);
        auto reduce = [&] {
#pragma unroll
          for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < 2; ++j) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o);
        };
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float p[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) p[e] = (x[j][e] + x[j][4 + e]) + (x[j][8 + e] + x[j][12 + e]);
          sum[j] = (p[0] + p[1]) + (p[2] + p[3]);
        }
        reduce();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float mean = sum[j] * (1.0f / kC);
          float p[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            x[j][e] -= mean;
            p[e & 3] = fmaf(x[j][e], x[j][e], p[e & 3]);
          }
          sum[j] = (p[0] + p[1]) + (p[2] + p[3]);
        }
        reduce();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float rstd = row0 + rb + 4 * j < rows ? rsqrtf(sum[j] * (1.0f / kC) + eps) : 0.f;
#pragma unroll
          for (int e = 0; e < 16; ++e) x[j][e] *= rstd;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4* g = reinterpret_cast<const float4*>(affine + 64 * i + 8 * piece);
          const float4 g0 = g[0], g1 = g[1], b0 = g[kC / 4], b1 = g[kC / 4 + 1];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int r = 32 * qw + r0 + rb + 4 * j;       // row inside the tile
            const float* v = &x[j][8 * i];
            *reinterpret_cast<uint4*>(sa + i * 16384 + r * 128 + ((piece ^ (r & 7)) << 4)) =
                make_uint4(pack_f16x2(fmaf(v[0], g0.x, b0.x), fmaf(v[1], g0.y, b0.y)), pack_f16x2(fmaf(v[2], g0.z, b0.z), fmaf(v[3], g0.w, b0.w)),
                           pack_f16x2(fmaf(v[4], g1.x, b1.x), fmaf(v[5], g1.y, b1.y)), pack_f16x2(fmaf(v[6], g1.z, b1.z), fmaf(v[7], g1.w, b1.w)));
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.a_full[ab]);
    }
  } else {
    // ------------------------------------------------------------------ SwiGLU in registers
    // Two groups of four warps, each on every other chunk and its H buffer.  A thread owns its row's 64 hidden values of the chunk,
    // so nothing is exchanged between threads.  The 16 values of a step are h, packed into 8 columns over a values read before.
    const int hb = warp >> 2, qw = warp & 3;
    const uint32_t t_h = tmem_base + ((uint32_t)(32 * qw) << 16) + 128 * hb;
    int n = 0;                                        // chunks of this group so far
    bool ok = true;
    for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
      for (int c = hb; c < kTrChunks; c += 2, ++n) {
        ok = mbar_wait_warp(&bars.h_full[hb], n & 1, 64u);
        if (!ok) break;
        tc_fence_after();
        uint32_t a[2][16], b[2][16];
        tmem_ld16(t_h, a[0]);
        tmem_ld16(t_h + 64, b[0]);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          tmem_wait_ld();
          if (p < 3) {
            tmem_ld16(t_h + 16 * (p + 1), a[(p + 1) & 1]);
            tmem_ld16(t_h + 64 + 16 * (p + 1), b[(p + 1) & 1]);
          }
          uint32_t w[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            // silu(a) * b / 2 = a' b' (1 + tanh a') with a' = a / 2, b' = b / 2 as the accumulators hold them:
            // one special-function op, one multiplication and one fused multiply-add per element
            const float a0 = __uint_as_float(a[p & 1][2 * e]), a1 = __uint_as_float(a[p & 1][2 * e + 1]);
            const float h0 = a0 * __uint_as_float(b[p & 1][2 * e]), h1 = a1 * __uint_as_float(b[p & 1][2 * e + 1]);
            w[e] = pack_f16x2(fmaf(h0, tanh_fast(a0), h0), fmaf(h1, tanh_fast(a1), h1));
          }
          tmem_st8(t_h + 8 * p, w);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.p_ready[hb]);
      }
    }
  }

  tc_fence_before();
  cta_teardown_sync();
  if (warp == 16) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

PX_DEFINE_FAMILY_HOOKS(transition)

template <typename Tz>
static int32_t launch_transition(const void* x_in, void* x_out, const float* ln_w, const float* ln_b, const px_bf16* w_a,
                                 const px_bf16* w_b, const px_bf16* w_o, int64_t rows, int32_t add_residual, float eps,
                                 cudaStream_t st) {
  CUtensorMap ma, mb, mo, mx, mr;
  // W_a, W_b: [512 rows][128 k] fp16, box [64 rows][64 k]; W_o: [128 rows][512 k], box [128 rows][64 k]
  if (!make_map_3d(&ma, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w_a, 128, 512, 1, 256, 512 * 256, 64, 64,
                   CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_map_3d(&mb, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w_b, 128, 512, 1, 256, 512 * 256, 64, 64,
                   CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_map_3d(&mo, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w_o, 512, 128, 1, 1024, 128 * 1024, 64, 128,
                   CU_TENSOR_MAP_SWIZZLE_128B))
    return PX_ERR_LAUNCH;
  // output and residual rows: box [32 rows][128 bytes]
  constexpr uint64_t kRow = 128 * sizeof(Tz);
  constexpr CUtensorMapDataType kType = sizeof(Tz) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  for (int i = 0; i < 2; ++i)
    if (!make_map_3d(i ? &mr : &mx, kType, i ? x_in : x_out, 128, (uint64_t)rows, 1, kRow, (uint64_t)rows * kRow, 128 / sizeof(Tz), 32,
                     CU_TENSOR_MAP_SWIZZLE_128B))
      return PX_ERR_LAUNCH;
  const size_t smem = TransLayout::total + 1024;
  static SmemLimit limit;
  if (!limit.set(transition_tc_kernel<Tz>, smem)) return PX_ERR_LAUNCH;
  const int64_t n_tiles = (rows + 127) / 128;
  const int grid = even_grid(n_tiles, sm_count());
  return launch_pdl(transition_tc_kernel<Tz>, dim3(grid), kTrThreads, smem, st, ma, mb, mo, mx, mr, (const Tz*)x_in, ln_w, ln_b,
                    (long long)rows, (int)n_tiles, (int)add_residual, (int)(sizeof(Tz) == 2 || x_in != x_out), eps)
             ? PX_OK
             : PX_ERR_LAUNCH;
}

}  // namespace px

using namespace px;

extern "C" int32_t px_transition(const void* x_in, void* x_out, int32_t dtype, const float* ln_w, const float* ln_b,
                                 const px_bf16* w_a, const px_bf16* w_b, const px_bf16* w_o, int64_t rows,
                                 int32_t add_residual, float eps, void* stream) {
  if (!x_in || !x_out || !ln_w || !ln_b || !w_a || !w_b || !w_o || rows < 0) return PX_ERR_BAD_ARG;
  if (((uintptr_t)x_in | (uintptr_t)x_out | (uintptr_t)w_a | (uintptr_t)w_b | (uintptr_t)w_o) & 15) return PX_ERR_BAD_ARG;
  if (rows == 0) return PX_OK;
  if (rows > 0x7fffff00) return PX_ERR_UNSUPPORTED;       // rows are counted in 32 bits (a terabyte of fp32)
  if (dtype == PX_F32)
    return launch_transition<float>(x_in, x_out, ln_w, ln_b, w_a, w_b, w_o, rows, add_residual, eps, (cudaStream_t)stream);
  if (dtype == PX_BF16)
    return launch_transition<bf16>(x_in, x_out, ln_w, ln_b, w_a, w_b, w_o, rows, add_residual, eps, (cudaStream_t)stream);
  return PX_ERR_UNSUPPORTED;
}
