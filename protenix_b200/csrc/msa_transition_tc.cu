// SwiGLU transition of the MSA embedding, m += W_out( silu(W_a LN(m)) * (W_b LN(m)) ) for rows of 64 channels, hidden width 256,
// in fp32-grade arithmetic on the 5th-generation tensor cores: both products take operands split into three bf16 values
// (px_split.cuh), six partial products each.  98 kFLOP a row: the library's fp32 GEMMs with the passes around them took 1.4 ms at
// 393216 rows; 6 x that on the tensor core is 0.16 ms at its measured rate, and the rows (256 bytes in and out) 31 us.
//
// Persistent kernel, one CTA per SM, 128 rows per tile, three tiles in flight as in the pair transition:
//   warps 0..15   SwiGLU of a 64-wide hidden chunk (lane quarter x quarter of the columns): h = silu(a) b, split, written back over
//                 the chunk's accumulator as the A operand of the second product (three planes of 32 columns)
//   warps 16..19  LayerNorm: 16 lanes a row, split rows written as three swizzled planes (two buffers)
//   warps 20..23  output: accumulators + residual, staged so that a warp's accesses cover 64 contiguous bytes of 8 rows
//   warps 24, 27  TMA producers of the weight chunks ([W_a; W_b] two stages, W_out one; they come from L2 for every tile)
//   warps 25, 26  MMA issuers of the first product (M=128, N=128) and of the second (M=128, N=64)
// The tensor core truncates on accumulation: the first product adds its corrections before its leading terms, the second has
// an accumulator for each.  Tensor memory: H (2 x 128) | out, corrections (2 x 128).  Every wait is bounded.
#include "px_split.cuh"

namespace px {

constexpr int kMtC = 64, kMtHid = 256, kMtChunks = kMtHid / 64;
constexpr int kMtABytes = 3 * 128 * 128;       // [3 planes][128 rows][64 k]
constexpr int kMtW1Bytes = 3 * 128 * 128;      // [3][a 64 | b 64 rows][64 k]
constexpr int kMtW2Bytes = 3 * 64 * 128;       // [3][64 outputs][64 hidden]
constexpr int kMtGate = 16;                    // SwiGLU warps
constexpr int kMtWarps = kMtGate + 12, kMtThreads = 32 * kMtWarps;

struct MtBars {
  uint64_t a_full[2], a_free[2], w1_full[2], w1_empty[2], w2_full, w2_empty, h_full[2], h_free[2], p_ready[2], out_full[2], out_free[2];
  uint32_t tmem_base;
};
struct MtLayout {
  static constexpr int a = 0;
  static constexpr int w1 = a + 2 * kMtABytes;
  static constexpr int w2 = w1 + 2 * kMtW1Bytes;
  static constexpr int stg = w2 + kMtW2Bytes;        // 4 warps x [32 rows][16 fp32]
  static constexpr int bars = stg + 4 * 2048;
  static constexpr int total = bars + (int)sizeof(MtBars);
};
static_assert(MtLayout::total + 1024 <= 232448, "shared memory budget");

// The partial products (i, j): corrections, then the leading one.
__device__ constexpr int kMtI[6] = {0, 2, 1, 0, 1, 0}, kMtJ[6] = {2, 0, 1, 1, 0, 0};

__global__ void __launch_bounds__(kMtThreads, 1)
msa_transition_tc_kernel(const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_w2, float* m,
                         const float* __restrict__ ln_w, const float* __restrict__ ln_b, long long rows, int n_tiles, float eps) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  MtBars& bars = *reinterpret_cast<MtBars*>(sm + MtLayout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int first_tile = blockIdx.x, tile_step = gridDim.x;

  const bool skip = cta_begin();
  if (threadIdx.x == 32) prefetch_maps(map_w1, map_w2);
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars.a_full[b], 4);
      mbar_init(&bars.a_free[b], 1);
      mbar_init(&bars.w1_full[b], 1);
      mbar_init(&bars.w1_empty[b], 1);
      mbar_init(&bars.h_full[b], 1);
      mbar_init(&bars.h_free[b], 1);
      mbar_init(&bars.p_ready[b], kMtGate);
      mbar_init(&bars.out_full[b], 1);
      mbar_init(&bars.out_free[b], 4);
    }
    mbar_init(&bars.w2_full, 1);
    mbar_init(&bars.w2_empty, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kMtGate + 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (!cta_ready(skip, warp == kMtGate + 8, bars.tmem_base, 512u)) return;
  const uint32_t tmem_base = bars.tmem_base;

  if (warp >= kMtGate + 8) {
    if (!elect_lane()) {
      // nothing: one elected lane of each control warp works
    } else if (warp == kMtGate + 8) {
      int j = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
        for (int c = 0; c < kMtChunks && ok; ++c, ++j) {
          ok = mbar_wait(&bars.w1_empty[j & 1], ((j >> 1) & 1) ^ 1, 1u);
          if (!ok) break;
          mbar_expect_tx(&bars.w1_full[j & 1], kMtW1Bytes);
          tma_load_3d(smem_u32(sm + MtLayout::w1 + (j & 1) * kMtW1Bytes), &map_w1, &bars.w1_full[j & 1], 0, 128 * c, 0);
        }
      }
    } else if (warp == kMtGate + 11) {
      int j = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
        for (int c = 0; c < kMtChunks && ok; ++c, ++j) {
          ok = mbar_wait(&bars.w2_empty, (j & 1) ^ 1, 1u);
          if (!ok) break;
          mbar_expect_tx(&bars.w2_full, kMtW2Bytes);
          tma_load_3d(smem_u32(sm + MtLayout::w2), &map_w2, &bars.w2_full, 64 * c, 0, 0);
        }
      }
    } else if (warp == kMtGate + 9) {
      // ---------------------------------------------------------------- first product: H = A [W_a; W_b]_c^T
      constexpr uint32_t idesc = umma_idesc_bf16(128, 128);
      int j = 0, k = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step, ++k) {
        const int ab = k & 1;
        ok = mbar_wait(&bars.a_full[ab], (k >> 1) & 1, 2u);
        const uint32_t a_addr = smem_u32(sm + MtLayout::a + ab * kMtABytes);
        for (int c = 0; c < kMtChunks && ok; ++c, ++j) {
          const int b = j & 1;
          ok = mbar_wait(&bars.w1_full[b], (j >> 1) & 1, 4u) && mbar_wait(&bars.h_free[b], ((j >> 1) & 1) ^ 1, 4u);
          if (!ok) break;
          tc_fence_after();
          const uint32_t w_addr = smem_u32(sm + MtLayout::w1 + b * kMtW1Bytes);
#pragma unroll
          for (int t = 0; t < 6; ++t) {
            const uint64_t da = umma_desc_sw128(a_addr + kMtI[t] * (128 * 128)), dw = umma_desc_sw128(w_addr + kMtJ[t] * (128 * 128));
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) umma_bf16(tmem_base + 128 * b, da + 2 * ks, dw + 2 * ks, idesc, (t | ks) ? 1u : 0u);
          }
          umma_commit(&bars.h_full[b]);
          umma_commit(&bars.w1_empty[b]);
        }
        if (ok) umma_commit(&bars.a_free[ab]);
      }
    } else {
      // ---------------------------------------------------------------- second product: OUT += h W_out,c^T
      constexpr uint32_t idesc = umma_idesc_bf16(128, 64);
      int j = 0, k = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step, ++k) {
        const int ob = k & 1;
        ok = mbar_wait(&bars.out_free[ob], ((k >> 1) & 1) ^ 1, 8u);
        for (int c = 0; c < kMtChunks && ok; ++c, ++j) {
          const int b = j & 1;
          ok = mbar_wait(&bars.w2_full, j & 1, 4u) && mbar_wait(&bars.p_ready[b], (j >> 1) & 1, 8u);
          if (!ok) break;
          tc_fence_after();
          const uint32_t w_addr = smem_u32(sm + MtLayout::w2), out = tmem_base + 256 + 128 * ob;
#pragma unroll
          for (int t = 0; t < 6; ++t) {
            const uint64_t dw = umma_desc_sw128(w_addr + kMtJ[t] * (64 * 128));
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_bf16_ts(out + (t == 5 ? 0 : 64), tmem_base + 128 * b + 32 * kMtI[t] + 8 * ks, dw + 2 * ks, idesc,
                           (c || ks || (t != 5 && t)) ? 1u : 0u);
          }
          umma_commit(&bars.h_free[b]);
          umma_commit(&bars.w2_empty);
        }
        if (ok) umma_commit(&bars.out_full[ob]);
      }
    }
  } else if (warp >= kMtGate + 4) {
    // ------------------------------------------------------------------ output rows: residual + store
    const int qw = warp - kMtGate - 4;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * qw) << 16);
    unsigned char* stg = sm + MtLayout::stg + qw * 2048;     // rows of 64 bytes, 16-byte pieces swizzled by row pair
    const int rsub = lane >> 2, piece = lane & 3;
    int k = 0;
    for (int tile = first_tile; tile < n_tiles; tile += tile_step, ++k) {
      const int ob = k & 1;
      const long long row0 = (long long)tile * 128 + 32 * qw;
      bool ok = mbar_wait(&bars.out_full[ob], (k >> 1) & 1, 32u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {                          // 16 channels at a time
        uint32_t r[16], e[16];
        float4 res[4];
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const long long row = row0 + 8 * it + rsub;
          res[it] = row < rows ? *reinterpret_cast<const float4*>(m + (size_t)row * kMtC + 16 * q + 4 * piece) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        tmem_ld16(lane_addr + 256 + 128 * ob + 16 * q, r);
        tmem_ld16(lane_addr + 256 + 128 * ob + 64 + 16 * q, e);
        tmem_wait_ld();
        if (q == 3) {                                        // this warp has read its part of the accumulators
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.out_free[ob]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<float4*>(stg + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) =
              make_float4(__uint_as_float(r[4 * c]) + __uint_as_float(e[4 * c]), __uint_as_float(r[4 * c + 1]) + __uint_as_float(e[4 * c + 1]),
                          __uint_as_float(r[4 * c + 2]) + __uint_as_float(e[4 * c + 2]),
                          __uint_as_float(r[4 * c + 3]) + __uint_as_float(e[4 * c + 3]));
        __syncwarp();
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const int rl = 8 * it + rsub;
          const long long row = row0 + rl;
          float4 v = *reinterpret_cast<const float4*>(stg + rl * 64 + ((piece ^ ((rl >> 1) & 3)) << 4));
          if (row < rows) {
            v.x += res[it].x, v.y += res[it].y, v.z += res[it].z, v.w += res[it].w;
            *reinterpret_cast<float4*>(m + (size_t)row * kMtC + 16 * q + 4 * piece) = v;
          }
        }
        __syncwarp();
      }
    }
  } else if (warp >= kMtGate) {
    // ------------------------------------------------------------------ LayerNorm -> split, swizzled A operand
    const int qw = warp - kMtGate, li = lane & 15, sub = lane >> 4;
    const float4 g4 = ln_w ? *reinterpret_cast<const float4*>(ln_w + 4 * li) : make_float4(1.f, 1.f, 1.f, 1.f);
    const float4 b4 = ln_b ? *reinterpret_cast<const float4*>(ln_b + 4 * li) : make_float4(0.f, 0.f, 0.f, 0.f);
    int k = 0;
    for (int tile = first_tile; tile < n_tiles; tile += tile_step, ++k) {
      const int ab = k & 1;
      const long long row0 = (long long)tile * 128 + 32 * qw;
      float4 v[8];                                           // half of the warp's 32 rows, two rows a load
      auto request = [&](int j1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const long long row = row0 + 2 * (j1 + j) + sub;
          v[j] = row < rows ? *reinterpret_cast<const float4*>(m + (size_t)row * kMtC + 4 * li) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      };
      request(0);
      bool ok = mbar_wait(&bars.a_free[ab], ((k >> 1) & 1) ^ 1, 16u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      unsigned char* sa = sm + MtLayout::a + ab * kMtABytes;
#pragma unroll 1
      for (int j1 = 0; j1 < 16; j1 += 8) {
        if (j1) request(j1);
#pragma unroll
      for (int j0 = 0; j0 < 8; j0 += 4) {
        float s[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = (v[j0 + j].x + v[j0 + j].y) + (v[j0 + j].z + v[j0 + j].w);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
          for (int j = 0; j < 4; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float4& x = v[j0 + j];
          const float mean = s[j] * (1.0f / kMtC);
          x.x -= mean, x.y -= mean, x.z -= mean, x.w -= mean;
          s[j] = fmaf(x.x, x.x, x.y * x.y) + fmaf(x.z, x.z, x.w * x.w);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
          for (int j = 0; j < 4; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 x = v[j0 + j];
          const float rstd = rsqrtf(s[j] * (1.0f / kMtC) + eps);
          const int r = 32 * qw + 2 * (j1 + j0 + j) + sub;
          uint32_t lo[3], hi[3];
          split3x2(fmaf(x.x * rstd, g4.x, b4.x), fmaf(x.y * rstd, g4.y, b4.y), lo);
          split3x2(fmaf(x.z * rstd, g4.z, b4.z), fmaf(x.w * rstd, g4.w, b4.w), hi);
#pragma unroll
          for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint2*>(sa + p * (128 * 128) + r * 128 + (((li >> 1) ^ (r & 7)) << 4) + (li & 1) * 8) = make_uint2(lo[p], hi[p]);
        }
      }
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.a_full[ab]);
    }
  } else {
    // ------------------------------------------------------------------ SwiGLU in registers
    const int part = warp >> 2, qw = warp & 3;               // 16 of the chunk's 64 columns, lane quarter
    const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * qw) << 16);
    int j = 0;
    bool ok = true;
    for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
      for (int c = 0; c < kMtChunks && ok; ++c, ++j) {
        const int hb = j & 1;
        const uint32_t t_h = lane_addr + 128 * hb;
        ok = mbar_wait(&bars.h_full[hb], (j >> 1) & 1, 64u);
        ok = named_barrier_all(2, 32 * kMtGate, ok);         // all of these warps go on, or none
        if (!ok) break;
        tc_fence_after();
        uint32_t w[3][8], a[16], b[16];
        tmem_ld16(t_h + 16 * part, a);
        tmem_ld16(t_h + 64 + 16 * part, b);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float a0 = __uint_as_float(a[2 * e]), a1 = __uint_as_float(a[2 * e + 1]);
          const float h0 = a0 / (1.0f + expf(-a0)) * __uint_as_float(b[2 * e]);
          const float h1 = a1 / (1.0f + expf(-a1)) * __uint_as_float(b[2 * e + 1]);
          uint32_t p[3];
          split3x2(h0, h1, p);
          w[0][e] = p[0], w[1][e] = p[1], w[2][e] = p[2];
        }
        named_barrier(2, 32 * kMtGate);                      // everybody has read H: h goes over its first 96 columns
#pragma unroll
        for (int p = 0; p < 3; ++p) tmem_st8(t_h + 32 * p + 8 * part, w[p]);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.p_ready[hb]);
      }
    }
  }

  tc_fence_before();
  cta_teardown_sync();
  if (warp == kMtGate + 8) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

PX_DEFINE_FAMILY_HOOKS(msa_transition)

constexpr int64_t kMtW1Elems = 3ll * 2 * kMtHid * kMtC, kMtW2Elems = 3ll * kMtC * kMtHid;

}  // namespace px

using namespace px;

extern "C" int64_t px_msa_transition_weights_bytes(void) { return (kMtW1Elems + kMtW2Elems) * 2; }

extern "C" int32_t px_msa_transition_prepare(const float* w_a, const float* w_b, const float* w_out, void* prepared, void* stream) {
  if (!w_a || !w_b || !w_out || !prepared || ((uintptr_t)prepared & 15)) return PX_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  bf16* p = (bf16*)prepared;
  split_weight_kernel<<<kMtHid, 64, 0, st>>>(w_a, p, kMtHid, kMtC, 2 * kMtHid, 64, 128, 0);
  split_weight_kernel<<<kMtHid, 64, 0, st>>>(w_b, p, kMtHid, kMtC, 2 * kMtHid, 64, 128, 64);
  split_weight_kernel<<<kMtC, 128, 0, st>>>(w_out, p + kMtW1Elems, kMtC, kMtHid, kMtC, kMtC, kMtC, 0);
  return cudaGetLastError() == cudaSuccess ? PX_OK : PX_ERR_LAUNCH;
}

extern "C" int32_t px_msa_transition(float* m, const void* prepared, const float* ln_w, const float* ln_b, int64_t rows, float eps,
                                     void* stream) {
  if (!m || !prepared || rows < 0 || (((uintptr_t)m | (uintptr_t)prepared | (uintptr_t)ln_w | (uintptr_t)ln_b) & 15)) return PX_ERR_BAD_ARG;
  if (rows == 0) return PX_OK;
  const int64_t n_tiles = (rows + 127) / 128;
  if (n_tiles > 0x7fffffff) return PX_ERR_UNSUPPORTED;
  CUtensorMap m1, m2;
  const bf16* p = (const bf16*)prepared;
  if (!make_plane_map(&m1, p, 2 * kMtHid, kMtC, 128) || !make_plane_map(&m2, p + kMtW1Elems, kMtC, kMtHid, 64)) return PX_ERR_LAUNCH;
  const size_t smem = MtLayout::total + 1024;
  static SmemLimit limit;
  const int grid = even_grid(n_tiles, sm_count());
  return limit.set(msa_transition_tc_kernel, smem) &&
                 launch_pdl(msa_transition_tc_kernel, dim3(grid), kMtThreads, smem, (cudaStream_t)stream, m1, m2, m, ln_w, ln_b,
                            (long long)rows, (int)n_tiles, eps)
             ? PX_OK
             : PX_ERR_LAUNCH;
}
