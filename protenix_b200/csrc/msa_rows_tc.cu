// Row-wise steps of the MSA stack on an fp32 MSA embedding m [S][N][64] (c_m = 64), each one pass over m:
//   opm_prep    a_t, b_t [(i, c)][s] fp16 = mask * LN(m) W_1^T, LN(m) W_2^T (32 columns each): the operands of px_opm_outer
//   values      v [8 heads][3][j][8 s + c] = LN(m) W_mv^T as three bf16 planes: the right-hand side of the pair-weighted average
//   gate_out    m += W_out( sigmoid(LN(m) W_mg^T) * wv ), wv [8][i][8 s + c] as the average leaves it (msa_average_tc.cu)
// Each is LayerNorm and one or two 64 x 64 products per row in fp32-grade arithmetic on the 5th-generation tensor cores (px_split.cuh).
// As fp32 FMAs from shared memory they were bound by its bandwidth (88 % of its peak, DRAM at 21 %).
// S = 1024, N = 384 (100 MB of m): opm_prep 121 -> 58 us, values 106 -> 66 (250 MB, 3.8 TB/s), gate_out 212 -> 101.
//
// Persistent, one CTA per SM, a tile = one token i and 128 sequences: with the token fixed, what leaves transposed are runs of
// 32 sequences per warp, and a warp's rows of the average 1 KB of one head.
//   warps 0..7    a thread owns one sequence and 32 of the 64 columns: result from tensor memory to its place; for gate_out the gated
//                 average, split, as the A operand of the second product (tensor memory)
//   warps 8..11   gate_out: + residual, staged so that a warp's accesses cover 64 contiguous bytes of 8 rows
//   warps 12..19  LayerNorm: 16 lanes a row, the next tile's rows requested ahead; split rows as swizzled planes (two buffers)
//   warps 20, 21  MMA issuers of the two products (24 MMAs each; the weights stay resident)
// The tensor core truncates on accumulation: leading products and corrections have an accumulator each.  Tensor memory: first
// product 2 x 128 | second product 128 | gated rows 96.  Every wait is bounded.
#include "px_split.cuh"

namespace px {

enum { kMrPrep = 0, kMrValues = 1, kMrGate = 2 };
constexpr int kMrC = 64;
constexpr int kMrThreads = 32 * 22;
constexpr int kMrABytes = 3 * 128 * 128;       // [3 planes][128 rows][64 k]
constexpr int kMrWBytes = 3 * kMrC * 128;      // [3][64 outputs][64 k]
constexpr uint32_t kMrColD2 = 256, kMrColA2 = 384;

struct MrBars {
  uint64_t a_full[2], a_free[2], d_full[2], d_free[2], p_ready, p_free, o_full, o_free, w_full;
  uint32_t tmem_base;
};
struct MrLayout {
  static constexpr int w = 2 * kMrABytes;
  static constexpr int w2 = w + kMrWBytes;
  static constexpr int stg = w2 + kMrWBytes;         // 4 warps x [32 rows][16 fp32]
  static constexpr int bars = stg + 4 * 2048;
  static constexpr int total = bars + (int)sizeof(MrBars);
};
static_assert(MrLayout::total + 1024 <= 232448, "shared memory budget");

struct MrArgs {
  const float *m, *gamma, *beta;
  const float* mask;                 // prep: [S][N] or null
  __half *a_t, *b_t;
  bf16* v;                           // values
  const float* wv;                   // gate_out
  float* m_out;
  int n, s_rows, ld, n_tiles;
  float eps;
};

// One issuing thread's share: the six partial products of A (its planes at a(i) for plane i) and the weight planes at `w`, N = 64.
template <typename Issue>
__device__ __forceinline__ void mr_products(uint32_t w, uint32_t d, Issue issue) {
  constexpr uint32_t kI = 0x010210u, kJ = 0x001012u;     // (0,2) (1,1) (2,0) (0,1) (1,0) (0,0): nibble t from the right
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const int i = (kI >> (4 * t)) & 15, j = (kJ >> (4 * t)) & 15;
    const uint64_t dw = umma_desc_sw128(w + j * (kMrC * 128));
    const bool lead = i + j == 0;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) issue(d + (lead ? 0 : 64), i, ks, dw + 2 * ks, (uint32_t)(ks > 0 || (!lead && t > 0)));
  }
}

template <int kMode>
__global__ void __launch_bounds__(kMrThreads, 1)
msa_rows_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2, const MrArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  MrBars& bars = *reinterpret_cast<MrBars*>(sm + MrLayout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int first_tile = blockIdx.x, tile_step = gridDim.x;

  const bool skip = cta_begin();
  if (threadIdx.x == 32) {
    prefetch_maps(map_w);
    if (kMode == kMrGate) prefetch_maps(map_w2);
  }
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars.a_full[b], 8);
      mbar_init(&bars.a_free[b], 1);
      mbar_init(&bars.d_full[b], 1);
      mbar_init(&bars.d_free[b], 8);
    }
    mbar_init(&bars.p_ready, 8);
    mbar_init(&bars.p_free, 1);
    mbar_init(&bars.o_full, 1);
    mbar_init(&bars.o_free, 4);
    mbar_init(&bars.w_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 20) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (!cta_ready(skip, warp == 20, bars.tmem_base, 512u)) return;
  const uint32_t tmem_base = bars.tmem_base;

  if (warp >= 20) {
    constexpr uint32_t idesc = umma_idesc_bf16(128, kMrC);
    if (!elect_lane() || (warp == 21 && kMode != kMrGate)) {
      // nothing: one elected lane of each control warp works
    } else if (warp == 20) {
      mbar_expect_tx(&bars.w_full, kMode == kMrGate ? 2 * kMrWBytes : kMrWBytes);
      tma_load_3d(smem_u32(sm + MrLayout::w), &map_w, &bars.w_full, 0, 0, 0);
      if (kMode == kMrGate) tma_load_3d(smem_u32(sm + MrLayout::w2), &map_w2, &bars.w_full, 0, 0, 0);
      bool ok = mbar_wait(&bars.w_full, 0, 4u);
      int k = 0;
      for (int tile = first_tile; tile < g.n_tiles && ok; tile += tile_step, ++k) {
        const int b = k & 1;
        ok = mbar_wait(&bars.a_full[b], (k >> 1) & 1, 2u) && mbar_wait(&bars.d_free[b], ((k >> 1) & 1) ^ 1, 4u);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a = smem_u32(sm + b * kMrABytes);
        mr_products(smem_u32(sm + MrLayout::w), tmem_base + 128 * b, [&](uint32_t d, int i, int ks, uint64_t dw, uint32_t acc) {
          umma_bf16(d, umma_desc_sw128(a + i * (128 * 128)) + 2 * ks, dw, idesc, acc);
        });
        umma_commit(&bars.d_full[b]);
        umma_commit(&bars.a_free[b]);
      }
    } else {
      bool ok = mbar_wait(&bars.w_full, 0, 4u);
      int k = 0;
      for (int tile = first_tile; tile < g.n_tiles && ok; tile += tile_step, ++k) {
        ok = mbar_wait(&bars.p_ready, k & 1, 8u) && mbar_wait(&bars.o_free, (k & 1) ^ 1, 8u);
        if (!ok) break;
        tc_fence_after();
        mr_products(smem_u32(sm + MrLayout::w2), tmem_base + kMrColD2, [&](uint32_t d, int i, int ks, uint64_t dw, uint32_t acc) {
          umma_bf16_ts(d, tmem_base + kMrColA2 + 32 * i + 8 * ks, dw, idesc, acc);
        });
        umma_commit(&bars.o_full);
        umma_commit(&bars.p_free);
      }
    }
  } else if (warp >= 12) {
    // ------------------------------------------------------------------ LayerNorm -> split, swizzled A operand
    const int lw = warp - 12, li = lane & 15, sub = lane >> 4;
    const float4 g4 = g.gamma ? *reinterpret_cast<const float4*>(g.gamma + 4 * li) : make_float4(1.f, 1.f, 1.f, 1.f);
    const float4 b4 = g.beta ? *reinterpret_cast<const float4*>(g.beta + 4 * li) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v[8];                                             // the warp's 16 rows, two at a time
    auto request = [&](int tile) {
      const int i = tile % g.n, s0 = (tile / g.n) * 128 + 16 * lw + sub;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int s = s0 + 2 * j;
        v[j] = s < g.s_rows ? *reinterpret_cast<const float4*>(g.m + ((size_t)s * g.n + i) * kMrC + 4 * li) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    if (first_tile < g.n_tiles) request(first_tile);
    int k = 0;
    for (int tile = first_tile; tile < g.n_tiles; tile += tile_step, ++k) {
      const int b = k & 1;
      float s[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] = (v[j].x + v[j].y) + (v[j].z + v[j].w);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float mean = s[j] * (1.0f / kMrC);
        v[j].x -= mean, v[j].y -= mean, v[j].z -= mean, v[j].w -= mean;
        s[j] = fmaf(v[j].x, v[j].x, v[j].y * v[j].y) + fmaf(v[j].z, v[j].z, v[j].w * v[j].w);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
      bool ok = mbar_wait(&bars.a_free[b], ((k >> 1) & 1) ^ 1, 16u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      unsigned char* sa = sm + b * kMrABytes;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float rstd = rsqrtf(s[j] * (1.0f / kMrC) + g.eps);
        const int r = 16 * lw + 2 * j + sub;
        uint32_t lo[3], hi[3];
        split3x2(fmaf(v[j].x * rstd, g4.x, b4.x), fmaf(v[j].y * rstd, g4.y, b4.y), lo);
        split3x2(fmaf(v[j].z * rstd, g4.z, b4.z), fmaf(v[j].w * rstd, g4.w, b4.w), hi);
#pragma unroll
        for (int p = 0; p < 3; ++p)
          *reinterpret_cast<uint2*>(sa + p * (128 * 128) + r * 128 + (((li >> 1) ^ (r & 7)) << 4) + (li & 1) * 8) = make_uint2(lo[p], hi[p]);
      }
      if (tile + tile_step < g.n_tiles) request(tile + tile_step);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.a_full[b]);
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ gate_out: residual + store
    if (kMode == kMrGate) {
      const int qw = warp - 8, rsub = lane >> 2, piece = lane & 3;
      const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * qw) << 16) + kMrColD2;
      unsigned char* stg = sm + MrLayout::stg + qw * 2048;   // rows of 64 bytes, 16-byte pieces swizzled by row pair
      int k = 0;
      for (int tile = first_tile; tile < g.n_tiles; tile += tile_step, ++k) {
        const int i = tile % g.n, s0 = (tile / g.n) * 128 + 32 * qw;
        bool ok = mbar_wait(&bars.o_full, k & 1, 32u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {                        // 16 channels at a time
          uint32_t r[16], e[16];
          float4 res[4];
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int s = s0 + 8 * it + rsub;
            res[it] = s < g.s_rows ? *reinterpret_cast<const float4*>(g.m + ((size_t)s * g.n + i) * kMrC + 16 * q + 4 * piece)
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
          }
          tmem_ld16(lane_addr + 16 * q, r);
          tmem_ld16(lane_addr + 64 + 16 * q, e);
          tmem_wait_ld();
          if (q == 3) {                                      // this warp has read its part of the accumulators
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.o_free);
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
            const int rl = 8 * it + rsub, s = s0 + rl;
            float4 o = *reinterpret_cast<const float4*>(stg + rl * 64 + ((piece ^ ((rl >> 1) & 3)) << 4));
            if (s < g.s_rows) {
              o.x += res[it].x, o.y += res[it].y, o.z += res[it].z, o.w += res[it].w;
              *reinterpret_cast<float4*>(g.m_out + ((size_t)s * g.n + i) * kMrC + 16 * q + 4 * piece) = o;
            }
          }
          __syncwarp();
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ first product's result
    const int half = warp >> 2, qw = warp & 3;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * qw) << 16);
    int k = 0;
    for (int tile = first_tile; tile < g.n_tiles; tile += tile_step, ++k) {
      const int b = k & 1, i = tile % g.n, s = (tile / g.n) * 128 + 32 * qw + lane;
      const bool in = s < g.s_rows;
      float4 wv[8];                                          // gate_out: the average's 4 heads x 8 channels of this half
      if (kMode == kMrGate) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          wv[e] = in ? __ldcs(reinterpret_cast<const float4*>(g.wv + (((size_t)(4 * half + (e >> 1)) * g.n + i) * g.s_rows + s) * 8 + 4 * (e & 1)))
                     : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      const float mk = kMode == kMrPrep ? (!in ? 0.f : g.mask ? __ldg(g.mask + (size_t)s * g.n + i) : 1.f) : 1.f;
      bool ok = mbar_wait(&bars.d_full[b], (k >> 1) & 1, 64u);
      if (kMode == kMrGate) ok = ok && mbar_wait(&bars.p_free, (k & 1) ^ 1, 64u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_d = lane_addr + 128 * b + 32 * half;
#pragma unroll
      for (int q = 0; q < 2; ++q) {                          // 16 columns at a time
        uint32_t x[16], e[16];
        tmem_ld16(t_d + 16 * q, x);
        tmem_ld16(t_d + 64 + 16 * q, e);
        tmem_wait_ld();
        float v[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] = __uint_as_float(x[c]) + __uint_as_float(e[c]);
        if (q == 1) {                                        // this warp has read its part of the accumulators
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.d_free[b]);
        }
        if (kMode == kMrPrep) {
          // a warp's 32 sequences of one column are 64 bytes; ld: S rounded up to 8, the padding zero
          if (s < g.ld) {
            __half* dst = (half ? g.b_t : g.a_t) + ((size_t)i * 32 + 16 * q) * g.ld + s;
#pragma unroll
            for (int c = 0; c < 16; ++c) dst[(size_t)c * g.ld] = __float2half_rn(in ? v[c] * mk : 0.f);
          }
        } else {
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {                   // eight columns are a head
            if (kMode == kMrGate) {
              const float4 lo = wv[4 * q + 2 * hh], hi = wv[4 * q + 2 * hh + 1];
              const float w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
              for (int c = 0; c < 8; ++c) v[8 * hh + c] = w[c] / (1.0f + expf(-v[8 * hh + c]));
            }
            uint32_t p[4][3];
#pragma unroll
            for (int c = 0; c < 4; ++c) split3x2(v[8 * hh + 2 * c], v[8 * hh + 2 * c + 1], p[c]);
            if (kMode == kMrValues) {
              const int h = 4 * half + 2 * q + hh;
              if (in) {
#pragma unroll
                for (int pl = 0; pl < 3; ++pl)
                  *reinterpret_cast<uint4*>(g.v + (((size_t)(h * 3 + pl) * g.n + i) * g.s_rows + s) * 8) =
                      make_uint4(p[0][pl], p[1][pl], p[2][pl], p[3][pl]);
              }
            } else {
              // columns 32 half + 16 q + 8 hh .. of the gated average: two to a tensor-memory column
#pragma unroll
              for (int pl = 0; pl < 3; ++pl) {
                const uint32_t r[4] = {p[0][pl], p[1][pl], p[2][pl], p[3][pl]};
                tmem_st4(lane_addr + kMrColA2 + 32 * pl + 16 * half + 8 * q + 4 * hh, r);
              }
            }
          }
        }
      }
      if (kMode == kMrGate) {
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.p_ready);
      }
    }
  }

  tc_fence_before();
  cta_teardown_sync();
  if (warp == 20) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

PX_DEFINE_FAMILY_HOOKS(msa_rows)

template <int kMode>
static int32_t launch_msa_rows(const void* w, const void* w2, MrArgs g, int64_t s_rows, int64_t n, cudaStream_t st) {
  if (!g.m || !w || (((uintptr_t)g.m | (uintptr_t)w | (uintptr_t)w2 | (uintptr_t)g.gamma | (uintptr_t)g.beta) & 15) || s_rows <= 0 ||
      n <= 0 || s_rows > (1 << 20) || n > 32768)
    return PX_ERR_BAD_ARG;
  const int64_t n_tiles = (s_rows + 127) / 128 * n;
  CUtensorMap mw, mw2;
  if (!make_plane_map(&mw, (const bf16*)w, kMrC, kMrC, kMrC) || !make_plane_map(&mw2, (const bf16*)(w2 ? w2 : w), kMrC, kMrC, kMrC))
    return PX_ERR_LAUNCH;
  g.n = (int)n, g.s_rows = (int)s_rows, g.n_tiles = (int)n_tiles;      // at most 2^13 * 2^15 tiles
  const size_t smem = MrLayout::total + 1024;
  static SmemLimit limit;
  const int grid = even_grid(n_tiles, sm_count());
  return limit.set(msa_rows_tc_kernel<kMode>, smem) &&
                 launch_pdl(msa_rows_tc_kernel<kMode>, dim3((unsigned)grid), kMrThreads, smem, st, mw, mw2, g)
             ? PX_OK
             : PX_ERR_LAUNCH;
}

}  // namespace px

using namespace px;

extern "C" int64_t px_msa_rows_weights_bytes(void) { return 3ll * kMrC * kMrC * 2; }

extern "C" int32_t px_msa_rows_prepare(const float* w_a, const float* w_b, void* prepared, void* stream) {
  if (!w_a || !prepared || ((uintptr_t)prepared & 15)) return PX_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int rows = w_b ? kMrC / 2 : kMrC;
  split_weight_kernel<<<rows, 64, 0, st>>>(w_a, (bf16*)prepared, rows, kMrC, kMrC, rows, rows, 0);
  if (w_b) split_weight_kernel<<<rows, 64, 0, st>>>(w_b, (bf16*)prepared, rows, kMrC, kMrC, rows, rows, rows);
  return cudaGetLastError() == cudaSuccess ? PX_OK : PX_ERR_LAUNCH;
}

extern "C" int32_t px_msa_opm_prep(const float* m, const float* mask, const float* ln_w, const float* ln_b, const void* prepared,
                                   px_f16* a_t, px_f16* b_t, int64_t s_rows, int64_t n, int64_t ld, float eps, void* stream) {
  if (!a_t || !b_t || ld != (s_rows + 7) / 8 * 8) return PX_ERR_BAD_ARG;
  MrArgs g = {};
  g.m = m, g.gamma = ln_w, g.beta = ln_b, g.mask = mask, g.a_t = (__half*)a_t, g.b_t = (__half*)b_t, g.ld = (int)ld, g.eps = eps;
  return launch_msa_rows<kMrPrep>(prepared, nullptr, g, s_rows, n, (cudaStream_t)stream);
}

extern "C" int32_t px_msa_values(const float* m, const float* ln_w, const float* ln_b, const void* prepared, px_bf16* v,
                                 int64_t s_rows, int64_t n, float eps, void* stream) {
  if (!v || ((uintptr_t)v & 15)) return PX_ERR_BAD_ARG;
  MrArgs g = {};
  g.m = m, g.gamma = ln_w, g.beta = ln_b, g.v = (bf16*)v, g.eps = eps;
  return launch_msa_rows<kMrValues>(prepared, nullptr, g, s_rows, n, (cudaStream_t)stream);
}

extern "C" int32_t px_msa_gate_out(float* m, const float* wv, const float* ln_w, const float* ln_b, const void* prepared_g,
                                   const void* prepared_out, int64_t s_rows, int64_t n, float eps, void* stream) {
  if (!wv || !prepared_out || ((uintptr_t)wv & 15)) return PX_ERR_BAD_ARG;
  MrArgs g = {};
  g.m = m, g.m_out = m, g.gamma = ln_w, g.beta = ln_b, g.wv = wv, g.eps = eps;
  return launch_msa_rows<kMrGate>(prepared_g, prepared_out, g, s_rows, n, (cudaStream_t)stream);
}
