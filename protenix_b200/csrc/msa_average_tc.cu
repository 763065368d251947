// Pair-weighted average of the MSA stack in fp32-grade arithmetic on the 5th-generation tensor cores:
//   wv[h][i][n] = sum_j softmax_j(logits[h][i])[j] v[h][j][n],   n = 8 s + c (8 sequences' channels a head: 8 S columns).
// Weights and values come as three bf16 planes (px_split.cuh), six partial products each: at S = 1024, N = 384 the six take 71 us at
// the tensor core's measured rate, the library's fp32 products took 356.
//
// msa_weights     one CTA per row: softmax of the logits, written as planes [8][3][N][ld], K-major operand (ld = N rounded up to 8)
// msa_average     persistent, one CTA per SM, tiles of 128 rows i x 128 columns n, 64 keys j at a time.  The values arrive as they
//                 lie, [64 j][64 n] boxes, and are used as an MN-major operand.  A stage holds the three planes of both operands
//                 (96 KB, two stages): 39 bytes a clock from L2 against 2400 clocks of loads and products, so wider tiles, which
//                 would leave one stage, gain nothing.
//   warps 0..3    epilogue: the accumulators' sum, staged so that a warp stores 128 contiguous bytes of four rows at a time
//   warp 4        TMA producer;  warps 5..7 MMA issuers: (0,0) | (0,1) (1,0) (1,1) | (0,2) (2,0)
// The tensor core truncates on accumulation: the leading products take turns on two accumulators, the corrections have one for each
// issuer.  Tensor memory: 4 x 128.  Every wait is bounded.
#include "px_split.cuh"

namespace px {

constexpr int kMvABytes = 3 * 128 * 128;       // [3 planes][128 i][64 j] bf16
constexpr int kMvBHalf = 3 * 64 * 128;         // [3 planes][64 j][64 n]
constexpr int kMvStageBytes = kMvABytes + 2 * kMvBHalf;
constexpr int kMvStages = 2;
constexpr int kMvThreads = 256;
constexpr int kMvHeads = 8;

struct MvBars {
  uint64_t full[kMvStages], empty[kMvStages], acc_full, acc_free;
  uint32_t tmem_base;
};
struct MvLayout {
  static constexpr int stg = kMvStages * kMvStageBytes;      // 4 warps x [32 rows][32 fp32]
  static constexpr int bars = stg + 4 * 4096;
  static constexpr int total = bars + (int)sizeof(MvBars);
};
static_assert(MvLayout::total + 1024 <= 232448, "shared memory budget");

// softmax of one row of logits [rows][n] -> planes: row r = h n + i goes to [h][p][i]
__global__ void __launch_bounds__(128) msa_weights_kernel(const float* __restrict__ logits, bf16* __restrict__ w, int n, int ld) {
  __shared__ float part[8];
  pdl_wait();
  const int i = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* x = logits + ((size_t)h * n + i) * n;
  float mx = -INFINITY;
  for (int j = threadIdx.x; j < n; j += 128) mx = fmaxf(mx, x[j]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) part[warp] = mx;
  __syncthreads();
  mx = fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3]));
  float sum = 0.f;
  for (int j = threadIdx.x; j < n; j += 128) sum += expf(x[j] - mx);
  sum = warp_sum(sum);
  if (lane == 0) part[4 + warp] = sum;
  __syncthreads();
  sum = (part[4] + part[5]) + (part[6] + part[7]);
  for (int j = 2 * threadIdx.x; j < ld; j += 256) {          // the padding of a row is zero
    uint32_t b[3];
    split3x2(j < n ? expf(x[j] - mx) / sum : 0.f, j + 1 < n ? expf(x[j + 1] - mx) / sum : 0.f, b);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(w + (((size_t)h * 3 + p) * n + i) * ld + j) = b[p];
  }
}

__global__ void __launch_bounds__(kMvThreads, 1)
msa_average_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_v, float* __restrict__ out,
                      int n, int cols, int tiles_m, int tiles_n, int n_tiles, int chunks) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  MvBars& bars = *reinterpret_cast<MvBars*>(sm + MvLayout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int first_tile = blockIdx.x, tile_step = gridDim.x;

  const bool skip = cta_begin();
  if (threadIdx.x == 32) prefetch_maps(map_w, map_v);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMvStages; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 3);
    }
    mbar_init(&bars.acc_full, 3);
    mbar_init(&bars.acc_free, 4);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (!cta_ready(skip, warp == 4, bars.tmem_base, 512u)) return;
  const uint32_t tmem_base = bars.tmem_base;

  if (warp >= 4) {
    if (!elect_lane()) {
      // nothing: one elected lane of each control warp works
    } else if (warp == 4) {
      int it = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
        const int i0 = (tile % tiles_m) * 128, rest = tile / tiles_m, n0 = (rest % tiles_n) * 128, h = rest / tiles_n;
        for (int c = 0; c < chunks; ++c, ++it) {
          const int s = it % kMvStages;
          ok = mbar_wait(&bars.empty[s], ((it / kMvStages) & 1) ^ 1, 1u);
          if (!ok) break;
          mbar_expect_tx(&bars.full[s], kMvStageBytes);
          const uint32_t dst = smem_u32(sm + s * kMvStageBytes);
          tma_load_3d(dst, &map_w, &bars.full[s], 64 * c, i0, 3 * h);
          tma_load_3d(dst + kMvABytes, &map_v, &bars.full[s], n0, 64 * c, 3 * h);
          tma_load_3d(dst + kMvABytes + kMvBHalf, &map_v, &bars.full[s], n0 + 64, 64 * c, 3 * h);
        }
      }
    } else {
      constexpr uint32_t idesc = umma_idesc_bf16(128, 128, false, true);
      const int who = warp - 5;                              // planes (a, b) packed as digits of a list
      const int count = who == 0 ? 1 : who == 1 ? 3 : 2;
      const uint32_t list = who == 0 ? 0x00u : who == 1 ? 0x011011u : 0x2002u;   // (0,0) | (1,1) (1,0) (0,1) | (0,2) (2,0)
      int it = 0, k = 0;
      bool ok = true;
      for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step, ++k) {
        ok = mbar_wait(&bars.acc_free, (k & 1) ^ 1, 8u);
        for (int c = 0; c < chunks && ok; ++c, ++it) {
          const int s = it % kMvStages;
          ok = mbar_wait(&bars.full[s], (it / kMvStages) & 1, 2u);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a = smem_u32(sm + s * kMvStageBytes), b = a + kMvABytes;
          for (int t = 0; t < count; ++t) {
            const uint32_t pair = (list >> (8 * t)) & 0xffu;
            const uint64_t da = umma_desc_sw128(a + (pair >> 4) * (128 * 128));
            const uint32_t db = b + (pair & 15) * (64 * 128);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              const uint32_t d = tmem_base + 128 * (who == 0 ? (ks & 1) : who + 1);
              umma_bf16(d, da + 2 * ks, umma_desc_mn_sw128(db + ks * 2048, kMvBHalf, 1024), idesc, c > 0 || (who == 0 ? ks > 1 : t + ks > 0));
            }
          }
          umma_commit(&bars.empty[s]);
        }
        if (ok) umma_commit(&bars.acc_full);
      }
    }
  } else {
    const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * warp) << 16);
    unsigned char* stg = sm + MvLayout::stg + warp * 4096;
    int k = 0;
    for (int tile = first_tile; tile < n_tiles; tile += tile_step, ++k) {
      const int i0 = (tile % tiles_m) * 128 + 32 * warp, rest = tile / tiles_m, n0 = (rest % tiles_n) * 128, h = rest / tiles_n;
      bool ok = mbar_wait(&bars.acc_full, k & 1, 4u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        uint32_t x[32], y[32], z[32];
        float v[32];
        tmem_ld32(lane_addr + 256 + 32 * q, x);              // corrections first
        tmem_ld32(lane_addr + 384 + 32 * q, y);
        tmem_ld32(lane_addr + 32 * q, z);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = (__uint_as_float(x[e]) + __uint_as_float(y[e])) + __uint_as_float(z[e]);
        tmem_ld32(lane_addr + 128 + 32 * q, x);
        tmem_wait_ld();
        if (q == 3) {                                        // this warp has read its part of the accumulators
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.acc_free);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<float4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) =
              make_float4(v[4 * c] + __uint_as_float(x[4 * c]), v[4 * c + 1] + __uint_as_float(x[4 * c + 1]),
                          v[4 * c + 2] + __uint_as_float(x[4 * c + 2]), v[4 * c + 3] + __uint_as_float(x[4 * c + 3]));
        __syncwarp();
        const int rsub = lane >> 3, piece = lane & 7, col = n0 + 32 * q + 4 * piece;   // cols is a multiple of 8
#pragma unroll
        for (int r8 = 0; r8 < 8; ++r8) {
          const int rl = 4 * r8 + rsub;
          if (i0 + rl < n && col < cols)
            *reinterpret_cast<float4*>(out + ((size_t)h * n + i0 + rl) * cols + col) =
                *reinterpret_cast<const float4*>(stg + rl * 128 + ((piece ^ (rl & 7)) << 4));
        }
        __syncwarp();
      }
    }
  }

  tc_fence_before();
  cta_teardown_sync();
  if (warp == 4) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

PX_DEFINE_FAMILY_HOOKS(msa_average)

}  // namespace px

using namespace px;

extern "C" int32_t px_msa_weights(const float* logits, px_bf16* w, int64_t n, int64_t ld, void* stream) {
  if (!logits || !w || ((uintptr_t)w & 15) || n <= 0 || n > 32768 || ld != (n + 7) / 8 * 8) return PX_ERR_BAD_ARG;
  return launch_pdl(msa_weights_kernel, dim3((unsigned)n, kMvHeads), 128, 0, (cudaStream_t)stream, logits, (bf16*)w, (int)n, (int)ld)
             ? PX_OK
             : PX_ERR_LAUNCH;
}

extern "C" int32_t px_msa_average(const px_bf16* w, const px_bf16* v, float* wv, int64_t s_rows, int64_t n, int64_t ld, void* stream) {
  if (!w || !v || !wv || (((uintptr_t)w | (uintptr_t)v | (uintptr_t)wv) & 15) || n <= 0 || n > 32768 || s_rows <= 0 ||
      s_rows > (1 << 20) || ld != (n + 7) / 8 * 8)
    return PX_ERR_BAD_ARG;
  const uint64_t cols = 8 * (uint64_t)s_rows;
  CUtensorMap mw, mv;
  // w [8 3][n][ld], box [3][128][64]; v [8 3][n][8 S], box [3][64][64]
  if (!make_map_3d(&mw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w, (uint64_t)n, (uint64_t)n, 3 * kMvHeads, (uint64_t)ld * 2,
                   (uint64_t)n * ld * 2, 64, 128, CU_TENSOR_MAP_SWIZZLE_128B, 3) ||
      !make_map_3d(&mv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, v, cols, (uint64_t)n, 3 * kMvHeads, cols * 2, (uint64_t)n * cols * 2, 64, 64,
                   CU_TENSOR_MAP_SWIZZLE_128B, 3))
    return PX_ERR_LAUNCH;
  const int64_t tiles_m = (n + 127) / 128, tiles_n = (int64_t)(cols + 127) / 128, n_tiles = tiles_m * tiles_n * kMvHeads;
  if (n_tiles > 0x7fffffff) return PX_ERR_UNSUPPORTED;
  const size_t smem = MvLayout::total + 1024;
  static SmemLimit limit;
  const int grid = even_grid(n_tiles, sm_count(), n % 128 ? tiles_m : 1);
  return limit.set(msa_average_tc_kernel, smem) &&
                 launch_pdl(msa_average_tc_kernel, dim3((unsigned)grid), kMvThreads, smem, (cudaStream_t)stream, mw, mv, wv, (int)n, (int)cols,
                            (int)tiles_m, (int)tiles_n, (int)n_tiles, (int)((n + 63) / 64))
             ? PX_OK
             : PX_ERR_LAUNCH;
}
