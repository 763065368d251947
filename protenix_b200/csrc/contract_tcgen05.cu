// Triangle-multiplication contraction on the 5th-generation tensor cores:
//   x[c][i][j] = 2^-6 sum_k a[c][i][k] * b[c][j][k]      (fp16 in, fp32 accumulate, fp16 out)
// The LayerNorm that consumes x does not see a common factor (its epsilon is scaled to match), and the factor 2^-6
// keeps sums over thousands of k inside the fp16 range.
//
// Bound by the operands' way from L2: a CTA of its own with a 128 x 256 tile takes 48 KB for every 512 cycles of products, 96 bytes a
// cycle, where all SMs together get about 44 each.  So two CTAs on neighbouring SMs share a 256 x 256 tile (cta_group::2): each
// loads its 128 rows of A and half of B's, 32 KB for the same products.  N = 437: 49.3 -> 45.5 us, 768: 120 -> 107, 1024: 265
// -> 235, outer product of 384 tokens and 1024 sequences: 266 -> 242; not everywhere, see pairs_pay.  Results leave by TMA: 16-byte stores of
// rows, half a sector each, took 37.7 us in place of 27.0 at N = 384, 131 in place of 114 at N = 768.
//
// Persistent kernel, one CTA per SM, 192 threads (in brackets: what the leader of a pair does for both):
//   warp 0      TMA producer: A tile [128 i][64 k] and B tile [256 (128) j][64 k] per k-block, 128-byte swizzle, a ring of stages
//               guarded by full/empty mbarriers [both CTAs' copies are counted by the leader's full barrier]
//   warp 1      MMA issuer: one thread issues tcgen05.mma (M=128 (256), N=256, K=16) four times per k-block; tcgen05.commit releases
//               the shared-memory stage and, after the last k-block, publishes the accumulator [in both CTAs]
//   warps 2..5  epilogue: tcgen05.ld of the fp32 accumulator (each warp its own 32 TMEM lanes = 32 rows), scale, convert to fp16,
//               staged in shared memory ([32 rows][64 columns], two buffers) and written by TMA
// The accumulator is double-buffered in TMEM (2 x 256 columns) so the epilogue of tile t overlaps the
// main loop of tile t+1.  Ragged edges need no predicates: the TMA zero-fills rows >= N and k >= ld on the way in and drops
// what lies outside on the way out.  Tiles are ordered channel-major so that a channel's operands (2 * N * ld * 2
// bytes) stay in L2 while its tiles are computed.
//
// Every wait on an mbarrier is bounded; a wait that runs out records a flag in g_tc_error, the
// role stops issuing work, and the kernel still frees its TMEM and returns.
#include "px_rowpipe.cuh"

namespace px {

constexpr int kTcBM = 128, kTcBN = 256, kTcBK = 64;        // of one CTA's accumulator
constexpr int kTcABytes = kTcBM * kTcBK * 2;
constexpr int kTcStgBytes = 32 * 128;                      // one staged block: [32 rows][64 columns] fp16
constexpr uint32_t kTcCols = 512;  // two 256-column fp32 accumulators
template <int kCtas>
struct TcShape {
  static constexpr int kBRows = kTcBN / kCtas;             // rows of B that a CTA loads
  static constexpr int kStageBytes = kTcABytes + kBRows * kTcBK * 2;
  static constexpr int kStages = kCtas == 2 ? 6 : 4;
  static constexpr int kStg = kStages * kStageBytes, kBars = kStg + 8 * kTcStgBytes;
};

struct TcBarriers {
  uint64_t full[6], empty[6], acc_full[2], acc_empty[2];
  uint32_t tmem_base, peer_stop;
};

// The forms of the tcgen05 and cluster instructions for a pair of CTAs.
__device__ __forceinline__ void tc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\n barrier.cluster.wait.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
// Into this CTA's shared memory, counted by a barrier of the pair (cluster address).
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this address in both CTAs.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

template <int kCtas>
__global__ void __launch_bounds__(192, 1)
trimul_contract_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                          const __grid_constant__ CUtensorMap map_x, int n, int ld_k, int ld, int tiles_i, int tiles_j, int total_tiles) {
  typedef TcShape<kCtas> Shape;
  constexpr bool kPair = kCtas == 2;
  constexpr int kStages = Shape::kStages;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // operand ring first (1024-byte aligned for the 128-byte swizzle), staging and barriers after it
  unsigned char* ring = smem_aligned(smem_raw);
  TcBarriers& bars = *reinterpret_cast<TcBarriers*>(ring + Shape::kBars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int nk = (ld_k + kTcBK - 1) / kTcBK;      // ld_k: extent of the contraction index; ld: row stride of x
  const uint32_t rank = kPair ? cluster_rank() : 0;
  const int first_tile = blockIdx.x / kCtas, tile_step = gridDim.x / kCtas;

  const bool skip = cta_begin();         // an earlier bounded wait gave up: do not start new work
  if (threadIdx.x == 32) prefetch_maps(map_a, map_b, map_x);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars.acc_full[b], 1);
      mbar_init(&bars.acc_empty[b], 4 * kCtas);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    if constexpr (kPair) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                   "r"(kTcCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                   "r"(kTcCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
  }
  bool stop;
  tc_fence_before();
  if constexpr (kPair) {
    // both CTAs work or neither does
    stop = __syncthreads_or(skip) != 0;
    if (threadIdx.x == 0)
      asm volatile("st.shared::cluster.u32 [%0], %1;\n" ::"r"(map_to_rank(smem_u32(&bars.peer_stop), rank ^ 1)), "r"((uint32_t)stop) : "memory");
    tc_cluster_sync();
    stop = stop || *reinterpret_cast<volatile uint32_t*>(&bars.peer_stop) != 0;
  } else {
    stop = __syncthreads_or(skip) != 0;
  }
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem_base = bars.tmem_base;

  auto tile_coords = [&](int tile, int& c, int& i0, int& j0) {
    const int per_c = tiles_i * tiles_j;
    c = tile / per_c;
    const int r = tile - c * per_c;
    i0 = (r / tiles_j) * (kTcBM * kCtas) + kTcBM * (int)rank;      // this CTA's rows
    j0 = (r % tiles_j) * kTcBN;
  };

  if (stop) {
    // nothing
  } else if (warp == 0) {
    uint32_t it = 0;
    bool ok = true;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
      int c, i0, j0;
      tile_coords(tile, c, i0, j0);
      for (int kt = 0; kt < nk && ok; ++kt, ++it) {
        const int s = it % kStages;
        const uint32_t ph = (it / kStages) & 1;
        ok = mbar_wait_warp(&bars.empty[s], ph ^ 1, 1u);
        if (!ok) break;
        if (elect_lane()) {
          const uint32_t sa = smem_u32(ring + s * Shape::kStageBytes);
          if constexpr (kPair) {
            if (rank == 0) mbar_expect_tx(&bars.full[s], 2 * Shape::kStageBytes);
            const uint32_t bar = map_to_rank(smem_u32(&bars.full[s]), 0);
            tma_load_3d_pair(sa, &map_a, bar, kt * kTcBK, i0, c);
            tma_load_3d_pair(sa + kTcABytes, &map_b, bar, kt * kTcBK, j0 + Shape::kBRows * (int)rank, c);
          } else {
            mbar_expect_tx(&bars.full[s], Shape::kStageBytes);
            tma_load_3d(sa, &map_a, &bars.full[s], kt * kTcBK, i0, c);
            tma_load_3d(sa + kTcABytes, &map_b, &bars.full[s], kt * kTcBK, j0, c);
          }
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      constexpr uint32_t idesc = umma_idesc_f16(kTcBM * kCtas, kTcBN);
      uint32_t it = 0, tcount = 0;
      bool ok = true;
      for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++tcount) {
        const uint32_t ab = tcount & 1, aph = (tcount >> 1) & 1;
        ok = mbar_wait_warp(&bars.acc_empty[ab], aph ^ 1, 2u);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + ab * kTcBN;
        for (int kt = 0; kt < nk; ++kt, ++it) {
          const int s = it % kStages;
          const uint32_t ph = (it / kStages) & 1;
          ok = mbar_wait_warp(&bars.full[s], ph, 4u);
          if (!ok) break;
          tc_fence_after();
          if (elect_lane()) {
            const uint32_t sa = smem_u32(ring + s * Shape::kStageBytes);
            const uint64_t da = umma_desc_sw128(sa), db = umma_desc_sw128(sa + kTcABytes);
#pragma unroll
            for (int k = 0; k < kTcBK / 16; ++k) {  // 16 fp16 = 32 bytes = 2 units of the start-address field
              if constexpr (kPair)
                umma_pair(d_tmem, da + 2 * k, db + 2 * k, idesc, (kt | k) ? 1u : 0u);
              else
                umma_bf16(d_tmem, da + 2 * k, db + 2 * k, idesc, (kt | k) ? 1u : 0u);
            }
            if constexpr (kPair)
              umma_commit_pair(&bars.empty[s]);
            else
              umma_commit(&bars.empty[s]);
            if (kt == nk - 1) {
              if constexpr (kPair)
                umma_commit_pair(&bars.acc_full[ab]);
              else
                umma_commit(&bars.acc_full[ab]);
            }
          }
          __syncwarp();
        }
        if (!ok) break;
      }
    }
  } else {
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    unsigned char* const stg = ring + Shape::kStg + q * 2 * kTcStgBytes;
    uint32_t tcount = 0, block = 0;                        // staged blocks so far
    bool ok = true;
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++tcount) {
      int c, i0, j0;
      tile_coords(tile, c, i0, j0);
      const uint32_t ab = tcount & 1, aph = (tcount >> 1) & 1;
      ok = mbar_wait(&bars.acc_full[ab], aph, 8u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int i = i0 + 32 * q;
#pragma unroll 1
      for (int cc = 0; cc < kTcBN / 64; ++cc) {
        if (j0 + 64 * cc >= ld || i >= n) break;           // warp-uniform; nothing of this block exists
        unsigned char* const buf = stg + (block++ & 1) * kTcStgBytes;
        if (lane == 0) tma_store_wait_read<1>();           // the store before last has read this buffer
        __syncwarp();
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          uint32_t r[32];
          tmem_ld32(tmem_base + ((uint32_t)(32 * q) << 16) + ab * kTcBN + cc * 64 + hh * 32, r);
          tmem_wait_ld();
          constexpr float sc = PX_TRIMUL_X_SCALE;
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 o;
            o.x = pack_f16x2(sc * __uint_as_float(r[8 * v + 0]), sc * __uint_as_float(r[8 * v + 1]));
            o.y = pack_f16x2(sc * __uint_as_float(r[8 * v + 2]), sc * __uint_as_float(r[8 * v + 3]));
            o.z = pack_f16x2(sc * __uint_as_float(r[8 * v + 4]), sc * __uint_as_float(r[8 * v + 5]));
            o.w = pack_f16x2(sc * __uint_as_float(r[8 * v + 6]), sc * __uint_as_float(r[8 * v + 7]));
            *reinterpret_cast<uint4*>(buf + lane * 128 + (((4 * hh + v) ^ (lane & 7)) << 4)) = o;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          tma_store_3d(&map_x, smem_u32(buf), j0 + 64 * cc, i, c);
          tma_store_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (kPair)
          mbar_arrive_cluster(map_to_rank(smem_u32(&bars.acc_empty[ab]), 0));
        else
          mbar_arrive(&bars.acc_empty[ab]);
      }
    }
    if (lane == 0) tma_store_wait_read<0>();
  }

  // teardown: everybody meets, then the allocating warp frees the tensor memory
  __syncwarp();
  tc_fence_before();
  cta_teardown_sync();
  if constexpr (kPair) tc_cluster_sync();          // nobody leaves while its pair may still signal or read it
  if (warp == 0) {
    tc_fence_after();
    if constexpr (kPair)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTcCols) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTcCols) : "memory");
  }
  if constexpr (kPair) tc_cluster_sync();
}

// [channels][n rows][ld k] fp16 tensor, box = [1][box_rows][64], 128-byte swizzle, zero fill outside.
static bool make_operand_map(CUtensorMap* map, const void* base, int64_t channels, int64_t n, int64_t ld,
                             uint32_t box_rows) {
  return make_map_3d(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, base, (uint64_t)ld, (uint64_t)n, (uint64_t)channels,
                     (uint64_t)ld * 2, (uint64_t)n * ld * 2, kTcBK, box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

PX_DEFINE_FAMILY_HOOKS(contract)

// x[c] [rows_a][ld] = 2^-6 a[c] b[c]^T, a [channels][rows_a][ld_k], b [channels][rows_b][ld_k]
template <int kCtas>
static int32_t launch_contract(const void* a, const void* b, void* x, int64_t channels, int64_t rows_a, int64_t rows_b, int64_t ld_k,
                               int64_t ld, cudaStream_t st) {
  typedef TcShape<kCtas> Shape;
  CUtensorMap ma, mb, mx;
  if (!make_operand_map(&ma, a, channels, rows_a, ld_k, kTcBM) || !make_operand_map(&mb, b, channels, rows_b, ld_k, Shape::kBRows) ||
      !make_operand_map(&mx, x, channels, rows_a, ld, 32))
    return PX_ERR_LAUNCH;
  const int64_t tiles_i = (rows_a + kTcBM * kCtas - 1) / (kTcBM * kCtas), tiles_j = (rows_b + kTcBN - 1) / kTcBN;
  const int64_t total = tiles_i * tiles_j * channels;
  if (total > 0x7fffffff) return PX_ERR_UNSUPPORTED;
  const int64_t room = sm_count() / kCtas;
  const bool ragged = rows_a % (kTcBM * kCtas) || rows_b % kTcBN;
  const int64_t period = !ragged ? 1 : channels > 1 ? tiles_i * tiles_j : tiles_j;
  const size_t smem = Shape::kBars + sizeof(TcBarriers) + 1024;
  static_assert(Shape::kBars + sizeof(TcBarriers) + 1024 <= 232448, "shared memory budget");
  static SmemLimit limit;
  if (!limit.set(trimul_contract_tc_kernel<kCtas>, smem)) return PX_ERR_LAUNCH;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = kCtas, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(even_grid(total, room, period) * kCtas));
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = kCtas > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, trimul_contract_tc_kernel<kCtas>, ma, mb, mx, (int)rows_a, (int)ld_k, (int)ld, (int)tiles_i, (int)tiles_j,
                         (int)total) == cudaSuccess)
    return PX_OK;
  cudaGetLastError();
  return PX_ERR_LAUNCH;
}

// A pair fetches a third less per product and takes longer to hand a tile over, so it pays where the way from L2 bounds the
// tile: with a contraction long enough, the longer the better operand rows lie.  Rows of whole 128-byte lines come fastest, rows of whole
// 32-byte sectors next, and others touch a sector more for every 128 bytes (us, single | paired; outer products of 300
// tokens: 256 sequences 57.7 | 68.6, 448 78.6 | 80.3, 512 87.5 | 83.8, 1024 149 | 136; 240 0.97, 272 1.04 and 304 1.06 times as
// fast in pairs; 136 70.0 | 70.5, 152 74.1 | 72.0, 500 134 | 110).  Few 128-row tiles leave half a pair idle on an odd last one (128 channels, N = 384: 31.1
// | 37.2, 512: 45.5 | 47.5, 640: 84.5 | 88.4, 768: 120 | 107, 832: 182 | 177, 850: 284 | 239, 1152: 375 | 370, 1400: 1069
// | 816; straddling rows, 390: 47.5 | 43.4, 520: 81.8 | 79.1, 344: 38.9 | 39.2), and with less than two tiles to an SM there is nothing to
// hand over beside (outer products of 64 tokens, 1024 sequences: 16.5 | 17.4; 92, 400: 16.9 | 18.5; 100, 1000: 41.2 | 35.1).
static bool pairs_pay(int64_t channels, int64_t rows_a, int64_t rows_b, int64_t ld_k) {
  const int64_t t = (rows_a + kTcBM - 1) / kTcBM, tiles = channels * t * ((rows_b + kTcBN - 1) / kTcBN);
  const bool lines = ld_k % 64 == 0, sectors = ld_k % 16 == 0;
  return t >= (sectors ? 6 : 4) && ld_k >= (lines ? 448 : sectors ? 272 : 152) && tiles >= 2 * sm_count();
}

}  // namespace px

using namespace px;

extern "C" int32_t px_trimul_contract(const px_bf16* a, const px_bf16* b, px_bf16* x, int64_t channels, int64_t n,
                                      int64_t ld, void* stream) {
  if (!a || !b || !x || channels <= 0 || channels > 65535 || n <= 0 || n > 32768 || ld != px_ld(n))
    return PX_ERR_BAD_ARG;
  if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)x) & 15) return PX_ERR_BAD_ARG;
  return (pairs_pay(channels, n, n, ld) ? launch_contract<2> : launch_contract<1>)(a, b, x, channels, n, n, ld, ld, (cudaStream_t)stream);
}

// The same kernel for the outer product of the MSA module: one "channel", a_t [rows_a][ld_k] against
// b_t [rows_b][ld_k] (rows = 32 x tokens), contraction over the ld_k (padded) MSA rows; x is [rows_a][rows_b].
extern "C" int32_t px_opm_outer(const px_f16* a_t, const px_f16* b_t, px_f16* x, int64_t rows_a, int64_t rows_b,
                                int64_t ld_k, void* stream) {
  if (!a_t || !b_t || !x || rows_a <= 0 || rows_a > (1 << 20) || rows_b <= 0 || rows_b > (1 << 20) || rows_b % 8 ||
      ld_k <= 0 || ld_k % 8 || ld_k > (1 << 20))
    return PX_ERR_BAD_ARG;
  if (((uintptr_t)a_t | (uintptr_t)b_t | (uintptr_t)x) & 15) return PX_ERR_BAD_ARG;
  return (pairs_pay(1, rows_a, rows_b, ld_k) ? launch_contract<2> : launch_contract<1>)(a_t, b_t, x, 1, rows_a, rows_b, ld_k, rows_b, (cudaStream_t)stream);
}
