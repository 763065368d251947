// The single-representation branch of a Pairformer block (c_s = 384, 16 heads x 24) in fp32-grade arithmetic:
//   s += W_o( softmax(q k^T / sqrt(24) + pair bias) v * sigmoid(W_g x) ),   x = LN(s)        (attention)
//   s += W_out( silu(W_a y) * (W_b y) ),                                    y = LN(s)        (transition)
//
// The matrix products run on the 5th-generation tensor cores with every fp32 operand written as the sum of three bf16
// values (8 + 8 + 8 significant bits) and the six partial products that reach 2^-24 accumulated in fp32: no operand
// bit of an fp32 product is given up, and the range is that of fp32.  Six bf16 products cost 1/6 of the bf16 rate,
// which is still five times that of the fp32 pipe.  Seven launches:
//   split_rows        LayerNorm of s, written as three bf16 planes [3][N][384]
//   split_gemm QKVG   [q | k | v | g] = x W^T, q scaled, sigmoid(g), fp32 [N][1536]
//   single_attention  flash attention on the fp32 pipe (3.6 GFLOP at N = 1536), gated, written as three planes
//   split_gemm RES    s1 = s + o W_o^T
//   split_rows        LayerNorm of s1
//   split_gemm SWIGLU h = silu(a) * b, a and b interleaved in the weight rows, written as three planes [3][N][1536]
//   split_gemm RES    s2 = s1 + h W_out^T, the contraction split over a cluster of four CTAs
// At N tokens each product has N/128 x (outputs/64) tiles: far too few to fill the chip at any N, so every launch is
// bound by the latency of one tile (load, 16 MMAs per 64 inputs, epilogue); hence narrow 64-column tiles, no
// persistence, and the split contraction where it is 1536 long.  The epilogue is as long as the products (64 columns of a row, half
// of them through expf and a division, six accumulators): sixteen warps, 16 columns a thread, and stores from shared memory.  Four
// warps of 64 columns a thread, storing their rows, against that, each kernel alone at N = 384: QKVG 13.5 -> 9.3 us, SWIGLU 16.1 -> 10.5,
// RES 9.9 -> 7.8 and 10.4 -> 9.9.
#include <initializer_list>

#include "px_split.cuh"

namespace px {

constexpr int kSc = 384;                  // single channels
constexpr int kSh = 16, kSd = 24;         // heads x head width
constexpr int kSf = 4 * kSc;              // hidden width of the transition; also q | k | v | g
constexpr int kSgBN = 64;                 // output columns of a tile
constexpr int kSgABytes = 3 * 128 * 128;  // three planes of [128 rows][64 k] bf16
constexpr int kSgWBytes = 3 * kSgBN * 128;
constexpr int kSgStageBytes = kSgABytes + kSgWBytes;
constexpr int kSgStages = 3;
// Tensor memory: the leading products (plane 0 x plane 0) go round four accumulators, the corrections of order 2^-8 and of order
// 2^-16 have one each.  The tensor core truncates when it adds to an accumulator, a bias that grows with the number of additions: one
// accumulator for all 144 steps of K = 384 gave a relative error of 4.3e-6 on s; with these it is 2.0e-7 (fp32 GEMMs
// of the library: 3.5e-7 to 4.8e-7).
// The planes of W lie behind one another, so that neighbouring partial products with one plane of A are one product of 128 columns:
// A0 W0 (48 cycles of the tensor pipe a step), A0 [W1 W2] (64), A1 [W0 W1] (64), A2 W0 (48), where six products of 64 columns, read
// from shared memory one by one, took 288: 0.4 to 0.8 us of 11 to 15 a kernel at N = 128, and the error was 2.4e-7.
constexpr int kSgMain = 4;
constexpr int kSgCorr = kSgBN * kSgMain;  // columns of the corrections: order 2^-8, then order 2^-16
constexpr int kSgAcc = kSgMain + 2;
constexpr int kSgEpilogue = 4;            // first of the epilogue's warps
constexpr int kSgEpiWarps = 16;           // four for every 32 rows of the tile, 16 columns each
constexpr uint32_t kSgCols = 512;
constexpr int kSgThreads = 32 * (kSgEpilogue + kSgEpiWarps);
constexpr int kSgSplit = 4;               // CTAs of a cluster that share a contraction of 1536

enum { kSgQkvg = 0, kSgRes = 1, kSgSwiglu = 2 };

struct SgBars {
  uint64_t full[kSgStages], empty[kSgStages], acc_full;
  uint32_t tmem_base;
};

// LayerNorm of rows of 384, written as three bf16 planes; one warp per row, the row in registers.
template <typename T>
__global__ void __launch_bounds__(128) split_rows_kernel(const T* __restrict__ x, const float* __restrict__ gamma,
                                                         const float* __restrict__ beta, bf16* __restrict__ out, int rows,
                                                         float eps) {
  pdl_wait();
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  float4 v[3];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    v[i] = ld4<T>(x + (size_t)row * kSc + 128 * i + 4 * lane);
    s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
  }
  const float mean = warp_sum(s) * (1.0f / kSc);
  float q = 0.f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    v[i].x -= mean, v[i].y -= mean, v[i].z -= mean, v[i].w -= mean;
    q += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
  }
  const float rstd = rsqrtf(warp_sum(q) * (1.0f / kSc) + eps);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int c = 128 * i + 4 * lane;
    const float4 g = ld4<float>(gamma + c), b = ld4<float>(beta + c);
    uint32_t lo[3], hi[3];
    split3x2(fmaf(v[i].x * rstd, g.x, b.x), fmaf(v[i].y * rstd, g.y, b.y), lo);
    split3x2(fmaf(v[i].z * rstd, g.z, b.z), fmaf(v[i].w * rstd, g.w, b.w), hi);
#pragma unroll
    for (int p = 0; p < 3; ++p)
      *reinterpret_cast<uint2*>(out + ((size_t)p * rows + row) * kSc + c) = make_uint2(lo[p], hi[p]);
  }
}

struct SgArgs {
  const float* bias;      // QKVG: bias of q [384]
  float* out_f;           // QKVG: [rows][1536]
  bf16* out_planes;       // SWIGLU: [3][rows][1536]
  const void* res;        // RES: residual and output [rows][384] of type T
  void* out;
  int rows, chunks;       // chunks of 64 inputs per CTA
  float scale;            // QKVG: factor of q
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\n barrier.cluster.wait.aligned;\n" ::: "memory");
}

// One 128 x 64 tile of a split product per cluster (of gridDim.z CTAs, each with its share of the contraction).
// Warp 0: TMA producer (three planes of A and of W per 64 inputs), warp 1: MMA issuer, warps 4..19: epilogue, a thread 16 columns of a
// row, which leave through shared memory so that the stores of a warp are runs of 64 to 256 bytes.
template <int kMode, typename T>
__global__ void __launch_bounds__(kSgThreads, 1)
split_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const SgArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* ring = smem_aligned(smem_raw);
  SgBars& bars = *reinterpret_cast<SgBars*>(ring + kSgStages * kSgStageBytes);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * kSgBN, m0 = blockIdx.y * 128, kc0 = blockIdx.z * g.chunks;

  const bool stop = cta_begin();                 // an earlier bounded wait gave up: do no work, but meet the barriers
  if (threadIdx.x == 32) prefetch_maps(map_a, map_w);
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSgStages; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 1);
    }
    mbar_init(&bars.acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                 "r"(kSgCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  const bool skip = __syncthreads_or(stop) != 0;
  tc_fence_after();
  // the weights of the first stages do not wait for the kernel before this one
  const int early = g.chunks < kSgStages ? g.chunks : kSgStages;
  if (threadIdx.x == 0 && !skip) {
    for (int i = 0; i < early; ++i) {
      mbar_expect_tx(&bars.full[i], kSgStageBytes);
      tma_load_3d(smem_u32(ring + i * kSgStageBytes) + kSgABytes, &map_w, &bars.full[i], (kc0 + i) * 64, n0, 0);
    }
  }
  __syncwarp();
  pdl_wait();
  const uint32_t tmem_base = bars.tmem_base;
  bool ok = !skip;

  if (warp == 0) {
    for (int i = 0; i < g.chunks && ok; ++i) {
      const int s = i % kSgStages;
      if (!mbar_wait_warp(&bars.empty[s], ((i / kSgStages) & 1) ^ 1, 1u)) break;
      if (elect_lane()) {
        const uint32_t dst = smem_u32(ring + s * kSgStageBytes);
        if (i >= early) {
          mbar_expect_tx(&bars.full[s], kSgStageBytes);
          tma_load_3d(dst + kSgABytes, &map_w, &bars.full[s], (kc0 + i) * 64, n0, 0);
        }
        tma_load_3d(dst, &map_a, &bars.full[s], (kc0 + i) * 64, m0, 0);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc1 = umma_idesc_bf16(128, kSgBN), idesc2 = umma_idesc_bf16(128, 2 * kSgBN);
    bool done = ok;
    for (int i = 0; i < g.chunks && done; ++i) {
      const int s = i % kSgStages;
      done = mbar_wait_warp(&bars.full[s], (i / kSgStages) & 1, 2u);
      if (!done) break;
      tc_fence_after();
      if (elect_lane()) {
        const uint32_t a = smem_u32(ring + s * kSgStageBytes), w = a + kSgABytes;
        const uint64_t a0 = umma_desc_sw128(a), a1 = umma_desc_sw128(a + 128 * 128), a2 = umma_desc_sw128(a + 2 * 128 * 128);
        const uint64_t w0 = umma_desc_sw128(w), w1 = umma_desc_sw128(w + kSgBN * 128);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {           // the terms above 2^-24 of the product: planes i + j <= 2
          const int step = 4 * i + ks;
          umma_bf16(tmem_base + kSgBN * ks, a0 + 2 * ks, w0 + 2 * ks, idesc1, i > 0);
          umma_bf16(tmem_base + kSgCorr, a0 + 2 * ks, w1 + 2 * ks, idesc2, step > 0);
          umma_bf16(tmem_base + kSgCorr, a1 + 2 * ks, w0 + 2 * ks, idesc2, 1u);
          umma_bf16(tmem_base + kSgCorr + kSgBN, a2 + 2 * ks, w0 + 2 * ks, idesc1, 1u);
        }
        umma_commit(&bars.empty[s]);
        if (i == g.chunks - 1) umma_commit(&bars.acc_full);
      }
      __syncwarp();
    }
  } else if (warp >= kSgEpilogue) {
    // thread: row r of the tile (its tensor-memory lane), columns c0 .. c0 + 7 and c1 .. c1 + 7
    const int q = warp & 3, r = 32 * q + lane, part = (warp - kSgEpilogue) >> 2, tid = threadIdx.x - 32 * kSgEpilogue;
    const int c0 = kMode == kSgSwiglu ? 8 * part : 16 * part, c1 = kMode == kSgSwiglu ? kSgBN / 2 + 8 * part : c0 + 8;
    ok = ok && mbar_wait(&bars.acc_full, 0, 4u);
    ok = __all_sync(0xffffffffu, ok);
    float v[16];
    if (ok) {
      tc_fence_after();
      const uint32_t t = tmem_base + ((uint32_t)(32 * q) << 16);
      uint32_t x[2][16];
#pragma unroll
      for (int p = kSgAcc - 1; p > 0; p -= 2) {    // corrections first
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          tmem_ld8(t + (p - i) * kSgBN + c0, x[i]);
          tmem_ld8(t + (p - i) * kSgBN + c1, x[i] + 8);
        }
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          v[e] = p == kSgAcc - 1 ? __uint_as_float(x[0][e]) : v[e] + __uint_as_float(x[0][e]);
          v[e] += __uint_as_float(x[1][e]);
        }
      }
      // the ring is idle: every product of this CTA is complete.  Rows of 16 pieces of 16 bytes, swizzled by row
      uint4* const stg = reinterpret_cast<uint4*>(ring);
      if (kMode == kSgSwiglu) {                    // columns 0..31: a, 32..63: b of hidden units n0/2 ..; pieces: plane, eight units
        uint32_t w[4][3];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float a0 = v[2 * e], a1 = v[2 * e + 1];
          split3x2(a0 / (1.0f + expf(-a0)) * v[8 + 2 * e], a1 / (1.0f + expf(-a1)) * v[8 + 2 * e + 1], w[e]);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) stg[r * 16 + ((4 * p + part) ^ (r & 15))] = make_uint4(w[0][p], w[1][p], w[2][p], w[3][p]);
      } else {
        if (kMode == kSgQkvg) {
          const int kind = n0 / kSc;               // q, k, v or g: a tile of 64 lies in one of them
          if (kind == 0) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = (v[e] + __ldg(g.bias + n0 + c0 + e)) * g.scale;
          } else if (kind == 3) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = 1.0f / (1.0f + expf(-v[e]));
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
          stg[r * 16 + ((4 * part + e) ^ (r & 15))] = make_uint4(__float_as_uint(v[4 * e]), __float_as_uint(v[4 * e + 1]),
                                                                 __float_as_uint(v[4 * e + 2]), __float_as_uint(v[4 * e + 3]));
      }
    }
    if (kMode != kSgRes) {
      ok = named_barrier_all(1, 32 * kSgEpiWarps, ok);
      if (ok) {
        const uint4* const stg = reinterpret_cast<const uint4*>(ring);
        constexpr int kPieces = kMode == kSgSwiglu ? 12 : 16;
#pragma unroll
        for (int i = 0; i < 128 * kPieces; i += 32 * kSgEpiWarps) {
          // SWIGLU: the planes one after the other, four pieces a row
          const int at = i + tid, p = kMode == kSgSwiglu ? at >> 9 : 0;
          const int rr = kMode == kSgSwiglu ? (at & 511) >> 2 : at >> 4, c = kMode == kSgSwiglu ? at & 3 : at & 15, row = m0 + rr;
          if (row < g.rows) {
            const uint4 o = stg[rr * 16 + ((4 * p + c) ^ (rr & 15))];
            if (kMode == kSgSwiglu)
              *reinterpret_cast<uint4*>(g.out_planes + ((size_t)p * g.rows + row) * kSf + n0 / 2 + 8 * c) = o;
            else
              *reinterpret_cast<uint4*>(g.out_f + (size_t)row * kSf + n0 + 4 * c) = o;
          }
        }
      }
    }
  }
  if (kMode == kSgRes) {
    __syncwarp();
    cluster_sync();                                // every CTA's partial tile is in its shared memory
    if (warp >= kSgEpilogue && ok) {
      // each CTA sums and writes its share of the rows; a thread takes 16 bytes of a row at a time
      const int split = gridDim.z, per = 128 / split, tid = threadIdx.x - 32 * kSgEpilogue;
      for (int i = tid; i < per * (kSgBN / 4); i += 32 * kSgEpiWarps) {
        const int r = blockIdx.z * per + i / (kSgBN / 4), c = i % (kSgBN / 4), row = m0 + r;
        const uint32_t src = smem_u32(ring) + (r * (kSgBN / 4) + (c ^ (r & 15))) * 16;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p = 0; p < split; ++p) {
          uint32_t peer;
          float4 x;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(peer) : "r"(src), "r"(p));
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                       : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                       : "r"(peer)
                       : "memory");
          sum.x += x.x, sum.y += x.y, sum.z += x.z, sum.w += x.w;
        }
        if (row < g.rows) {
          // the update is rounded to the type of s before it is added, as the module's composition does
          const size_t at = (size_t)row * kSc + n0 + 4 * c;
          const float4 z = ld4<T>(reinterpret_cast<const T*>(g.res) + at);
          T* o = reinterpret_cast<T*>(g.out) + at;
          o[0] = T(z.x + float(T(sum.x))), o[1] = T(z.y + float(T(sum.y)));
          o[2] = T(z.z + float(T(sum.z))), o[3] = T(z.w + float(T(sum.w)));
        }
      }
    }
    __syncwarp();
    cluster_sync();                                // nobody leaves while a peer may still read its shared memory
  }
  tc_fence_before();
  cta_teardown_sync();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kSgCols) : "memory");
  }
}

// Attention of one head and 32 queries over tiles of 64 keys, online softmax, fp32 throughout.  qkvg [n][1536] (q
// scaled, g already a sigmoid), bias [16][n][n]; out: gated result as three planes [3][n][384].
// Two groups of 128 threads take every other key tile and merge at the end (one group per CTA left an SM with five
// warps at N = 384: 23 us).  A thread owns 4 queries x 4 keys of the logits; of the product with the values 4 queries
// x 3 channels over half the keys of a tile.
constexpr int kSaQ = 32, kSaK = 64, kSaLd = kSaK + 4, kSaGroups = 2;

struct SaTile {
  float k[kSd][kSaLd], v[kSd][kSaLd], p[kSaQ][kSaLd];
};

__global__ void __launch_bounds__(128 * kSaGroups, 2)
single_attention_kernel(const float* __restrict__ qkvg, const float* __restrict__ bias, bf16* __restrict__ out, int n) {
  extern __shared__ __align__(16) unsigned char sa_raw[];
  pdl_wait();
  float(*qs)[kSaQ] = reinterpret_cast<float(*)[kSaQ]>(sa_raw);
  const int grp = threadIdx.x >> 7, tid = threadIdx.x & 127, ty = tid >> 4, tx = tid & 15;
  SaTile& t = reinterpret_cast<SaTile*>(sa_raw + kSd * kSaQ * 4)[grp];
  const int h = blockIdx.y, q0 = blockIdx.x * kSaQ;
  const float* base = qkvg + h * kSd;
  for (int i = threadIdx.x; i < kSaQ * (kSd / 4); i += 128 * kSaGroups) {
    const int r = i & 31, d4 = i >> 5;
    const float4 x = (q0 + r < n) ? ld4<float>(base + (size_t)(q0 + r) * kSf + 4 * d4) : make_float4(0.f, 0.f, 0.f, 0.f);
    qs[4 * d4][r] = x.x, qs[4 * d4 + 1][r] = x.y, qs[4 * d4 + 2][r] = x.z, qs[4 * d4 + 3][r] = x.w;
  }
  float4 kr[3], vr[3];
  auto load_kv = [&](int k0) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int i = tid + 128 * j, k = k0 + (i & 63), d4 = i >> 6;
      kr[j] = vr[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < n) {
        const float* row = base + (size_t)k * kSf + 4 * d4;
        kr[j] = ld4<float>(row + kSc);
        vr[j] = ld4<float>(row + 2 * kSc);
      }
    }
  };
  const int khalf = tx >> 3, dg = 3 * (tx & 7);
  float m[4], l[4], o[4][3];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY, l[i] = 0.f;
    o[i][0] = o[i][1] = o[i][2] = 0.f;
  }
  load_kv(kSaK * grp);
  __syncthreads();
  for (int k0 = kSaK * grp; k0 < n; k0 += kSaK * kSaGroups) {
    named_barrier(1 + grp, 128);                   // the previous tile has been used
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int i = tid + 128 * j, k = i & 63, d = 4 * (i >> 6);
      t.k[d][k] = kr[j].x, t.k[d + 1][k] = kr[j].y, t.k[d + 2][k] = kr[j].z, t.k[d + 3][k] = kr[j].w;
      t.v[d][k] = vr[j].x, t.v[d + 1][k] = vr[j].y, t.v[d + 2][k] = vr[j].z, t.v[d + 3][k] = vr[j].w;
    }
    float s[4][4];
    const int kc = k0 + 4 * tx;
#pragma unroll
    for (int i = 0; i < 4; ++i) {                  // the pair bias starts the sum
      const int qi = q0 + 4 * ty + i;
      const float* b = bias + ((size_t)h * n + (qi < n ? qi : 0)) * n + kc;
      if ((n & 3) == 0 && kc < n) {
        const float4 b4 = __ldg(reinterpret_cast<const float4*>(b));
        s[i][0] = b4.x, s[i][1] = b4.y, s[i][2] = b4.z, s[i][3] = b4.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) s[i][e] = kc + e < n ? __ldg(b + e) : -INFINITY;
      }
    }
    named_barrier(1 + grp, 128);
    if (k0 + kSaK * kSaGroups < n) load_kv(k0 + kSaK * kSaGroups);
#pragma unroll
    for (int d = 0; d < kSd; ++d) {
      const float4 a = *reinterpret_cast<const float4*>(&qs[d][4 * ty]), b = *reinterpret_cast<const float4*>(&t.k[d][4 * tx]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[i][e] = fmaf(av[i], bv[e], s[i][e]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float mx = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      const float mn = fmaxf(m[i], mx), alpha = expf(m[i] - mn);
      m[i] = mn;
#pragma unroll
      for (int e = 0; e < 4; ++e) s[i][e] = expf(s[i][e] - mn);
      l[i] = l[i] * alpha + ((s[i][0] + s[i][1]) + (s[i][2] + s[i][3]));
      o[i][0] *= alpha, o[i][1] *= alpha, o[i][2] *= alpha;
      *reinterpret_cast<float4*>(&t.p[4 * ty + i][4 * tx]) = make_float4(s[i][0], s[i][1], s[i][2], s[i][3]);
    }
    __syncwarp();                                  // the 16 threads of four queries sit in one warp
#pragma unroll
    for (int k = 0; k < kSaK / 2; k += 4) {
      float4 p[4], w[3];
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(&t.p[4 * ty + i][32 * khalf + k]);
#pragma unroll
      for (int e = 0; e < 3; ++e) w[e] = *reinterpret_cast<const float4*>(&t.v[dg + e][32 * khalf + k]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 3; ++e)
          o[i][e] = fmaf(p[i].x, w[e].x, fmaf(p[i].y, w[e].y, fmaf(p[i].z, w[e].z, fmaf(p[i].w, w[e].w, o[i][e]))));
    }
    __syncwarp();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int x = 8; x > 0; x >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], x);
#pragma unroll
    for (int e = 0; e < 3; ++e) o[i][e] += __shfl_xor_sync(0xffffffffu, o[i][e], 8);
  }
  // group 1 hands its (m, l, o) to group 0 through its tile memory
  float* part = &reinterpret_cast<SaTile*>(sa_raw + kSd * kSaQ * 4)[1].p[0][0];
  __syncthreads();
  if (grp == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float* r = part + (4 * ty + i) * (kSd + 2);
      if (tx == 0) r[kSd] = m[i], r[kSd + 1] = l[i];
      if (khalf == 0) r[dg] = o[i][0], r[dg + 1] = o[i][1], r[dg + 2] = o[i][2];
    }
  }
  __syncthreads();
  if (grp != 0 || khalf != 0) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int qi = q0 + 4 * ty + i;
    if (qi >= n) continue;
    const float* r = part + (4 * ty + i) * (kSd + 2);
    const float mn = fmaxf(m[i], r[kSd]), a0 = expf(m[i] - mn), a1 = expf(r[kSd] - mn);   // m[0] is finite, m[1] may not be
    const float inv = 1.0f / (l[i] * a0 + r[kSd + 1] * a1);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      bf16 b[3];
      split3((o[i][e] * a0 + r[dg + e] * a1) * inv * __ldg(base + (size_t)qi * kSf + 3 * kSc + dg + e), b);
#pragma unroll
      for (int p = 0; p < 3; ++p) out[((size_t)p * n + qi) * kSc + h * kSd + dg + e] = b[p];
    }
  }
}

PX_DEFINE_FAMILY_HOOKS(single)

// Prepared weights: planes of [q|k|v|g] (1536 x 384), W_o (384 x 384), [a|b] interleaved (3072 x 384), W_out (384 x 1536)
constexpr int64_t kSwQkvg = 0, kSwO = kSwQkvg + 3ll * kSf * kSc, kSwAb = kSwO + 3ll * kSc * kSc,
                  kSwOut = kSwAb + 3ll * 2 * kSf * kSc, kSwEnd = kSwOut + 3ll * kSc * kSf;

template <int kMode, typename T>
static bool launch_split_gemm(const bf16* a, const bf16* w, int64_t w_rows, int64_t k, int split, SgArgs g, cudaStream_t st) {
  CUtensorMap ma, mw;
  if (!make_plane_map(&ma, a, g.rows, k, 128) || !make_plane_map(&mw, w, w_rows, k, kSgBN)) return false;
  constexpr size_t smem = (size_t)kSgStages * kSgStageBytes + sizeof(SgBars) + 1024;
  static_assert(smem <= 232448, "shared memory budget");
  static SmemLimit limit;
  if (!limit.set(split_gemm_tc_kernel<kMode, T>, smem)) return false;
  g.chunks = (int)(k / 64 / split);
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = (unsigned)split;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(w_rows / kSgBN), (unsigned)((g.rows + 127) / 128), (unsigned)split);
  cfg.blockDim = dim3(kSgThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = split > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, split_gemm_tc_kernel<kMode, T>, ma, mw, g) == cudaSuccess;
}

// The two parts of the branch: what needs s alone, and what needs the pair bias.
struct SingleWs {
  bf16* xp;        // [3][n][384]: LN(s), the attention's result, LN(s1)
  float* qkvg;     // [n][1536]; later the hidden planes [3][n][1536]
};
static SingleWs single_ws(void* ws, int n) { return {(bf16*)ws, (float*)((unsigned char*)ws + (size_t)3 * n * kSc * 2)}; }

template <typename T>
static int32_t single_project(const void* s, const bf16* w, const float* ln_w, const float* ln_b, const float* q_bias, void* ws, int n,
                              float eps, cudaStream_t st) {
  const SingleWs b = single_ws(ws, n);
  SgArgs g = {};
  g.rows = n;
  if (!launch_pdl(split_rows_kernel<T>, dim3((unsigned)((n + 3) / 4)), 128, 0, st, (const T*)s, ln_w, ln_b, b.xp, n, eps)) return PX_ERR_LAUNCH;
  g.bias = q_bias, g.out_f = b.qkvg, g.scale = 1.0f / sqrtf((float)kSd);
  return launch_split_gemm<kSgQkvg, T>(b.xp, w + kSwQkvg, kSf, kSc, 1, g, st) ? PX_OK : PX_ERR_LAUNCH;
}

template <typename T>
static int32_t single_finish(const void* s, void* s_out, const bf16* w, const float* ln_w, const float* ln_b, const float* bias, void* ws,
                             int n, float eps, cudaStream_t st) {
  const SingleWs b = single_ws(ws, n);
  SgArgs g = {};
  g.rows = n;
  constexpr int sa_smem = kSd * kSaQ * 4 + kSaGroups * (int)sizeof(SaTile);
  static SmemLimit limit;
  if (!limit.set(single_attention_kernel, sa_smem) ||
      !launch_pdl(single_attention_kernel, dim3((unsigned)((n + kSaQ - 1) / kSaQ), kSh), 128 * kSaGroups, sa_smem, st, b.qkvg, bias, b.xp, n))
    return PX_ERR_LAUNCH;
  g.res = s, g.out = s_out;
  if (!launch_split_gemm<kSgRes, T>(b.xp, w + kSwO, kSc, kSc, 2, g, st)) return PX_ERR_LAUNCH;
  if (!launch_pdl(split_rows_kernel<T>, dim3((unsigned)((n + 3) / 4)), 128, 0, st, (const T*)s_out, ln_w, ln_b, b.xp, n, eps))
    return PX_ERR_LAUNCH;
  g.out_planes = (bf16*)b.qkvg;
  if (!launch_split_gemm<kSgSwiglu, T>(b.xp, w + kSwAb, 2 * kSf, kSc, 1, g, st)) return PX_ERR_LAUNCH;
  g.res = s_out, g.out = s_out;
  return launch_split_gemm<kSgRes, T>((bf16*)b.qkvg, w + kSwOut, kSc, kSf, kSgSplit, g, st) ? PX_OK : PX_ERR_LAUNCH;
}

static bool single_args_ok(int64_t n, std::initializer_list<const void*> pointers) {
  uintptr_t bits = 0;
  for (const void* p : pointers) {
    if (!p) return false;
    bits |= (uintptr_t)p;
  }
  return n > 0 && n <= 32768 && !(bits & 15);
}

}  // namespace px

using namespace px;

extern "C" int64_t px_single_weights_bytes(void) { return kSwEnd * 2; }

extern "C" int64_t px_single_workspace_bytes(int64_t n) { return n <= 0 ? 0 : (3ll * kSc * 2 + 3ll * kSf * 2) * n; }

extern "C" int32_t px_single_prepare(const float* w_q, const float* w_k, const float* w_v, const float* w_g, const float* w_o,
                                     const float* w_a, const float* w_b, const float* w_out, void* prepared, void* stream) {
  if (!w_q || !w_k || !w_v || !w_g || !w_o || !w_a || !w_b || !w_out || !prepared || ((uintptr_t)prepared & 15))
    return PX_ERR_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  bf16* p = (bf16*)prepared;
  const float* qkvg[4] = {w_q, w_k, w_v, w_g};
  for (int i = 0; i < 4; ++i)
    split_weight_kernel<<<kSc, 128, 0, st>>>(qkvg[i], p + kSwQkvg, kSc, kSc, kSf, kSc, kSc, i * kSc);
  split_weight_kernel<<<kSc, 128, 0, st>>>(w_o, p + kSwO, kSc, kSc, kSc, kSc, kSc, 0);
  split_weight_kernel<<<kSf, 128, 0, st>>>(w_a, p + kSwAb, kSf, kSc, 2 * kSf, 32, 64, 0);
  split_weight_kernel<<<kSf, 128, 0, st>>>(w_b, p + kSwAb, kSf, kSc, 2 * kSf, 32, 64, 32);
  split_weight_kernel<<<kSc, 256, 0, st>>>(w_out, p + kSwOut, kSc, kSf, kSc, kSc, kSc, 0);
  return cudaGetLastError() == cudaSuccess ? PX_OK : PX_ERR_LAUNCH;
}

extern "C" int32_t px_single_project(const void* s, int32_t s_dtype, const void* prepared, const float* ln_att_w,
                                     const float* ln_att_b, const float* q_bias, void* workspace, int64_t workspace_bytes, int64_t n,
                                     float eps_att, void* stream) {
  if (!single_args_ok(n, {s, prepared, ln_att_w, ln_att_b, q_bias, workspace})) return PX_ERR_BAD_ARG;
  if (workspace_bytes < px_single_workspace_bytes(n)) return PX_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const bf16* w = (const bf16*)prepared;
  switch (s_dtype) {
    case PX_F32: return single_project<float>(s, w, ln_att_w, ln_att_b, q_bias, workspace, (int)n, eps_att, st);
    case PX_BF16: return single_project<bf16>(s, w, ln_att_w, ln_att_b, q_bias, workspace, (int)n, eps_att, st);
    case PX_F16: return single_project<__half>(s, w, ln_att_w, ln_att_b, q_bias, workspace, (int)n, eps_att, st);
    default: return PX_ERR_UNSUPPORTED;
  }
}

extern "C" int32_t px_single_finish(const void* s, void* s_out, int32_t s_dtype, const void* prepared, const float* ln_tr_w,
                                    const float* ln_tr_b, const float* pair_bias, void* workspace, int64_t workspace_bytes, int64_t n,
                                    float eps_tr, void* stream) {
  if (!single_args_ok(n, {s, s_out, prepared, ln_tr_w, ln_tr_b, pair_bias, workspace})) return PX_ERR_BAD_ARG;
  if (workspace_bytes < px_single_workspace_bytes(n)) return PX_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const bf16* w = (const bf16*)prepared;
  switch (s_dtype) {
    case PX_F32: return single_finish<float>(s, s_out, w, ln_tr_w, ln_tr_b, pair_bias, workspace, (int)n, eps_tr, st);
    case PX_BF16: return single_finish<bf16>(s, s_out, w, ln_tr_w, ln_tr_b, pair_bias, workspace, (int)n, eps_tr, st);
    case PX_F16: return single_finish<__half>(s, s_out, w, ln_tr_w, ln_tr_b, pair_bias, workspace, (int)n, eps_tr, st);
    default: return PX_ERR_UNSUPPORTED;
  }
}
