// Triangle attention core on the 5th-generation tensor cores (4 heads x 32).
//
//   o[u][q][h*32+d] = softmax_k( q[u,h,q,:] . k[u,h,k,:] + bias[h][q][k] + mask_bias[u][k] ) v[u,h,k,d]
//
// q, k, v and o are fp16 (projections of standardised rows and convex combinations of them: far inside its range;
// fp16 keeps three more bits than bf16), the pair bias, the logits, the softmax and the accumulators fp32.
//
// One CTA = (head h, 128 queries, 6 attended rows u; 3 for part of the last wave, then one row a group), 16 warps:
//   warps 0..11   three softmax groups of four warps; group g owns rows u0+2g, u0+2g+1, each thread one query row and
//                 the softmax denominator of it.  The pair bias does not depend on u: all six rows use the same tile.
//   warps 12..14  one control warp per group, whose elected lane issues.  It loads the group's Q tiles once
//                 and, per work item, a K tile [64 keys][32] (64-byte swizzle) and a transposed V tile
//                 [32 d][64 keys] (128-byte swizzle) into the group's 4-stage ring; copies the pair bias of the first 32
//                 keys into the group's S buffer in tensor memory and adds Q K^T (M=128, N=64, K=32) to it; and, once the
//                 group has written P (fp16) into its P buffer, issues O_u += P V with P as the TMEM-resident A operand
//                 (M=128, N=32, K=64).  S of the next item is issued as soon as the group has pulled the current S into
//                 registers, so it is ready when the group comes back.  The bias of the other 32 keys is added by the softmax
//                 threads, which leave zeros in those columns for the next product.
//   warp 15       loads the pair-bias tiles [128 q][64 k] fp32 (two 128-byte-swizzled boxes, 2-deep ring).
// Tensor memory: S (3 x 64) | P (3 x 32, two fp16 per column) | O (6 x 32).
//
// It runs beyond 1024 keys and where there are no more units (128 queries of a head x 6 rows) than SMs; in between, px_flash_units.cuh does the
// same with several units a CTA.  Figures from 129 to 1024 tokens in this file are from when this kernel ran there, too.
//
// What bounds it (per item of 128 queries x 64 keys, 770 cycles at N = 768): no unit alone, but the chain of a group's item.  Tensor
// pipe 416 (a copy of 8 columns takes 64 cycles, S 96, P V 64), special-function unit 384, issue slots 440; without any load of K, V
// and bias the time is the same.  So nothing waits on the chain that can wait beside it: the other half of the bias is fetched
// before S is waited for, and the store of the zeros is waited for behind the tile maximum (N = 200 30.5 -> 29.8 us, 384 110.2 -> 106.7,
// 768 677 -> 653, 1536 4.98 -> 4.80 ms; either alone less than 1 %).  Taken against the standing maximum before it is checked,
// the logits need fewer steps on the chain, but 709 us at N = 768; P handed over behind the loads of the next S 685; bias held for both rows 662.
// Hence, too, the bias split in halves: all 64 columns copied
// make the tensor pipe 80 % busy and S late (N = 384 118.7 us against 110.4, N = 1536 level), none copied is 48 more
// instructions of 400 per softmax thread (123.5, 5.61 ms against 5.06).  24 or 40 columns: as 32 within 1 %.  Writing the bias
// into S from the softmax threads for the next item: 5.32 ms (a store and its wait are on the group's chain).  Four groups of
// one row: 5.15 to 7.0 ms.  Exponentials without the cubic 5.52, every third pair 5.02, every second 5.26, a quartic 5.08.
//
// Softmax is online in base 2 with a lazy reference maximum: the reference only moves (and O_u is rescaled
// through TMEM) when the tile maximum exceeds it by more than 8, so probabilities stay below 2^8.
// Exponentials are fp32 (three pairs in four by ex2, the fourth by a cubic on the FMA pipe); P is their rounding to
// fp16, the denominators sum the fp32 values.  Every mbarrier wait is bounded.
#include <math_constants.h>

#include <type_traits>

#include "px_rowpipe.cuh"

namespace px {

constexpr int kFH = 4, kFD = 32;
constexpr int kFGroups = 3;               // softmax groups per CTA
constexpr int kFRpg = 2;                  // attended rows per group
constexpr int kFRows = kFGroups * kFRpg;  // attended rows per CTA
constexpr int kFKT = 64;                  // keys per work item
constexpr int kFCopied = 32;              // columns of S that are laid out with the pair bias before the product (a copy into tensor memory)
constexpr int kFStages = 4;               // K/V ring of each group (work items = (key tile, row))
constexpr int kFQBytes = 128 * 64;        // [128][32] fp16
constexpr int kFKBytes = kFKT * 64;       // [64][32] fp16
constexpr int kFVBox = 32 * 128;          // the TMA box of the value tile: 32 rows x 64 keys
constexpr int kFVBytes = 32 * 128;        // [32 d][64 keys] fp16
constexpr int kFStageBytes = kFKBytes + kFVBytes;
constexpr int kFBiasBytes = 128 * kFKT * 4;
constexpr int kFON = 32;                  // columns of an O accumulator
constexpr uint32_t kFCols = 512;
constexpr int kFColS = 0, kFColP = kFGroups * kFKT, kFColO = kFColP + kFGroups * (kFKT / 2);  // TMEM column map
constexpr float kRescaleGap = 8.0f;
constexpr int kFThreads = 32 * (4 * kFGroups + 4);
static_assert(kFColO + kFRows * kFON <= 512, "tensor memory budget");
static_assert(kFCopied == 32 && kFKT == 64, "the copied columns are one box of the bias tile, the others one store");

struct FlashBars {
  uint64_t q_full[kFGroups], kv_full[kFGroups][kFStages], bias_full[2], bias_empty[2], s_full[kFGroups],
      s_free[kFGroups], p_ready[kFGroups], pv_done[kFGroups];
  uint32_t tmem_base;
};

struct FlashLayout {
  static constexpr int q = 0;
  static constexpr int kv = q + kFRows * kFQBytes;
  static constexpr int bias = kv + kFGroups * kFStages * kFStageBytes;
  static constexpr int bars = bias + 2 * kFBiasBytes;
  static constexpr int total = bars + (int)sizeof(FlashBars);
};
static_assert(FlashLayout::kv % 1024 == 0 && FlashLayout::bias % 1024 == 0 && kFStageBytes % 1024 == 0, "swizzle alignment");

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// 2^x for two arguments on the FMA pipe (the special-function unit delivers 16 ex2 per clock and SM and is the
// busiest unit of this kernel): x = n + f with n = round(x) taken from the mantissa after adding 1.5 * 2^23,
// 2^f by a cubic on [-0.5, 0.5] (relative error 7.5e-5, below the fp16 rounding of P), 2^n added into the exponent
// field.  Arguments below -126 (masked or padded keys) give 2^-126.
constexpr int kFPolyEvery = 4;   // every fourth pair of exponentials takes this path
__device__ __forceinline__ void exp2_poly2(float x0, float x1, float& p0, float& p1) {
  constexpr float kMagic = 12582912.f;
  constexpr float c0 = 0.9999280571937561f, c1 = 0.6932610273361206f, c2 = 0.2426111102104187f, c3 = 0.05517144873738289f;
  x0 = fmaxf(x0, -126.f);
  x1 = fmaxf(x1, -126.f);
  float t0 = x0, t1 = x1;
  add2(t0, t1, kMagic, kMagic);
  float n0 = t0, n1 = t1;
  add2(n0, n1, -kMagic, -kMagic);
  float f0, f1, q0, q1;
  fma2(f0, f1, n0, n1, -1.f, -1.f, x0, x1);
  fma2(q0, q1, f0, f1, c3, c3, c2, c2);
  fma2(q0, q1, q0, q1, f0, f1, c1, c1);
  fma2(q0, q1, q0, q1, f0, f1, c0, c0);
  p0 = __int_as_float(__float_as_int(q0) + (__float_as_int(t0) << 23));
  p1 = __int_as_float(__float_as_int(q1) + (__float_as_int(t1) << 23));
}

// kHalves: the grid ends with CTAs of one row per group.  kBrief: the last key tile has 32 keys at most, its other half is left out.
template <bool kHalves, bool kBrief>
__global__ void __launch_bounds__(kFThreads, 1)
triatt_flash_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ CUtensorMap map_o, const float* __restrict__ mb,
                       int n_u, int n, int ldm, int nkt, int whole) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  FlashBars& bars = *reinterpret_cast<FlashBars*>(sm + FlashLayout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  // The last rows first: their q, k and v were written last and may still lie in L2.
  // kHalves: slices of the grid from `whole` on have one row per group, two of them share the rows of one (see px_triatt_flash).
  const int q0 = blockIdx.x * 128, h = blockIdx.y, behind = kHalves ? (int)blockIdx.z - whole : -1;
  const int halves = kHalves ? ((int)gridDim.z - whole) >> 1 : 0;
  const int u0 = !kHalves ? (gridDim.z - 1 - blockIdx.z) * kFRows
                 : behind < 0 ? (halves - 1 - behind) * kFRows : halves * kFRows - (behind + 1) * kFGroups;
  if (kHalves && u0 >= n_u) return;      // the second half of the last rows, where they are three at most

  const bool skip = cta_begin();         // an earlier bounded wait gave up: do not start new work
  if (threadIdx.x == 32) prefetch_maps(map_q, map_k, map_v, map_b, map_o);
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars.bias_full[b], 1);
      mbar_init(&bars.bias_empty[b], 5 * kFGroups);     // four softmax warps and the copies of each group
    }
    for (int g = 0; g < kFGroups; ++g) {
      mbar_init(&bars.q_full[g], 1);
      for (int s = 0; s < kFStages; ++s) mbar_init(&bars.kv_full[g][s], 1);
      mbar_init(&bars.s_full[g], 1);
      mbar_init(&bars.s_free[g], 4);
      mbar_init(&bars.p_ready[g], 4);
      mbar_init(&bars.pv_done[g], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 4 * kFGroups) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&bars.tmem_base)),
                 "r"(kFCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (!cta_ready(skip, warp == 4 * kFGroups, bars.tmem_base, kFCols)) return;
  const uint32_t tmem_base = bars.tmem_base;

  const auto rows = [&](auto per_group) {
  constexpr int kRpg = decltype(per_group)::value;     // attended rows per group
  if (warp >= 4 * kFGroups) {
    // ------------------------------------------------------------------ control warp of group g
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n");   // registers go to the softmax warpgroups
    const int g = warp - 4 * kFGroups;
    if (g == kFGroups) {
      // ---------------------------------------------------------------- pair-bias loader (all six rows share a tile)
      for (int kt = 0; kt < nkt; ++kt) {
        const int b = kt & 1;
        if (!mbar_wait_warp(&bars.bias_empty[b], ((kt >> 1) & 1) ^ 1, 1u)) break;
        // the first tile does not share its way with the second: -0.4 % from N = 384 on
        if (kt == 1 && !mbar_wait_warp(&bars.bias_full[0], 0, 1u)) break;
        if (elect_lane()) {
          mbar_expect_tx(&bars.bias_full[b], kFBiasBytes);
          for (int c = 0; c < kFKT / 32; ++c)
            tma_load_3d(smem_u32(sm + FlashLayout::bias + b * kFBiasBytes + c * (128 * 128)), &map_b, &bars.bias_full[b],
                        kt * kFKT + c * 32, q0, h);
        }
        __syncwarp();
      }
    } else {
      constexpr uint32_t idesc_s = umma_idesc_f16(128, kFKT), idesc_o = umma_idesc_f16(128, kFON);
      const int n_items = nkt * kRpg;              // work item i = (key tile i / 2, row i % 2 of the group)
      const uint32_t q_addr = smem_u32(sm + FlashLayout::q + g * kRpg * kFQBytes);
      const uint32_t ring = smem_u32(sm + FlashLayout::kv + g * kFStages * kFStageBytes);
      const uint32_t d_s = tmem_base + kFColS + kFKT * g, d_p = tmem_base + kFColP + (kFKT / 2) * g;
      const uint32_t d_o = tmem_base + kFColO + kFON * kRpg * g;
      const int uh0 = (u0 + g * kRpg) * kFH + h;   // rows past n_u: coordinate beyond the tensor -> zero fill
      auto load_kv = [&](int i) {                   // K and V tiles of item i into stage i % kFStages (one lane)
        const int s = i % kFStages, kt = i / kRpg, uh = uh0 + (i % kRpg) * kFH;
        mbar_expect_tx(&bars.kv_full[g][s], kFKBytes + kFVBox);
        tma_load_3d(ring + s * kFStageBytes, &map_k, &bars.kv_full[g][s], 0, kt * kFKT, uh);
        tma_load_3d(ring + s * kFStageBytes + kFKBytes, &map_v, &bars.kv_full[g][s], kt * kFKT, 0, uh);
      };
      auto issue_s = [&](int i) {                   // S(i) = bias + Q_r K^T
        const int s = i % kFStages, kt = i / kRpg, r = i % kRpg;
        if (r == 0 && !mbar_wait_warp(&bars.bias_full[kt & 1], (kt >> 1) & 1, 64u)) return false;
        if (!mbar_wait_warp(&bars.kv_full[g][s], (i / kFStages) & 1, 8u)) return false;
        tc_fence_after();
        if (elect_lane()) {
          const uint32_t tile = smem_u32(sm + FlashLayout::bias + (kt & 1) * kFBiasBytes);
#pragma unroll
          for (int c = 0; c < kFCopied / 8; ++c)    // 32 bytes (8 columns) of the 128-byte rows of the tile's first box
            tmem_copy_128x256b(d_s + 8 * c, umma_desc_sw128(tile) + 2 * c);
          const uint64_t dq = umma_desc_sw64(q_addr + r * kFQBytes), dk = umma_desc_sw64(ring + s * kFStageBytes);
          umma_bf16(d_s, dq, dk, idesc_s, 1u);
          umma_bf16(d_s, dq + 2, dk + 2, idesc_s, 1u);
          umma_commit(&bars.s_full[g]);
          if (r == kRpg - 1) umma_commit(&bars.bias_empty[kt & 1]);   // this group is done with the bias tile
        }
        __syncwarp();
        return true;
      };
      if (elect_lane()) {
        mbar_expect_tx(&bars.q_full[g], kRpg * kFQBytes);
        for (int r = 0; r < kRpg; ++r) tma_load_3d(q_addr + r * kFQBytes, &map_q, &bars.q_full[g], 0, q0, uh0 + r * kFH);
        for (int i = 0; i < kFStages - 1 && i < n_items; ++i) load_kv(i);   // first use of these stages
      }
      __syncwarp();
      bool ok = mbar_wait_warp(&bars.q_full[g], 0, 4u) && mbar_wait_warp(&bars.s_free[g], 0, 2u) && issue_s(0);
      for (int i = 0; i < n_items && ok; ++i) {
        const int kt = i / kRpg, r = i % kRpg;
        if (i + 1 < n_items) {                      // next S as soon as the group holds the current one in registers
          ok = mbar_wait_warp(&bars.s_free[g], (i + 1) & 1, 2u) && issue_s(i + 1);
          if (!ok) break;
        }
        if (i + kFStages - 1 < n_items) {           // refill: that stage was last read by P.V of item i-1
          if (i >= 1) ok = mbar_wait_warp(&bars.pv_done[g], (i - 1) & 1, 32u);
          if (!ok) break;
          if (elect_lane()) load_kv(i + kFStages - 1);
          __syncwarp();
        }
        ok = mbar_wait_warp(&bars.p_ready[g], i & 1, 16u);
        if (!ok) break;
        tc_fence_after();
        if (elect_lane()) {
          const uint64_t dv = umma_desc_sw128(ring + (i % kFStages) * kFStageBytes + kFKBytes);
#pragma unroll
          for (int ks = 0; ks < kFKT / 16; ++ks) {  // 16 keys per step: 8 TMEM columns of P, 32 bytes of the value rows
            if (kBrief && ks == kFKT / 32 && kt == nkt - 1) break;
            umma_bf16_ts(d_o + kFON * r, d_p + 8 * ks, dv + 2 * ks, idesc_o, (kt | ks) ? 1u : 0u);
          }
          umma_commit(&bars.pv_done[g]);
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax groups
    asm volatile("setmaxnreg.inc.sync.aligned.u32 160;\n");
    const int g = warp >> 2, qw = warp & 3;
    const int row = 32 * qw + lane;                 // query row inside the tile = TMEM lane
    const uint32_t lane_addr = (uint32_t)(32 * qw) << 16;
    const uint32_t t_s = tmem_base + lane_addr + kFColS + kFKT * g;
    const uint32_t t_p = tmem_base + lane_addr + kFColP + (kFKT / 2) * g;
    const uint32_t t_o = tmem_base + lane_addr + kFColO + kFON * kRpg * g;
    const int ug = u0 + kRpg * g;                  // first row of this group
    unsigned long long flag_word[kRpg];            // bit kt & 63: some key of tile kt has a mask bias other than zero
    float m_ref[kRpg], l_sum[kRpg];             // reference maximum and denominator of this thread's query per row
#pragma unroll
    for (int r = 0; r < kRpg; ++r) {
      flag_word[r] = 0;
      m_ref[r] = -CUDART_INF_F;
      l_sum[r] = 0.f;
    }
    // the product adds to what S holds: the columns without the bias start from zero (the store is waited for by the caller)
    auto clear_rest = [&] {
      uint32_t zero[kFKT - kFCopied];
#pragma unroll
      for (int e = 0; e < kFKT - kFCopied; ++e) zero[e] = 0u;
      tmem_st32(t_s + kFCopied, zero);
    };
    clear_rest();
    tmem_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&bars.s_free[g]);
    const auto mask_flags = [&](int kt) {
      if ((kt & 63) == 0) {
        for (int r = 0; r < kRpg; ++r) flag_word[r] = 0;
        // A load covers two tiles (ldm is a multiple of 128), eight are in flight beside the first TMA loads and products (two
        // in flight: 6.17 ms at N = 1536, against 5.88).  As a kernel of its own this cost a launch: 16.6 us together at
        // N = 128 against 12.6, 143 against 136 at N = 384.
        const int left = min(nkt - kt, 64);
#pragma unroll 1
        for (int t0 = 0; t0 < left; t0 += 8) {
          float4 m4[kRpg][4];
#pragma unroll
          for (int r = 0; r < kRpg; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              m4[r][j] = t0 + 2 * j < left ? __ldg(reinterpret_cast<const float4*>(mb + (size_t)((ug + r < n_u) ? ug + r : 0) * ldm +
                                                                                   (kt + t0 + 2 * j) * kFKT) + lane)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int r = 0; r < kRpg; ++r) {
            unsigned bits = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const unsigned b = __ballot_sync(0xffffffffu, m4[r][j].x != 0.f || m4[r][j].y != 0.f || m4[r][j].z != 0.f || m4[r][j].w != 0.f);
              bits |= (((b & 0xffffu) ? 1u : 0u) | ((b >> 16) ? 2u : 0u)) << (2 * j);
            }
            flag_word[r] |= (unsigned long long)bits << t0;
          }
        }
      }
    };
    // The items of key tile kt, of which the first `keys` exist: 64, or 32 where a last tile has no more.
    const auto items = [&](int kt, auto keys) {
      constexpr int kKeys = decltype(keys)::value;
#pragma unroll
      for (int r = 0; r < kRpg; ++r) {
        const int i = kt * kRpg + r;               // this group's work item
        // a wait that gave up is voted on once per item, below: what is computed till then goes nowhere
        bool ok = r == 0 ? mbar_wait(&bars.bias_full[kt & 1], (kt >> 1) & 1, 64u) : true;
        // The pair bias of the columns that were not copied (128-byte rows, 16-byte pieces swizzled by row) is fetched before S is waited
        // for, so that it is at hand when S comes.
        float4 b4[(kFKT - kFCopied) / 4];
        const float* brow = reinterpret_cast<const float*>(sm + FlashLayout::bias + (kt & 1) * kFBiasBytes) + row * 32;
#pragma unroll
        for (int c = kFCopied / 4; c < kKeys / 4; ++c)
          b4[c - kFCopied / 4] = *reinterpret_cast<const float4*>(brow + (c >> 3) * (128 * 32) + (((c & 7) ^ (row & 7)) << 2));
        ok = mbar_wait(&bars.s_full[g], i & 1, 128u) && ok;
        __syncwarp();
        tc_fence_after();
        float s[kKeys];
#pragma unroll
        for (int c = kKeys - 32; c >= 0; c -= 32) {  // the zeros are stored while the first half is on its way
          tmem_ld32(t_s + c, *reinterpret_cast<uint32_t(*)[32]>(&s[c]));
          tmem_wait_ld();
          if (kKeys == kFKT && c) clear_rest();      // (a tile of 32 keys is the last)
        }
#pragma unroll
        for (int c = kFCopied / 4; c < kKeys / 4; ++c) {
          add2(s[4 * c + 0], s[4 * c + 1], b4[c - kFCopied / 4].x, b4[c - kFCopied / 4].y);
          add2(s[4 * c + 2], s[4 * c + 3], b4[c - kFCopied / 4].z, b4[c - kFCopied / 4].w);
        }
        if ((flag_word[r] >> (kt & 63)) & 1ull) {     // warp-uniform
          const int u = (ug + r < n_u) ? ug + r : 0;
          const float4* mrow = reinterpret_cast<const float4*>(mb + (size_t)u * ldm + kt * kFKT);
#pragma unroll
          for (int c4 = 0; c4 < kKeys / 4; ++c4) {
            const float4 m4 = __ldg(mrow + c4);
            add2(s[4 * c4 + 0], s[4 * c4 + 1], m4.x, m4.y);
            add2(s[4 * c4 + 2], s[4 * c4 + 3], m4.z, m4.w);
          }
        }
        // tile maximum: independent chains of 16, so the reduction costs about 8 dependent steps
        float mq[kKeys / 16];
#pragma unroll
        for (int c = 0; c < kKeys / 16; ++c) {
          mq[c] = max3(s[16 * c], s[16 * c + 1], s[16 * c + 2]);
#pragma unroll
          for (int e = 3; e + 1 < 16; e += 2) mq[c] = max3(mq[c], s[16 * c + e], s[16 * c + e + 1]);
          mq[c] = fmaxf(mq[c], s[16 * c + 15]);
        }
        float mt = fmaxf(mq[0], mq[1]);
        if constexpr (kKeys == 64) mt = fmaxf(mt, fmaxf(mq[2], mq[3]));
        // S is in registers and its columns are zero again: the next S may be computed.  Said only here, when the store of the zeros has long
        // arrived, so that nobody waits for it; the next S has the time of the exponentials to come.
        if (kKeys == kFKT) tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.s_free[g]);
        // Does the reference maximum have to move?  Rare after the first tiles.  The exponentials need only this thread's own answer;
        // the warp's (tensor memory is rescaled by whole warps) is asked for beside them.
        const bool up = mt > m_ref[r] + kRescaleGap;
        const bool move = __any_sync(0xffffffffu, up) && kt > 0;     // first tile: the P.V product overwrites O
        const float m_old = m_ref[r];
        m_ref[r] = up ? mt : m_old;
        uint32_t w[kKeys / 2];
        float l0 = 0.f, l1 = 0.f;
        {
          const float nm = -m_ref[r];
#pragma unroll
          for (int e = 0; e < kKeys / 2; ++e) {
            // fp32 exponentials; P is their rounding to nearest fp16 (one conversion per pair), which is unbiased,
            // so the denominator can sum the fp32 values themselves.
            add2(s[2 * e], s[2 * e + 1], nm, nm);
            float p0, p1;
            if (e % kFPolyEvery == kFPolyEvery - 1) {
              exp2_poly2(s[2 * e], s[2 * e + 1], p0, p1);
            } else {
              p0 = fast_exp2(s[2 * e]);
              p1 = fast_exp2(s[2 * e + 1]);
            }
            w[e] = pack_f16x2(p0, p1);
            add2(l0, l1, p0, p1);
          }
        }
        // P.V of the previous item must be through before O is rescaled or the P buffer overwritten
        if (i >= 1) ok = mbar_wait(&bars.pv_done[g], (i - 1) & 1, 256u) && ok;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) return false;
        tc_fence_after();
        if (move) {
          const float alpha = fast_exp2(m_old - m_ref[r]);
          l_sum[r] *= alpha;
#pragma unroll
          for (int c = 0; c < kFON / 16; ++c) {
            uint32_t a[16];
            tmem_ld16(t_o + kFON * r + 16 * c, a);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) a[e] = __float_as_uint(__uint_as_float(a[e]) * alpha);
            tmem_st16(t_o + kFON * r + 16 * c, a);
          }
        }
        l_sum[r] += l0 + l1;
        if constexpr (kKeys == 64)
          tmem_st32(t_p, w);
        else
          tmem_st16(t_p, w);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bars.p_ready[g]);
          // Done with the bias tile.  Only here, where every value read from it has been used: signalled right behind the loads, while
          // these were generic ones, the next tile now and then overtook them (one row in 10^8 wrong).
          if (r == kRpg - 1) mbar_arrive(&bars.bias_empty[kt & 1]);
        }
      }
      return true;
    };
    bool ok = true;
    for (int kt = 0; kt < nkt - (kBrief ? 1 : 0) && ok; ++kt) {
      mask_flags(kt);
      ok = items(kt, std::integral_constant<int, kFKT>{});
    }
    if (kBrief && ok) {
      mask_flags(nkt - 1);
      ok = items(nkt - 1, std::integral_constant<int, kFKT / 2>{});
    }
    // ---- epilogue: o = O / denominator for this group's rows
    ok = ok && mbar_wait(&bars.pv_done[g], (nkt * kRpg - 1) & 1, 512u);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      // the rows leave by TMA from the place of their queries, which every product has read: a warp's 32 queries of one row are
      // 2 KB there (64-byte swizzle).  Written by their threads, 16 bytes at 256-byte distances, they took 4 % of the kernel at
      // N = 384 (135 us against 129) and 1.6 % at N = 1536 (5.89 ms against 5.79).
#pragma unroll
      for (int r = 0; r < kRpg; ++r) {
        uint32_t a[32];
        tmem_ld32(t_o + kFON * r, a);
        tmem_wait_ld();
        unsigned char* tile = sm + FlashLayout::q + (g * kRpg + r) * kFQBytes;
        const float inv = 1.0f / l_sum[r];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint4 pk;
          pk.x = pack_f16x2(__uint_as_float(a[8 * v + 0]) * inv, __uint_as_float(a[8 * v + 1]) * inv);
          pk.y = pack_f16x2(__uint_as_float(a[8 * v + 2]) * inv, __uint_as_float(a[8 * v + 3]) * inv);
          pk.z = pack_f16x2(__uint_as_float(a[8 * v + 4]) * inv, __uint_as_float(a[8 * v + 5]) * inv);
          pk.w = pack_f16x2(__uint_as_float(a[8 * v + 6]) * inv, __uint_as_float(a[8 * v + 7]) * inv);
          *reinterpret_cast<uint4*>(tile + row * 64 + ((v ^ ((row >> 1) & 3)) << 4)) = pk;
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0 && ug + r < n_u && q0 + 32 * qw < n) {
          tma_store_3d(&map_o, smem_u32(tile + 32 * qw * 64), h * kFD, q0 + 32 * qw, ug + r);
          tma_store_commit();
        }
      }
      if (lane == 0) tma_store_wait_read<0>();
    }
  }
  };
  if (kHalves && behind >= 0)
    rows(std::integral_constant<int, 1>{});
  else
    rows(std::integral_constant<int, kFRpg>{});

  tc_fence_before();
  cta_teardown_sync();
  if (warp == 4 * kFGroups) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kFCols) : "memory");
  }
}

}  // namespace px

#include "px_flash_units.cuh"

namespace px {

PX_DEFINE_FAMILY_HOOKS(flash)

}  // namespace px

using namespace px;

extern "C" int64_t px_ld_mask(int64_t n) { return (n + 127) / 128 * 128; }

extern "C" int32_t px_triatt_flash(const px_f16* q, const px_f16* k, const px_f16* v, const float* bias,
                                   const float* mask_bias, px_f16* o, int64_t n_u, int64_t n,
                                   int64_t ldm, void* stream) {
  if (!q || !k || !v || !bias || !mask_bias || !o || n_u <= 0 || n <= 0 || n_u > 32768 || n > 32768 ||
      ldm != px_ld_mask(n))
    return PX_ERR_BAD_ARG;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)bias | (uintptr_t)mask_bias | (uintptr_t)o) & 15)
    return PX_ERR_BAD_ARG;
  const int64_t ldt = px_ld(n);
  const int nkt = (int)((n + kFKT - 1) / kFKT);
  CUtensorMap mq, mk, mv, mbias, mo;
  const uint64_t uh = (uint64_t)n_u * kFH;
  // q, k: [n_u*4][n][32] fp16, box [1][128][32], 64-byte swizzle
  if (!make_map_3d(&mq, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, q, kFD, (uint64_t)n, uh, kFD * 2, (uint64_t)n * kFD * 2, kFD,
                   128, CU_TENSOR_MAP_SWIZZLE_64B) ||
      !make_map_3d(&mk, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, k, kFD, (uint64_t)n, uh, kFD * 2, (uint64_t)n * kFD * 2, kFD,
                   kFKT, CU_TENSOR_MAP_SWIZZLE_64B) ||
      // v (transposed): [n_u*4][32][n keys, row stride ldt] fp16, box [1][32][64], 128-byte swizzle
      !make_map_3d(&mv, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, v, (uint64_t)n, kFD, uh, (uint64_t)ldt * 2,
                   (uint64_t)kFD * ldt * 2, 64, kFD, CU_TENSOR_MAP_SWIZZLE_128B) ||
      // pair bias: [4][n q][n k, row stride ldm] fp32, box [1][128][32], 128-byte swizzle
      !make_map_3d(&mbias, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, bias, (uint64_t)n, (uint64_t)n, kFH, (uint64_t)ldm * 4,
                   (uint64_t)n * ldm * 4, 32, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
      // o: [n_u][n][128] fp16, box [1][32][32], 64-byte swizzle
      !make_map_3d(&mo, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, o, kC, (uint64_t)n, (uint64_t)n_u, kC * 2, (uint64_t)n * kC * 2, kFD, 32,
                   CU_TENSOR_MAP_SWIZZLE_64B))
    return PX_ERR_LAUNCH;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = FlashLayout::total + 1024;
  // CTAs of six rows (two a group); where what is left of them for the last wave fits the SMs twice, that in CTAs of three (one a
  // group; whole slices of the grid), so that the wave ends in little more than half the time: N = 100 10.2 -> 7.8 us and, one unit a CTA as
  // well, 160 23.9 -> 20.8, 256 41.5 -> 37.6, 384 106.4 -> 101.6, 512 218.5 -> 213.  CTAs of three only: 384 125, 768 805 against 653.  Each
  // number of rows has its own code (as a run-time number, which leaves no parity known to the compiler, 15 % slower).
  const int64_t per = (n + 127) / 128 * kFH, slices = (n_u + kFRows - 1) / kFRows, room = sm_count(), left = per * slices % room;
  const int64_t halves = 2 * left <= room ? (left + per - 1) / per : 0, whole = slices - halves;
  // A last key tile of 32 keys at most is worked off by its half, in kernels of their own (the branch costs the others 1 %): N = 150
  // 20.6 -> 19.2 us, 200 29.8 -> 28.1, 224 36.1 -> 34.1, 528 298 -> 291 (one unit a CTA), 1056 1824 -> 1812, 1300 level.
  const bool brief = (n - 1) % kFKT < kFKT / 2;
  // Up to 1024 keys CTAs work on several units; with more, a unit is so long that its beginning and end do not pay for the slower items.  How
  // many units an SM gets makes no difference.  One unit a CTA | several, us, rows x keys: 160 x 160 19.1 | 17.1, 384 x 384 98.7 | 92.4, 2000 x 384
  // 468 | 427, 7000 x 150 630 | 512, 768 x 768 631 | 628, 96 x 768 95.8 | 96.0, 3000 x 768 2564 | 2493, 1024 x 1024 1474 | 1460, 128 x 1024
  // 207 | 207, 2000 x 1024 3010 | 2984; 1088 x 1088 1856 | 1889, 137 x 1100 264 | 273, 1100 x 1100 1931 | 1988, 1300 x 1300 3311 | 3418, 96 x 1536
  // 318 | 326, 192 x 1536 614 | 615, 384 x 1536 1171 | 1195, 1536 x 1536 4824 | 5053, 256 x 2048 1467 | 1514, 512 x 2048 2973 | 3110.
  const int64_t units = per * slices;
  if (units > room && n <= 1024) {
    const int64_t halved = 2 * left <= room ? left : 0;
    const auto kernel = halved ? (brief ? triatt_flash_units_tc_kernel<true, true> : triatt_flash_units_tc_kernel<true, false>)
                               : (brief ? triatt_flash_units_tc_kernel<false, true> : triatt_flash_units_tc_kernel<false, false>);
    constexpr size_t bytes = FlashUnitLayout::total + 1024;
    static SmemLimit limit[4];
    if (!limit[2 * (halved > 0) + brief].set(kernel, bytes)) return PX_ERR_LAUNCH;
    return launch_pdl(kernel, dim3((unsigned)room), kFThreads, bytes, st, mq, mk, mv, mbias, mo, mask_bias, (int)n_u, (int)n, (int)ldm, nkt,
                      (int)(units - halved), (int)halved)
               ? PX_OK
               : PX_ERR_LAUNCH;
  }
  const auto kernel = halves ? (brief ? triatt_flash_tc_kernel<true, true> : triatt_flash_tc_kernel<true, false>)
                             : (brief ? triatt_flash_tc_kernel<false, true> : triatt_flash_tc_kernel<false, false>);
  static SmemLimit limit[4];
  if (!limit[2 * (halves > 0) + brief].set(kernel, smem)) return PX_ERR_LAUNCH;
  return launch_pdl(kernel, dim3((unsigned)((n + 127) / 128), kFH, (unsigned)(whole + 2 * halves)), kFThreads, smem, st, mq, mk, mv, mbias,
                    mo, mask_bias, (int)n_u, (int)n, (int)ldm, nkt, (int)whole)
             ? PX_OK
             : PX_ERR_LAUNCH;
}
