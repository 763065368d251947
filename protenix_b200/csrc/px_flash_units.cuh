// The attention core of flash_tcgen05.cu with CTAs that work on several units (128 queries of a head x 6 rows) one after the other: roles,
// work items, tensor memory and arithmetic are the same, and so are the results, to the bit.
//
// A CTA's beginning and end (set-up, queries and first tiles on their way, the last product, the rows on theirs, its successor's launch)
// take 4 to 5 us, as long as five items.  Here the next unit's queries are asked for when the last S of this one is there, its first K, V
// and bias tiles while its last items are worked on, and the rows of O leave through a staging area of their own, one row a group; to make
// room for it the K/V ring has three stages.  Groups go on to the next unit each by itself.
// Alone, us, one unit a CTA | this: N = 160 19.3 | 17.3, 200 28.1 | 26.4, 256 37.3 | 34.0, 300 72.2 | 64.9, 384 101.5 | 93.3, 437 161 | 154,
// 512 213 | 205, 768 650 | 631, 1024 1471 | 1466; beyond, its items take 3 % longer (more state beside the logits) and the one with a unit a CTA
// is launched (figures at the rule, px_triatt_flash).  Flags of 32 tiles at a time in place of 64 gave 1 to 2 % with the coordinates worked out
// anew for the rows of O; kept instead, as they are now, 0.5 % (N = 437 154.3 -> 153.1, 512 208.4 -> 207.4).  Runs of neighbouring units per CTA
// in place of every 148th: 693 at N = 768 (K and V are not shared in L2); rings of three K and four V tiles with barriers of their own: 655.
// The control warps' first unit taken as a whole one, as it always is, in place of the test for it: 1.5 % slower at 96 rows of 768.
#pragma once

namespace px {

constexpr int kFuStages = 3;

struct FlashUnitBars {
  uint64_t q_full[kFGroups], kv_full[kFGroups][kFuStages], bias_full[2], bias_empty[2], s_full[kFGroups], s_free[kFGroups],
      p_ready[kFGroups], pv_done[kFGroups];
  uint32_t tmem_base;
};
struct FlashUnitLayout {
  static constexpr int q = 0;
  static constexpr int kv = q + kFRows * kFQBytes;
  static constexpr int bias = kv + kFGroups * kFuStages * kFStageBytes;
  static constexpr int out = bias + 2 * kFBiasBytes;          // one row of O per group on its way out
  static constexpr int bars = out + kFGroups * kFQBytes;
  static constexpr int total = bars + (int)sizeof(FlashUnitBars);
};
static_assert(FlashUnitLayout::kv % 1024 == 0 && FlashUnitLayout::bias % 1024 == 0 && FlashUnitLayout::out % 1024 == 0, "swizzle alignment");
static_assert(FlashUnitLayout::total + 1024 <= 232448, "shared memory budget");

// What a CTA works on: 128 queries of a head, and rows u0 .. of one or two per group.
struct FlashUnit {
  int q0, h, u0;
};
// Units 0 .. whole - 1 are worked on whole, at least one by every CTA (whole >= gridDim.x).  kHalves: `halves` more are shared by two CTAs each,
// one row per group.  kBrief: the last key tile has 32 keys at most, its other half is left out.
template <bool kHalves, bool kBrief>
__global__ void __launch_bounds__(kFThreads, 1)
triatt_flash_units_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                       const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ CUtensorMap map_o, const float* __restrict__ mb,
                       int n_u, int n, int ldm, int nkt, int whole, int halves) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  FlashUnitBars& bars = *reinterpret_cast<FlashUnitBars*>(sm + FlashUnitLayout::bars);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int tiles_q = (n + 127) / 128, chunks = (n_u + kFRows - 1) / kFRows;
  // Unit `unit`, or the first or second three rows of it.  The last rows first: their q, k and v were written last and may still lie in L2.
  const auto unit_at = [&](int unit, int second) {
    const int rest = unit / tiles_q;
    return FlashUnit{(unit - rest * tiles_q) * 128, rest % kFH, (chunks - 1 - rest / kFH) * kFRows + (second ? kFGroups : 0)};
  };
  // this CTA's half unit, if it has one (the second half of the last rows may not exist)
  const int half_unit = whole + ((int)blockIdx.x >> 1), second = blockIdx.x & 1;
  const bool has_half = kHalves && (int)blockIdx.x < 2 * halves && unit_at(half_unit, second).u0 < n_u;

  const bool skip = cta_begin();         // an earlier bounded wait gave up: do not start new work
  if (threadIdx.x == 32) prefetch_maps(map_q, map_k, map_v, map_b, map_o);
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars.bias_full[b], 1);
      mbar_init(&bars.bias_empty[b], 5 * kFGroups);     // four softmax warps and the copies of each group
    }
    for (int g = 0; g < kFGroups; ++g) {
      mbar_init(&bars.q_full[g], 1);
      for (int s = 0; s < kFuStages; ++s) mbar_init(&bars.kv_full[g][s], 1);
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

  if (warp >= 4 * kFGroups) {
    // ------------------------------------------------------------------ control warp of group g
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;\n");   // registers go to the softmax warpgroups
    const int g = warp - 4 * kFGroups;
    if (g == kFGroups) {
      // ---------------------------------------------------------------- pair-bias loader (all rows of a unit share a tile)
      int t = 0;                                      // bias tiles so far
      bool ok = true;
      const auto tiles = [&](const FlashUnit& w) {
        for (int kt = 0; kt < nkt; ++kt, ++t) {
          const int b = t & 1;
          if (!mbar_wait_warp(&bars.bias_empty[b], ((t >> 1) & 1) ^ 1, 1u)) return false;
          // the first tile does not share its way with the second: -0.4 % from N = 384 on
          if (t == 1 && !mbar_wait_warp(&bars.bias_full[0], 0, 1u)) return false;
          if (elect_lane()) {
            mbar_expect_tx(&bars.bias_full[b], kFBiasBytes);
            for (int c = 0; c < kFKT / 32; ++c)
              tma_load_3d(smem_u32(sm + FlashUnitLayout::bias + b * kFBiasBytes + c * (128 * 128)), &map_b, &bars.bias_full[b],
                          kt * kFKT + c * 32, w.q0, w.h);
          }
          __syncwarp();
        }
        return true;
      };
      for (int unit = blockIdx.x; unit < whole && ok; unit += gridDim.x) ok = tiles(unit_at(unit, 0));
      if (has_half && ok) tiles(unit_at(half_unit, second));
    } else {
      constexpr uint32_t idesc_s = umma_idesc_f16(128, kFKT), idesc_o = umma_idesc_f16(128, kFON);
      const uint32_t ring = smem_u32(sm + FlashUnitLayout::kv + g * kFuStages * kFStageBytes);
      const uint32_t q_base = smem_u32(sm + FlashUnitLayout::q);
      const uint32_t d_s = tmem_base + kFColS + kFKT * g, d_p = tmem_base + kFColP + (kFKT / 2) * g;
      int done = 0, tiles = 0, units = 0;           // items, bias tiles and units before this one
      int stage = 0;                                // ring stage of the item at hand, counted on from item to item (a division is on
      uint32_t round = 0;                           // the way of every product) with the parity of its use
      // K and V tiles of work item i = (key tile i / rpg, row i % rpg of the group) of a unit into stage `s` (one lane); rows past
      // n_u: coordinate beyond the tensor -> zero fill
      auto load_kv = [&](const FlashUnit& w, int rpg, int i, int s) {
        const int kt = rpg == 2 ? i >> 1 : i, uh = (w.u0 + g * rpg + (rpg == 2 ? i & 1 : 0)) * kFH + w.h;
        mbar_expect_tx(&bars.kv_full[g][s], kFKBytes + kFVBox);
        tma_load_3d(ring + s * kFStageBytes, &map_k, &bars.kv_full[g][s], 0, kt * kFKT, uh);
        tma_load_3d(ring + s * kFStageBytes + kFKBytes, &map_v, &bars.kv_full[g][s], kt * kFKT, 0, uh);
      };
      auto load_q = [&](const FlashUnit& w, int rpg) {
        mbar_expect_tx(&bars.q_full[g], rpg * kFQBytes);
        for (int r = 0; r < rpg; ++r)
          tma_load_3d(q_base + (g * kFRpg + r) * kFQBytes, &map_q, &bars.q_full[g], 0, w.q0, (w.u0 + g * rpg + r) * kFH + w.h);
      };
      // The products of a unit; its Q and first K and V tiles have been asked for, those of the next unit (nrpg rows a group, 0: none) are
      // while this one's last items are worked on.
      auto products = [&](auto per_group, const FlashUnit& w, const FlashUnit& nw, int nrpg) {
        constexpr int kRpg = decltype(per_group)::value;
        const int n_items = nkt * kRpg;
        // a group keeps its places for queries and O whatever the unit: the others may still be at the unit before
        const uint32_t q_addr = q_base + g * kFRpg * kFQBytes, d_o = tmem_base + kFColO + kFON * kFRpg * g;
        auto issue_s = [&](int i, int s, uint32_t parity) {     // S(i) = bias + Q_r K^T
          const int kt = i / kRpg, r = i % kRpg, t = tiles + kt;
          if (r == 0 && !mbar_wait_warp(&bars.bias_full[t & 1], (t >> 1) & 1, 64u)) return false;
          if (!mbar_wait_warp(&bars.kv_full[g][s], parity, 8u)) return false;
          tc_fence_after();
          if (elect_lane()) {
            const uint32_t tile = smem_u32(sm + FlashUnitLayout::bias + (t & 1) * kFBiasBytes);
#pragma unroll
            for (int b = 0; b < kFCopied / 8; ++b)  // 32 bytes (8 columns) of the 128-byte rows of the tile's first box
              tmem_copy_128x256b(d_s + 8 * b, umma_desc_sw128(tile) + 2 * b);
            const uint64_t dq = umma_desc_sw64(q_addr + r * kFQBytes), dk = umma_desc_sw64(ring + s * kFStageBytes);
            umma_bf16(d_s, dq, dk, idesc_s, 1u);
            umma_bf16(d_s, dq + 2, dk + 2, idesc_s, 1u);
            umma_commit(&bars.s_full[g]);
            if (r == kRpg - 1) umma_commit(&bars.bias_empty[t & 1]);   // this group is done with the bias tile
          }
          __syncwarp();
          return true;
        };
        bool ok = mbar_wait_warp(&bars.q_full[g], units & 1, 4u) && mbar_wait_warp(&bars.s_free[g], done & 1, 2u) && issue_s(0, stage, round);
        for (int i = 0; i < n_items && ok; ++i) {
          const int kt = i / kRpg, r = i % kRpg, c = done + i, s = stage, before = s ? s - 1 : kFuStages - 1;
          stage = s + 1 == kFuStages ? 0 : s + 1;
          round ^= stage == 0;
          if (i + 1 < n_items) {                    // next S as soon as the group holds the current one in registers
            ok = mbar_wait_warp(&bars.s_free[g], (c + 1) & 1, 2u) && issue_s(i + 1, stage, round);
            if (!ok) break;
          }
          if (i + 1 == n_items && nrpg) {           // the queries have been read for the last time once the last S is there
            ok = mbar_wait_warp(&bars.s_full[g], c & 1, 4u);
            if (!ok) break;
            if (elect_lane()) load_q(nw, nrpg);
            __syncwarp();
          }
          const int ahead = i + kFuStages - 1;       // refill: that stage was last read by P.V of the item before
          if (ahead < n_items || ahead - n_items < nkt * nrpg) {
            if (c >= 1) ok = mbar_wait_warp(&bars.pv_done[g], (c - 1) & 1, 32u);
            if (!ok) break;
            if (elect_lane()) {
              if (ahead < n_items)
                load_kv(w, kRpg, ahead, before);
              else
                load_kv(nw, nrpg, ahead - n_items, before);
            }
            __syncwarp();
          }
          ok = mbar_wait_warp(&bars.p_ready[g], c & 1, 16u);
          if (!ok) break;
          tc_fence_after();
          if (elect_lane()) {
            const uint64_t dv = umma_desc_sw128(ring + s * kFStageBytes + kFKBytes);
#pragma unroll
            for (int ks = 0; ks < kFKT / 16; ++ks) {  // 16 keys per step: 8 TMEM columns of P, 32 bytes of the value rows
              if (kBrief && ks == kFKT / 32 && kt == nkt - 1) break;
              umma_bf16_ts(d_o + kFON * r, d_p + 8 * ks, dv + 2 * ks, idesc_o, (kt | ks) ? 1u : 0u);
            }
            umma_commit(&bars.pv_done[g]);
          }
          __syncwarp();
        }
        done += n_items, tiles += nkt, ++units;
        return ok;
      };
      const FlashUnit half = has_half ? unit_at(half_unit, second) : FlashUnit{0, 0, 0};
      int unit = blockIdx.x;
      FlashUnit w = unit < whole ? unit_at(unit, 0) : half;
      int rpg = unit < whole ? kFRpg : has_half ? 1 : 0;
      if (rpg && elect_lane()) {
        load_q(w, rpg);
        for (int i = 0; i < kFuStages - 1 && i < nkt * rpg; ++i) load_kv(w, rpg, i, i);   // first use of these stages
      }
      __syncwarp();
      bool ok = true;
      while (rpg == kFRpg && ok) {
        unit += gridDim.x;
        const FlashUnit nw = unit < whole ? unit_at(unit, 0) : half;
        const int nrpg = unit < whole ? kFRpg : has_half ? 1 : 0;
        ok = products(std::integral_constant<int, kFRpg>{}, w, nw, nrpg);
        w = nw, rpg = nrpg;
      }
      if (kHalves && rpg == 1 && ok) products(std::integral_constant<int, 1>{}, w, w, 0);
    }
  } else {
    // ------------------------------------------------------------------ softmax groups
    asm volatile("setmaxnreg.inc.sync.aligned.u32 160;\n");
    const int g = warp >> 2, qw = warp & 3;
    const int row = 32 * qw + lane;                 // query row inside the tile = TMEM lane
    const uint32_t lane_addr = (uint32_t)(32 * qw) << 16;
    const uint32_t t_s = tmem_base + lane_addr + kFColS + kFKT * g;
    const uint32_t t_p = tmem_base + lane_addr + kFColP + (kFKT / 2) * g;
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
    int tiles = 0;                                  // bias tiles before this unit (the items before it are an even number)
    const auto softmax = [&](auto per_group, int unit, int second) {
    const FlashUnit w = unit_at(unit, second);
    constexpr int kRpg = decltype(per_group)::value;     // attended rows per group
    const uint32_t t_o = tmem_base + lane_addr + kFColO + kFON * kFRpg * g;
    const int ug = w.u0 + kRpg * g;                 // first row of this group
    unsigned flag_word[kRpg];                       // bit kt & 31: some key of tile kt has a mask bias other than zero
    float m_ref[kRpg], l_sum[kRpg];                 // reference maximum and denominator of this thread's query per row
#pragma unroll
    for (int r = 0; r < kRpg; ++r) {
      flag_word[r] = 0;
      m_ref[r] = -CUDART_INF_F;
      l_sum[r] = 0.f;
    }
    const auto mask_flags = [&](int kt) {
      if ((kt & 31) == 0) {
        for (int r = 0; r < kRpg; ++r) flag_word[r] = 0;
        // A load covers two tiles (ldm is a multiple of 128), eight are in flight (figures in flash_tcgen05.cu).
        const int left = min(nkt - kt, 32);
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
            flag_word[r] |= bits << t0;
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
        const int tt = tiles + kt;
        bool ok = r == 0 ? mbar_wait(&bars.bias_full[tt & 1], (tt >> 1) & 1, 64u) : true;
        // The pair bias of the columns that were not copied (128-byte rows, 16-byte pieces swizzled by row) is fetched before S is waited
        // for, so that it is at hand when S comes.
        float4 b4[(kFKT - kFCopied) / 4];
        const float* brow = reinterpret_cast<const float*>(sm + FlashUnitLayout::bias + ((tiles + kt) & 1) * kFBiasBytes) + row * 32;
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
          if (c == kKeys - 32) clear_rest();
        }
#pragma unroll
        for (int c = kFCopied / 4; c < kKeys / 4; ++c) {
          add2(s[4 * c + 0], s[4 * c + 1], b4[c - kFCopied / 4].x, b4[c - kFCopied / 4].y);
          add2(s[4 * c + 2], s[4 * c + 3], b4[c - kFCopied / 4].z, b4[c - kFCopied / 4].w);
        }
        if ((flag_word[r] >> (kt & 31)) & 1) {     // warp-uniform
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
        tmem_wait_st();
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
        if (r > 0 || kt + tiles > 0) ok = mbar_wait(&bars.pv_done[g], (i - 1) & 1, 256u) && ok;
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
          if (r == kRpg - 1) mbar_arrive(&bars.bias_empty[(tiles + kt) & 1]);
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
    tiles += nkt;
    // ---- epilogue: o = O / denominator for this group's rows.  They leave by TMA, a row at a time through the group's staging area: a
    // warp's 32 queries are 2 KB there (64-byte swizzle).  The first of two rows has been complete since the last item's P was stored.
#pragma unroll
    for (int r = 0; r < kRpg; ++r) {
      if (r == kRpg - 1) {
        ok = ok && mbar_wait(&bars.pv_done[g], (nkt * kRpg - 1) & 1, 512u);
        ok = __all_sync(0xffffffffu, ok);
      }
      if (!ok) return false;
      tc_fence_after();
      uint32_t a[32];
      tmem_ld32(t_o + kFON * r, a);
      tmem_wait_ld();
      if (lane == 0) tma_store_wait_read<0>();      // the row before has left the staging area
      __syncwarp();
      unsigned char* tile = sm + FlashUnitLayout::out + g * kFQBytes;
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
      if (lane == 0 && ug + r < n_u && w.q0 + 32 * qw < n) {
        tma_store_3d(&map_o, smem_u32(tile + 32 * qw * 64), w.h * kFD, w.q0 + 32 * qw, ug + r);
        tma_store_commit();
      }
    }
    return true;
    };
    bool ok = true;
    for (int unit = blockIdx.x; unit < whole && ok; unit += gridDim.x) ok = softmax(std::integral_constant<int, kFRpg>{}, unit, 0);
    if (kHalves && has_half && ok) softmax(std::integral_constant<int, 1>{}, half_unit, second);
    if (lane == 0) tma_store_wait_read<0>();
  }

  tc_fence_before();
  cta_teardown_sync();
  if (warp == 4 * kFGroups) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kFCols) : "memory");
  }
}

}  // namespace px
