// Pieces shared by the persistent, TMA-fed row kernels (LayerNorm'd 128-channel rows times resident weights).
//
// Operand formats.  Rows of a bf16 pair tensor are multiplied as they are stored, against bf16 weights.  For an fp32
// pair tensor the kernels read a standardised fp16 copy of the rows, (x - mean) * rstd, that px_standardise_rows
// writes (a standardised row lies within +-sqrt(128), so fp16's range is safe and its three extra mantissa bits cut
// the operand rounding error eightfold), against fp16 weights; such rows carry mean 0 and deviation 1, so their
// correction step only adds the beta term.  `kF16` names the format of a product's operands; the correction step
// is a separate MMA and always takes bf16 head/tail pairs.
//
// LayerNorm is not applied to the operand.  With W' = W diag(gamma), s = W' 1, t = W beta and std = 1/rstd,
//     W LN(x) = rstd * ( W' x - mean * s + std * t ),
// so the tensor core multiplies the rows exactly as they are stored (bf16 rows go from global memory to the swizzled
// operand by TMA without passing through registers).  The two correction terms ride along as one extra K step of 16:
// the row side holds (-mean, std) and the weight side (s, t), each split into a bf16 head and tail so that the
// products carry about 17 bits.  What is left for the epilogue is one multiplication by the row's rstd.
#pragma once
#include "px_tcgen05.cuh"

namespace px {

constexpr int kPanelBytes = 128 * 128;        // [128 rows][64 k] bf16, 128-byte swizzle
constexpr int kOperandBytes = 2 * kPanelBytes;  // [128 rows][128 k] as two k panels

__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 -> one bf16x2 word (one conversion instruction; measured at 64 lanes per clock and SM on B200, half the
// FMA rate and four times the special-function rate).
__device__ __forceinline__ uint32_t pack_bf16x2_int(float lo, float hi) { return pack_bf16x2(lo, hi); }

// Byte offset of the 16-byte piece holding channels 8*piece16..8*piece16+7 of row r inside a [128][128] operand.
__device__ __forceinline__ int operand_piece_offset(int r, int piece16, int panel_bytes = kPanelBytes) {
  return (piece16 >> 3) * panel_bytes + r * 128 + (((piece16 & 7) ^ (r & 7)) << 4);
}

// bf16 head and tail of an fp32 value: head + tail carries about 17 significant bits.
__device__ __forceinline__ void split_bf16(float v, uint32_t& head, uint32_t& tail) {
  const bf16 h = __float2bfloat16_rn(v);
  const bf16 t = __float2bfloat16_rn(v - __bfloat162float(h));
  head = (uint32_t)__bfloat16_as_ushort(h);
  tail = (uint32_t)__bfloat16_as_ushort(t);
}

// Row r of a correction panel ([rows][16 k] bf16, 32-byte swizzle).  One 8-wide half of the row (`khalf`: k = 0..7 or
// k = 8..15) pairs up x with the other side's first value in its k = 0..3 and y with its second value in k = 4..7;
// `weight_side` picks the interleaving so that the four head/tail products of each pair meet:
// row side (xh, xh, xl, xl, yh, yh, yl, yl), weight side (xh, xl, xh, xl, yh, yl, yh, yl).
// The other half of the row is zeroed when `zero_other` is set (it must never hold anything but finite values).
__device__ __forceinline__ void write_correction_row(unsigned char* panel, int r, float x, float y, bool weight_side,
                                                     int khalf = 0, bool zero_other = true) {
  uint32_t xh, xl, yh, yl;
  split_bf16(x, xh, xl);
  split_bf16(y, yh, yl);
  uint4 v;
  if (weight_side) {
    v.x = xh | (xl << 16), v.y = v.x, v.z = yh | (yl << 16), v.w = v.z;
  } else {
    v.x = xh | (xh << 16), v.y = xl | (xl << 16), v.z = yh | (yh << 16), v.w = yl | (yl << 16);
  }
  const int sw = ((r >> 2) & 1) ^ khalf;
  *reinterpret_cast<uint4*>(panel + r * 32 + (sw << 4)) = v;
  if (zero_other) *reinterpret_cast<uint4*>(panel + r * 32 + ((sw ^ 1) << 4)) = make_uint4(0u, 0u, 0u, 0u);
}

// 16-bit weight values -> fp32 (`kF16`: the weights are fp16, otherwise bf16).
template <bool kF16>
__device__ __forceinline__ float4 load4_w16(const uint16_t* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack16x2<kF16>(u.x), b = unpack16x2<kF16>(u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}

// Folds gamma (and `scale`) into rows [row_begin, row_begin + count) of a [*][128] 16-bit weight (format kInF16) and
// writes them in the operand format kOutF16 as rows dst_row0.. of a K-major swizzled operand with `panel_bytes` per
// 64-wide k panel; the matching rows of the correction panel `extra` receive (s, t): s = sum_c W'[row][c] over the
// rounded values, t = scale * sum_c W[row][c] * beta[c].  Warp-per-row; called by `nwarps` warps with consecutive
// `warp` numbers.  gamma == nullptr: no LayerNorm to fold (plain copy with `scale`, no correction row).
template <bool kInF16, bool kOutF16>
__device__ __forceinline__ void fold_weight_rows(unsigned char* dst, unsigned char* extra, int dst_row0, int panel_bytes,
                                                 const bf16* __restrict__ W, int row_begin, int count,
                                                 const float* __restrict__ gamma, const float* __restrict__ beta,
                                                 float scale, int warp, int nwarps, int lane, int khalf = 0) {
  const float4 g4 = gamma ? *reinterpret_cast<const float4*>(gamma + 4 * lane) : make_float4(1.f, 1.f, 1.f, 1.f);
  const float4 b4 = gamma ? *reinterpret_cast<const float4*>(beta + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
  for (int i = warp; i < count; i += nwarps) {
    const float4 w = load4_w16<kInF16>(reinterpret_cast<const uint16_t*>(W) + (size_t)(row_begin + i) * kC + 4 * lane);
    const uint32_t lo = pack16x2<kOutF16>(w.x * g4.x * scale, w.y * g4.y * scale);
    const uint32_t hi = pack16x2<kOutF16>(w.z * g4.z * scale, w.w * g4.w * scale);
    const int r = i + dst_row0;
    *reinterpret_cast<uint2*>(dst + operand_piece_offset(r, lane >> 1, panel_bytes) + (lane & 1) * 8) = make_uint2(lo, hi);
    if (gamma) {
      const float2 f0 = unpack16x2<kOutF16>(lo), f1 = unpack16x2<kOutF16>(hi);
      const float s = warp_sum(f0.x + f0.y + f1.x + f1.y);
      const float t = warp_sum(w.x * b4.x + w.y * b4.y + w.z * b4.z + w.w * b4.w) * scale;
      if (lane == 0) write_correction_row(extra, r, s, t, true, khalf);
    }
  }
}

// Folded weights.  Folding 256 rows takes a CTA 5 to 6 us (global loads, two warp sums a row), a third of a row kernel at
// N = 128, and it is the same work on every launch.  A caller that keeps the weights folds them once (`fold_kernel` writes the
// image of the operands as they lie in shared memory, for each variant of CTA); the row kernels then fetch the image with one
// bulk copy that overlaps the end of the kernel before them.  Without an image the CTA folds the weights itself.
__device__ __forceinline__ void folded_load(unsigned char* dst, const unsigned char* image, uint32_t bytes, uint64_t* bar) {
  mbar_expect_tx(bar, bytes);
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_u32(dst)),
               "l"(image), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
constexpr int kFoldThreads = 768;
// One CTA per variant: weights.fold(sm, variant, warp, warps, lane, tid, threads) writes W::kBytes bytes at sm.
template <typename W>
__global__ void __launch_bounds__(kFoldThreads, 1) fold_kernel(const W weights, unsigned char* __restrict__ image) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* sm = smem_aligned(smem_raw);
  weights.fold(sm, blockIdx.x, threadIdx.x >> 5, kFoldThreads / 32, threadIdx.x & 31, threadIdx.x, kFoldThreads);
  __syncthreads();
  for (int i = threadIdx.x; i < W::kBytes / 16; i += kFoldThreads)
    reinterpret_cast<uint4*>(image + (size_t)blockIdx.x * W::kBytes)[i] = reinterpret_cast<const uint4*>(sm)[i];
}
template <typename W>
static bool launch_fold(const W& weights, int variants, void* image, cudaStream_t st) {
  static SmemLimit limit;
  if (!limit.set(fold_kernel<W>, W::kBytes + 1024)) return false;
  fold_kernel<W><<<variants, kFoldThreads, W::kBytes + 1024, st>>>(weights, (unsigned char*)image);
  return cudaGetLastError() == cudaSuccess;
}
// In a row kernel, after cta_ready: folds the weights here unless their image is on its way.  `full` is what the issuing threads
// wait for before their first product.
template <typename W>
__device__ __forceinline__ void fold_here(const W& weights, const unsigned char* image, unsigned char* sm, int variant,
                                          uint64_t* full) {
  if (image) return;
  weights.fold(sm, variant, threadIdx.x >> 5, blockDim.x >> 5, threadIdx.x & 31, threadIdx.x, blockDim.x);
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) mbar_arrive(full);
}

// TMA store of a 3-D box from shared memory (bulk async group of the calling thread).
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];\n"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(x), "r"(y), "r"(z)
               : "memory");
}
// The same, adding to what is there (fp32).
__device__ __forceinline__ void tma_add_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];\n"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
// Waits until at most N of this thread's store groups still read their shared-memory source.  Enough at the end of a kernel, too:
// what shared memory held is on its way, and the grid is not complete before it has arrived.
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;\n" ::"n"(N) : "memory");
}
// Barrier over `threads` threads that also returns whether `ok` held on all of them, so that a group can leave a
// loop together after one of its waits ran out.
__device__ __forceinline__ bool named_barrier_all(int id, int threads, bool ok) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.b32 q, %1, 0;\n bar.red.and.pred p, %2, %3, q;\n selp.b32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)ok), "r"(id), "r"(threads)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void named_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// ---------------------------------------------------------------------------------------------------------------
// Row tiles: the part of the pipeline that is the same for every kernel that consumes LayerNorm'd pair rows.
// A tile is 128 pair elements: 128 consecutive t of one u, or two runs of 64, each of one u; element (u, t) is row u*n_t + t of z, or row
// t*n_u + u when the two indices are exchanged (`swap`).  A stage of the ring holds the tile as two k panels of 128 rows.
//   * producer thread: TMA loads of the rows (bf16 rows of z, or the standardised fp16 copy of an fp32 z);
//   * statistics threads: mean and variance of the row as it lies in the stage (bf16 rows), correction row (-mean, std),
//     and whatever the kernel wants per row.  For standardised rows the statistics are known: (0, 1).  A product Z Z^T
//     with the sums of squares on its diagonal took 600 cycles of the tensor pipe a tile, and 144 columns of tensor memory that
//     now hold a second set of accumulators for bf16 rows, too.
// What bounds these kernels from N = 384 on is the way of a tile from memory, 2 us under load: three stages where they fit
// (with the statistics as they are now; projections of the triangle multiplication, bf16 N = 768 132 -> 117 us, N = 437 55.3 -> 47.5;
// fp16 N = 384 in a stack 36.4 -> 31.8; two stages and a second staging buffer 148 at N = 768 where three took 136).  The projections of
// the triangle attention, which write three times what they read, take two from the size on where the rows exceed L2 (triatt_in_tc.cu).
// ---------------------------------------------------------------------------------------------------------------
constexpr int kTileBytes = kOperandBytes;
constexpr int kTileExtra = 128 * 32;           // [128 rows][16 k] correction panel

// Slots of everything written per tile by the statistics warps (scales, correction rows, the a_ready barrier): read after the
// stage is freed, by an epilogue that may run two tiles behind the products when the accumulators are double-buffered.  Slot
// k % slots is rewritten for tile k + slots, whose stage is the one of tile k + 2, and handed out only after the products of
// that tile, which are issued after the correction step of tile k and wait for the epilogue of tile k (at the latest) to have
// read its scales and its accumulator.
constexpr int tile_slots(int stages) { return stages + 2; }
// The correction rows of standardised rows are all alike: one panel serves every tile.
constexpr int tile_extras(int stages, bool standardised) { return standardised ? 1 : tile_slots(stages); }

// Barriers that say a tile has arrived: of every one, each set of statistics warps sees all phases or none (a wait on a parity tells a
// phase from the one before only; tile k + 1 may arrive before tile k), so two sets need an even number of them.
constexpr int tile_fulls(int stages, int sets) { return sets == 2 && stages % 2 ? 2 * stages : stages; }

template <int kStages, int kFulls = kStages>
struct TileBars {
  // raw_full: tile in shared memory (which of them is tile k's, for every load and every wait: TileCtx::full); a_ready: statistics,
  // correction rows and scales written; a_empty: every MMA that reads the stage is complete (one commit per issuing thread)
  uint64_t raw_full[kFulls], a_ready[tile_slots(kStages)], a_empty[kStages];
};
// kStandardised: the rows are a standardised fp16 copy (otherwise bf16 rows of z).  kSets: of statistics warps for bf16 rows
// (tile_stats_loop).
template <int kStages_, bool kStandardised_, int kRun_ = 128, int kSets_ = 1>
struct TileCtx {
  static constexpr int kStages = kStages_, kSlots = tile_slots(kStages_), kSets = kStandardised_ ? 1 : kSets_;
  static constexpr int kFulls = tile_fulls(kStages_, kSets_);
  static constexpr bool kStandardised = kStandardised_;
  static constexpr int kRun = kRun_;          // elements of a run: 128 or 64
  unsigned char* tiles;     // kStages x kTileBytes
  unsigned char* extras;    // tile_extras() x kTileExtra (the correction step of a tile runs after its stage is freed)
  TileBars<kStages_, kFulls>* bars;
  int first_tile, tile_step, n_tiles, runs_t, n_u, n_t, swap;   // runs_t: runs that cover the t of one u
  __device__ __forceinline__ uint64_t* full(int k) const { return &bars->raw_full[k % kFulls]; }
  __device__ __forceinline__ uint32_t full_parity(int k) const { return (k / kFulls) & 1; }
  __device__ __forceinline__ unsigned char* extra(int k) const { return extras + (kStandardised ? 0 : (k % kSlots) * kTileExtra); }
};

// Statistics warps: a thread per row where there is nothing to measure, two for bf16 rows.
constexpr int tile_stats_warps(bool standardised) { return standardised ? 4 : 8; }
// readers: how many arrivals free a stage besides those of the statistics warps.
template <typename Ctx>
__device__ __forceinline__ void tile_bars_init(const Ctx& c, int readers) {
  constexpr int kWarps = tile_stats_warps(Ctx::kStandardised) / Ctx::kSets;       // of a set
  for (int s = 0; s < Ctx::kFulls; ++s) mbar_init(&c.bars->raw_full[s], 1);
  for (int s = 0; s < Ctx::kStages; ++s) mbar_init(&c.bars->a_empty[s], readers + kWarps);
  for (int s = 0; s < Ctx::kSlots; ++s) mbar_init(&c.bars->a_ready[s], kWarps);
}

// Run number `run`: which u, and its first t.  With runs of 64 tile k is made of the runs 2 k and 2 k + 1, which lie behind one another or are
// the end of one u and the beginning of the next; the second run of the last tile may be none (u = n_u: loads give zeros, nothing is
// stored).  In tiles of 128 t of one u a length just above a multiple of 128 pays for half a tile more.
struct Run {
  int u, t;
};
template <int kRun>
__device__ __forceinline__ Run run_at(int run, int runs_t) {
  const int u = run / runs_t;
  return {u, (run - u * runs_t) * kRun};
}
static inline int64_t runs_of(int64_t n_t, int run) { return (n_t + run - 1) / run; }
static inline int64_t tiles_of(int64_t n_u, int64_t n_t, int run) { return (n_u * runs_of(n_t, run) * run + 127) / 128; }
// Tiles of unlike size (ragged runs) recur every so many (for even_grid).
static inline int64_t tile_period(int64_t n_u, int64_t n_t, int run) {
  const int64_t runs = runs_of(n_t, run);
  return n_u == 1 || n_t % run == 0 ? 1 : run == 64 && runs % 2 == 0 ? runs / 2 : runs;
}

// Where consecutive rows of tiles lie behind one another in every tensor of a kernel (rows of z as they are, and no pad columns), the
// tiles need not end with each row (both output stages of the triangle multiplication, its outgoing projection and the output stage of the
// starting node, us a block of a stack: 160 tokens 205.3 -> 196.5, 200 260.5 -> 252.5, 400 914 -> 873; where fewer tiles leave SMs free, the single
// branch has them).  Outgoing projection: as one row unless n_t is a multiple of 64 (lengths of an odd number of 64 take two runs a tile, below).
static inline bool one_row_pays(int64_t n_u, int64_t n_t) { return n_u > 1 && n_t % 64 != 0; }

// How an output stage cuts its tiles: each u by itself (kRows), runs of 64, or as one row where that is possible; whichever makes fewer tiles,
// and runs of 64, with their twice as many loads and stores, only where one row does not.  us, rows | runs | one row: triangle multiplication
// N = 150 bf16 17.1 | 14.4 | - (pad columns), 160 17.0 | 14.4 | 14.3, 400 39.7 | 37.2 | 34.7, 1096 219 | 219 | 212, fp32 264 25.8 | 23.3 | 21.1;
// starting node 300 fp32 25.6 | 23.4 | 21.6, bf16 448 48.8 | 45.5 | 44.4, whole tiles (N = 768) 104 | 107.
// fp32 rows are the exception at both ends.  Where most SMs are idle anyway, an SM's tile should be small: N = 24 11.1 | 11.4 | 11.8, 64 11.5 |
// 11.9 | 11.9, 100 level, 120 12.7 | 12.8 | 12.4.  From `most` tiles an SM on the time is that of their memory traffic, which the same SMs
// ask for in fewer places at once when all tiles are full: triangle attention 320 26.6 | 24.8 | 24.4, 400 47.7 | 47.9 | 49.0, 437 54.8 | 56.4 |
// 56.9, 776 148 | 151 | 157, triangle multiplication 520 78.8 | 77.0 | 77.0, 680 120 | 120 | 122, 1000 241 | 241 | 246.  most = 0: none.
enum class Cut { kRows, kRuns, kOneRow };
static inline Cut output_cut(int64_t n_u, int64_t n_t, bool can_be_one_row, int64_t most) {
  const int64_t rows = tiles_of(n_u, n_t, 128), room = sm_count();
  if (most && (3 * rows <= 2 * room || rows > most * room)) return Cut::kRows;
  if (can_be_one_row && tiles_of(1, n_u * n_t, 128) < rows) return Cut::kOneRow;
  return rows > room && tiles_of(n_u, n_t, 64) < rows ? Cut::kRuns : Cut::kRows;
}

// Projections (a pair of CTAs a tile): tiles of two runs where the last pair is through in fewer of them.  They load and store twice as many
// pieces, which costs whole tiles 2 (fp16) to 6 % (bf16), hence up to 1024.  Incoming projection of the triangle multiplication, us, one run
// of 128 | two of 64: bf16 N = 136 16.6 | 15.9, 264 28.0 | 25.9, 437 51.9 | 49.3, 700 119 | 118; fp16 192 17.9 | 16.2, 437 47.2 | 46.0, 700
// 110 | 99; whole tiles 384 31.7 | 33.3; no fewer a pair: 55 rows of 437 bf16 15.6 | 16.0, fp16 14.7 | 15.2, 110 rows 19.8 | 20.4, 18.7 | 19.0.
// With one tile a pair there is nothing in it but the fewer of them to start (N = 56 level, 64 12.4 | 11.9).
static inline bool two_runs_pay(int64_t n_u, int64_t n_t) {
  const int64_t rows = tiles_of(n_u, n_t, 128), runs = tiles_of(n_u, n_t, 64), room = sm_count() / 2;
  return n_u > 1 && n_t < 1024 && runs < rows && (rows <= room || (runs + room - 1) / room < (rows + room - 1) / room);
}

// One warp: TMA loads of the tiles (boxes of a run).
template <typename Ctx>
__device__ __forceinline__ void tile_producer_loop(const Ctx& c, const CUtensorMap* map_z) {
  int k = 0;
  for (int tile = c.first_tile; tile < c.n_tiles; tile += c.tile_step, ++k) {
    const int s = k % Ctx::kStages, n = k / Ctx::kStages;
    if (!mbar_wait_warp(&c.bars->a_empty[s], (n & 1) ^ 1, 1u)) break;
    if (elect_lane()) {
      uint64_t* const full = c.full(k);
      mbar_expect_tx(full, kOperandBytes);
      const uint32_t dst = smem_u32(c.tiles + s * kTileBytes);
      constexpr int kPer = 128 / Ctx::kRun;
      for (int h = 0; h < kPer; ++h) {
        const Run r = run_at<Ctx::kRun>(kPer * tile + h, c.runs_t);
        for (int p = 0; p < 2; ++p)
          tma_load_3d(dst + p * kPanelBytes + h * (Ctx::kRun * 128), map_z, full, 64 * p, c.swap ? r.u : r.t, c.swap ? r.t : r.u);
      }
    }
    __syncwarp();
  }
}

// Mean and variance of row r of a bf16 tile.  Two neighbouring lanes share a row, eight 16-byte pieces each (lane 1 begins at another
// piece, so that the two meet different banks), and sum d and d^2 of d = x - x0 in fp32: about one of its values, nothing cancels
// however far the row lies from zero.
__device__ __forceinline__ void bf16_row_stats(const unsigned char* tile, int r, int half, float& mean, float& var) {
  const float x0 = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(tile + operand_piece_offset(r, 0))).x;
  float s0 = 0.f, s1 = 0.f, q0 = 0.f, q1 = 0.f;
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    const uint4 v = *reinterpret_cast<const uint4*>(tile + operand_piece_offset(r, 8 * half + (p ^ (4 * half))));
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 x = unpack_bf16x2(w[e]);
      add2(x.x, x.y, -x0, -x0);
      add2(s0, s1, x.x, x.y);
      fma2(q0, q1, x.x, x.y, x.x, x.y, q0, q1);
    }
  }
  float sum = s0 + s1, sq = q0 + q1;
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sq += __shfl_xor_sync(0xffffffffu, sq, 1);
  const float m = sum * (1.0f / kC);
  var = fmaxf(sq * (1.0f / kC) - m * m, 0.f);
  mean = x0 + m;
}

// The statistics warps (`sw` = 0..3, or 0..7 for bf16 rows).  per_row(k, u, t, r, rstd, fetched) is called once per
// tile and row with the row's 1/std, before a_ready is signalled.  `kStandardised`: the rows are a standardised copy
// (mean 0, deviation 1 by construction), so the correction row is (0, 1), written once, and the factor is 1.
// fetched: what ahead(u, t) loaded from global memory a tile earlier, so that nothing waits for it between the arrival of a tile and the
// hand-over.  after(u, t) follows once the stage and the statistics have been handed over: for what nothing in the kernel waits for.
// A tile's statistics are a chain of 1.3 us (arrival, loads, sums, square roots, hand-over).  In the projections of the triangle
// multiplication a tile lasts about as long: two sets of four warps work on two tiles there, each lane on two rows of its tile at once.
// Eight warps on one tile, with the load of the mask on the chain, against that (outgoing, us): bf16 N = 200 15.2 -> 14.5, 384 36.2 -> 31.0,
// 437 47.0 -> 42.8, 768 118 -> 105.5, 1536 477 -> 424 (the mask alone 111 at 768; without any statistics 96); fp16 rows, which only had
// the mask there, 384 28.9 -> 27.8, 768 98 -> 94.5, 1536 388 -> 377.  In the output stage of the triangle attention, whose tiles
// last longer than their statistics, all eight work on one tile (two sets | one set: N = 128 11.5 | 11.1, 384 30.9 | 29.9, 768 108.7 | 105,
// 1536 398 | 392), and so they do in the pair bias (128 5.5 | 5.3, 256 7.7 | 7.4, 1024 56 | 55) and the recycling update (level).
// Projections of the triangle attention: by the number of tiles (triatt_in_tc.cu).
struct TileNothingAhead {
  __device__ __forceinline__ float operator()(int, int) const { return 0.f; }
};
struct TileNothingAfter {
  __device__ __forceinline__ void operator()(int, int) const {}
};
template <typename Ctx, typename PerRow, typename Ahead = TileNothingAhead, typename After = TileNothingAfter>
__device__ __forceinline__ void tile_stats_loop(const Ctx& c, float eps, int sw, int lane, PerRow per_row, Ahead ahead = Ahead(),
                                                After after = After()) {
  constexpr bool kStandardised = Ctx::kStandardised;
  constexpr int kSets = Ctx::kSets, kRows = kSets;
  const int set = kSets == 2 ? sw >> 2 : 0, half = kStandardised ? 0 : lane & 1;
  const int r0 = kStandardised ? 32 * sw + lane : 16 * (kSets == 2 ? sw & 3 : sw) + (lane >> 1);      // two sets: and r0 + 64
  const auto where = [&](int tile, int j) {           // (u, t) of row j of this lane
    constexpr int kPer = 128 / Ctx::kRun;
    const int row = r0 + 64 * j;
    Run r = run_at<Ctx::kRun>(kPer * tile + (kPer == 2 ? row >> 6 : 0), c.runs_t);
    r.t += row % Ctx::kRun;
    return r;
  };
  float next[kRows];
  const auto fetch = [&](int tile) {
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const Run r = where(tile, j);
      next[j] = tile < c.n_tiles ? ahead(r.u, r.t) : 0.f;
    }
  };
  fetch(c.first_tile + set * c.tile_step);
  int k = set;
  for (int tile = c.first_tile + set * c.tile_step; tile < c.n_tiles; tile += kSets * c.tile_step, k += kSets) {
    const int s = k % Ctx::kStages;
    float fetched[kRows], mean[kRows], var[kRows];
#pragma unroll
    for (int j = 0; j < kRows; ++j) fetched[j] = next[j];
    fetch(tile + kSets * c.tile_step);
    // for standardised rows the arrival of the tile only paces this loop, so that the slots it writes are those of tiles in flight
    if (!mbar_wait_warp(c.full(k), c.full_parity(k), 16u)) break;
    if constexpr (!kStandardised) {
#pragma unroll
      for (int j = 0; j < kRows; ++j) bf16_row_stats(c.tiles + s * kTileBytes, r0 + 64 * j, half, mean[j], var[j]);
    }
#pragma unroll
    for (int j = 0; j < kRows; ++j) {
      const float rstd = kStandardised ? 1.f : rsqrtf(var[j] + eps);
      // rstd * (W'x - mean * s + std * t): the row side of the correction step holds (-mean, std)
      if (kStandardised ? k == 0 : half == 0)
        write_correction_row(c.extra(k), r0 + 64 * j, kStandardised ? -0.f : -mean[j], kStandardised ? 1.f : sqrtf(var[j] + eps), false);
      if (half == 0) {
        const Run r = where(tile, j);
        per_row(k, r.u, r.t, r0 + 64 * j, rstd, fetched[j]);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(&c.bars->a_ready[k % Ctx::kSlots]);
      mbar_arrive(&c.bars->a_empty[s]);                 // after the last use of what was read from the stage
    }
    if (half == 0) {
#pragma unroll
      for (int j = 0; j < kRows; ++j) {
        const Run r = where(tile, j);
        after(r.u, r.t);
      }
    }
  }
}

// One warp: for every tile, 8 MMAs M=128 (rows) x N (weight rows of `w_addr`, two k panels of w_panel bytes) into
// tensor-memory column d_tmem, then the correction step against the weight-side panel at wx_addr.  acc_full/acc_free
// hand the accumulator back and forth with the epilogue warps: arrays of n_acc barriers, tile k uses accumulator
// k % n_acc at d_tmem + (k % n_acc) * acc_cols (n_acc = 1 or 2).
template <typename Ctx>
__device__ __forceinline__ void tile_product_loop(const Ctx& c, uint32_t d_tmem, uint32_t w_addr, int w_panel,
                                                  uint32_t wx_addr, uint32_t idesc, uint64_t* w_full,
                                                  uint64_t* acc_full, uint64_t* acc_free, int n_acc = 1,
                                                  uint32_t acc_cols = 0) {
  if (!mbar_wait_warp(w_full, 0, 4u)) return;    // the resident weights
  const uint64_t wx_desc = umma_desc_sw32(wx_addr);
  // the correction step multiplies bf16 head/tail pairs whatever the format of the main operands; M and N as `idesc`
  const uint32_t idesc_corr = idesc | (1u << 7) | (1u << 10);
  int k = 0;
  for (int tile = c.first_tile; tile < c.n_tiles; tile += c.tile_step, ++k) {
    const int s = k % Ctx::kStages;
    const int ab = n_acc == 2 ? (k & 1) : 0, an = n_acc == 2 ? (k >> 1) : k;
    const uint32_t d = d_tmem + ab * acc_cols;
    if (!mbar_wait_warp(c.full(k), c.full_parity(k), 4u) || !mbar_wait_warp(&acc_free[ab], (an & 1) ^ 1, 8u)) break;
    tc_fence_after();
    if (elect_lane()) {
      const uint32_t a_addr = smem_u32(c.tiles + s * kTileBytes);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks)
        umma_bf16(d, umma_desc_sw128(a_addr + (ks >> 2) * kPanelBytes) + 2 * (ks & 3),
                  umma_desc_sw128(w_addr + (ks >> 2) * w_panel) + 2 * (ks & 3), idesc, ks ? 1u : 0u);
      // this warp's reads of the stage end here: the producer may refill it while the statistics of the tile are on their way
      umma_commit(&c.bars->a_empty[s]);
    }
    __syncwarp();
    if (!mbar_wait_warp(&c.bars->a_ready[k % Ctx::kSlots], (k / Ctx::kSlots) & 1, 4u)) break;   // needs the statistics
    tc_fence_after();
    if (elect_lane()) {
      umma_bf16(d, umma_desc_sw32(smem_u32(c.extra(k))), wx_desc, idesc_corr, 1u);
      umma_commit(&acc_full[ab]);
    }
    __syncwarp();
  }
}

// fp32 output rows through TMA: a warp's [32 rows][32 channels] block in a private 4 KB staging area (rows of 128 bytes, 128-byte
// swizzle), then stored, or added to the tensor where the residual is the output itself: the sum (one fp32 rounding, as
// before) is formed in L2 and the rows of z never come to the SM.  N = 768, against the plain accesses below: triangle multiplication
// 187 -> 144 us, attention 187 -> 141 (starting) and 189 -> 165 (ending), transition 316 -> 273.
__device__ __forceinline__ void rows_bulk_out(unsigned char* stg, const float (&v)[32], const CUtensorMap* map, bool add, int x, int y,
                                              int z, bool any, int lane) {
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<float4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) =
        make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  __syncwarp();
  if (lane == 0 && any) {
    if (add)
      tma_add_3d(map, smem_u32(stg), x, y, z);
    else
      tma_store_3d(map, smem_u32(stg), x, y, z);
    tma_store_commit();
  }
}

// fp32 output rows, coalesced.  A thread of the epilogue owns one row (its accumulator lane) and 32 consecutive
// channels of it; written as they are, a warp's store would touch 32 rows 512 bytes apart.  Instead the warp passes
// its [32 rows][32 channels] block through a private 4 KB staging area (rows of 128 bytes, 16-byte pieces swizzled
// by row) and reads it back with 8 lanes per row, so that every global access of the warp covers four rows x 128
// contiguous bytes.  `res` holds the residual values of the same block in the read-back arrangement, loaded by
// rows_out_request before the accumulator is waited for (zeros without a residual).
struct RowsOutReq {
  float4 v[8];
};
// first_row: index (inside the tensor, in rows of 128 channels) of the warp's row 0; row_stride: distance in rows
// between consecutive rows of the warp (1, or n_u for a column slab); rows_valid: how many of the 32 rows exist.
__device__ __forceinline__ void rows_out_request(RowsOutReq& rq, const float* __restrict__ z, long long first_row,
                                                 long long row_stride, int rows_valid, int chan0, int lane, bool want) {
  const int rsub = lane >> 3, piece = lane & 7;
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int rl = 4 * it + rsub;
    rq.v[it] = (want && rl < rows_valid)
                   ? __ldg(reinterpret_cast<const float4*>(z + (size_t)(first_row + rl * row_stride) * kC + chan0) + piece)
                   : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
__device__ __forceinline__ void rows_out_store(unsigned char* stg, const float (&v)[32], const RowsOutReq& rq,
                                               float* __restrict__ out, long long first_row, long long row_stride,
                                               int rows_valid, int chan0, int lane) {
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<float4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) =
        make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
  __syncwarp();
  const int rsub = lane >> 3, piece = lane & 7;
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int rl = 4 * it + rsub;
    float4 o = *reinterpret_cast<const float4*>(stg + rl * 128 + ((piece ^ (rl & 7)) << 4));
    if (rl < rows_valid) {
      o.x += rq.v[it].x, o.y += rq.v[it].y, o.z += rq.v[it].z, o.w += rq.v[it].w;
      *(reinterpret_cast<float4*>(out + (size_t)(first_row + rl * row_stride) * kC + chan0) + piece) = o;
    }
  }
  __syncwarp();
}

}  // namespace px
