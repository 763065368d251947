// tcgen05 / TMA / mbarrier building blocks shared by the sm_100a tensor-core kernels.
#pragma once
#include <cuda.h>

#include "px_common.cuh"

namespace px {

// Flags recorded by bounded waits that ran out, and the limit of a wait in clock cycles (2^28: about 0.14 s at
// 1.9 GHz; tests shorten it).  One copy of each per translation unit.
static __device__ unsigned int g_tc_error = 0;
static __device__ long long g_wait_limit = 1ll << 28;

// True once any bounded wait of this translation unit's kernels has given up (until the host reads the word).
__device__ __forceinline__ bool tc_error_seen() { return *reinterpret_cast<volatile unsigned int*>(&g_tc_error) != 0; }

// Called by every thread at the top of a kernel: whether a wait has run out before.  The answer is not needed before
// cta_ready, so the read of the flag overlaps the set-up.
__device__ __forceinline__ bool cta_begin() { return tc_error_seen(); }
__device__ __forceinline__ void tc_fence_before();
__device__ __forceinline__ void tc_fence_after();
// The barrier after the set-up, and the wait for the kernels before this one.  False (for every thread of the CTA): a wait ran
// out earlier and the CTA shall do no work, so that a failure holds the GPU for one wait limit and not one per CTA; its tensor
// memory is given back here by the warp that allocated it.
// before_wait(): work that needs nothing of earlier kernels (loads of the resident weights).
struct Nothing {
  __device__ __forceinline__ void operator()() const {}
};
template <typename F = Nothing>
__device__ __forceinline__ bool cta_ready(bool skip, bool alloc_warp, const uint32_t& tmem_base, uint32_t cols, F before_wait = F()) {
  tc_fence_before();
  const bool stop = __syncthreads_or(skip) != 0;
  tc_fence_after();
  if (!stop) before_wait();
  pdl_wait();
  if (stop && alloc_warp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(cols) : "memory");
  return !stop;
}

// Called by every thread at the end of a kernel, in place of the closing __syncthreads(): copies that a wait gave up on have
// landed by now (see mbar_wait).
__device__ __forceinline__ void cta_teardown_sync() { __syncthreads(); }

// Asks for the descriptors of a kernel's TMA copies (one thread, before pdl_wait): the first copy through each would fetch it
// from global memory, after the kernel before has ended.
template <typename... Maps>
__device__ __forceinline__ void prefetch_maps(const Maps&... maps) {
  const CUtensorMap* list[] = {&maps...};
#pragma unroll
  for (const CUtensorMap* m : list) asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

// Index of this warp, in a form that the compiler knows to be the same for all its lanes.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
// True for one lane of a whole warp (always the same one).  The operands of tcgen05 and TMA instructions are warp-uniform;
// behind elect.sync the compiler knows that one lane issues them.  Issued behind `lane == 0` they cost 100 to 170 cycles each
// and bounded every kernel with short products: transition of 1024 tokens 433 -> 407 us, of 384 77 -> 69, MSA transition
// 230 -> 181, single-branch projections 28 -> 22, flash attention at N = 1536 5.95 -> 5.83 ms, a block at N = 128 202 -> 195 us.
__device__ __forceinline__ bool elect_lane() {
  uint32_t pred = 0;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n @p mov.s32 %0, 1;\n}\n" : "+r"(pred));
  return pred != 0;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait for the phase with the given parity; false = gave up (error flag set, copies in flight have landed).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned int code) {
  const uint32_t addr = smem_u32(bar);
  {
    // fast path: the phase is often complete already, and a plain test costs one shared-memory round trip
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  const long long t0 = clock64();
  for (;;) {
    uint32_t done;
    // the hardware suspends the thread until the phase completes or the hint (in ns) runs out, so a waiting
    // warp does not spend issue slots on polling
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity), "r"(1000000u)
        : "memory");
    if (done) return true;
    if (tc_error_seen()) break;          // another wait gave up: this one would only repeat its limit
    if (clock64() - t0 > *reinterpret_cast<volatile long long*>(&g_wait_limit)) {
      atomicOr(&g_tc_error, code);
      break;
    }
  }
  // Copies may still be in flight towards this CTA's shared memory, so whoever gives up lingers before it goes on to the end of the
  // kernel, where everything is freed.  (Looking at the flag there instead cost every launch a trip to L2.)
  const long long t1 = clock64();
  while (clock64() - t1 < 200000) {
  }
  return false;
}

// The same for a whole warp: all lanes wait and get one answer.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, unsigned int code) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, code)) != 0;
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// Asks L2 for what a load with these coordinates will bring.
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* map, int x, int y, int z) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];\n"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z)
               : "memory");
}

// K-major operand tile, rows of 64 bf16 (128 bytes), 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// K-major operand tile, rows of 32 bf16 (64 bytes), 64-byte swizzle, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
// K-major operand tile, rows of 16 bf16 (32 bytes), 32-byte swizzle, 8-row groups 256 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw32(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(256 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)6 << 61);
}
// MN-major operand tile (the M or N index is the contiguous one): per k a run of 64 bf16 (128 bytes), 128-byte
// swizzle; groups of 8 k are `sbo` bytes apart, blocks of 64 along M/N are `lbo` bytes apart.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Instruction descriptor of kind::f16 with bf16 A and B (both K-major) and fp32 D, M x N tile.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n, bool a_mn_major = false, bool b_mn_major = false) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// The same for any pair of 16-bit operand formats (fp16 or bf16 per operand) and fp32 D.
__host__ __device__ constexpr uint32_t umma_idesc_16(int m, int n, bool a_f16, bool b_f16, bool a_mn_major = false,
                                                     bool b_mn_major = false) {
  return (1u << 4) | ((a_f16 ? 0u : 1u) << 7) | ((b_f16 ? 0u : 1u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n, bool a_mn_major = false, bool b_mn_major = false) {
  return umma_idesc_16(m, n, true, true, a_mn_major, b_mn_major);
}
// D[tmem] (+)= A[smem] * B[smem]   (kind::f16 covers fp16 and bf16 operands; the instruction descriptor says which)
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]   (A: 128 lanes x K, two bf16 per 32-bit column)
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 128 lanes x 32 bytes from shared memory (addressed like one K step of a K-major operand) into 8 columns of tensor memory; runs
// in order with the products that the same thread issues.
__device__ __forceinline__ void tmem_copy_128x256b(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::1.128x256b [%0], %1;\n" ::"r"(taddr), "l"(desc) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}


__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (the library does not link libcuda).
static inline EncodeTiledFn tensor_map_encoder() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// 3-D tiled map: dims/strides innermost first (strides in bytes for dims 1 and 2), zero fill outside.
static inline bool make_map_3d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t d0, uint64_t d1,
                               uint64_t d2, uint64_t s1, uint64_t s2, uint32_t b0, uint32_t b1,
                               CUtensorMapSwizzle swz, uint32_t b2 = 1) {
  EncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {d0, d1, d2};
  const cuuint64_t strides[2] = {s1, s2};
  const cuuint32_t box[3] = {b0, b1, b2};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, dt, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Reads and clears this translation unit's flag word (synchronises the device).
static inline int read_clear_tc_error(unsigned int* out) {
  unsigned int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(v)) != cudaSuccess) return -1;
  if (v && cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(zero)) != cudaSuccess) return -1;
  *out = v;
  return 0;
}

// Host hooks of one translation unit: <family>_error_flags() returns (and clears) the wait codes its kernels
// recorded (0x80000000 when the word could not be read), <family>_set_wait_limit() replaces the limit of its waits.
#define PX_DEFINE_FAMILY_HOOKS(family)                                                              \
  unsigned int family##_error_flags() {                                                             \
    unsigned int v = 0;                                                                             \
    return read_clear_tc_error(&v) == 0 ? v : 0x80000000u;                                          \
  }                                                                                                 \
  int family##_set_wait_limit(long long cycles) {                                                   \
    return cudaMemcpyToSymbol(g_wait_limit, &cycles, sizeof(cycles)) == cudaSuccess ? 0 : -1;       \
  }

}  // namespace px
