// Shared device helpers for the sm_100a Pairformer kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <numeric>

#include "../../include/px_b200.h"

namespace px {

typedef __nv_bfloat16 bf16;

constexpr int kC = 128;        // pair channels handled by the fused kernels
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The first 1024-byte boundary of the dynamic shared memory.  As an offset from the array, so that the compiler still sees shared
// memory behind every pointer made from it: rounded through an integer, all plain accesses were generic ones (slower, counted
// with global memory, and not in order with the mbarrier operations behind them).
__device__ __forceinline__ unsigned char* smem_aligned(unsigned char* raw) { return raw + ((0u - smem_u32(raw)) & 1023u); }

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// Two fp32 -> one f16x2 word (round to nearest; values beyond the fp16 range saturate to +-65504 instead of inf).
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float2 unpack_f16x2(uint32_t u) {
  return __half22float2(*reinterpret_cast<const __half2*>(&u));
}
// The two 16-bit operand formats of the tensor-core kernels: bf16 (kF16 = false) and fp16 (kF16 = true).
template <bool kF16>
__device__ __forceinline__ uint32_t pack16x2(float lo, float hi) {
  return kF16 ? pack_f16x2(lo, hi) : pack_bf16x2(lo, hi);
}
template <bool kF16>
__device__ __forceinline__ float2 unpack16x2(uint32_t u);
template <>
__device__ __forceinline__ float2 unpack16x2<true>(uint32_t u) {
  return unpack_f16x2(u);
}
// bf16 -> fp32 is a 16-bit shift: spelled out so that it runs on the integer pipe, not the conversion unit
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}

template <>
__device__ __forceinline__ float2 unpack16x2<false>(uint32_t u) {
  return unpack_bf16x2(u);
}

// Packed fp32 arithmetic (sm_100): two elements per issue slot.  Pays where the issue slots are the scarce resource
// (flash attention: -7 %); the SwiGLU of the transition kernel got 22 % slower with it and stays scalar.
// (a0, a1) += (b0, b1) as one packed instruction: half the issue slots of two scalar additions.
__device__ __forceinline__ void add2(float& a0, float& a1, float b0, float b1) {
  asm("{\n .reg .b64 x, y;\n mov.b64 x, {%0, %1};\n mov.b64 y, {%2, %3};\n add.f32x2 x, x, y;\n mov.b64 {%0, %1}, x;\n}\n"
      : "+f"(a0), "+f"(a1)
      : "f"(b0), "f"(b1));
}

// (d0, d1) = (a0, a1) * (b0, b1) + (c0, c1) as one packed instruction.
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b0, float b1, float c0, float c1) {
  asm("{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mov.b64 c, {%6, %7};\n"
      " fma.rn.f32x2 d, a, b, c;\n mov.b64 {%0, %1}, d;\n}\n"
      : "=f"(d0), "=f"(d1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- typed access to the residual stream (fp32 or bf16 storage) -------------------------
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
  uint2 u = *reinterpret_cast<const uint2*>(p);
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}

// Programmatic dependent launch: a kernel launched with launch_pdl may start while the one before it drains, and waits here,
// before it touches anything that earlier kernels wrote or read, until those are complete.  Its launch, barrier set-up,
// tensor-memory allocation and fetch of the resident weights then overlap that end (a block at N = 128: 28 launches, 278 us
// without, 225 us with).  Nothing signals its dependents early (griddepcontrol.launch_dependents at the top of every kernel
// measured 235 us, and 1.5 % more at N = 1536: what starts early takes room from what runs).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Launch that may overlap the end of the kernel before it (see pdl_wait).
template <typename... Params, typename... Args>
static inline bool launch_pdl(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}

// cudaFuncSetAttribute for the dynamic shared memory of one kernel, once per device (one object per kernel).
struct SmemLimit {
  std::atomic<unsigned long long> done{0};
  template <typename F>
  bool set(F* kernel, size_t bytes) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const unsigned long long bit = 1ull << (dev & 63);
    if (dev < 64 && (done.load(std::memory_order_relaxed) & bit)) return true;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return false;
    done.fetch_or(bit, std::memory_order_relaxed);
    return true;
  }
};

// Number of SMs of the current device (cached per device ordinal).
static inline int sm_count() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// Size of the current device's L2 in bytes (cached per device ordinal).
static inline int64_t l2_bytes() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 126 << 20;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrL2CacheSize, dev) != cudaSuccess || n <= 0) n = 126 << 20;
    cached[dev] = n;
  }
  return cached[dev];
}

// CTAs (or pairs of them) of a persistent kernel that deals out `tiles` in turn: as few of the `room` that fit as end with the same
// number of tiles each.  The others would only end a tile earlier, and they keep CTAs of another stream (the single branch) from
// the SMs and ask L2 for more at once: pair path at N = 200 249 -> 246 us a block, with the single branch beside it 288 -> 285.
// `period`: tiles of unlike size (the ragged edge) recur every so many tiles; 1 if there are none.  A number of CTAs that shares a
// factor with it deals some of them the small tiles only, so it is raised to one that does not, if that still fits.  All SMs | even
// alone | this: contraction N = 300 21.1 | 21.1 | 17.6 us, 520 76.1 | 89.1 | 74.7, 600 92.5 | 98.0 | 90.5; projections of the triangle
// attention N = 132 9.7 | 9.7 | 9.0, output stage N = 400 39.0 | 40.2 | 38.8.
static inline int even_grid(int64_t tiles, int64_t room, int64_t period = 1) {
  const int64_t rounds = (tiles + room - 1) / room;
  int64_t grid = (tiles + rounds - 1) / rounds;
  while (rounds > 1 && grid < room && std::gcd(grid, period) != 1) ++grid;
  return (int)grid;
}

}  // namespace px
