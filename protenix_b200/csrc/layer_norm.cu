// Stand-alone LayerNorm forward over the last axis (general width, fp32 / bf16 / fp16).
//
// HBM-bound: 2 * cols * sizeof(T) algorithmic bytes per row.  One warp owns a row; the row is
// held in registers between the statistics and the write-back (cols <= 32*VEC*kMaxIt), so x is
// read from HBM exactly once.  VEC is the widest vector (up to 16 bytes) that divides cols.
// Rows that fit 4..32 lanes x 16 bytes (the pair representation's 128 channels in any of the three types, the
// template embedder's 64) take ln_fwd_rows16: every lane moves 16 bytes, a warp works on 32/LANES rows at once.
#include <cuda_fp16.h>

#include "px_common.cuh"

namespace px {

template <typename T>
struct Cvt;
template <>
struct Cvt<float> {
  static __device__ __forceinline__ float to_f(float v) { return v; }
  static __device__ __forceinline__ float from_f(float v) { return v; }
};
template <>
struct Cvt<bf16> {
  static __device__ __forceinline__ float to_f(bf16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ bf16 from_f(float v) { return __float2bfloat16_rn(v); }
};
template <>
struct Cvt<__half> {
  static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from_f(float v) { return __float2half_rn(v); }
};

template <typename T, int VEC>
struct alignas(sizeof(T) * VEC) Vec {
  T v[VEC];
};

// Scale and offset come in the type of x or as the fp32 parameters themselves; the latter are rounded to the type of x
// here, which gives what a cast before the call gives and saves its launches.
template <typename T, typename P>
__device__ __forceinline__ float param(P v) { return Cvt<T>::to_f(Cvt<T>::from_f(Cvt<P>::to_f(v))); }

constexpr int kMaxIt = 8;

// Launch of 256 threads a CTA that overlaps the end of the kernel before it (see pdl_wait): [384, 384] fp32 8.5 -> 7.9 us a call, forward
// and backward of [768^2, 128] bf16 141.9 -> 136.8.
template <typename... Params, typename... Args>
static cudaError_t pdl(void (*kernel)(Params...), unsigned grid, size_t smem, cudaStream_t st, Args... args) {
  return launch_pdl(kernel, dim3(grid), 256, smem, st, args...) ? cudaSuccess : cudaErrorLaunchFailure;
}

// Register-resident path: cols <= 32 * VEC * kMaxIt.
template <typename T, int VEC, typename P>
__global__ void __launch_bounds__(256) ln_fwd_cached(const T* __restrict__ x, const P* __restrict__ gamma,
                                                     const P* __restrict__ beta, T* __restrict__ y,
                                                     float* __restrict__ mean_out, float* __restrict__ invvar_out,
                                                     int64_t rows, int cols, float eps) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int nvec = cols / VEC;
  const float inv_c = 1.0f / (float)cols;
  for (int64_t row = warp0; row < rows; row += nwarps) {
    const Vec<T, VEC>* xr = reinterpret_cast<const Vec<T, VEC>*>(x + row * cols);
    float v[kMaxIt][VEC];
    float s = 0.f;
#pragma unroll
    for (int it = 0; it < kMaxIt; ++it) {
      int i = lane + 32 * it;
      if (i < nvec) {
        Vec<T, VEC> t = xr[i];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          v[it][e] = Cvt<T>::to_f(t.v[e]);
          s += v[it][e];
        }
      } else {
#pragma unroll
        for (int e = 0; e < VEC; ++e) v[it][e] = 0.f;
      }
    }
    const float mean = warp_sum(s) * inv_c;
    float q = 0.f;
#pragma unroll
    for (int it = 0; it < kMaxIt; ++it) {
      if (lane + 32 * it < nvec) {
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          float d = v[it][e] - mean;
          q += d * d;
        }
      }
    }
    const float var = fmaxf(warp_sum(q) * inv_c, 0.f);
    const float rstd = rsqrtf(var + eps);
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      if (invvar_out) invvar_out[row] = rstd;
    }
    Vec<T, VEC>* yr = reinterpret_cast<Vec<T, VEC>*>(y + row * cols);
#pragma unroll
    for (int it = 0; it < kMaxIt; ++it) {
      int i = lane + 32 * it;
      if (i < nvec) {
        Vec<P, VEC> g, b;
        Vec<T, VEC> o;
        if (gamma) g = reinterpret_cast<const Vec<P, VEC>*>(gamma)[i];
        if (beta) b = reinterpret_cast<const Vec<P, VEC>*>(beta)[i];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          float r = (v[it][e] - mean) * rstd;
          if (gamma) r *= param<T, P>(g.v[e]);
          if (beta) r += param<T, P>(b.v[e]);
          o.v[e] = Cvt<T>::from_f(r);
        }
        yr[i] = o;
      }
    }
  }
}

// Rows of exactly LANES x 16 bytes, LANES a power of two <= 32: a group of LANES lanes owns a row.  The rows in flight
// stay packed as loaded and are converted once per pass (sum, squares, output): held as floats they took 100 registers
// and a third of the warps (68 us on [768^2, 128] bf16).  Every CTA is resident, and the rows of the next round are requested
// before this one's are reduced: 51.6 us with statistics ([768^2, 128] bf16, kernel alone), 53.7 without that and with three CTAs to an SM,
// 20 % more with it and three CTAs.  From 1000 to 100 000 rows the two are within 4 % of each other either way.
constexpr int kLnFwdOcc = 2, kLnFwdGroups = 4;           // CTAs per SM, row groups in flight per warp
template <typename T, int LANES, typename P>
__global__ void __launch_bounds__(256, kLnFwdOcc) ln_fwd_rows16(const T* __restrict__ x, const P* __restrict__ gamma,
                                                                const P* __restrict__ beta, T* __restrict__ y,
                                                                float* __restrict__ mean_out, float* __restrict__ invvar_out,
                                                                int64_t rows, float eps) {
  pdl_wait();
  constexpr int VEC = 16 / (int)sizeof(T), kCols = VEC * LANES, kR = 32 / LANES, kB = kLnFwdGroups;
  const int lane = threadIdx.x & 31, sub = lane / LANES, li = lane % LANES;
  const int64_t warp0 = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  float g[VEC], b[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    g[e] = gamma ? param<T, P>(gamma[li * VEC + e]) : 1.f;
    b[e] = beta ? param<T, P>(beta[li * VEC + e]) : 0.f;
  }
  uint4 next[kB];                                          // the rows of the next round, on their way while this one's are worked on
  auto request = [&](int64_t r0) {
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const int64_t row = r0 + j * kR + sub;
      next[j] = row < rows ? __ldcs(reinterpret_cast<const uint4*>(x + row * kCols) + li) : make_uint4(0, 0, 0, 0);
    }
  };
  request(warp0 * (kB * kR));
  for (int64_t r0 = warp0 * (kB * kR); r0 < rows; r0 += nwarps * (kB * kR)) {
    uint4 raw[kB];
    float acc[kB], mean[kB];
#pragma unroll
    for (int j = 0; j < kB; ++j) raw[j] = next[j];
    request(r0 + nwarps * (kB * kR));
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const Vec<T, VEC> t = *reinterpret_cast<const Vec<T, VEC>*>(&raw[j]);
      acc[j] = 0.f;
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[j] += Cvt<T>::to_f(t.v[e]);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < kB; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const Vec<T, VEC> t = *reinterpret_cast<const Vec<T, VEC>*>(&raw[j]);
      mean[j] = acc[j] * (1.0f / kCols);
      acc[j] = 0.f;
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float d = Cvt<T>::to_f(t.v[e]) - mean[j];
        acc[j] = fmaf(d, d, acc[j]);
      }
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < kB; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const int64_t row = r0 + j * kR + sub;
      if (row < rows) {
        const Vec<T, VEC> t = *reinterpret_cast<const Vec<T, VEC>*>(&raw[j]);
        const float rstd = rsqrtf(acc[j] * (1.0f / kCols) + eps);
        if (li == 0) {
          if (mean_out) mean_out[row] = mean[j];
          if (invvar_out) invvar_out[row] = rstd;
        }
        Vec<T, VEC> o;
#pragma unroll
        for (int e = 0; e < VEC; ++e) o.v[e] = Cvt<T>::from_f(fmaf((Cvt<T>::to_f(t.v[e]) - mean[j]) * rstd, g[e], b[e]));
        __stcs(reinterpret_cast<uint4*>(y + row * kCols) + li, *reinterpret_cast<const uint4*>(&o));
      }
    }
  }
}

template <typename T, int LANES, typename P>
static cudaError_t launch_rows16(const void* x, const void* g, const void* b, void* y, float* mean, float* invvar,
                                 int64_t rows, float eps, cudaStream_t st) {
  const int64_t rows_per_cta = 8 * kLnFwdGroups * (32 / LANES);
  int64_t ctas = (rows + rows_per_cta - 1) / rows_per_cta;
  const int64_t cap = 148 * kLnFwdOcc;
  if (ctas > cap) ctas = cap;
  return pdl(ln_fwd_rows16<T, LANES, P>, (unsigned)ctas, 0, st, (const T*)x, (const P*)g, (const P*)b, (T*)y, mean, invvar, rows, eps);
}

// Wide rows: three passes over the row (the second and third hit L1/L2).
template <typename T, typename P>
__global__ void __launch_bounds__(256) ln_fwd_wide(const T* __restrict__ x, const P* __restrict__ gamma,
                                                   const P* __restrict__ beta, T* __restrict__ y,
                                                   float* __restrict__ mean_out, float* __restrict__ invvar_out,
                                                   int64_t rows, int cols, float eps) {
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const float inv_c = 1.0f / (float)cols;
  for (int64_t row = warp0; row < rows; row += nwarps) {
    const T* xr = x + row * cols;
    float s = 0.f;
    for (int i = lane; i < cols; i += 32) s += Cvt<T>::to_f(xr[i]);
    const float mean = warp_sum(s) * inv_c;
    float q = 0.f;
    for (int i = lane; i < cols; i += 32) {
      float d = Cvt<T>::to_f(xr[i]) - mean;
      q += d * d;
    }
    const float rstd = rsqrtf(fmaxf(warp_sum(q) * inv_c, 0.f) + eps);
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      if (invvar_out) invvar_out[row] = rstd;
    }
    T* yr = y + row * cols;
    for (int i = lane; i < cols; i += 32) {
      float r = (Cvt<T>::to_f(xr[i]) - mean) * rstd;
      if (gamma) r *= param<T, P>(gamma[i]);
      if (beta) r += param<T, P>(beta[i]);
      yr[i] = Cvt<T>::from_f(r);
    }
  }
}

template <typename T, int VEC, typename P>
static cudaError_t launch_cached(const void* x, const void* g, const void* b, void* y, float* mean, float* invvar,
                                 int64_t rows, int cols, float eps, cudaStream_t st) {
  const int warps_per_cta = 8;
  int64_t ctas = (rows + warps_per_cta - 1) / warps_per_cta;
  const int64_t cap = 148 * 8 * 4;  // a few waves of resident CTAs; warps stride over the rows
  if (ctas > cap) ctas = cap;
  return pdl(ln_fwd_cached<T, VEC, P>, (unsigned)ctas, 0, st, (const T*)x, (const P*)g, (const P*)b, (T*)y, mean, invvar, rows, cols, eps);
}

template <typename T, typename P>
static cudaError_t dispatch(const void* x, const void* g, const void* b, void* y, float* mean, float* invvar,
                            int64_t rows, int cols, float eps, cudaStream_t st) {
  constexpr int kMaxVec = 16 / (int)sizeof(T);
  auto aligned = [&](int vec) {
    uintptr_t m = (uintptr_t)(sizeof(T) * vec) - 1;
    return cols % vec == 0 && cols <= 32 * vec * kMaxIt && !((uintptr_t)x & m) && !((uintptr_t)y & m) &&
           !((uintptr_t)g & (sizeof(P) * vec - 1)) && !((uintptr_t)b & (sizeof(P) * vec - 1));
  };
  if (cols % kMaxVec == 0 && aligned(kMaxVec)) {       // rows of 4..32 lanes x 16 bytes
    switch (cols / kMaxVec) {
      case 32: return launch_rows16<T, 32, P>(x, g, b, y, mean, invvar, rows, eps, st);
      case 16: return launch_rows16<T, 16, P>(x, g, b, y, mean, invvar, rows, eps, st);
      case 8: return launch_rows16<T, 8, P>(x, g, b, y, mean, invvar, rows, eps, st);
      case 4: return launch_rows16<T, 4, P>(x, g, b, y, mean, invvar, rows, eps, st);
      default: break;
    }
  }
  if (kMaxVec >= 8 && aligned(8) && cols >= 32 * 8)
    return launch_cached<T, (kMaxVec >= 8 ? 8 : 1), P>(x, g, b, y, mean, invvar, rows, cols, eps, st);
  if (aligned(4)) return launch_cached<T, 4, P>(x, g, b, y, mean, invvar, rows, cols, eps, st);
  if (aligned(2)) return launch_cached<T, 2, P>(x, g, b, y, mean, invvar, rows, cols, eps, st);
  if (aligned(1)) return launch_cached<T, 1, P>(x, g, b, y, mean, invvar, rows, cols, eps, st);
  const int warps_per_cta = 8;
  int64_t ctas = (rows + warps_per_cta - 1) / warps_per_cta;
  if (ctas > 148 * 32) ctas = 148 * 32;
  ln_fwd_wide<T, P><<<(unsigned)ctas, 256, 0, st>>>((const T*)x, (const P*)g, (const P*)b, (T*)y, mean, invvar, rows,
                                                 cols, eps);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------------------------
// Backward.  With xhat = (x - mean) * invvar and g = dy * gamma (g = dy without a scale):
//   dx = invvar * (g - mean_c(g) - xhat * mean_c(g * xhat)),   dgamma = sum_rows dy * xhat,   dbeta = sum_rows dy.
// HBM-bound: dy and x in, dx out.  Rows of up to LANES x IT x 16 bytes stay in registers: a group of LANES lanes owns a
// row, a lane always the same columns, so it sums its columns' dgamma and dbeta in registers over all its rows; lane
// groups, warps and CTAs are combined once at the end (shuffles, shared memory, one atomic per column and CTA into an
// fp32 scratch, which a second kernel converts).  The row-by-row form below, with a shared-memory atomic per element,
// took 234 us on [768^2, 128] bf16 where the three tensors take 69 us at the copy rate; it is left for wider rows.
// Two CTAs to an SM and two (fp32 three) row groups a warp, the next round's requested before this one's are reduced: [768^2, 128]
// bf16 85 us, fp32 147; without the early request and with three groups 91 and 153, with it and three groups 98 in bf16, two 155 in fp32.
constexpr int kLnBwdOcc = 2;
constexpr int ln_bwd_groups(int it, int bytes) { return it == 1 ? (bytes == 4 ? 3 : 2) : it == 2 ? 2 : 1; }
template <typename T, typename P, int LANES, int IT>
__global__ void __launch_bounds__(256, IT == 1 ? kLnBwdOcc : 1) ln_bwd_rows(const T* __restrict__ dy, const T* __restrict__ x,
                                                   const float* __restrict__ mean, const float* __restrict__ invvar,
                                                   const P* __restrict__ gamma, T* __restrict__ dx,
                                                   float* __restrict__ scratch, long long rows, int cols) {
  pdl_wait();
  constexpr int VEC = 16 / (int)sizeof(T), kR = 32 / LANES;
  constexpr int kB = ln_bwd_groups(IT, (int)sizeof(T));                  // row groups in flight per warp
  extern __shared__ float ln_bwd_sums[];                 // [8 warps][2][cols]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / LANES, li = lane % LANES;
  const int nvec = cols / VEC;
  const float inv_cols = 1.0f / (float)cols;
  float gm[IT][VEC], dg[IT][VEC], db[IT][VEC];
#pragma unroll
  for (int i = 0; i < IT; ++i)
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const int v = li + LANES * i;
      gm[i][e] = gamma && v < nvec ? param<T, P>(gamma[v * VEC + e]) : 1.f;
      dg[i][e] = db[i][e] = 0.f;
    }
  const long long step = (long long)gridDim.x * 8 * kR * kB;
  // the rows of the next round are on their way while this one's are worked on
  uint4 nx[kB][IT], ny[kB][IT];
  float nmu[kB], nrs[kB];
  auto request = [&](long long r0) {
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const long long row = r0 + j * kR + sub;
      const bool in = row < rows;
      nmu[j] = in ? __ldg(mean + row) : 0.f;
      nrs[j] = in ? __ldg(invvar + row) : 0.f;
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        const int v = li + LANES * i;
        const bool have = in && v < nvec;                // absent values count as zero everywhere
        nx[j][i] = have ? __ldcs(reinterpret_cast<const uint4*>(x + (size_t)row * cols) + v) : make_uint4(0, 0, 0, 0);
        ny[j][i] = have ? __ldcs(reinterpret_cast<const uint4*>(dy + (size_t)row * cols) + v) : make_uint4(0, 0, 0, 0);
      }
    }
  };
  const long long begin = ((long long)blockIdx.x * 8 + warp) * (kR * kB);
  request(begin);
  for (long long r0 = begin; r0 < rows; r0 += step) {
    uint4 rx[kB][IT], ry[kB][IT];
    float mu[kB], rs[kB];
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      mu[j] = nmu[j], rs[j] = nrs[j];
#pragma unroll
      for (int i = 0; i < IT; ++i) rx[j][i] = nx[j][i], ry[j][i] = ny[j][i];
    }
    request(r0 + step);
    float s1[kB], s2[kB];
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      s1[j] = s2[j] = 0.f;
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        const Vec<T, VEC> xv = *reinterpret_cast<const Vec<T, VEC>*>(&rx[j][i]), yv = *reinterpret_cast<const Vec<T, VEC>*>(&ry[j][i]);
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          const float d = Cvt<T>::to_f(yv.v[e]), xh = (Cvt<T>::to_f(xv.v[e]) - mu[j]) * rs[j], g = d * gm[i][e];
          s1[j] += g;
          s2[j] = fmaf(g, xh, s2[j]);
          dg[i][e] = fmaf(d, xh, dg[i][e]);
          db[i][e] += d;
        }
      }
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        s1[j] += __shfl_xor_sync(0xffffffffu, s1[j], o);
        s2[j] += __shfl_xor_sync(0xffffffffu, s2[j], o);
      }
#pragma unroll
    for (int j = 0; j < kB; ++j) {
      const long long row = r0 + j * kR + sub;
      const float m1 = s1[j] * inv_cols, m2 = s2[j] * inv_cols;
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        const int v = li + LANES * i;
        if (row < rows && v < nvec) {
          const Vec<T, VEC> xv = *reinterpret_cast<const Vec<T, VEC>*>(&rx[j][i]), yv = *reinterpret_cast<const Vec<T, VEC>*>(&ry[j][i]);
          Vec<T, VEC> o;
#pragma unroll
          for (int e = 0; e < VEC; ++e) {
            const float xh = (Cvt<T>::to_f(xv.v[e]) - mu[j]) * rs[j];
            o.v[e] = Cvt<T>::from_f(rs[j] * (Cvt<T>::to_f(yv.v[e]) * gm[i][e] - m1 - xh * m2));
          }
          __stcs(reinterpret_cast<uint4*>(dx + (size_t)row * cols) + v, *reinterpret_cast<const uint4*>(&o));
        }
      }
    }
  }
  if (!scratch) return;
#pragma unroll
  for (int i = 0; i < IT; ++i)
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
#pragma unroll
      for (int o = LANES; o < 32; o <<= 1) {
        dg[i][e] += __shfl_xor_sync(0xffffffffu, dg[i][e], o);
        db[i][e] += __shfl_xor_sync(0xffffffffu, db[i][e], o);
      }
      const int v = li + LANES * i;
      if (sub == 0 && v < nvec) {
        ln_bwd_sums[(2 * warp) * cols + v * VEC + e] = dg[i][e];
        ln_bwd_sums[(2 * warp + 1) * cols + v * VEC + e] = db[i][e];
      }
    }
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * cols; c += blockDim.x) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += ln_bwd_sums[2 * w * cols + c];
    atomicAdd(&scratch[c], t);
  }
}

// Wide or unaligned rows: one warp per row, two passes over it (the second is served by L1/L2), the column sums of a
// CTA's rows collected in shared memory.
template <typename T, typename P>
__global__ void __launch_bounds__(256) ln_bwd_wide(const T* __restrict__ dy, const T* __restrict__ x,
                                                     const float* __restrict__ mean, const float* __restrict__ invvar,
                                                     const P* __restrict__ gamma, T* __restrict__ dx,
                                                     float* __restrict__ scratch, long long rows, int cols) {
  extern __shared__ float ln_bwd_sums[];                 // [2][cols]: dgamma, dbeta partial sums of this CTA
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  if (scratch) {
    for (int c = threadIdx.x; c < 2 * cols; c += blockDim.x) ln_bwd_sums[c] = 0.f;
    __syncthreads();
  }
  const float inv_cols = 1.0f / (float)cols;
  for (long long row = (long long)blockIdx.x * warps + warp; row < rows; row += (long long)gridDim.x * warps) {
    const T* xr = x + (size_t)row * cols;
    const T* dyr = dy + (size_t)row * cols;
    const float mu = mean[row], rs = invvar[row];
    float s1 = 0.f, s2 = 0.f;
    for (int c = lane; c < cols; c += 32) {
      const float g = Cvt<T>::to_f(dyr[c]) * (gamma ? param<T, P>(gamma[c]) : 1.0f);
      s1 += g;
      s2 += g * ((Cvt<T>::to_f(xr[c]) - mu) * rs);
    }
    s1 = warp_sum(s1) * inv_cols;
    s2 = warp_sum(s2) * inv_cols;
    T* dxr = dx + (size_t)row * cols;
    for (int c = lane; c < cols; c += 32) {
      const float d = Cvt<T>::to_f(dyr[c]), xh = (Cvt<T>::to_f(xr[c]) - mu) * rs;
      const float g = d * (gamma ? param<T, P>(gamma[c]) : 1.0f);
      dxr[c] = Cvt<T>::from_f(rs * (g - s1 - xh * s2));
      if (scratch) {
        atomicAdd(&ln_bwd_sums[c], d * xh);
        atomicAdd(&ln_bwd_sums[cols + c], d);
      }
    }
  }
  if (scratch) {
    __syncthreads();
    for (int c = threadIdx.x; c < 2 * cols; c += blockDim.x) atomicAdd(&scratch[c], ln_bwd_sums[c]);
  }
}

// A kernel and not a memset: between kernels alone a launch overlaps the end of the kernel before it.
__global__ void __launch_bounds__(256) ln_bwd_zero_kernel(float* __restrict__ scratch, int n) {
  pdl_wait();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) scratch[i] = 0.f;
}

// The sums are rounded to the type of x, whatever the type of the gradients (fp32 parameters of a 16-bit x).
template <typename T, typename P>
__global__ void ln_bwd_finish_kernel(const float* __restrict__ scratch, P* __restrict__ dgamma, P* __restrict__ dbeta,
                                     int cols) {
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  if (dgamma) dgamma[c] = Cvt<P>::from_f(Cvt<T>::to_f(Cvt<T>::from_f(scratch[c])));
  if (dbeta) dbeta[c] = Cvt<P>::from_f(Cvt<T>::to_f(Cvt<T>::from_f(scratch[cols + c])));
}

template <typename T, typename P, int LANES, int IT>
static cudaError_t launch_bwd_rows(const void* dy, const void* x, const float* mean, const float* invvar, const void* gamma,
                                   void* dx, float* scratch, long long rows, int cols, int sms, cudaStream_t st) {
  constexpr int kB = ln_bwd_groups(IT, (int)sizeof(T)), kRows = 8 * (32 / LANES) * kB;
  const size_t smem = scratch ? (size_t)16 * cols * sizeof(float) : 0;
  const long long want = (rows + kRows - 1) / kRows;
  const int grid = (int)(want < kLnBwdOcc * sms ? want : (long long)kLnBwdOcc * sms);   // resident CTAs: every extra one adds 2 * cols atomics
  return pdl(ln_bwd_rows<T, P, LANES, IT>, (unsigned)grid, smem, st, (const T*)dy, (const T*)x, mean, invvar, (const P*)gamma, (T*)dx,
             scratch, rows, cols);
}

template <typename T, typename P>
static cudaError_t dispatch_bwd(const void* dy, const void* x, const float* mean, const float* invvar, const void* gamma,
                                void* dx, void* dgamma, void* dbeta, float* scratch, long long rows, int cols,
                                cudaStream_t st) {
  const bool sums = dgamma || dbeta;
  if (!sums) scratch = nullptr;
  if (sums) {
    const cudaError_t e = pdl(ln_bwd_zero_kernel, (unsigned)((2 * cols + 255) / 256), 0, st, scratch, 2 * cols);
    if (e != cudaSuccess) return e;
  }
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (rows > 0) {
    constexpr int kVec = 16 / (int)sizeof(T);
    const int nvec = cols % kVec == 0 && !(((uintptr_t)dy | (uintptr_t)x | (uintptr_t)dx) & 15) ? cols / kVec : 1 << 30;
    cudaError_t e;
    // the registers of a lane hold IT vectors of x, dy, gamma and both sums: up to 16 columns
    if (nvec <= 8) e = launch_bwd_rows<T, P, 8, 1>(dy, x, mean, invvar, gamma, dx, scratch, rows, cols, sms, st);
    else if (nvec <= 16) e = launch_bwd_rows<T, P, 16, 1>(dy, x, mean, invvar, gamma, dx, scratch, rows, cols, sms, st);
    else if (nvec <= 32) e = launch_bwd_rows<T, P, 32, 1>(dy, x, mean, invvar, gamma, dx, scratch, rows, cols, sms, st);
    else if (nvec <= 64) e = launch_bwd_rows<T, P, 32, 2>(dy, x, mean, invvar, gamma, dx, scratch, rows, cols, sms, st);
    else if (kVec == 4 && nvec <= 96) e = launch_bwd_rows<T, P, 32, (kVec == 4 ? 3 : 1)>(dy, x, mean, invvar, gamma, dx, scratch, rows, cols, sms, st);
    else {
      const size_t smem = sums ? (size_t)2 * cols * sizeof(float) : 0;
      if (smem > 48 * 1024 &&
          cudaFuncSetAttribute(ln_bwd_wide<T, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return cudaErrorInvalidValue;
      const long long want = (rows + 7) / 8;
      const int grid = (int)(want < 4ll * sms ? want : 4ll * sms);
      ln_bwd_wide<T, P><<<grid, 256, smem, st>>>((const T*)dy, (const T*)x, mean, invvar, (const P*)gamma, (T*)dx, scratch, rows,
                                                 cols);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) return e;
  }
  if (sums)
    return pdl(ln_bwd_finish_kernel<T, P>, (unsigned)((cols + 255) / 256), 0, st, (const float*)scratch, (P*)dgamma, (P*)dbeta, cols);
  return cudaSuccess;
}

// Calls f<T, P> for the type of x and of the parameters (that of x, or fp32).
#define PX_LN_DISPATCH(f, ...)                                                                    \
  (dtype == PX_F32    ? f<float, float>(__VA_ARGS__)                                              \
   : dtype == PX_BF16 ? (params == PX_F32 ? f<bf16, float>(__VA_ARGS__) : f<bf16, bf16>(__VA_ARGS__)) \
                      : (params == PX_F32 ? f<__half, float>(__VA_ARGS__) : f<__half, __half>(__VA_ARGS__)))

static bool ln_types_ok(int dtype, int params) {
  return (dtype == PX_F32 || dtype == PX_BF16 || dtype == PX_F16) && (params == dtype || params == PX_F32);
}

}  // namespace px

extern "C" int32_t px_layer_norm_bwd_params(const void* dy, const void* x, const float* mean, const float* invvar,
                                            const void* gamma, void* dx, void* dgamma, void* dbeta, float* scratch,
                                            int64_t rows, int64_t cols, int32_t dtype, int32_t params, void* stream) {
  using namespace px;
  if (cols <= 0 || cols > 16384 || rows < 0) return PX_ERR_BAD_ARG;
  if ((dgamma || dbeta) && !scratch) return PX_ERR_BAD_ARG;
  if (rows > 0 && (!dy || !x || !mean || !invvar || !dx)) return PX_ERR_BAD_ARG;
  if (!ln_types_ok(dtype, params)) return PX_ERR_UNSUPPORTED;
  // rows == 0 still runs the (empty) reduction so that the parameter gradients come out as zeros
  const cudaError_t e = PX_LN_DISPATCH(dispatch_bwd, dy, x, mean, invvar, gamma, dx, dgamma, dbeta, scratch, rows, (int)cols,
                                       (cudaStream_t)stream);
  return e == cudaSuccess ? PX_OK : PX_ERR_LAUNCH;
}

extern "C" int32_t px_layer_norm_bwd(const void* dy, const void* x, const float* mean, const float* invvar,
                                     const void* gamma, void* dx, void* dgamma, void* dbeta, float* scratch,
                                     int64_t rows, int64_t cols, int32_t dtype, void* stream) {
  return px_layer_norm_bwd_params(dy, x, mean, invvar, gamma, dx, dgamma, dbeta, scratch, rows, cols, dtype, dtype, stream);
}

extern "C" int32_t px_layer_norm_fwd_params(const void* x, const void* gamma, const void* beta, void* y, float* mean,
                                            float* invvar, int64_t rows, int64_t cols, float eps, int32_t dtype,
                                            int32_t params, void* stream) {
  using namespace px;
  if (rows == 0 && cols > 0) return PX_OK;  // empty input: nothing to launch, pointers may be null
  if (!x || !y || rows < 0 || cols <= 0 || cols > (1 << 30)) return PX_ERR_BAD_ARG;
  if (!ln_types_ok(dtype, params)) return PX_ERR_UNSUPPORTED;
  const cudaError_t e =
      PX_LN_DISPATCH(dispatch, x, gamma, beta, y, mean, invvar, rows, (int)cols, eps, (cudaStream_t)stream);
  return e == cudaSuccess ? PX_OK : PX_ERR_LAUNCH;
}

extern "C" int32_t px_layer_norm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean,
                                     float* invvar, int64_t rows, int64_t cols, float eps, int32_t dtype,
                                     void* stream) {
  return px_layer_norm_fwd_params(x, gamma, beta, y, mean, invvar, rows, cols, eps, dtype, dtype, stream);
}
