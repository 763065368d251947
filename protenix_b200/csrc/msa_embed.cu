// MSA embedding: m[s][i] = W[:, class] + W[:, 32] * has_deletion + W[:, 33] * deletion_value + s_proj[i] for the selected sequences,
// W [64][34] the weight of the linear layer over one_hot(class) | has_deletion | deletion_value.
// The one-hot product selects a column: nothing is multiplied out.  16 threads a row, four channels each, W transposed in shared
// memory; HBM-bound by the 256 bytes written per row.  With the one-hot tensor, the concatenation, a library GEMM over 34 inputs and
// the sum as separate passes 230 us at 1024 x 384, 33 us here.
#include "px_common.cuh"

namespace px {

constexpr int kMeClasses = 32, kMeIn = kMeClasses + 2, kMeC = 64, kMeLd = kMeC + 4;

__global__ void __launch_bounds__(256)
msa_embed_kernel(const long long* __restrict__ msa, const float* __restrict__ has_deletion, const float* __restrict__ deletion_value,
                 const long long* __restrict__ index, const float* __restrict__ w, const float* __restrict__ s_proj,
                 float* __restrict__ m, int s_rows, int n) {
  __shared__ __align__(16) float wt[kMeIn][kMeLd];
  pdl_wait();
  for (int i = threadIdx.x; i < kMeIn * kMeC; i += 256) wt[i % kMeIn][i / kMeIn] = w[i];
  __syncthreads();
  const int c = 4 * (threadIdx.x & 15), sub = threadIdx.x >> 4;
  const float4 wh = *reinterpret_cast<const float4*>(&wt[kMeClasses][c]), wd = *reinterpret_cast<const float4*>(&wt[kMeClasses + 1][c]);
  // blockIdx.y: a sequence; four tokens a step, so that the chain index -> class -> column is four wide
  for (int s = blockIdx.y; s < s_rows; s += gridDim.y) {
    const size_t src = (size_t)index[s] * n;
    for (int i0 = blockIdx.x * 64 + sub; i0 < n; i0 += gridDim.x * 64) {
      long long cls[4];
      float h[4], d[4];
      float4 p[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + 16 * j;
        cls[j] = -1, h[j] = d[j] = 0.f;
        p[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n) {
          cls[j] = msa[src + i], h[j] = has_deletion[src + i], d[j] = deletion_value[src + i];
          p[j] = *reinterpret_cast<const float4*>(s_proj + (size_t)i * kMeC + c);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + 16 * j;
        // a class outside the alphabet has no embedding
        const float4 e = cls[j] >= 0 && cls[j] < kMeClasses ? *reinterpret_cast<const float4*>(&wt[cls[j]][c]) : make_float4(NAN, NAN, NAN, NAN);
        if (i < n)
          *reinterpret_cast<float4*>(m + ((size_t)s * n + i) * kMeC + c) =
              make_float4(fmaf(wd.x, d[j], fmaf(wh.x, h[j], e.x)) + p[j].x, fmaf(wd.y, d[j], fmaf(wh.y, h[j], e.y)) + p[j].y,
                          fmaf(wd.z, d[j], fmaf(wh.z, h[j], e.z)) + p[j].z, fmaf(wd.w, d[j], fmaf(wh.w, h[j], e.w)) + p[j].w);
      }
    }
  }
}

}  // namespace px

extern "C" int32_t px_msa_embed(const int64_t* msa, const float* has_deletion, const float* deletion_value, const int64_t* index,
                                const float* w, const float* s_proj, float* m, int64_t s_rows, int64_t n, void* stream) {
  if (!msa || !has_deletion || !deletion_value || !index || !w || !s_proj || !m || s_rows < 0 || n <= 0 || n > 32768 ||
      s_rows > (1 << 20) || (((uintptr_t)s_proj | (uintptr_t)m) & 15))
    return PX_ERR_BAD_ARG;
  if (s_rows == 0) return PX_OK;
  const int64_t x = (n + 63) / 64, room = (8 * px::sm_count() + x - 1) / x;      // eight CTAs resident per SM
  return px::launch_pdl(px::msa_embed_kernel, dim3((unsigned)x, (unsigned)(s_rows < room ? s_rows : room)), 256, 0, (cudaStream_t)stream,
                        (const long long*)msa, has_deletion, deletion_value, (const long long*)index, w, s_proj, m, (int)s_rows, (int)n)
             ? PX_OK
             : PX_ERR_LAUNCH;
}
