// Row-wise steps of the MSA stack on an fp32 MSA embedding m [S][N][64] (c_m = 64), each one pass over m:
//   msa_opm_prep    a_t, b_t [(i, c)][s] fp16 = mask * LN(m) W_1^T, LN(m) W_2^T (32 columns each): the operands of px_opm_outer
//   msa_values      v [8 heads][3][j][8 s + c] = LN(m) W_mv^T as three bf16 planes: the right-hand side of the pair-weighted average
//   msa_gate_out    m += W_out( sigmoid(LN(m) W_mg^T) * wv ), wv [8][i][8 s + c] as the average leaves it (msa_average_tc.cu)
// Each is LayerNorm and one or two 64 x 64 products per row (8192 FLOP against 256 bytes read), in fp32 on the FMA pipe as before;
// what they replace were library GEMMs with the LayerNorm, the mask, the gate, the residual and the permutations as separate
// passes over tensors of m's size (100 MB at S = 1024, N = 384).
//
// CTA = one token and 128 sequences, 256 threads.  The rows (256 bytes each, N * 256 apart) go through the LayerNorm into shared
// memory, 16 lanes a row; a thread then owns 8 rows x 4 columns of the product (per 4 inputs: 8 broadcast and 4 contiguous
// 16-byte reads against 128 FMAs).  With the token fixed, the transposed results are runs of 128 sequences: 256 bytes of
// fp16 per (i, c), 2 KB per head and plane.
#include "px_split.cuh"

namespace px {

constexpr int kMrRows = 128, kMrC = 64, kMrLd = kMrC + 4;
constexpr int kMrThreads = 256;

struct MrSmem {
  float x[kMrRows][kMrLd];      // LN(m), later the gated average
  float w[kMrC][kMrC];          // [input][output]
};

__device__ __forceinline__ float group16_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// w[k][n] = W[n][k] for a row-major [64 outputs][64 inputs] weight.
__device__ __forceinline__ void load_w(MrSmem& sm, const float* __restrict__ w) {
  for (int i = threadIdx.x; i < kMrC * kMrC / 4; i += kMrThreads) {
    const int n = i & 63, k = 4 * (i >> 6);
    const float4 v = __ldg(reinterpret_cast<const float4*>(w + n * kMrC + k));
    sm.w[k][n] = v.x, sm.w[k + 1][n] = v.y, sm.w[k + 2][n] = v.z, sm.w[k + 3][n] = v.w;
  }
}

// LayerNorm of the CTA's rows (sequences s0.., token i) into sm.x; rows past the end are zero.
__device__ __forceinline__ void load_rows(MrSmem& sm, const float* __restrict__ m, const float* __restrict__ gamma,
                                          const float* __restrict__ beta, int n, int i, int s0, int s_rows, float eps) {
  const int li = threadIdx.x & 15, g = threadIdx.x >> 4;
  const float4 gm = gamma ? *reinterpret_cast<const float4*>(gamma + 4 * li) : make_float4(1.f, 1.f, 1.f, 1.f);
  const float4 bt = beta ? *reinterpret_cast<const float4*>(beta + 4 * li) : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int s = s0 + 16 * j + g;
    v[j] = s < s_rows ? *reinterpret_cast<const float4*>(m + ((size_t)s * n + i) * kMrC + 4 * li) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float mean = group16_sum((v[j].x + v[j].y) + (v[j].z + v[j].w)) * (1.0f / kMrC);
    v[j].x -= mean, v[j].y -= mean, v[j].z -= mean, v[j].w -= mean;
    const float var = group16_sum(fmaf(v[j].x, v[j].x, v[j].y * v[j].y) + fmaf(v[j].z, v[j].z, v[j].w * v[j].w)) * (1.0f / kMrC);
    const float rstd = rsqrtf(var + eps);
    const bool in = s0 + 16 * j + g < s_rows;
    const float4 o = make_float4(fmaf(v[j].x * rstd, gm.x, bt.x), fmaf(v[j].y * rstd, gm.y, bt.y), fmaf(v[j].z * rstd, gm.z, bt.z),
                                 fmaf(v[j].w * rstd, gm.w, bt.w));
    *reinterpret_cast<float4*>(&sm.x[16 * j + g][4 * li]) = in ? o : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// acc[a][b] = row ty + 16 a, column 4 tx + b of x w.
__device__ __forceinline__ void product(const MrSmem& sm, float (&acc)[8][4], int ty, int tx) {
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
#pragma unroll 4
  for (int k = 0; k < kMrC; k += 4) {
    float4 w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = *reinterpret_cast<const float4*>(&sm.w[k + e][4 * tx]);
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const float4 x = *reinterpret_cast<const float4*>(&sm.x[ty + 16 * a][k]);
      const float xe[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[a][0] = fmaf(xe[e], w[e].x, acc[a][0]);
        acc[a][1] = fmaf(xe[e], w[e].y, acc[a][1]);
        acc[a][2] = fmaf(xe[e], w[e].z, acc[a][2]);
        acc[a][3] = fmaf(xe[e], w[e].w, acc[a][3]);
      }
    }
  }
}

__global__ void __launch_bounds__(kMrThreads, 3)
msa_opm_prep_kernel(const float* __restrict__ m, const float* __restrict__ mask, const float* __restrict__ gamma,
                    const float* __restrict__ beta, const float* __restrict__ w_1, const float* __restrict__ w_2,
                    __half* __restrict__ a_t, __half* __restrict__ b_t, int n, int s_rows, int ld, float eps) {
  extern __shared__ __align__(16) unsigned char mr_raw[];
  MrSmem& sm = *reinterpret_cast<MrSmem*>(mr_raw);
  pdl_wait();
  const int i = blockIdx.x, s0 = blockIdx.y * kMrRows, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int j = threadIdx.x; j < kMrC * kMrC / 4; j += kMrThreads) {   // columns 0..31 from W_1, 32..63 from W_2
    const int c = j & 63, k = 4 * (j >> 6);
    const float4 v = __ldg(reinterpret_cast<const float4*>((c < 32 ? w_1 + c * kMrC : w_2 + (c - 32) * kMrC) + k));
    sm.w[k][c] = v.x, sm.w[k + 1][c] = v.y, sm.w[k + 2][c] = v.z, sm.w[k + 3][c] = v.w;
  }
  load_rows(sm, m, gamma, beta, n, i, s0, s_rows, eps);
  __syncthreads();
  float acc[8][4];
  product(sm, acc, ty, tx);
  __syncthreads();
  // transposed through shared memory: [64 columns][128 sequences] fp16, rows of 136
  __half* t = reinterpret_cast<__half*>(&sm.x[0][0]);
  constexpr int kT = kMrRows + 8;
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int s = s0 + ty + 16 * a;
    const float mk = mask && s < s_rows ? __ldg(mask + (size_t)s * n + i) : 1.f;
#pragma unroll
    for (int b = 0; b < 4; ++b) t[(4 * tx + b) * kT + ty + 16 * a] = __float2half_rn(acc[a][b] * mk);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < kMrC * (kMrRows / 8); j += kMrThreads) {   // ld: S rounded up to 8, the padding zero
    const int c = j >> 4, s = s0 + 8 * (j & 15);
    if (s < ld) {
      __half* dst = (c < 32 ? a_t : b_t) + ((size_t)i * 32 + (c & 31)) * ld + s;
      *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(t + c * kT + 8 * (j & 15));
    }
  }
}

__global__ void __launch_bounds__(kMrThreads, 3)
msa_values_kernel(const float* __restrict__ m, const float* __restrict__ gamma, const float* __restrict__ beta,
                  const float* __restrict__ w, bf16* __restrict__ v, int n, int s_rows, float eps) {
  extern __shared__ __align__(16) unsigned char mr_raw[];
  MrSmem& sm = *reinterpret_cast<MrSmem*>(mr_raw);
  pdl_wait();
  const int i = blockIdx.x, s0 = blockIdx.y * kMrRows, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_w(sm, w);
  load_rows(sm, m, gamma, beta, n, i, s0, s_rows, eps);
  __syncthreads();
  float acc[8][4];
  product(sm, acc, ty, tx);
  __syncthreads();                                   // x and w have been read
  // [plane][head][128 sequences][8 channels], heads 2080 bytes apart
  unsigned char* t = mr_raw;
  constexpr int kHead = kMrRows * 16 + 32;
  static_assert(24 * kHead <= (int)sizeof(MrSmem), "staging");
  const int h = tx >> 1, c = 4 * (tx & 1);           // columns 4 tx.. = head tx / 2, channels 4 (tx & 1)..
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    uint32_t lo[3], hi[3];
    split3x2(acc[a][0], acc[a][1], lo);
    split3x2(acc[a][2], acc[a][3], hi);
#pragma unroll
    for (int p = 0; p < 3; ++p)
      *reinterpret_cast<uint2*>(t + (p * 8 + h) * kHead + (ty + 16 * a) * 16 + 2 * c) = make_uint2(lo[p], hi[p]);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < 24 * kMrRows; j += kMrThreads) {
    const int ph = j / kMrRows, s = j % kMrRows;     // ph = 8 plane + head
    if (s0 + s < s_rows)
      *reinterpret_cast<uint4*>(v + ((((size_t)(ph & 7) * 3 + (ph >> 3)) * n + i) * s_rows + s0 + s) * 8) =
          *reinterpret_cast<const uint4*>(t + ph * kHead + s * 16);
  }
}

__global__ void __launch_bounds__(kMrThreads, 3)
msa_gate_out_kernel(float* __restrict__ m, const float* __restrict__ wv, const float* __restrict__ gamma,
                    const float* __restrict__ beta, const float* __restrict__ w_g, const float* __restrict__ w_out, int n,
                    int s_rows, float eps) {
  extern __shared__ __align__(16) unsigned char mr_raw[];
  MrSmem& sm = *reinterpret_cast<MrSmem*>(mr_raw);
  pdl_wait();
  const int i = blockIdx.x, s0 = blockIdx.y * kMrRows, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_w(sm, w_g);
  load_rows(sm, m, gamma, beta, n, i, s0, s_rows, eps);
  __syncthreads();
  float acc[8][4];
  product(sm, acc, ty, tx);
  __syncthreads();                                   // x and w have been read
  const int h = tx >> 1, c = 4 * (tx & 1);
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int s = s0 + ty + 16 * a;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s < s_rows) o = __ldcs(reinterpret_cast<const float4*>(wv + (((size_t)h * n + i) * s_rows + s) * 8 + c));
    o.x *= 1.0f / (1.0f + expf(-acc[a][0])), o.y *= 1.0f / (1.0f + expf(-acc[a][1]));
    o.z *= 1.0f / (1.0f + expf(-acc[a][2])), o.w *= 1.0f / (1.0f + expf(-acc[a][3]));
    *reinterpret_cast<float4*>(&sm.x[ty + 16 * a][4 * tx]) = o;
  }
  load_w(sm, w_out);
  __syncthreads();
  product(sm, acc, ty, tx);
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    const int s = s0 + ty + 16 * a;
    if (s < s_rows) {
      float4* p = reinterpret_cast<float4*>(m + ((size_t)s * n + i) * kMrC + 4 * tx);
      float4 r = *p;
      r.x += acc[a][0], r.y += acc[a][1], r.z += acc[a][2], r.w += acc[a][3];
      *p = r;
    }
  }
}

static bool mr_ok(const void* m, int64_t s_rows, int64_t n) {
  return m && !((uintptr_t)m & 15) && s_rows > 0 && n > 0 && s_rows <= (1 << 20) && n <= 32768 && (s_rows + kMrRows - 1) / kMrRows <= 65535;
}
static dim3 mr_grid(int64_t s_rows, int64_t n) { return dim3((unsigned)n, (unsigned)((s_rows + kMrRows - 1) / kMrRows)); }

}  // namespace px

using namespace px;

extern "C" int32_t px_msa_opm_prep(const float* m, const float* mask, const float* ln_w, const float* ln_b, const float* w_1,
                                   const float* w_2, px_f16* a_t, px_f16* b_t, int64_t s_rows, int64_t n, int64_t ld, float eps,
                                   void* stream) {
  if (!mr_ok(m, s_rows, n) || !w_1 || !w_2 || !a_t || !b_t || ld != (s_rows + 7) / 8 * 8) return PX_ERR_BAD_ARG;
  if (((uintptr_t)ln_w | (uintptr_t)ln_b | (uintptr_t)w_1 | (uintptr_t)w_2 | (uintptr_t)a_t | (uintptr_t)b_t) & 15) return PX_ERR_BAD_ARG;
  static SmemLimit limit;
  return limit.set(msa_opm_prep_kernel, sizeof(MrSmem)) &&
                 launch_pdl(msa_opm_prep_kernel, mr_grid(s_rows, n), kMrThreads, sizeof(MrSmem), (cudaStream_t)stream, m, mask, ln_w,
                            ln_b, w_1, w_2, (__half*)a_t, (__half*)b_t, (int)n, (int)s_rows, (int)ld, eps)
             ? PX_OK
             : PX_ERR_LAUNCH;
}

extern "C" int32_t px_msa_values(const float* m, const float* ln_w, const float* ln_b, const float* w, px_bf16* v, int64_t s_rows,
                                 int64_t n, float eps, void* stream) {
  if (!mr_ok(m, s_rows, n) || !w || !v || (((uintptr_t)ln_w | (uintptr_t)ln_b | (uintptr_t)w | (uintptr_t)v) & 15)) return PX_ERR_BAD_ARG;
  static SmemLimit limit;
  return limit.set(msa_values_kernel, sizeof(MrSmem)) &&
                 launch_pdl(msa_values_kernel, mr_grid(s_rows, n), kMrThreads, sizeof(MrSmem), (cudaStream_t)stream, m, ln_w, ln_b, w,
                            (bf16*)v, (int)n, (int)s_rows, eps)
             ? PX_OK
             : PX_ERR_LAUNCH;
}

extern "C" int32_t px_msa_gate_out(float* m, const float* wv, const float* ln_w, const float* ln_b, const float* w_g,
                                   const float* w_out, int64_t s_rows, int64_t n, float eps, void* stream) {
  if (!mr_ok(m, s_rows, n) || !wv || !w_g || !w_out) return PX_ERR_BAD_ARG;
  if (((uintptr_t)ln_w | (uintptr_t)ln_b | (uintptr_t)wv | (uintptr_t)w_g | (uintptr_t)w_out) & 15) return PX_ERR_BAD_ARG;
  static SmemLimit limit;
  return limit.set(msa_gate_out_kernel, sizeof(MrSmem)) &&
                 launch_pdl(msa_gate_out_kernel, mr_grid(s_rows, n), kMrThreads, sizeof(MrSmem), (cudaStream_t)stream, m, wv, ln_w, ln_b,
                            w_g, w_out, (int)n, (int)s_rows, eps)
             ? PX_OK
             : PX_ERR_LAUNCH;
}
