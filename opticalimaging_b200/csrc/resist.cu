// The parts of an optimisation iteration outside the transforms: the sigmoid resist loss with its image gradient, the
// field weights of a new source, and the source gradient from the field dot products.  The reference composes the first
// from torch operations behind its image (CalculateAerialImage_SOCS.py:3-11); as such a composition it was a dozen passes
// over the images and as many launches (8 images of 1024 x 1024: 107 us forward and backward, now 41 and 4 for the s that a
// recorded backward pass needs), the other two about twenty launches on a few hundred values.
//
// Bound: memory for the loss (image and target in, gradient and s out), the launch for the others.
#include "oi_common.cuh"
#include <algorithm>
#include <cstdint>

namespace oi {

constexpr int RL_T = 256, RL_BLOCKS = 148 * 8;

// loss += (s - t)^2, s = 1 / (1 + exp(-a (I - thr))) over images [batch][nz][n] against targets [batch][n]; with grad,
// grad = 2 (s - t) a s (1 - s), and with resist, resist = s.  Sums in FP64, per block to partial[blockIdx.x].
template <int V>
__global__ void __launch_bounds__(RL_T) resist_loss_kernel(const float* __restrict__ image, const float* __restrict__ target,
                                                           int nz, long long n, long long total, float a, float thr,
                                                           float* __restrict__ grad, float* __restrict__ resist,
                                                           double* __restrict__ partial) {
  __shared__ double sh[RL_T / 32];
  double acc = 0.0;
  auto one = [&](float I, float t, float& s) {
    s = 1.f / (1.f + expf(-(a * (I - thr))));
    const float r = s - t;
    acc += (double)r * (double)r;
    return 2.f * r * a * (s * (1.f - s));
  };
  for (long long e = ((long long)blockIdx.x * RL_T + threadIdx.x) * V; e < total; e += (long long)gridDim.x * RL_T * V) {
    const long long plane = e / n, t0 = (plane / nz) * n + (e - plane * n);
    if constexpr (V == 4) {
      const float4 I = *(const float4*)(image + e), t = *(const float4*)(target + t0);
      float4 s;
      const float4 g = make_float4(one(I.x, t.x, s.x), one(I.y, t.y, s.y), one(I.z, t.z, s.z), one(I.w, t.w, s.w));
      if (grad) *(float4*)(grad + e) = g;
      if (resist) *(float4*)(resist + e) = s;
    } else {
      float s;
      const float g = one(image[e], target[t0], s);
      if (grad) grad[e] = g;
      if (resist) resist[e] = s;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < RL_T / 32; ++i) acc += sh[i];
    partial[blockIdx.x] = acc;
  }
}

__global__ void __launch_bounds__(RL_T) resist_sum_kernel(const double* __restrict__ partial, int count, float* loss) {
  __shared__ double sh[RL_T];
  double s = 0.0;
  for (int i = threadIdx.x; i < count; i += RL_T) s += partial[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = RL_T / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = (float)sh[0];
}

// Block-wide sum, the same value in every thread.
__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (int i = 0; i < (int)blockDim.x / 32; ++i) s += sh[i];
  return s;
}

// weights[z][(p S + j) E + e] = n v_j / sum v, one block per plane z; fields = P S E.
__global__ void __launch_bounds__(512) source_weights_kernel(const double* __restrict__ v, int S, int E, int fields, double n,
                                                             float* __restrict__ weights) {
  __shared__ double sh[16];
  double s = 0.0;
  for (int j = threadIdx.x; j < S; j += 512) s += v[j];
  s = block_sum(s, sh);
  for (int k = threadIdx.x; k < fields; k += 512) weights[(long long)blockIdx.x * fields + k] = (float)(n / s * v[k / E % S]);
}

// out[b][j] = (n d_j - n / W sum_i d_i v_i) / W, d_j the sum of dots[b][z][(p S + j) E + e] over z, p, e; W = sum v.  One block
// per image b.
__global__ void __launch_bounds__(512) source_gradient_kernel(const float* __restrict__ dots, int nz, int P, int S, int E,
                                                              const double* __restrict__ v, double n, float* __restrict__ out) {
  __shared__ double sh[16];
  const float* d = dots + (long long)blockIdx.x * nz * P * S * E;
  auto sum = [&](int j) {
    double s = 0.0;
    for (int zp = 0; zp < nz * P; ++zp)
      for (int e = 0; e < E; ++e) s += (double)d[((long long)zp * S + j) * E + e];
    return s;
  };
  double w = 0.0, g = 0.0;
  for (int j = threadIdx.x; j < S; j += 512) {
    w += v[j];
    g += sum(j) * v[j];
  }
  w = block_sum(w, sh);
  g = block_sum(g, sh) * n / w;
  for (int j = threadIdx.x; j < S; j += 512) out[(long long)blockIdx.x * S + j] = (float)((n * sum(j) - g) / w);
}

}  // namespace oi

extern "C" int oi_resist_loss_workspace(long long* bytes) {
  using namespace oi;
  if (!bytes) return fail(OI_EINVAL, "oi_resist_loss_workspace: null bytes");
  *bytes = sizeof(double) * RL_BLOCKS;
  return OI_OK;
}

extern "C" int oi_resist_loss_terms(const float* image, const float* target, int batch, int nz, long long n, float steepness,
                                    float threshold, float* grad, float* resist, float* loss, void* work,
                                    long long work_bytes, void* stream) {
  using namespace oi;
  if (!image || !target || !loss || !work || batch <= 0 || nz <= 0 || n <= 0)
    return fail(OI_EINVAL, "oi_resist_loss: bad arguments");
  if (work_bytes < (long long)sizeof(double) * RL_BLOCKS)
    return fail(OI_ERANGE, "oi_resist_loss: %lld workspace bytes given, %lld needed", work_bytes, (long long)sizeof(double) * RL_BLOCKS);
  cudaStream_t s = (cudaStream_t)stream;
  const long long total = (long long)batch * nz * n;
  const bool v4 = n % 4 == 0 && ((uintptr_t)image | (uintptr_t)target | (uintptr_t)grad | (uintptr_t)resist) % 16 == 0;
  const int blocks = (int)std::min((long long)RL_BLOCKS, (long long)ceil_div(total, RL_T * (v4 ? 4 : 1)));
  auto kern = v4 ? resist_loss_kernel<4> : resist_loss_kernel<1>;
  kern<<<blocks, RL_T, 0, s>>>(image, target, nz, n, total, steepness, threshold, grad, resist, (double*)work);
  note_launch();
  if (int rc = check_launch("oi_resist_loss")) return rc;
  resist_sum_kernel<<<1, RL_T, 0, s>>>((const double*)work, blocks, loss);
  note_launch();
  return check_launch("oi_resist_loss/sum");
}

extern "C" int oi_resist_loss(const float* image, const float* target, int batch, int nz, long long n, float steepness,
                              float threshold, float* grad, float* loss, void* work, long long work_bytes, void* stream) {
  return oi_resist_loss_terms(image, target, batch, nz, n, steepness, threshold, grad, nullptr, loss, work, work_bytes, stream);
}

extern "C" int oi_source_weights(const double* values, int points, int fields_per_point, int fields, int nz, double index_image,
                                 float* weights, void* stream) {
  using namespace oi;
  if (!values || !weights || points <= 0 || fields_per_point <= 0 || nz <= 0 || fields <= 0 ||
      fields % (points * fields_per_point))
    return fail(OI_EINVAL, "oi_source_weights: bad arguments (points=%d per point=%d fields=%d)", points, fields_per_point, fields);
  source_weights_kernel<<<(unsigned)nz, 512, 0, (cudaStream_t)stream>>>(values, points, fields_per_point, fields, index_image, weights);
  note_launch();
  return check_launch("oi_source_weights");
}

extern "C" int oi_source_gradient(const float* dots, int batch, int nz, int states, int points, int fields_per_point,
                                  const double* values, double index_image, float* out, void* stream) {
  using namespace oi;
  if (!dots || !values || !out || batch <= 0 || nz <= 0 || states <= 0 || points <= 0 || fields_per_point <= 0)
    return fail(OI_EINVAL, "oi_source_gradient: bad arguments");
  source_gradient_kernel<<<(unsigned)batch, 512, 0, (cudaStream_t)stream>>>(dots, nz, states, points, fields_per_point, values,
                                                                            index_image, out);
  note_launch();
  return check_launch("oi_source_gradient");
}
