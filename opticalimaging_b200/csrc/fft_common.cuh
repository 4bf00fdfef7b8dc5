// Device helpers shared by the coarse-grid kernels (coherent_fft.cu, adjoint.cu): the 32-point transform in registers and
// the inverse four-step gather of a band-limited input.
#pragma once
#include "oi_common.cuh"

namespace oi {
namespace cg {

// cos(2 pi t / 32), t = 0..15 (exact decimal expansions of the standard values); sin via the quarter shift
__host__ __device__ constexpr float c32(int t) {
  return t == 0 ? 1.0f : t == 1 ? 0.980785280403230449f : t == 2 ? 0.923879532511286756f
       : t == 3 ? 0.831469612302545237f : t == 4 ? 0.707106781186547524f : t == 5 ? 0.555570233019602225f
       : t == 6 ? 0.382683432365089772f : t == 7 ? 0.195090322016128268f : t == 8 ? 0.0f
       : t == 9 ? -0.195090322016128268f : t == 10 ? -0.382683432365089772f : t == 11 ? -0.555570233019602225f
       : t == 12 ? -0.707106781186547524f : t == 13 ? -0.831469612302545237f : t == 14 ? -0.923879532511286756f
       : -0.980785280403230449f;
}
__host__ __device__ constexpr float s32(int t) { return t <= 8 ? c32(8 - t) : c32(t - 8); }
__host__ __device__ constexpr int brev5(int i) {
  return ((i & 1) << 4) | ((i & 2) << 2) | (i & 4) | ((i & 8) >> 2) | ((i & 16) >> 4);
}

// 32-point DFT with exp(SIGN 2 pi i k n / 32) in registers, decimation in frequency: v[i] = X[brev5(i)].
template <int SIGN>
__device__ __forceinline__ void dft32(float2 (&v)[32]) {
#pragma unroll
  for (int len = 32; len >= 2; len >>= 1) {
    const int half = len >> 1, step = 32 / len;
#pragma unroll
    for (int blk = 0; blk < 32; blk += len) {
#pragma unroll
      for (int j = 0; j < half; ++j) {
        float2 u = v[blk + j], w = v[blk + j + half];
        v[blk + j] = make_float2(u.x + w.x, u.y + w.y);
        float2 d = make_float2(u.x - w.x, u.y - w.y);
        const int t = j * step;
        if (t == 0) {
          v[blk + j + half] = d;
        } else if (t == 8) {
          v[blk + j + half] = SIGN > 0 ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);  // * (+-i)
        } else {
          const float c = c32(t), s = SIGN * s32(t);
          v[blk + j + half] = make_float2(d.x * c - d.y * s, d.x * s + d.y * c);
        }
      }
    }
  }
}
__device__ __forceinline__ void ifft32(float2 (&v)[32]) { dft32<-1>(v); }

// The coarse grids' geometry (M = 32 N1, 64 or 128 points per axis).  A band of b frequencies fits when 2 b - 1 <= M,
// so b <= B = 16 N1.  A band inside [-B/2, B/2) is kept wrapped, frequency m at place m mod B; any other is shifted
// there first: that only turns the phase of the field, which neither |E|^2 nor the adjoint's products see.
// A gather term then needs no bounds, and frequency 0, the largest by far, meets no rounded twiddle.
template <int N1> struct Axis {
  static constexpr int M = 32 * N1, B = 16 * N1;
  static constexpr int BAND_LD = B + 2;     // row of a band array: eight rows' values fall on eight bank pairs
  static constexpr int FIELD_LD = M + N1;   // row of a row-transformed array: as many rows as a half warp holds
  // where band index 0 (frequency m0) goes: index i of b is at (place0 + i) mod B
  __host__ __device__ static int place0(int m0, int b) { return (m0 >= -B / 2 && m0 + b <= B / 2 ? m0 : -B / 2) & (B - 1); }
};

// tw[t][n1] = exp(-2 pi i m n1 / M), 32 x N1, from w[j] = exp(+2 pi i j / M): m = t, or for B = 32 the frequency at place t.
template <int N1>
__device__ __forceinline__ void build_twiddles(float2* tw, const float2* w, int tid, int nthreads) {
  constexpr int M = 32 * N1;
  for (int e = tid; e < 32 * N1; e += nthreads) {
    const int t = e / N1, m = N1 == 2 && t >= 16 ? t - 32 : t;
    const float2 v = __ldg(w + ((m * (e % N1)) & (M - 1)));
    tw[e] = make_float2(v.x, -v.y);
  }
}

// Thread n1 of N1: z[i] = X[n1 + N1 brev5(i)], X[s] = sum_p src[p * stride] exp(-2 pi i m(p) s / M), p < B, m(p) = p below
// B / 2, else p - B.
template <int N1>
__device__ __forceinline__ void band_ifft(float2 (&z)[32], const float2* src, int stride, const float2* tw, int n1) {
  static_assert(N1 == 2 || N1 == 4, "coarse grids of 64 or 128");
  // the place t + 32 holds frequency t - 32: exp(+2 pi i 32 n1 / 128) = 1, i, -1, -i
  const float2 w1 = make_float2(n1 == 0 ? 1.f : n1 == 2 ? -1.f : 0.f, n1 == 1 ? 1.f : n1 == 3 ? -1.f : 0.f);
#pragma unroll
  for (int t = 0; t < 32; ++t) {
    float2 acc = src[t * stride];
    if (N1 == 4) cfma(acc, src[(t + 32) * stride], w1);
    z[t] = t == 0 ? acc : cmul(acc, tw[t * N1 + n1]);
  }
  ifft32(z);
}

}  // namespace cg
}  // namespace oi
