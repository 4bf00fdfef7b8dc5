// FFT form of the two N-point transforms of the imaging path, FP32 on the CUDA cores:
//   forward  mask -> band spectrum      (Scatter.CalculateSpectrum, Scatter.py:10-35, on the band only)
//   inverse  intensity spectrum -> image (the final synthesis of CalculateAerialImage_SOCS.py:7-10)
//
// Four-step decomposition N = 32 * N1 (N1 = 8, 16, 32, 64 for N = 256 .. 2048), x = n1 + N1 n2, k = k2 + 32 k1:
//   X[k2 + 32 k1] = sum_n1 W_N1^{k1 n1} W_N^{k2 n1} [ sum_n2 x[n1 + N1 n2] W_32^{k2 n2} ]
// Each of the N1 threads of a group owns one n1 and runs the 32-point transform in registers; the groups
// exchange through shared memory.  Only the band is wanted, so:
//   forward: the outer N1-term sum is evaluated for the band bins only (59 of 1024 at configuration 3);
//   inverse: the input is zero outside the band, so the first N1-term stage sums the few non-zero k1 only.
// Real rows travel in pairs as one complex row (x = a + i b); the forward pass separates the two spectra,
// the inverse pass builds one Hermitian spectrum per row so that the real and imaginary parts of one complex
// transform are the two output rows.
//
// Memory: the forward row pass reads each mask row once (coalesced: thread n1 reads x[n1 + N1 n2]) and writes
// the band columns transposed, [b][ic][y], so the column pass reads contiguous columns; the inverse passes
// write [b][qc][y] then rows [b][y][x], again coalesced.
#include "tc_common.cuh"
#include <cstdint>

namespace oi {

// cos / sin of 2 pi t / 32 for t = 0..15 (exact decimal expansions of the standard values)
__host__ __device__ constexpr float c32(int t) {
  return t == 0 ? 1.0f : t == 1 ? 0.980785280403230449f : t == 2 ? 0.923879532511286756f
       : t == 3 ? 0.831469612302545237f : t == 4 ? 0.707106781186547524f : t == 5 ? 0.555570233019602225f
       : t == 6 ? 0.382683432365089772f : t == 7 ? 0.195090322016128268f : t == 8 ? 0.0f
       : t == 9 ? -0.195090322016128268f : t == 10 ? -0.382683432365089772f : t == 11 ? -0.555570233019602225f
       : t == 12 ? -0.707106781186547524f : t == 13 ? -0.831469612302545237f : t == 14 ? -0.923879532511286756f
       : -0.980785280403230449f;
}
__host__ __device__ constexpr float s32(int t) { return t <= 8 ? c32(8 - t) : c32(t - 8); }
__host__ __device__ constexpr int bitrev5(int i) {
  return ((i & 1) << 4) | ((i & 2) << 2) | (i & 4) | ((i & 8) >> 2) | ((i & 16) >> 4);
}

// d * exp(SIGN 2 pi i t / 32), t a compile-time constant after unrolling
template <int SIGN>
__device__ __forceinline__ float2 rot32(float2 d, int t) {
  if (t == 0) return d;
  if (t == 8) return SIGN > 0 ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
  const float c = c32(t), s = SIGN * s32(t);
  return make_float2(d.x * c - d.y * s, d.x * s + d.y * c);
}

// In-register 32-point DFT, X[k] = sum_n v[n] exp(SIGN 2 pi i k n / 32), decimation in frequency.
// Natural-order input; on return v[i] = X[bitrev5(i)].
template <int SIGN>
__device__ __forceinline__ void fft32(float2 (&v)[32]) {
#pragma unroll
  for (int len = 32; len >= 2; len >>= 1) {
    const int half = len >> 1, step = 32 / len;
#pragma unroll
    for (int blk = 0; blk < 32; blk += len) {
#pragma unroll
      for (int j = 0; j < half; ++j) {
        float2 u = v[blk + j], w = v[blk + j + half];
        v[blk + j] = make_float2(u.x + w.x, u.y + w.y);
        v[blk + j + half] = rot32<SIGN>(make_float2(u.x - w.x, u.y - w.y), j * step);
      }
    }
  }
}

template <typename K>
static int set_smem(K kern, size_t bytes, const char* what) {
  return ensure_smem((const void*)kern, bytes, what);
}

template <int KIND> __device__ __forceinline__ float load_real(const void* f, long long i);
template <> __device__ __forceinline__ float load_real<OI_FIELD_REAL_F32>(const void* f, long long i) {
  return __ldg((const float*)f + i);
}
template <> __device__ __forceinline__ float load_real<OI_FIELD_U8>(const void* f, long long i) {
  return (float)__ldg((const uint8_t*)f + i);
}

// Twiddle tables, laid out so that a warp reading one k for all n1 touches consecutive entries:
//   t2[k2][n1] = W_N^{k2 n1}  (32 x N1)      t1[k1][n1] = W_N1^{k1 n1} = W_N^{32 k1 n1}  (N1 x N1)
// with W_N = exp(+2 pi i / N).  The four N-point kernels read them from global memory (one table per N, built
// by oi_twiddle: warp-coalesced, L1-resident); the coarse-spectrum kernel builds them in shared memory from the
// 1-D table W_M^j.  (Reading a 1-D table at index k n1 mod N across a warp is a stride-k access, up to 32-way
// bank conflicts.)
template <int N1>
__device__ __forceinline__ void build_tables(const float2* __restrict__ wn_g, float2* t2, float2* t1, int tid,
                                             int nthreads) {
  constexpr int N = 32 * N1;
  for (int e = tid; e < 32 * N1; e += nthreads) {
    const int k2 = e / N1, n1 = e % N1;
    t2[e] = __ldg(wn_g + ((k2 * n1) & (N - 1)));
  }
  for (int e = tid; e < N1 * N1; e += nthreads) {
    const int k1 = e / N1, n1 = e % N1;
    t1[e] = __ldg(wn_g + ((32 * k1 * n1) & (N - 1)));
  }
}
template <int N1>
constexpr int table_f2() { return 32 * N1 + N1 * N1; }

template <int SIGN>
__device__ __forceinline__ float2 sgn(float2 w) { return SIGN > 0 ? w : make_float2(w.x, -w.y); }

// Stage 2 + transpose: z holds the bit-reversed 32-point result of thread n1; multiply by W_N^{n1 k2} and
// store to ys[k2][n1] (row stride N1 + 1).
template <int SIGN, int N1>
__device__ __forceinline__ void twiddle_store(const float2 (&z)[32], const float2* t2, int n1, float2* ys) {
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int k2 = bitrev5(i);
    ys[k2 * (N1 + 1) + n1] = cmul(z[i], sgn<SIGN>(t2[k2 * N1 + n1]));
  }
}

// Z[k] = sum_n1 W_N1^{k1 n1} ys[k2][n1]  (forward outer stage for one bin k = k2 + 32 k1)
template <int SIGN, int N1>
__device__ __forceinline__ float2 outer_bin(const float2* ys, const float2* t1, int k) {
  const int k2 = k & 31, k1 = k >> 5;
  const float2* row = ys + k2 * (N1 + 1);
  const float2* tw = t1 + k1 * N1;
  float2 acc = make_float2(0.f, 0.f);
#pragma unroll 8
  for (int n1 = 0; n1 < N1; ++n1) cfma(acc, row[n1], sgn<SIGN>(tw[n1]));
  return acc;
}
// --------------------------------------------------------------------------------- forward, rows
// cos(2 pi t / 64) for t = 0..16 (exact decimal expansions of the standard values; the even ones are c32's), and for any
// t >= 0.  Inlined without recursion, so that a constant t leaves a constant.
__host__ __device__ __forceinline__ constexpr float c64q(int t) {
  return t == 16 ? 0.0f : t % 2 == 0 ? c32(t / 2) : t == 1 ? 0.995184726672196886f : t == 3 ? 0.956940335732208865f
       : t == 5 ? 0.881921264348355029f : t == 7 ? 0.773010453362736960f : t == 9 ? 0.634393284163645498f
       : t == 11 ? 0.471396736825997649f : t == 13 ? 0.290284677254462367f : 0.098017140329560602f;
}
__host__ __device__ __forceinline__ constexpr float c64h(int t) { return t > 16 ? -c64q(32 - t) : c64q(t); }   // t <= 32
__host__ __device__ __forceinline__ constexpr float c64(int t) { return (t & 63) > 32 ? c64h(64 - (t & 63)) : c64h(t & 63); }
__host__ __device__ __forceinline__ constexpr float s64(int t) { return c64(t + 48); }

// The outer sums of the bins k2 + 32 k1, -H <= k1 < H, from one row of twiddled values: out[k1 + H] = sum over the NT values
// n1 of row[n1] exp(+2 pi i k1 n1 / N1).  The row is read once for all 2 H bins and the twiddles are constants; +k1 and -k1
// share their products with cos and sin.
template <int N1, int H, int NT>
__device__ __forceinline__ void outer_sums(float2 (&out)[2 * H], const float2* row) {
  float2 a0 = make_float2(0.f, 0.f), last = a0, ca[H], sa[H];
#pragma unroll
  for (int p = 0; p < H; ++p) ca[p] = sa[p] = a0;
#pragma unroll
  for (int n1 = 0; n1 < NT; ++n1) {
    const float2 y = row[n1];
    a0.x += y.x;
    a0.y += y.y;
#pragma unroll
    for (int p = 1; p < H; ++p) {
      const float c = c64(64 / N1 * p * n1), s = s64(64 / N1 * p * n1);
      ca[p].x = fmaf(y.x, c, ca[p].x);
      ca[p].y = fmaf(y.y, c, ca[p].y);
      sa[p].x = fmaf(y.x, s, sa[p].x);
      sa[p].y = fmaf(y.y, s, sa[p].y);
    }
    cfma(last, y, make_float2(c64(64 / N1 * H * n1), -s64(64 / N1 * H * n1)));   // k1 = -H
  }
  out[0] = last;
  out[H] = a0;
#pragma unroll
  for (int p = 1; p < H; ++p) {
    out[H + p] = make_float2(ca[p].x - sa[p].y, ca[p].y + sa[p].x);
    out[H - p] = make_float2(ca[p].x + sa[p].y, ca[p].y - sa[p].x);
  }
}

// Real masks (float32 or uint8): field rows [nrows = batch*ny][N], two rows per group as one complex row.  Complex fields
// [batch][ny][N][nch]: rows (b, y, c), c fastest (the channels of a row share its cache lines), one per group.
// -> t[(b, c)][ic][y], ic over the band m0c .. m0c+bc-1.  Z is evaluated on the contiguous frequency range u0 .. u0+nu-1
// that holds the band and, for real rows, its mirror; H: that range lies within [-32 H, 32 H) (0: any).
// Bound: instruction issue (about 1500 a warp for two rows of 1024) and latency: 24 warps an SM, all their registers.
// With one bin per thread at a time, its twiddles read from global memory, the outer sums cost twice the loads and
// stalled on them: 4 masks of 2048 x 2048, 117 columns: 41.0 -> 30.3 us; 8 of 1024, 59: 14.2 -> 12.2.
// Two fields of 512 x 512 x 3 complex: 41.5 (as a dense product) -> 6.7 us.
template <int N1, int KIND, int H>
__global__ void __launch_bounds__(256, H == 4 ? 2 : 3) fft_rows_fwd_kernel(const void* __restrict__ field, long long nrows, int ny, int nch,
                                                           const float2* __restrict__ wn_g, int m0c, int bc, int u0,
                                                           int nu, float2* __restrict__ t, int nparts,
                                                           long long pstride) {
  // nparts > 1 (float32 only): the field is the sum of nparts arrays pstride elements apart
  constexpr bool CPLX = KIND == OI_FIELD_COMPLEX_C64;
  constexpr int N = 32 * N1, G = 256 / N1, PER = CPLX ? 1 : 2;  // G groups per block, PER rows each
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const float2* t2 = wn_g;                    // global [32][N1], read through L1 (warp-coalesced)
  const float2* t1 = wn_g + 32 * N1;          // global [N1][N1]
  float2* ys = (float2*)smem_raw;             // [G][32][N1+1]
  float2* zs = ys + G * 32 * (N1 + 1);        // [G][nu]
  const int tid = threadIdx.x, g = tid / N1, n1 = tid % N1;
  const long long r0 = (long long)blockIdx.x * (PER * G) + PER * g;
  float2 z[32];
  if constexpr (CPLX) {
    if (r0 < nrows) {
      const float2* f = (const float2*)field + (r0 / nch * N + n1) * nch + r0 % nch;
      const long long step = (long long)N1 * nch;
#pragma unroll
      for (int n2 = 0; n2 < 32; ++n2) z[n2] = __ldg(f + n2 * step);
    } else {
#pragma unroll
      for (int n2 = 0; n2 < 32; ++n2) z[n2] = make_float2(0.f, 0.f);
    }
  } else {
    if (r0 + 1 < nrows) {
      const long long o0 = r0 * N, o1 = o0 + N;
#pragma unroll
      for (int n2 = 0; n2 < 32; ++n2)
        z[n2] = make_float2(load_real<KIND>(field, o0 + n1 + N1 * n2), load_real<KIND>(field, o1 + n1 + N1 * n2));
      for (int p = 1; p < nparts; ++p) {
        const long long op = p * pstride;
#pragma unroll
        for (int n2 = 0; n2 < 32; ++n2) {
          z[n2].x += load_real<KIND>(field, op + o0 + n1 + N1 * n2);
          z[n2].y += load_real<KIND>(field, op + o1 + n1 + N1 * n2);
        }
      }
    } else {
#pragma unroll
      for (int n2 = 0; n2 < 32; ++n2) z[n2] = make_float2(0.f, 0.f);
    }
  }
  fft32<+1>(z);
  float2* yg = ys + g * 32 * (N1 + 1);
  twiddle_store<+1, N1>(z, t2, n1, yg);
  __syncthreads();
  float2* zg = zs + g * nu;
  if constexpr (H == 0) {
    for (int q = n1; q < nu; q += N1) zg[q] = outer_bin<+1, N1>(yg, t1, (u0 + q) & (N - 1));
  } else {
    // k2 = n1 + N1 j, all N1 terms; N1 = 64: k2 = n1 % 32, the upper half of the threads the upper half of the terms, whose
    // twiddles are those of the lower half times (-1)^k1
    constexpr int NT = N1 < 32 ? N1 : 32;
    const bool upper = N1 == 64 && n1 >= 32;
#pragma unroll
    for (int k2 = n1 & 31; k2 < 32; k2 += NT) {
      float2 o[2 * H];
      outer_sums<N1, H, NT>(o, yg + k2 * (N1 + 1) + (upper ? 32 : 0));
      if constexpr (N1 == 64) {
        if (upper) {
#pragma unroll
          for (int i = 0; i < 2 * H; ++i) {
            const int q = k2 + 32 * (i - H) - u0;
            const float sg = (i - H) & 1 ? -1.f : 1.f;
            if (q >= 0 && q < nu) zg[q] = make_float2(sg * o[i].x, sg * o[i].y);
          }
        }
        __syncthreads();
      }
      if (!upper) {
#pragma unroll
        for (int i = 0; i < 2 * H; ++i) {
          const int q = k2 + 32 * (i - H) - u0;
          if (q < 0 || q >= nu) continue;
          if (N1 == 64) {
            const float2 v = zg[q];
            o[i].x += v.x;
            o[i].y += v.y;
          }
          zg[q] = o[i];
        }
      }
    }
  }
  __syncthreads();
  const long long rblk = (long long)blockIdx.x * (PER * G);
  if constexpr (CPLX) {
    for (int e = tid; e < bc * G; e += 256) {
      const int ic = e / G, gg = e % G;
      const long long r = rblk + gg;
      if (r >= nrows) continue;
      const long long line = r / nch, b = line / ny;
      t[((b * nch + r % nch) * bc + ic) * (long long)ny + line - b * ny] = zs[gg * nu + (m0c + ic - u0)];
    }
    return;
  }
  // separate the two real rows and write t[b][ic][y] with y fastest (2G consecutive rows of one image)
  for (int e = tid; e < bc * 2 * G; e += 256) {
    const int ic = e / (2 * G), rr = e % (2 * G), gg = rr >> 1;
    const long long r = rblk + rr;
    if (r >= nrows) continue;
    const int m = m0c + ic;
    const float2 zp = zs[gg * nu + (m - u0)], zm = zs[gg * nu + (-m - u0)];
    float2 v;
    if ((rr & 1) == 0) v = make_float2(0.5f * (zp.x + zm.x), 0.5f * (zp.y - zm.y));   // (Z(m) + conj Z(-m)) / 2
    else v = make_float2(0.5f * (zp.y + zm.y), -0.5f * (zp.x - zm.x));               // (Z(m) - conj Z(-m)) / 2i
    const long long b = r / ny;
    const int y = (int)(r - b * ny);
    t[(b * bc + ic) * (long long)ny + y] = v;
  }
}

// ------------------------------------------------------------------------------ forward, columns
// t[b][ic][y] (N = ny) -> band[b][ir][ic] = scale * sum_y t exp(+2 pi i (m0r+ir) y / ny).
// COLS_SYM: t holds the non-negative columns kx = 0 .. bc-1 of a real mask's row transform and the band is the
// symmetric bco x br band (m0c = -(bco-1)/2, m0r = -(br-1)/2): column kx lands at ic = kx + (bco-1)/2 and, for
// kx > 0, its mirror band[-ky][-kx] = conj(band[ky][kx]) at row br-1-ir, column (bco-1)/2 - kx.
// Blocks of COLS_T threads (G = COLS_T / N1 columns each, 32 KB of t): the block's columns are contiguous in t
// and are staged into shared memory by 16-byte asynchronous copies (cp.async, completed per thread: no waits on
// another thread's progress), from where each thread reads its 32 strided values; the twiddled rows then reuse
// the same shared memory.  At the symmetric band's 30 columns per image a batch of 64 has 1920 columns: 480
// blocks, all resident at once.
// COLS_COARSE: the bins stay in shared memory and go on to GRAD_M points, band[col][s] = sum_q bin(q) exp(-2 pi i q s /
// GRAD_M), |q| <= (br-1) / 2 < GRAD_M / 2 (wn_m: that transform's tables), four threads per column.
constexpr int COLS_T = 128, GRAD_M = 128;
enum ColsMode { COLS_BAND, COLS_SYM, COLS_COARSE };

template <int N1, int H>
__device__ __forceinline__ void inverse_gather(float2 (&z)[32], const float2* cq, int qmax, const float2* t2, const float2* t1,
                                               int n1);

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// H: the bins lie within [-32 H, 32 H) (0: any); they come from outer_sums, as the row pass's (one bin per thread at a time
// with loaded twiddles: 8 images of 1024 x 1024, 59 x 59 band 5.4 us, now 4.0; 4 of 2048, 117 x 117 10.0, now 6.1).
template <int N1, ColsMode MODE, int H>
__global__ void __launch_bounds__(COLS_T, H == 4 ? 4 : 6) fft_cols_fwd_kernel(const float2* __restrict__ t, long long ncols, int bc,
                                                              const float2* __restrict__ wn_g, int m0r, int br,
                                                              float scale, float2* __restrict__ band, int bco,
                                                              int dbl_from, const float2* __restrict__ wn_m) {
  constexpr int N = 32 * N1, G = COLS_T / N1;
  constexpr bool SYM = MODE == COLS_SYM;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const float2* t2 = wn_g;
  const float2* t1 = wn_g + 32 * N1;
  float2* ys = (float2*)smem_raw;
  const int tid = threadIdx.x, g = tid / N1, n1 = tid % N1;
  const long long col0 = (long long)blockIdx.x * G, col = col0 + g;
  pdl_trigger();
  pdl_wait();   // t comes from the row pass
  {
    const long long cols = ncols - col0 < G ? ncols - col0 : G;
    const int chunks = (int)(cols * N / 2);   // 16-byte pieces of the block's contiguous columns
    const float4* src = (const float4*)(t + col0 * N);
    float4* dst = (float4*)smem_raw;
    for (int c = tid; c < chunks; c += COLS_T) cp_async16(dst + c, src + c);
    cp_async_wait_all();
    __syncthreads();
  }
  float2 z[32];
  if (col < ncols) {
    const float2* stg = ys + g * N;
#pragma unroll
    for (int n2 = 0; n2 < 32; ++n2) z[n2] = stg[n1 + N1 * n2];
  } else {
#pragma unroll
    for (int n2 = 0; n2 < 32; ++n2) z[n2] = make_float2(0.f, 0.f);
  }
  __syncthreads();   // the stage is overwritten by the twiddled rows below
  fft32<+1>(z);
  float2* yg = ys + g * 32 * (N1 + 1);
  twiddle_store<+1, N1>(z, t2, n1, yg);
  __syncthreads();
  const bool live = col < ncols;
  const long long b = live ? col / bc : 0;
  const int ic = (int)(col - b * bc), half = (bco - 1) / 2;
  // columns ic >= dbl_from are doubled (a Hermitian half-spectrum standing for both halves)
  const float sc = !SYM && ic >= dbl_from ? 2.f * scale : scale;
  float2* cs = ys + G * 32 * (N1 + 1 + (N1 == 64 ? 2 * H : 0));   // [G][br], COLS_COARSE only
  auto put = [&](int ir, float2 v) {
    if (MODE == COLS_COARSE) {
      cs[g * br + ir] = make_float2(v.x * sc, v.y * sc);
    } else if (!SYM) {
      band[(b * br + ir) * (long long)bc + ic] = make_float2(v.x * sc, v.y * sc);
    } else {
      band[(b * br + ir) * (long long)bco + half + ic] = make_float2(v.x * sc, v.y * sc);
      if (ic > 0) band[(b * br + br - 1 - ir) * (long long)bco + half - ic] = make_float2(v.x * sc, -v.y * sc);
    }
  };
  if constexpr (H == 0) {
    if (!live) return;
    for (int ir = n1; ir < br; ir += N1) put(ir, outer_bin<+1, N1>(yg, t1, (m0r + ir) & (N - 1)));
  } else {
    // k2 = n1 + N1 j, all N1 terms; N1 = 64: half of the terms per thread, met in shared memory (as in the row pass)
    constexpr int NT = N1 < 32 ? N1 : 32;
    const bool upper = N1 == 64 && n1 >= 32;
    float2* zs = ys + G * 32 * (N1 + 1);   // [G][32][2 H], N1 = 64 only
#pragma unroll
    for (int k2 = n1 & 31; k2 < 32; k2 += NT) {
      float2 o[2 * H];
      outer_sums<N1, H, NT>(o, yg + k2 * (N1 + 1) + (upper ? 32 : 0));
      if constexpr (N1 == 64) {
        if (upper) {
#pragma unroll
          for (int i = 0; i < 2 * H; ++i) zs[(g * 32 + k2) * 2 * H + i] = o[i];
        }
        __syncthreads();
        if (upper) continue;
#pragma unroll
        for (int i = 0; i < 2 * H; ++i) {
          const float2 v = zs[(g * 32 + k2) * 2 * H + i];
          const float sg = (i - H) & 1 ? -1.f : 1.f;
          o[i] = make_float2(fmaf(sg, v.x, o[i].x), fmaf(sg, v.y, o[i].y));
        }
      }
#pragma unroll
      for (int i = 0; i < 2 * H; ++i) {
        const int ir = k2 + 32 * (i - H) - m0r;
        if (live && ir >= 0 && ir < br) put(ir, o[i]);
      }
    }
  }
  if constexpr (MODE == COLS_COARSE) {
    constexpr int M1 = GRAD_M / 32;
    __syncthreads();
    const int gm = tid / M1, nm = tid % M1;
    if (gm >= G || col0 + gm >= ncols) return;
    inverse_gather<M1, 2>(z, cs + gm * br, (br - 1) / 2, wn_m, wn_m + 32 * M1, nm);
    float2* dst = band + (col0 + gm) * GRAD_M;
#pragma unroll
    for (int i = 0; i < 32; ++i) dst[nm + M1 * bitrev5(i)] = z[i];
  }
}

// v[i][qc][y] (qc < bc, y < GRAD_M; qc > 0 doubled) -> out[i][y][x] = sum_qc Re(v exp(-2 pi i qc x / GRAD_M)): 2 R rows per
// block, a thread per column x and row group; column x + GRAD_M / 2 differs by the sign of the odd terms.  One read of v per
// row and a table of GRAD_M twiddles; bound: latency.  8 images of 1024 x 1024, 59 x 59 band: the gradient's coarse copy was
// 5.5 (bins) + 16.7 (a DFT that summed each row's spectrum per block) us after its row pass, now 9.9 + 4.8.
template <int R>
__global__ void __launch_bounds__(GRAD_M) coarse_gradient_rows_kernel(const float2* __restrict__ v, int bc,
                                                                      const float2* __restrict__ wm, float* __restrict__ out) {
  constexpr int ROWS = 2 * R, X = GRAD_M / 2;
  __shared__ float2 vs[X][ROWS], tab[GRAD_M];   // bc <= X
  const int tid = threadIdx.x, y0 = blockIdx.x * ROWS;
  const long long i = blockIdx.y;
  tab[tid] = __ldg(wm + tid);
  for (int e = tid; e < bc * ROWS; e += GRAD_M) vs[e / ROWS][e % ROWS] = __ldg(v + (i * bc + e / ROWS) * GRAD_M + y0 + e % ROWS);
  __syncthreads();
  const int x = tid % X, g = tid / X * R;
  float acc[2][R] = {};   // sums of the even and the odd qc
  for (int q = 0; q < bc; q += 2) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (q + u >= bc) break;
      const float2 w = tab[((q + u) * x) & (GRAD_M - 1)];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float2 c = vs[q + u][g + r];
        acc[u][r] = fmaf(c.x, w.x, fmaf(c.y, w.y, acc[u][r]));
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float* o = out + (i * GRAD_M + y0 + g + r) * GRAD_M + x;
    o[0] = acc[0][r] + acc[1][r];
    o[X] = acc[0][r] - acc[1][r];
  }
}

// --------------------------------------------------------------------------- inverse, shared part
// Thread n1 of a group: z[k2] = W_N^{-k2 n1} sum_{k1} coef(k2 + 32 k1) W_N1^{-k1 n1} over the non-zero
// coefficients, which sit at frequencies q in [-qmax, qmax] (index q mod N); coef(q) = cq[q + qmax].
// H = 2, 4: |q| < 32 H, the inputs of k2 are q = k2 + 32 k1, -H <= k1 < H: 2 H predicated terms with their twiddles
// in registers and no runtime loops, so the 32 independent k2 chains interleave.  H = 0: any qmax.
template <int N1, int H>
__device__ __forceinline__ void inverse_gather(float2 (&z)[32], const float2* cq, int qmax, const float2* t2,
                                               const float2* t1, int n1) {
  constexpr int N = 32 * N1;
  if constexpr (H > 0) {
    float2 w[2 * H];   // W_N1^{-k1 n1}, k1 = -H .. H - 1
#pragma unroll
    for (int i = 0; i < 2 * H; ++i) w[i] = sgn<-1>(t1[((i - H) & (N1 - 1)) * N1 + n1]);
    const float2* c0 = cq + qmax;   // c0[q] = coefficient of frequency q
#pragma unroll
    for (int k2 = 0; k2 < 32; ++k2) {
      float2 acc = k2 <= qmax ? c0[k2] : make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 2 * H; ++i) {
        const int q = k2 + 32 * (i - H);
        if (i != H && q <= qmax && q >= -qmax) cfma(acc, c0[q], w[i]);
      }
      z[k2] = cmul(acc, sgn<-1>(t2[k2 * N1 + n1]));
    }
  } else {
#pragma unroll
    for (int k2 = 0; k2 < 32; ++k2) {
      float2 acc = make_float2(0.f, 0.f);
      for (int k1 = 0; k2 + 32 * k1 <= qmax; ++k1)  // q = k2 + 32 k1 >= 0
        cfma(acc, cq[k2 + 32 * k1 + qmax], sgn<-1>(t1[k1 * N1 + n1]));
      for (int k1 = N1 - 1; k1 > 0 && k2 + 32 * k1 >= N - qmax; --k1)  // q = k2 + 32 k1 - N < 0
        cfma(acc, cq[k2 + 32 * k1 - N + qmax], sgn<-1>(t1[k1 * N1 + n1]));
      z[k2] = cmul(acc, sgn<-1>(t2[k2 * N1 + n1]));
    }
  }
  fft32<-1>(z);
}
// The H of a band of b frequencies per side (qmax = b - 1).  For N1 = 8 (N = 256) 32 H must stay below N / 2 + 1.
__host__ __device__ constexpr int gather_blocks(int b) { return b <= 64 ? 2 : b <= 128 ? 4 : 0; }

// exp(-2 pi i b k / L) sums of L = 4 or 8 values (b = 0 .. L-1, natural order in and out)
__device__ __forceinline__ void dft_short(float2 (&v)[4]) {
  const float2 a = make_float2(v[0].x + v[2].x, v[0].y + v[2].y), b = make_float2(v[0].x - v[2].x, v[0].y - v[2].y);
  const float2 c = make_float2(v[1].x + v[3].x, v[1].y + v[3].y), d = make_float2(v[1].y - v[3].y, v[3].x - v[1].x);
  v[0] = make_float2(a.x + c.x, a.y + c.y);
  v[1] = make_float2(b.x + d.x, b.y + d.y);
  v[2] = make_float2(a.x - c.x, a.y - c.y);
  v[3] = make_float2(b.x - d.x, b.y - d.y);
}
__device__ __forceinline__ void dft_short(float2 (&v)[8]) {
  float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
  dft_short(e);
  dft_short(o);
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const float2 w = rot32<-1>(o[b], 4 * b);
    v[b] = make_float2(e[b].x + w.x, e[b].y + w.y);
    v[b + 4] = make_float2(e[b].x - w.x, e[b].y - w.y);
  }
}

// inverse_gather for |q| < 32 H in two steps: ys[k2][n1] (row stride N1 + 1; the group's own) = sum_k1 coef(k2 + 32 k1)
// W_N1^{-k1 n1} for all n1 of a k2 by one thread, 2 H inputs as N1 / (2 H) short transforms with constant twiddles; a
// barrier of the block; then each thread its column n1.  The gather's 2 H terms per value (8 H instructions with their
// loads) become about 8 and an exchange, and with fewer values live at a time three blocks of H = 4 share an SM's registers
// where two did.  Rows of 4 images of 2048 x 2048, 117 columns: 37.7 -> 27.1 us (30.9 with two blocks); of 8 of 1024 x 1024,
// 59 columns: 16.4 before and after.
template <int N1, int H>
__device__ __forceinline__ void inverse_outer(float2 (&z)[32], const float2* cq, int qmax, float2* ys, const float2* t2, int n1) {
  constexpr int L = 2 * H, A = N1 / L, NT = N1 < 32 ? N1 : 32, AT = N1 == 64 ? A / 2 : A;
  const bool upper = N1 == 64 && n1 >= 32;   // N1 = 64: two threads per k2, the upper one offset by AT in n1
  const float2* c0 = cq + qmax;
#pragma unroll
  for (int k2 = n1 & 31; k2 < 32; k2 += NT) {
    float2 c[L];
#pragma unroll
    for (int i = 0; i < L; ++i) {
      const int k1 = i < H ? i : i - L, q = k2 + 32 * k1;
      c[i] = q <= qmax && q >= -qmax ? c0[q] : make_float2(0.f, 0.f);
      if constexpr (N1 == 64) {
        const float2 r = cmul(c[i], make_float2(c64(64 / N1 * k1 * AT), -s64(64 / N1 * k1 * AT)));
        if (upper) c[i] = r;
      }
    }
    float2* row = ys + k2 * (N1 + 1) + (upper ? AT : 0);
#pragma unroll
    for (int a = 0; a < AT; ++a) {
      float2 v[L];
#pragma unroll
      for (int i = 0; i < L; ++i) {
        const int t = 64 / N1 * (i < H ? i : i - L) * a;
        v[i] = t == 0 ? c[i] : cmul(c[i], make_float2(c64(t), -s64(t)));
      }
      dft_short(v);
#pragma unroll
      for (int b = 0; b < L; ++b) row[a + A * b] = v[b];
    }
  }
  __syncthreads();
#pragma unroll
  for (int k2 = 0; k2 < 32; ++k2) z[k2] = cmul(ys[k2 * (N1 + 1) + n1], sgn<-1>(t2[k2 * N1 + n1]));
  fft32<-1>(z);
}
// complex values of ys for the 256 / N1 groups of a block
template <int N1, int H> __host__ __device__ constexpr int outer_f2() { return H ? 256 / N1 * 32 * (N1 + 1) : 0; }

// ------------------------------------------------------------------------------ inverse, columns
// ihat[i][jr][qc] (qr = jr - (br-1)) -> v[i][qc][y] = sum_qr ihat exp(-2 pi i qr y / ny)
template <int N1, int H>
__global__ void __launch_bounds__(256, 3) fft_cols_inv_kernel(const float2* __restrict__ ihat, long long ncols, int br,
                                                           int bc, const float2* __restrict__ wn_g,
                                                           float2* __restrict__ v) {
  constexpr int N = 32 * N1, G = 256 / N1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const float2* t2 = wn_g;
  const float2* t1 = wn_g + 32 * N1;
  const int nq = 2 * br - 1;
  float2* ys = (float2*)smem_raw;        // [G][32][N1 + 1] (H > 0)
  float2* cs = ys + outer_f2<N1, H>();   // [G][nq]
  const int tid = threadIdx.x, g = tid / N1, n1 = tid % N1;
  const long long col0 = (long long)blockIdx.x * G;
  for (int e = tid; e < G * nq; e += 256) {
    const int jr = e / G, gg = e % G;
    const long long col = col0 + gg;
    float2 c = make_float2(0.f, 0.f);
    if (col < ncols) {
      const long long i = col / bc;
      const int qc = (int)(col - i * bc);
      c = ihat[(i * nq + jr) * (long long)bc + qc];
    }
    cs[gg * nq + jr] = c;
  }
  __syncthreads();
  const long long col = col0 + g;
  float2 z[32];
  if constexpr (H > 0) inverse_outer<N1, H>(z, cs + g * nq, br - 1, ys + g * 32 * (N1 + 1), t2, n1);
  else inverse_gather<N1, H>(z, cs + g * nq, br - 1, t2, t1, n1);
  if (col >= ncols) return;
  float2* dst = v + col * N;
#pragma unroll
  for (int i = 0; i < 32; ++i) dst[n1 + N1 * bitrev5(i)] = z[i];
}

// ---------------------------------------------------------------- inverse, columns into V operand tiles
// The column pass of the tensor-core synthesis: for image i and band columns qc0 .. qc0+G-1 (G = max(8, 256/N1),
// zero beyond bc) the inverse column FFTs as fft_cols_inv_kernel, kept in shared memory, then written directly as
// the bf16 hi / lo V operand tiles of the row pass (rows y of 128-row blocks, K = re | im of 64 band columns,
// 128-byte swizzled: [hi: re | im][lo: re | im] x [128][64]) -- v itself never reaches global memory.
template <int N1, int G>
__global__ void __launch_bounds__(G * N1) cols_inv_tiles_kernel(const float2* __restrict__ ihat, int br, int bc,
                                                              int ny, const float2* __restrict__ wn_g,
                                                              unsigned char* __restrict__ tiles) {
  constexpr int N = 32 * N1, T = G * N1;
  constexpr uint32_t OPER = 128 * 128, TILE = 4 * OPER;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const float2* t2 = wn_g;
  const float2* t1 = wn_g + 32 * N1;
  const int nq = 2 * br - 1;
  float2* cs = (float2*)smem_raw;                        // [G][nq]
  float2* vs = cs + ((G * nq + 1) & ~1);                 // [G][N / 2]: one half of the rows, column-major so that
                                                         // consecutive lanes (rows) hit consecutive banks
  const int tid = threadIdx.x, g = tid / N1, n1 = tid % N1;
  const long long i = blockIdx.y;
  const int qc0 = blockIdx.x * G;
  pdl_trigger();
  pdl_wait();   // ihat comes from the coarse spectrum
  for (int e = tid; e < G * nq; e += T) {
    const int jr = e / G, gg = e % G, qc = qc0 + gg;
    cs[gg * nq + jr] = qc < bc ? ihat[(i * nq + jr) * (long long)bc + qc] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  float2 z[32];
  inverse_gather<N1, 2>(z, cs + g * nq, br - 1, t2, t1, n1);   // 2 br - 1 <= 128
  // z[k] is row n1 + N1 bitrev5(k): even k give the first half of the rows, odd k the second.  The rows are
  // transposed through shared memory one half at a time (half the buffer: more blocks per SM, one wave).
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h) __syncthreads();   // the first half has been stored
#pragma unroll
    for (int k = h; k < 32; k += 2) vs[g * (N / 2) + n1 + N1 * (bitrev5(k) - 16 * h)] = z[k];
    __syncthreads();
    // QPT band columns per store: 8 (one 16-byte chunk of the bf16 row) or, for G = 4, 4 (half a chunk)
    constexpr int QPT = G < 8 ? G : 8;
    for (int it = tid; it < (N / 2) * (G / QPT); it += T) {
      const int yh = it % (N / 2), gq = it / (N / 2), y = yh + h * (N / 2);
      const int qf = qc0 + QPT * gq, q = qf >> 3;
      const float2* src = vs + (QPT * gq) * (N / 2) + yh;
      float re[QPT], im[QPT];
#pragma unroll
      for (int e = 0; e < QPT; ++e) {
        const float2 x = src[e * (N / 2)];
        re[e] = x.x, im[e] = x.y;
      }
      uint32_t rh[QPT / 2], rl[QPT / 2], ih[QPT / 2], il[QPT / 2];
#pragma unroll
      for (int e = 0; e < QPT / 2; ++e) {
        tc::split2(re[2 * e], re[2 * e + 1], rh[e], rl[e]);
        tc::split2(im[2 * e], im[2 * e + 1], ih[e], il[e]);
      }
      const long long row = i * ny + y;
      unsigned char* o = tiles + (row >> 7) * TILE + tc::swz((int)(row & 127), q);
      if constexpr (QPT == 8) {
        *(uint4*)o = make_uint4(rh[0], rh[1], rh[2], rh[3]);
        *(uint4*)(o + OPER) = make_uint4(ih[0], ih[1], ih[2], ih[3]);
        *(uint4*)(o + 2 * OPER) = make_uint4(rl[0], rl[1], rl[2], rl[3]);
        *(uint4*)(o + 3 * OPER) = make_uint4(il[0], il[1], il[2], il[3]);
      } else {
        o += 2 * (qf & 7);   // the half of the chunk holding band columns qf .. qf + 3
        *(uint2*)o = make_uint2(rh[0], rh[1]);
        *(uint2*)(o + OPER) = make_uint2(ih[0], ih[1]);
        *(uint2*)(o + 2 * OPER) = make_uint2(rl[0], rl[1]);
        *(uint2*)(o + 3 * OPER) = make_uint2(il[0], il[1]);
      }
    }
  }
}

template <int N1, int G>
static int cols_inv_tiles(const float2* ihat, int count, int br, int bc, int ny, const float2* wn_y,
                          unsigned char* tiles, cudaStream_t s) {
  const size_t smem = sizeof(float2) * (((size_t)G * (2 * br - 1) + 1) & ~(size_t)1) + sizeof(float2) * 16 * N1 * G;
  int rc = set_smem(cols_inv_tiles_kernel<N1, G>, smem, "oi_coarse_to_image_tc/cols");
  if (rc) return rc;
  dim3 grid(64 / G, (unsigned)count);
  (void)launch_pdl(cols_inv_tiles_kernel<N1, G>, grid, dim3(G * N1), smem, s, ihat, br, bc, ny, wn_y, tiles);
  oi::note_launch();
  return check_launch("oi_coarse_to_image_tc/cols");
}

// --------------------------------------------------------------------------------- inverse, rows
// v[i][qc][y] (qc = 0..bc-1, qc > 0 doubled) -> out[i][y][x] = sum_qc Re(v exp(-2 pi i qc x / nx))
template <int N1, int H>
__global__ void __launch_bounds__(256, 3) fft_rows_inv_kernel(const float2* __restrict__ v, long long nrows, int ny,
                                                           int bc, const float2* __restrict__ wn_g,
                                                           float* __restrict__ out) {
  constexpr int N = 32 * N1, G = 256 / N1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const float2* t2 = wn_g;
  const float2* t1 = wn_g + 32 * N1;
  const int nq = 2 * bc - 1;
  float2* vs = (float2*)smem_raw;      // [bc][2G + 1] (padded against bank conflicts), then [G][32][N1 + 1] (H > 0)
  float2* cs = vs + max(bc * (2 * G + 1), outer_f2<N1, H>());   // [G][nq]
  const int tid = threadIdx.x, g = tid / N1, n1 = tid % N1;
  const long long rblk = (long long)blockIdx.x * (2 * G);
  for (int e = tid; e < bc * 2 * G; e += 256) {
    const int qc = e / (2 * G), rr = e % (2 * G);
    const long long r = rblk + rr;
    float2 c = make_float2(0.f, 0.f);
    if (r < nrows) {
      const long long i = r / ny;
      const int y = (int)(r - i * ny);
      c = v[(i * bc + qc) * (long long)ny + y];
    }
    vs[qc * (2 * G + 1) + rr] = c;
  }
  __syncthreads();
  // Hermitian spectra of the row pair packed as F_a + i F_b, q in [-(bc-1), bc-1]
  for (int e = tid; e < G * nq; e += 256) {
    const int gg = e / nq, j = e % nq, q = j - (bc - 1), aq = q < 0 ? -q : q;
    float2 a = vs[aq * (2 * G + 1) + 2 * gg], b = vs[aq * (2 * G + 1) + 2 * gg + 1];
    const float h = aq == 0 ? 1.0f : 0.5f;
    if (q < 0) {
      a.y = -a.y;
      b.y = -b.y;
    }
    cs[e] = make_float2(h * (a.x - b.y), h * (a.y + b.x));  // h (a + i b)
  }
  __syncthreads();
  const long long r0 = rblk + 2 * g;
  float2 z[32];
  if constexpr (H > 0) inverse_outer<N1, H>(z, cs + g * nq, bc - 1, vs + g * 32 * (N1 + 1), t2, n1);
  else inverse_gather<N1, H>(z, cs + g * nq, bc - 1, t2, t1, n1);
  if (r0 >= nrows) return;
  float* o0 = out + r0 * N;
  float* o1 = o0 + N;
  const bool second = r0 + 1 < nrows;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const int x = n1 + N1 * bitrev5(i);
    o0[x] = z[i].x;
    if (second) o1[x] = z[i].y;
  }
}

// ------------------------------------------------------- coarse intensity -> image columns, two passes
// Rows: U[i][qc][sr] = sum_sc (sum_p coarse[p][i][sr][sc]) exp(+2 pi i qc sc / mc), 0 <= qc < bc, mc = 32 N1C: PAIRS row
// pairs per block (one complex transform each), the partial sums added as the rows load, U written transposed.
// Columns: the mr-point transform of U's column (mr = 32 N1R), its 2 br - 1 bins scaled by 1 / (mr mc), qc > 0 doubled,
// and the ny-point inverse transform of those (ny = 32 N1) back into the same column: v[i][qc][y].
// Bound: latency; the point of the split is blocks.  One image used to be two blocks for the whole coarse spectrum:
// 8 images of 128 x 128, 12 parts, 59 x 59 band, 1024 rows: 20.1 (spectrum) + 8.5 (columns) us -> 5.3 + 9.5;
// 4 of 256 x 256, 37 parts, 117 x 117 band, 2048 rows: 58 + 9.4 + 39.6 -> 7.0 + 9.7.
constexpr int COARSE_T = 128;

template <int N1C, int PAIRS>
__global__ void __launch_bounds__(COARSE_T) coarse_rows_kernel(const float* __restrict__ coarse, int nparts,
                                                               long long pstride, int mr, int bc,
                                                               const float2* __restrict__ wc, int ny,
                                                               float2* __restrict__ u) {
  constexpr int MC = 32 * N1C, PER = 2 * PAIRS * MC / 4 / COARSE_T > 0 ? 2 * PAIRS * MC / 4 / COARSE_T : 1;
  constexpr int LOADERS = 2 * PAIRS * MC / 4 / PER;   // threads that load (all, except for few short rows)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* img = (float*)smem_raw;                      // [2 PAIRS][MC]
  float2* ys = (float2*)smem_raw + PAIRS * MC;        // [PAIRS][32][N1C + 1]
  const int tid = threadIdx.x, r0 = blockIdx.x * 2 * PAIRS;
  const long long i = blockIdx.y;
  if (tid < LOADERS) {
    const float4* src = (const float4*)(coarse + (i * mr + r0) * MC) + tid;
    float4 acc[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) acc[k] = __ldg(src + LOADERS * k);
#pragma unroll(PER <= 2 ? 8 / PER : 4)   // an Abbe image of a few fields per block has up to a hundred parts
    for (int p = 1; p < nparts; ++p) {
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const float4 x = __ldg(src + p * (pstride / 4) + LOADERS * k);
        acc[k].x += x.x;
        acc[k].y += x.y;
        acc[k].z += x.z;
        acc[k].w += x.w;
      }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) ((float4*)img)[tid + LOADERS * k] = acc[k];
  }
  __syncthreads();
  if (tid < PAIRS * N1C) {
    const int p = tid / N1C, n1 = tid % N1C;
    float2 z[32];
#pragma unroll
    for (int n2 = 0; n2 < 32; ++n2) z[n2] = make_float2(img[2 * p * MC + n1 + N1C * n2], img[(2 * p + 1) * MC + n1 + N1C * n2]);
    fft32<+1>(z);
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int k2 = bitrev5(k);
      ys[(p * 32 + k2) * (N1C + 1) + n1] = cmul(z[k], __ldg(wc + ((k2 * n1) & (MC - 1))));
    }
  }
  __syncthreads();
  for (int e = tid; e < PAIRS * bc; e += COARSE_T) {
    const int p = e % PAIRS, qc = e / PAIRS;
    const float2* y = ys + p * 32 * (N1C + 1);
    float2 zp = make_float2(0.f, 0.f), zm = zp;   // bins qc and -qc
#pragma unroll
    for (int n1 = 0; n1 < N1C; ++n1) {
      const float2 w = __ldg(wc + ((32 * (qc >> 5) * n1) & (MC - 1)));
      const int m = -qc & (MC - 1);
      cfma(zp, y[(qc & 31) * (N1C + 1) + n1], w);
      cfma(zm, y[(m & 31) * (N1C + 1) + n1], __ldg(wc + ((32 * (m >> 5) * n1) & (MC - 1))));
    }
    float2* o = u + (i * bc + qc) * (long long)ny + r0 + 2 * p;
    o[0] = make_float2(0.5f * (zp.x + zm.x), 0.5f * (zp.y - zm.y));
    o[1] = make_float2(0.5f * (zp.y + zm.y), -0.5f * (zp.x - zm.x));
  }
}

template <int N1R, int N1, int H>
__global__ void __launch_bounds__(COARSE_T) coarse_cols_kernel(long long ncols, int br, int bc, const float2* __restrict__ wr,
                                                               const float2* __restrict__ wn_g, float norm, float2* v) {
  constexpr int MR = 32 * N1R, N = 32 * N1, G = COARSE_T / N1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nq = 2 * br - 1;
  float2* us = (float2*)smem_raw;           // [G][MR]
  float2* ys = us + G * MR;                 // [G][32][N1R + 1]
  float2* cs = ys + G * 32 * (N1R + 1);     // [G][nq]
  __shared__ float2 t1[N1R * N1R];          // exp(+2 pi i k1 n1 / N1R)
  const int tid = threadIdx.x;
  const long long col0 = (long long)blockIdx.x * G;
  const int qc0 = (int)(col0 % bc);         // band column of the block's first
  if (tid < N1R * N1R) t1[tid] = __ldg(wr + ((32 * (tid / N1R) * (tid % N1R)) & (MR - 1)));
  for (int e = tid; e < G * MR; e += COARSE_T) {
    const int g = e / MR;
    us[e] = col0 + g < ncols ? v[(col0 + g) * N + e % MR] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  float2 z[32];
  if (tid < G * N1R) {
    const int g = tid / N1R, n1 = tid % N1R;
#pragma unroll
    for (int n2 = 0; n2 < 32; ++n2) z[n2] = us[g * MR + n1 + N1R * n2];
    fft32<+1>(z);
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int k2 = bitrev5(k);
      ys[(g * 32 + k2) * (N1R + 1) + n1] = cmul(z[k], __ldg(wr + ((k2 * n1) & (MR - 1))));
    }
  }
  __syncthreads();
  // thread: column g = tid / N1, bins tid % N1 + N1 i
  const int g = tid / N1, n1 = tid % N1;
  {
    const float s = (qc0 + g) % bc == 0 ? norm : 2.f * norm;
    const float2* yg = ys + g * 32 * (N1R + 1);
#pragma unroll 4
    for (int jr = n1; jr < nq; jr += N1) {
      const int k = (jr - (br - 1)) & (MR - 1);
      const float2* y = yg + (k & 31) * (N1R + 1);
      float2 a = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < N1R; ++i) cfma(a, y[i], t1[(k >> 5) * N1R + i]);
      cs[g * nq + jr] = make_float2(a.x * s, a.y * s);
    }
  }
  __syncthreads();
  if (col0 + g >= ncols) return;
  inverse_gather<N1, H>(z, cs + g * nq, br - 1, wn_g, wn_g + 32 * N1, n1);
  float2* dst = v + (col0 + g) * N;
#pragma unroll
  for (int i = 0; i < 32; ++i) dst[n1 + N1 * bitrev5(i)] = z[i];
}

// --------------------------------------------------------------- coarse intensity -> its spectrum
// For the tensor-core synthesis.  COARSE_PARTS blocks per coarse image, each for a range of the band columns qc (mr = mc =
// 128; U holds the block's columns only, so that two blocks fit an SM):
//   ihat[i][jr][qc] = (qc ? 2 : 1) / (mr mc) * sum_{sr,sc} coarse[i][sr][sc] exp(+2 pi i (qr sr/mr + qc sc/mc))
// for qr = jr - (br-1) in [-(br-1), br-1] and qc in [0, bc).  Row FFTs of the real image in pairs (two rows per
// complex transform), the band bins of each separated into U[sr][qc]; then column FFTs of U at the qr bins.
constexpr int COARSE_PARTS = 2, SPEC_N1 = 4, SPEC_M = 32 * SPEC_N1;
__global__ void __launch_bounds__(512) coarse_spec_fft_kernel(const float* __restrict__ coarse, int nparts,
                                                              long long part_stride, int br, int bc,
                                                              const float2* __restrict__ wr_g,
                                                              const float2* __restrict__ wc_g, int area_f2,
                                                              float2* __restrict__ ihat) {
  constexpr int N1R = SPEC_N1, N1C = SPEC_N1, MR = SPEC_M, MC = SPEC_M, T = 512;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* r2 = (float2*)smem_raw;      // row-axis (MR) tables: [32][N1R], [N1R][N1R]
  float2* r1 = r2 + 32 * N1R;
  float2* c2 = r1 + N1R * N1R;         // column-axis (MC) tables: [32][N1C], [N1C][N1C]
  float2* c1t = c2 + 32 * N1C;
  float2* area = c1t + N1C * N1C;      // [area_f2] union: coarse image / row transposes / column transposes
  float2* u = area + area_f2;          // [MR][cw]: this block's band columns
  const int tid = threadIdx.x;
  const long long img = blockIdx.x;
  // this block's band columns: blockIdx.y-th of gridDim.y equal ranges of [0, bc)
  const int cw = (bc + gridDim.y - 1) / gridDim.y, c0 = blockIdx.y * cw, c1 = min(bc, c0 + cw);
  build_tables<N1R>(wr_g, r2, r1, tid, T);
  build_tables<N1C>(wc_g, c2, c1t, tid, T);
  pdl_trigger();
  pdl_wait();   // the partial coarse images come from the coherent sum
  float* cimg = (float*)area;
  const float4* src = (const float4*)(coarse + img * (long long)MR * MC);
  constexpr int PER = MR * MC / 4 / T;   // float4 per thread
  float4 acc[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) acc[k] = __ldg(src + tid + T * k);
  for (int p = 1; p < nparts; ++p) {   // the partial sums, added in order; all loads of a part in flight together
    float4 x[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) x[k] = __ldg(src + p * (part_stride / 4) + tid + T * k);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      acc[k].x += x[k].x;
      acc[k].y += x[k].y;
      acc[k].z += x[k].z;
      acc[k].w += x[k].w;
    }
  }
#pragma unroll
  for (int k = 0; k < PER; ++k) ((float4*)cimg)[tid + T * k] = acc[k];
  __syncthreads();
  // row pass: pair p = rows (2p, 2p+1), thread n1
  const int p = tid / N1C, n1 = tid % N1C;
  const bool row_task = p < MR / 2;
  float2 z[32];
  if (row_task) {
#pragma unroll
    for (int n2 = 0; n2 < 32; ++n2)
      z[n2] = make_float2(cimg[(2 * p) * MC + n1 + N1C * n2], cimg[(2 * p + 1) * MC + n1 + N1C * n2]);
    fft32<+1>(z);
  }
  __syncthreads();  // the image is consumed; the area now holds row transposes
  if (row_task) twiddle_store<+1, N1C>(z, c2, n1, area + p * 32 * (N1C + 1));
  __syncthreads();
  for (int e = tid; e < (MR / 2) * (c1 - c0); e += T) {
    const int pp = e / (c1 - c0), qc = c0 + e % (c1 - c0);
    const float2* ys = area + pp * 32 * (N1C + 1);
    const float2 zp = outer_bin<+1, N1C>(ys, c1t, qc & (MC - 1));
    const float2 zm = outer_bin<+1, N1C>(ys, c1t, (-qc) & (MC - 1));
    u[(2 * pp) * cw + qc - c0] = make_float2(0.5f * (zp.x + zm.x), 0.5f * (zp.y - zm.y));
    u[(2 * pp + 1) * cw + qc - c0] = make_float2(0.5f * (zp.y + zm.y), -0.5f * (zp.x - zm.x));
  }
  __syncthreads();
  // column pass: column qc of U, thread n1r
  const int qc = c0 + tid / N1R, n1r = tid % N1R;
  const bool col_task = qc < c1;
  if (col_task) {
#pragma unroll
    for (int n2 = 0; n2 < 32; ++n2) z[n2] = u[(n1r + N1R * n2) * cw + qc - c0];
    fft32<+1>(z);
  }
  __syncthreads();  // row transposes are consumed; the area now holds column transposes
  if (col_task) twiddle_store<+1, N1R>(z, r2, n1r, area + (qc - c0) * 32 * (N1R + 1));
  __syncthreads();
  const int nq = 2 * br - 1;
  const float norm = 1.0f / ((float)MR * (float)MC);
  for (int e = tid; e < nq * (c1 - c0); e += T) {
    const int jr = e / (c1 - c0), c = c0 + e % (c1 - c0);
    const float2 v = outer_bin<+1, N1R>(area + (c - c0) * 32 * (N1R + 1), r1, (jr - (br - 1)) & (MR - 1));
    const float s = (c == 0 ? 1.0f : 2.0f) * norm;
    ihat[(img * nq + jr) * (long long)bc + c] = make_float2(v.x * s, v.y * s);
  }
}

static int launch_coarse_spec_fft(float* coarse, int nparts, int count, int br, int bc, const float2* wr,
                                  const float2* wc, float2* ihat, cudaStream_t s) {
  constexpr int N1R = SPEC_N1, N1C = SPEC_N1, MR = SPEC_M, MC = SPEC_M;
  const int cw = (bc + COARSE_PARTS - 1) / COARSE_PARTS;   // band columns per block (as in the kernel)
  const int rows_ys = (MR / 2) * 32 * (N1C + 1), c_f2 = MR * MC / 2, cols_ys = cw * 32 * (N1R + 1);
  const int area_f2 = max(rows_ys, max(c_f2, cols_ys));
  const size_t smem = sizeof(float2) * ((size_t)table_f2<N1R>() + table_f2<N1C>() + area_f2 + (size_t)MR * cw);
  auto kern = coarse_spec_fft_kernel;
  int rc = set_smem(kern, smem, "coarse spectrum fft");
  if (rc) return rc;
  (void)launch_pdl(kern, dim3((unsigned)count, COARSE_PARTS), dim3(512), smem, s, (const float*)coarse, nparts,
                   (long long)count * MR * MC, br, bc, wr, wc, area_f2, ihat);
  oi::note_launch();
  return check_launch("coarse spectrum fft");
}

template <int N1>
static size_t smem_rows_fwd(int nu) { return sizeof(float2) * ((256 / N1) * 32 * (N1 + 1) + (256 / N1) * nu); }
template <int N1, int H>
static size_t smem_cols_fwd() { return sizeof(float2) * ((COLS_T / N1) * 32 * (N1 + 1 + (N1 == 64 ? 2 * H : 0))); }


template <int N1, int KIND, int H>
static int rows_fwd_h(const void* field, long long nrows, int ny, int nch, int m0c, int bc, int u0, int nu, const float2* wn_x,
                      float2* t, cudaStream_t s, int nparts, long long pstride) {
  constexpr int ROWS = (KIND == OI_FIELD_COMPLEX_C64 ? 1 : 2) * (256 / N1);
  const size_t smem = smem_rows_fwd<N1>(nu);
  if (int rc = set_smem(fft_rows_fwd_kernel<N1, KIND, H>, smem, "oi_band_spectrum_fft/rows")) return rc;
  fft_rows_fwd_kernel<N1, KIND, H><<<(unsigned)ceil_div(nrows, ROWS), 256, smem, s>>>(field, nrows, ny, nch, wn_x, m0c, bc, u0,
                                                                                     nu, t, nparts, pstride);
  oi::note_launch();
  return check_launch("oi_band_spectrum_fft/rows");
}
template <int N1, int KIND>
static int rows_fwd(const void* field, int batch, int ny, int nch, int m0c, int bc, const float2* wn_x, float2* t, cudaStream_t s,
                    int nparts = 1, long long pstride = 0) {
  int u0 = m0c, u1 = m0c + bc - 1;
  if (KIND != OI_FIELD_COMPLEX_C64) {   // the band and its mirror
    u0 = min(m0c, -(m0c + bc - 1));
    u1 = max(m0c + bc - 1, -m0c);
  }
  const int nu = u1 - u0 + 1;
  const long long nrows = (long long)batch * ny * nch;
  auto within = [&](int h) { return u0 >= -32 * h && u1 < 32 * h; };
  if (within(1)) return rows_fwd_h<N1, KIND, 1>(field, nrows, ny, nch, m0c, bc, u0, nu, wn_x, t, s, nparts, pstride);
  if (within(2)) return rows_fwd_h<N1, KIND, 2>(field, nrows, ny, nch, m0c, bc, u0, nu, wn_x, t, s, nparts, pstride);
  if (within(4)) return rows_fwd_h<N1, KIND, 4>(field, nrows, ny, nch, m0c, bc, u0, nu, wn_x, t, s, nparts, pstride);
  return rows_fwd_h<N1, KIND, 0>(field, nrows, ny, nch, m0c, bc, u0, nu, wn_x, t, s, nparts, pstride);
}

// row transforms have length nx = 32 * N1; the column kernel picks its own N1 for ny
template <int N1>
static int band_fft(const void* field, int kind, int batch, int ny, int nch, int m0c, int bc, const float2* wn_x, float2* t,
                    cudaStream_t s, int nparts = 1, long long pstride = 0) {
  switch (kind) {
    case OI_FIELD_U8: return rows_fwd<N1, OI_FIELD_U8>(field, batch, ny, nch, m0c, bc, wn_x, t, s);
    case OI_FIELD_COMPLEX_C64: return rows_fwd<N1, OI_FIELD_COMPLEX_C64>(field, batch, ny, nch, m0c, bc, wn_x, t, s);
  }
  return rows_fwd<N1, OI_FIELD_REAL_F32>(field, batch, ny, nch, m0c, bc, wn_x, t, s, nparts, pstride);
}
static int band_rows(int nx1, const void* field, int kind, int batch, int ny, int nch, int m0c, int bc, const void* wn_x, float2* t,
                     cudaStream_t s, int nparts = 1, long long pstride = 0) {
  const float2* wx = (const float2*)wn_x;
  switch (nx1) {
    case 8: return band_fft<8>(field, kind, batch, ny, nch, m0c, bc, wx, t, s, nparts, pstride);
    case 16: return band_fft<16>(field, kind, batch, ny, nch, m0c, bc, wx, t, s, nparts, pstride);
    case 32: return band_fft<32>(field, kind, batch, ny, nch, m0c, bc, wx, t, s, nparts, pstride);
  }
  return band_fft<64>(field, kind, batch, ny, nch, m0c, bc, wx, t, s, nparts, pstride);
}

// bco: the output band width (SYM: bc = (bco + 1) / 2 input columns; else bco = bc)
template <int N1, ColsMode MODE, int H>
static int cols_fwd_h(const float2* t, long long ncols, int bc, const float2* wn_y, int m0r, int br, float scale,
                      float2* band, cudaStream_t s, int bco, int dbl_from, const float2* wn_m = nullptr) {
  constexpr int G = COLS_T / N1;
  const size_t smem = smem_cols_fwd<N1, H>() + (MODE == COLS_COARSE ? sizeof(float2) * G * br : 0);
  if (int rc = set_smem(fft_cols_fwd_kernel<N1, MODE, H>, smem, "oi_band_spectrum_fft/cols")) return rc;
  (void)launch_pdl(fft_cols_fwd_kernel<N1, MODE, H>, dim3((unsigned)ceil_div(ncols, G)), dim3(COLS_T), smem, s, t, ncols, bc,
                   wn_y, m0r, br, scale, band, bco, dbl_from, wn_m);
  oi::note_launch();
  return check_launch("oi_band_spectrum_fft/cols");
}
template <int N1, bool SYM = false>
static int cols_fwd(const float2* t, int batch, int bc, const float2* wn_y, int m0r, int br, float scale,
                    float2* band, cudaStream_t s, int bco = 0, int dbl_from = 0x7fffffff) {
  if ((uintptr_t)t % 16) return fail(OI_EINVAL, "oi_band_spectrum_fft/cols: scratch must be 16-byte aligned");
  const long long ncols = (long long)batch * bc;
  bco = SYM ? bco : bc;
  constexpr ColsMode MODE = SYM ? COLS_SYM : COLS_BAND;
  auto within = [&](int h) { return m0r >= -32 * h && m0r + br <= 32 * h; };
  if (within(1)) return cols_fwd_h<N1, MODE, 1>(t, ncols, bc, wn_y, m0r, br, scale, band, s, bco, dbl_from);
  if (within(2)) return cols_fwd_h<N1, MODE, 2>(t, ncols, bc, wn_y, m0r, br, scale, band, s, bco, dbl_from);
  if (within(4)) return cols_fwd_h<N1, MODE, 4>(t, ncols, bc, wn_y, m0r, br, scale, band, s, bco, dbl_from);
  return cols_fwd_h<N1, MODE, 0>(t, ncols, bc, wn_y, m0r, br, scale, band, s, bco, dbl_from);
}

// Columns of GRAD_M points from the columns of ny = 32 N1 in t (br frequencies per side, the positive columns doubled)
template <int N1>
static int cols_coarse(const float2* t, int count, int bc, const float2* wn_y, int br, float scale, const float2* wn_m, float2* v,
                       cudaStream_t s) {
  const long long ncols = (long long)count * bc;
  const int nq = 2 * br - 1;
  return br <= 32 ? cols_fwd_h<N1, COLS_COARSE, 1>(t, ncols, bc, wn_y, 1 - br, nq, scale, v, s, bc, 1, wn_m)
                  : cols_fwd_h<N1, COLS_COARSE, 2>(t, ncols, bc, wn_y, 1 - br, nq, scale, v, s, bc, 1, wn_m);
}

template <int N1, int H>
static int cols_inv_h(const float2* ihat, int count, int br, int bc, const float2* wn_y, float2* v, cudaStream_t s) {
  constexpr int G = 256 / N1;
  size_t smem = sizeof(float2) * (outer_f2<N1, H>() + G * (2 * br - 1));
  int rc = set_smem(fft_cols_inv_kernel<N1, H>, smem, "oi_coarse_to_image_fft/cols");
  if (rc) return rc;
  const long long ncols = (long long)count * bc;
  fft_cols_inv_kernel<N1, H><<<(unsigned)ceil_div(ncols, G), 256, smem, s>>>(ihat, ncols, br, bc, wn_y, v);
  oi::note_launch();
  return check_launch("oi_coarse_to_image_fft/cols");
}
template <int N1>
static int cols_inv(const float2* ihat, int count, int br, int bc, const float2* wn_y, float2* v, cudaStream_t s) {
  switch (gather_blocks(br)) {
    case 2: return cols_inv_h<N1, 2>(ihat, count, br, bc, wn_y, v, s);
    case 4: return cols_inv_h<N1, 4>(ihat, count, br, bc, wn_y, v, s);
  }
  return cols_inv_h<N1, 0>(ihat, count, br, bc, wn_y, v, s);
}

template <int N1, int H>
static int rows_inv_h(const float2* v, int count, int ny, int bc, const float2* wn_x, float* out, cudaStream_t s) {
  constexpr int G = 256 / N1;
  size_t smem = sizeof(float2) * (max(bc * (2 * G + 1), outer_f2<N1, H>()) + G * (2 * bc - 1));
  int rc = set_smem(fft_rows_inv_kernel<N1, H>, smem, "oi_coarse_to_image_fft/rows");
  if (rc) return rc;
  const long long nrows = (long long)count * ny;
  fft_rows_inv_kernel<N1, H><<<(unsigned)ceil_div(nrows, 2 * G), 256, smem, s>>>(v, nrows, ny, bc, wn_x, out);
  oi::note_launch();
  return check_launch("oi_coarse_to_image_fft/rows");
}
template <int N1>
static int rows_inv(const float2* v, int count, int ny, int bc, const float2* wn_x, float* out, cudaStream_t s) {
  switch (gather_blocks(bc)) {
    case 2: return rows_inv_h<N1, 2>(v, count, ny, bc, wn_x, out, s);
    case 4: return rows_inv_h<N1, 4>(v, count, ny, bc, wn_x, out, s);
  }
  return rows_inv_h<N1, 0>(v, count, ny, bc, wn_x, out, s);
}

// Coarse intensity (nparts partial sums of [count][32 N1R][32 N1C]) -> v, the first two passes of the synthesis; v holds
// count * bc columns of ny >= 32 N1R complex values and carries U between the two (same column, its first 32 N1R values).
template <int N1C>
static int coarse_rows(const float* coarse, int nparts, int count, int mr, int bc, const float2* wc, int ny, float2* v,
                       cudaStream_t s) {
  constexpr int MC = 32 * N1C;
  auto run = [&](auto kern, int pairs) {
    const size_t smem = sizeof(float2) * ((size_t)pairs * MC + pairs * 32 * (N1C + 1));
    if (int rc = set_smem(kern, smem, "coarse rows fft")) return rc;
    constexpr int MOST = 65535;   // images per launch: the grid's second dimension
    for (int i = 0; i < count; i += min(MOST, count - i)) {
      kern<<<dim3((unsigned)(mr / (2 * pairs)), (unsigned)min(MOST, count - i)), COARSE_T, smem, s>>>(
          coarse + (long long)i * mr * MC, nparts, (long long)count * mr * MC, mr, bc, wc, ny, v + (long long)i * bc * ny);
      oi::note_launch();
      if (int rc = check_launch("coarse rows fft")) return rc;
    }
    return (int)OI_OK;
  };
  // 16 rows per block write whole 128-byte lines; 8 or 4 rows while that leaves SMs (148) without a block
  if ((long long)count * mr / 16 >= 148) return run(coarse_rows_kernel<N1C, 8>, 8);
  if ((long long)count * mr / 8 >= 148) return run(coarse_rows_kernel<N1C, 4>, 4);
  return run(coarse_rows_kernel<N1C, 2>, 2);
}
template <int N1R, int N1, int H>
static int coarse_cols_h(int count, int br, int bc, const float2* wr, const float2* wn_y, float2* v, float norm, cudaStream_t s) {
  constexpr int G = COARSE_T / N1, MR = 32 * N1R;
  const size_t smem = sizeof(float2) * ((size_t)G * MR + G * 32 * (N1R + 1) + G * (2 * br - 1));
  auto kern = coarse_cols_kernel<N1R, N1, H>;
  if (int rc = set_smem(kern, smem, "coarse columns fft")) return rc;
  kern<<<(unsigned)ceil_div((long long)count * bc, G), COARSE_T, smem, s>>>((long long)count * bc, br, bc, wr, wn_y, norm, v);
  oi::note_launch();
  return check_launch("coarse columns fft");
}
template <int N1R>
static int coarse_cols(int count, int br, int bc, const float2* wr, const float2* wn_y, int ny1, float2* v, float norm,
                       cudaStream_t s) {
  constexpr int H = N1R == 8 ? 4 : 2;   // 2 br - 1 <= 32 N1R
  switch (ny1) {
    case 8: return coarse_cols_h<N1R, 8, H>(count, br, bc, wr, wn_y, v, norm, s);
    case 16: return coarse_cols_h<N1R, 16, H>(count, br, bc, wr, wn_y, v, norm, s);
    case 32: return coarse_cols_h<N1R, 32, H>(count, br, bc, wr, wn_y, v, norm, s);
  }
  return coarse_cols_h<N1R, 64, H>(count, br, bc, wr, wn_y, v, norm, s);
}

static int n1_of(int n) {
  switch (n) {
    case 256: return 8;
    case 512: return 16;
    case 1024: return 32;
    case 2048: return 64;
  }
  return 0;
}

}  // namespace oi

extern "C" int oi_fft_supported(int ny, int nx) {
  return oi::n1_of(ny) != 0 && oi::n1_of(nx) != 0 ? 1 : 0;
}

extern "C" int oi_band_spectrum_fft(const void* field, int kind, int batch, int ny, int nx, int m0r, int br, int m0c,
                                    int bc, const void* wn_x, const void* wn_y, float scale, void* scratch,
                                    void* band, void* stream) {
  using namespace oi;
  if (!field || !wn_x || !wn_y || !scratch || !band || batch <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_band_spectrum_fft: bad arguments");
  if (kind != OI_FIELD_REAL_F32 && kind != OI_FIELD_U8)
    return fail(OI_EINVAL, "oi_band_spectrum_fft: real float32 or uint8 masks only (kind=%d)", kind);
  const int nx1 = n1_of(nx), ny1 = n1_of(ny);
  if (!nx1 || !ny1) return fail(OI_ERANGE, "oi_band_spectrum_fft: grid %dx%d is not 256..2048, power of 2", ny, nx);
  const int maxc = max(abs(m0c), abs(m0c + bc - 1));
  if (2 * maxc >= nx || br > ny)
    return fail(OI_ERANGE, "oi_band_spectrum_fft: band (%d+%d, %d+%d) too wide for %dx%d", m0r, br, m0c, bc, ny, nx);
  cudaStream_t s = (cudaStream_t)stream;
  float2* t = (float2*)scratch;
  int rc = band_rows(nx1, field, kind, batch, ny, 1, m0c, bc, wn_x, t, s);
  if (rc) return rc;
  switch (ny1) {
    case 8: return cols_fwd<8>(t, batch, bc, (const float2*)wn_y, m0r, br, scale, (float2*)band, s);
    case 16: return cols_fwd<16>(t, batch, bc, (const float2*)wn_y, m0r, br, scale, (float2*)band, s);
    case 32: return cols_fwd<32>(t, batch, bc, (const float2*)wn_y, m0r, br, scale, (float2*)band, s);
    default: return cols_fwd<64>(t, batch, bc, (const float2*)wn_y, m0r, br, scale, (float2*)band, s);
  }
}

extern "C" int oi_band_spectrum_fft_c64(const void* field, int batch, int ny, int nx, int nch, int m0r, int br, int m0c, int bc,
                                        const void* wn_x, const void* wn_y, float scale, void* scratch, void* band,
                                        void* stream) {
  using namespace oi;
  if (!field || !wn_x || !wn_y || !scratch || !band || batch <= 0 || nch <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_band_spectrum_fft_c64: bad arguments");
  const int nx1 = n1_of(nx), ny1 = n1_of(ny);
  if (!nx1 || !ny1) return fail(OI_ERANGE, "oi_band_spectrum_fft_c64: grid %dx%d is not 256..2048, power of 2", ny, nx);
  const int maxc = max(abs(m0c), abs(m0c + bc - 1));
  if ((long long)batch * nch > 65535) return fail(OI_ERANGE, "oi_band_spectrum_fft_c64: batch too large");   // as oi_band_spectrum
  if (2 * maxc >= nx || br > ny)
    return fail(OI_ERANGE, "oi_band_spectrum_fft_c64: band (%d+%d, %d+%d) too wide for %dx%d", m0r, br, m0c, bc, ny, nx);
  cudaStream_t s = (cudaStream_t)stream;
  float2* t = (float2*)scratch;
  if (int rc = band_rows(nx1, field, OI_FIELD_COMPLEX_C64, batch, ny, nch, m0c, bc, wn_x, t, s)) return rc;
  const float2* wy = (const float2*)wn_y;
  switch (ny1) {
    case 8: return cols_fwd<8>(t, batch * nch, bc, wy, m0r, br, scale, (float2*)band, s);
    case 16: return cols_fwd<16>(t, batch * nch, bc, wy, m0r, br, scale, (float2*)band, s);
    case 32: return cols_fwd<32>(t, batch * nch, bc, wy, m0r, br, scale, (float2*)band, s);
    default: return cols_fwd<64>(t, batch * nch, bc, wy, m0r, br, scale, (float2*)band, s);
  }
}

// The Hermitian half-spectrum of a coarse intensity held as nparts partial sums (oi_coherent_coarse_fft's output,
// [nparts][count][mr][mc] float32): ihat[i][qr + br-1][qc] = w(qc) / (mr mc) sum_{y,x} (sum_p coarse[p][i][y][x])
// exp(+2 pi i (qr y / mr + qc x / mc)), |qr| < br, 0 <= qc < bc, w(0) = 1 and w(qc > 0) = 2 -- the input of
// oi_spectrum_to_image_fft.  The parts are summed in the row pass's loads; scratch: count * mr * bc complex.
extern "C" int oi_coarse_half_spectrum_fft(const float* coarse, int nparts, int count, int mr, int mc, int br, int bc,
                                           const void* wn_c, const void* wn_r, void* scratch, void* ihat,
                                           void* stream) {
  using namespace oi;
  if (!coarse || !wn_c || !wn_r || !scratch || !ihat || nparts <= 0 || count <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_coarse_half_spectrum_fft: bad arguments");
  const int nx1 = n1_of(mc), ny1 = n1_of(mr);
  if (!nx1 || !ny1)
    return fail(OI_ERANGE, "oi_coarse_half_spectrum_fft: coarse grid %dx%d is not 256..2048, power of 2", mr, mc);
  if (2 * (bc - 1) >= mc || 2 * br - 1 > mr)
    return fail(OI_ERANGE, "oi_coarse_half_spectrum_fft: band %dx%d too wide for %dx%d", br, bc, mr, mc);
  cudaStream_t s = (cudaStream_t)stream;
  float2* t = (float2*)scratch;
  float2* out = (float2*)ihat;
  const int nq = 2 * br - 1, m0r = -(br - 1);
  const float scale = 1.f / ((float)mr * (float)mc);
  const long long pstride = (long long)count * mr * mc;
  int rc = band_rows(nx1, coarse, OI_FIELD_REAL_F32, count, mr, 1, 0, bc, wn_c, t, s, nparts, pstride);
  if (rc) return rc;
  switch (ny1) {
    case 8: return cols_fwd<8>(t, count, bc, (const float2*)wn_r, m0r, nq, scale, out, s, 0, 1);
    case 16: return cols_fwd<16>(t, count, bc, (const float2*)wn_r, m0r, nq, scale, out, s, 0, 1);
    case 32: return cols_fwd<32>(t, count, bc, (const float2*)wn_r, m0r, nq, scale, out, s, 0, 1);
    default: return cols_fwd<64>(t, count, bc, (const float2*)wn_r, m0r, nq, scale, out, s, 0, 1);
  }
}

// out[i][s] = scale sum_{|qr| < br, |qc| < bc} ghat_i(q) exp(-2 pi i q.s / 128) on 128 x 128 points, ghat_i(q) = sum_r g_i(r)
// exp(+2 pi i q.r / N) over the ny x nx grid (256..2048, powers of two); br, bc <= 64.
extern "C" int oi_coarse_gradient_fft(const float* g, int count, int ny, int nx, int br, int bc, const void* wn_x,
                                      const void* wn_y, const void* wn_m, const void* wm, float scale, void* scratch,
                                      float* out, void* stream) {
  using namespace oi;
  if (!g || !wn_x || !wn_y || !wn_m || !wm || !scratch || !out || count <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_coarse_gradient_fft: bad arguments");
  const int nx1 = n1_of(nx), ny1 = n1_of(ny);
  if (!nx1 || !ny1) return fail(OI_ERANGE, "oi_coarse_gradient_fft: grid %dx%d is not 256..2048, power of 2", ny, nx);
  if (br > GRAD_M / 2 || bc > GRAD_M / 2 || count > 65535)
    return fail(OI_ERANGE, "oi_coarse_gradient_fft: band %dx%d or count %d out of range", br, bc, count);
  if ((uintptr_t)scratch % 16) return fail(OI_EINVAL, "oi_coarse_gradient_fft: scratch must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
  float2 *t = (float2*)scratch, *v = t + (long long)count * bc * ny;
  const float2 *wy = (const float2*)wn_y, *wv = (const float2*)wn_m;
  int rc = band_rows(nx1, g, OI_FIELD_REAL_F32, count, ny, 1, 0, bc, wn_x, t, s);
  if (rc) return rc;
  switch (ny1) {
    case 8: rc = cols_coarse<8>(t, count, bc, wy, br, scale, wv, v, s); break;
    case 16: rc = cols_coarse<16>(t, count, bc, wy, br, scale, wv, v, s); break;
    case 32: rc = cols_coarse<32>(t, count, bc, wy, br, scale, wv, v, s); break;
    default: rc = cols_coarse<64>(t, count, bc, wy, br, scale, wv, v, s); break;
  }
  if (rc) return rc;
  // four rows per block while that gives every SM (148) a block, else two
  if ((long long)count * (GRAD_M / 4) >= 148)
    coarse_gradient_rows_kernel<2><<<dim3(GRAD_M / 4, count), GRAD_M, 0, s>>>(v, bc, (const float2*)wm, out);
  else
    coarse_gradient_rows_kernel<1><<<dim3(GRAD_M / 2, count), GRAD_M, 0, s>>>(v, bc, (const float2*)wm, out);
  oi::note_launch();
  return check_launch("oi_coarse_gradient_fft/rows");
}

extern "C" int oi_coarse_to_image_fft(float* coarse, int nparts, int count, int mr, int mc, int br, int bc,
                                      const void* gc, const void* gr, const void* wm_r, const void* wm_c,
                                      const void* wn_y, const void* wn_x, int ny, int nx, void* scratch_ihat,
                                      void* scratch_v, float* out, void* stream) {
  using namespace oi;
  if (!coarse || !gc || !gr || !wn_y || !wn_x || !scratch_ihat || !scratch_v || !out || count <= 0 || nparts <= 0)
    return fail(OI_EINVAL, "oi_coarse_to_image_fft: bad arguments");
  const int nx1 = n1_of(nx), ny1 = n1_of(ny);
  if (!nx1 || !ny1) return fail(OI_ERANGE, "oi_coarse_to_image_fft: grid %dx%d is not 256..2048, power of 2", ny, nx);
  if (2 * br - 1 > ny || 2 * bc - 1 > nx) return fail(OI_ERANGE, "oi_coarse_to_image_fft: band too wide for grid");
  cudaStream_t s = (cudaStream_t)stream;
  int rc;
  float2* v = (float2*)scratch_v;
  auto small = [](int m) { return m == 64 || m == 128 || m == 256; };
  if (wm_r && wm_c && small(mr) && small(mc) && mr <= ny && 2 * br - 1 <= mr && 2 * bc - 1 <= mc &&
      (uintptr_t)coarse % alignof(float4) == 0) {
    const float2 *tr = (const float2*)wm_r, *tc = (const float2*)wm_c;
    rc = mc == 64    ? coarse_rows<2>(coarse, nparts, count, mr, bc, tc, ny, v, s)
         : mc == 128 ? coarse_rows<4>(coarse, nparts, count, mr, bc, tc, ny, v, s)
                     : coarse_rows<8>(coarse, nparts, count, mr, bc, tc, ny, v, s);
    if (rc) return rc;
    const float norm = 1.0f / ((float)mr * (float)mc);
    const float2* wy = (const float2*)wn_y;
    rc = mr == 64    ? coarse_cols<2>(count, br, bc, tr, wy, ny1, v, norm, s)
         : mr == 128 ? coarse_cols<4>(count, br, bc, tr, wy, ny1, v, norm, s)
                     : coarse_cols<8>(count, br, bc, tr, wy, ny1, v, norm, s);
    if (rc) return rc;
    switch (nx1) {
      case 8: return rows_inv<8>(v, count, ny, bc, (const float2*)wn_x, out, s);
      case 16: return rows_inv<16>(v, count, ny, bc, (const float2*)wn_x, out, s);
      case 32: return rows_inv<32>(v, count, ny, bc, (const float2*)wn_x, out, s);
      default: return rows_inv<64>(v, count, ny, bc, (const float2*)wn_x, out, s);
    }
  }
  rc = coarse_spectrum(coarse, count, mr, mc, br, bc, gc, gr, scratch_ihat, s, nparts, scratch_v,
                       (long long)count * bc * ny * (long long)sizeof(float2));
  if (rc) return rc;
  const float2* ih = (const float2*)scratch_ihat;
  switch (ny1) {
    case 8: rc = cols_inv<8>(ih, count, br, bc, (const float2*)wn_y, v, s); break;
    case 16: rc = cols_inv<16>(ih, count, br, bc, (const float2*)wn_y, v, s); break;
    case 32: rc = cols_inv<32>(ih, count, br, bc, (const float2*)wn_y, v, s); break;
    default: rc = cols_inv<64>(ih, count, br, bc, (const float2*)wn_y, v, s); break;
  }
  if (rc) return rc;
  switch (nx1) {
    case 8: return rows_inv<8>(v, count, ny, bc, (const float2*)wn_x, out, s);
    case 16: return rows_inv<16>(v, count, ny, bc, (const float2*)wn_x, out, s);
    case 32: return rows_inv<32>(v, count, ny, bc, (const float2*)wn_x, out, s);
    default: return rows_inv<64>(v, count, ny, bc, (const float2*)wn_x, out, s);
  }
}

extern "C" int oi_spectrum_to_image_fft(const void* ihat, int count, int br, int bc, const void* wn_y,
                                        const void* wn_x, int ny, int nx, void* scratch_v, float* out,
                                        void* stream) {
  using namespace oi;
  if (!ihat || !wn_y || !wn_x || !scratch_v || !out || count <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_spectrum_to_image_fft: bad arguments");
  const int nx1 = n1_of(nx), ny1 = n1_of(ny);
  if (!nx1 || !ny1) return fail(OI_ERANGE, "oi_spectrum_to_image_fft: grid %dx%d is not 256..2048, power of 2", ny, nx);
  if (2 * br - 1 > ny || 2 * bc - 1 > nx) return fail(OI_ERANGE, "oi_spectrum_to_image_fft: band too wide for grid");
  cudaStream_t s = (cudaStream_t)stream;
  const float2* ih = (const float2*)ihat;
  float2* v = (float2*)scratch_v;
  int rc;
  switch (ny1) {
    case 8: rc = cols_inv<8>(ih, count, br, bc, (const float2*)wn_y, v, s); break;
    case 16: rc = cols_inv<16>(ih, count, br, bc, (const float2*)wn_y, v, s); break;
    case 32: rc = cols_inv<32>(ih, count, br, bc, (const float2*)wn_y, v, s); break;
    default: rc = cols_inv<64>(ih, count, br, bc, (const float2*)wn_y, v, s); break;
  }
  if (rc) return rc;
  switch (nx1) {
    case 8: return rows_inv<8>(v, count, ny, bc, (const float2*)wn_x, out, s);
    case 16: return rows_inv<16>(v, count, ny, bc, (const float2*)wn_x, out, s);
    case 32: return rows_inv<32>(v, count, ny, bc, (const float2*)wn_x, out, s);
    default: return rows_inv<64>(v, count, ny, bc, (const float2*)wn_x, out, s);
  }
}

// Split-BF16x3 tensor-core form of oi_band_spectrum_fft: the row pass is oi_rows_fwd_tc (a DFT contraction
// on the tensor cores against the constant image `wconsts` of oi_rows_tc_constants(0, ...)), the column pass
// the FFT above.
extern "C" int oi_band_spectrum_tc(const void* field, int kind, int batch, int ny, int nx, int m0r, int br, int m0c,
                                   int bc, const void* wconsts, const void* wn_y, float scale, void* scratch,
                                   void* band, void* stream) {
  using namespace oi;
  if (!field || !wconsts || !wn_y || !scratch || !band || batch <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_band_spectrum_tc: bad arguments");
  const int ny1 = n1_of(ny);
  if (!ny1 || nx % 128 != 0 || nx > 4096)
    return fail(OI_ERANGE, "oi_band_spectrum_tc: grid %dx%d unsupported", ny, nx);
  if (bc > 64 || br > ny) return fail(OI_ERANGE, "oi_band_spectrum_tc: band %dx%d unsupported", br, bc);
  int rc = oi_rows_fwd_tc(field, kind, batch, ny, nx, m0c, bc, wconsts, scratch, stream);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  const float2* t = (const float2*)scratch;
  switch (ny1) {
    case 8: return cols_fwd<8>(t, batch, bc, (const float2*)wn_y, m0r, br, scale, (float2*)band, s);
    case 16: return cols_fwd<16>(t, batch, bc, (const float2*)wn_y, m0r, br, scale, (float2*)band, s);
    case 32: return cols_fwd<32>(t, batch, bc, (const float2*)wn_y, m0r, br, scale, (float2*)band, s);
    default: return cols_fwd<64>(t, batch, bc, (const float2*)wn_y, m0r, br, scale, (float2*)band, s);
  }
}

// oi_band_spectrum_tc for a symmetric band (m0r = -(br-1)/2, m0c = -(bc-1)/2, br and bc odd, bc <= 63): the row
// pass computes only the band's non-negative columns (oi_rows_fwd_tc_half against `hconsts` of
// oi_rows_tc_constants(2, nx, m0c, bc, ...)) and the column pass fills the negative ones from
// band[-ky][-kx] = conj(band[ky][kx]) (a real mask).  scratch: batch * ny * (bc+1)/2 complex.
extern "C" int oi_band_spectrum_tc_sym(const void* field, int kind, int batch, int ny, int nx, int br, int bc,
                                       const void* hconsts, const void* wn_y, float scale, void* scratch, void* band,
                                       void* stream) {
  using namespace oi;
  if (!field || !hconsts || !wn_y || !scratch || !band || batch <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_band_spectrum_tc_sym: bad arguments");
  const int ny1 = n1_of(ny);
  if (!ny1 || nx % 128 != 0 || nx > 4096)
    return fail(OI_ERANGE, "oi_band_spectrum_tc_sym: grid %dx%d unsupported", ny, nx);
  if (bc % 2 == 0 || br % 2 == 0 || bc > 63 || br > ny)
    return fail(OI_ERANGE, "oi_band_spectrum_tc_sym: band %dx%d is not an odd symmetric band of width <= 63", br, bc);
  const int bch = (bc + 1) / 2, m0r = -(br - 1) / 2;
  int rc = oi_rows_fwd_tc_half(field, kind, batch, ny, nx, bch, hconsts, scratch, stream);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  const float2* t = (const float2*)scratch;
  switch (ny1) {
    case 8: return cols_fwd<8, true>(t, batch, bch, (const float2*)wn_y, m0r, br, scale, (float2*)band, s, bc);
    case 16: return cols_fwd<16, true>(t, batch, bch, (const float2*)wn_y, m0r, br, scale, (float2*)band, s, bc);
    case 32: return cols_fwd<32, true>(t, batch, bch, (const float2*)wn_y, m0r, br, scale, (float2*)band, s, bc);
    default: return cols_fwd<64, true>(t, batch, bch, (const float2*)wn_y, m0r, br, scale, (float2*)band, s, bc);
  }
}

// Split-BF16x3 tensor-core form of oi_coarse_to_image_fft on the 128 x 128 coarse grid: fold, coarse spectrum
// and column pass as there; the row pass is oi_rows_inv_tc against `cconsts` of oi_rows_tc_constants(1, ...).
extern "C" int oi_coarse_to_image_tc(float* coarse, int nparts, int count, int br, int bc, const void* wm_r,
                                     const void* wm_c, const void* wn_y, const void* cconsts, int ny, int nx,
                                     void* scratch_ihat, void* scratch_v, void* scratch_tiles, float* out,
                                     void* stream) {
  using namespace oi;
  (void)scratch_v;
  if (!coarse || !wm_r || !wm_c || !wn_y || !cconsts || !scratch_ihat || !scratch_tiles || !out || count <= 0 ||
      nparts <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_coarse_to_image_tc: bad arguments");
  const int ny1 = n1_of(ny);
  if (!ny1 || nx % 128 != 0 || nx > 4096 || bc > 64 || 2 * br - 1 > 128 || 2 * br - 1 > ny)
    return fail(OI_ERANGE, "oi_coarse_to_image_tc: grid %dx%d / band %dx%d unsupported", ny, nx, br, bc);
  cudaStream_t s = (cudaStream_t)stream;
  float2* ih = (float2*)scratch_ihat;
  int rc = launch_coarse_spec_fft(coarse, nparts, count, br, bc, (const float2*)wm_r, (const float2*)wm_c, ih, s);
  if (rc) return rc;
  unsigned char* tiles = (unsigned char*)scratch_tiles;
  const float2* wy = (const float2*)wn_y;
  switch (ny1) {
    case 8: rc = cols_inv_tiles<8, 32>(ih, count, br, bc, ny, wy, tiles, s); break;
    case 16: rc = cols_inv_tiles<16, 16>(ih, count, br, bc, ny, wy, tiles, s); break;
    case 32: rc = cols_inv_tiles<32, 8>(ih, count, br, bc, ny, wy, tiles, s); break;
    default: rc = cols_inv_tiles<64, 8>(ih, count, br, bc, ny, wy, tiles, s); break;
  }
  if (rc) return rc;
  return rows_inv_from_tiles(tiles, count, ny, nx, cconsts, out, s);
}
