// Exact band-limited resampling of the coarse intensity to the output grid: the last step of both imaging
// paths (the fftshift + normalisation of CalculateAerialImage.py:89-92 and CalculateAerialImage_SOCS.py:10).
//
// The intensity of fields band-limited to Br x Bc has a spectrum supported on |qr| < Br, |qc| < Bc.  Its
// samples on the coarse Mr x Mc grid (Mr >= 2Br-1, Mc >= 2Bc-1) determine that spectrum exactly:
//   Ihat(q) = 1/(Mr Mc) sum_s coarse[s] exp(+2 pi i (qr sr/Mr + qc sc/Mc))             (spec kernel)
// (the coarse intensity may arrive as `nparts` partial sums laid out one after another; they are added here)
// and the output is its trigonometric polynomial evaluated on the Ny x Nx grid.  The intensity is real, so
// only qc >= 0 is kept (qc > 0 doubled) and the x synthesis is a real dot product:
//   V[y][qc]   = sum_qr Ihat(qr, qc) exp(-2 pi i qr y/Ny)
//   out[y][x]  = sum_qc Re(V[y][qc] exp(-2 pi i qc x/Nx))                                 (synth kernel)
#include "dft_gemm.cuh"

namespace oi {

constexpr int SP_QT = 16;  // qc per spec block

// grid (ceil(bc/16), count).  ihat[i][jr][qc], jr = qr + br - 1.
__global__ void __launch_bounds__(256) coarse_spec_kernel(const float* __restrict__ coarse, int mr, int mc, int br, int bc,
                                                          const float2* __restrict__ gc, const float2* __restrict__ gr,
                                                          float2* __restrict__ ihat) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* us = (float2*)smem_raw;  // [mr][SP_QT]
  const int tid = threadIdx.x, ql = tid % SP_QT, rg = tid / SP_QT;  // rg 0..15
  const int qc0 = blockIdx.x * SP_QT;
  const long long img = blockIdx.y;
  const float* cimg = coarse + img * (long long)mr * mc;
  const int qc = qc0 + ql;
  const int nq = 2 * br - 1;
  // U[sr][qc] = sum_sc coarse[sr][sc] gc[sc][qc]
  for (int sr = rg; sr < mr; sr += 16) {
    float2 u = make_float2(0.f, 0.f);
    if (qc < bc) {
      const float* row = cimg + (long long)sr * mc;
      for (int sc = 0; sc < mc; ++sc) {
        const float v = __ldg(row + sc);
        const float2 t = __ldg(gc + (long long)sc * bc + qc);
        u.x = fmaf(v, t.x, u.x);
        u.y = fmaf(v, t.y, u.y);
      }
    }
    us[sr * SP_QT + ql] = u;
  }
  __syncthreads();
  const float norm = (qc == 0 ? 1.0f : 2.0f) / ((float)mr * (float)mc);
  for (int jr = rg; jr < nq; jr += 16) {
    if (qc >= bc) continue;
    float2 acc = make_float2(0.f, 0.f);
    for (int sr = 0; sr < mr; ++sr) cfma(acc, __ldg(gr + (long long)sr * nq + jr), us[sr * SP_QT + ql]);
    ihat[(img * nq + jr) * (long long)bc + qc] = make_float2(acc.x * norm, acc.y * norm);
  }
}

// The same spectrum as two tile products (dft_gemm.cuh), U = coarse * gc and ihat = gr^T U, when the caller has room for
// U: the partial sums are added as the first product's operand is read.  Four 128 x 128 coarse images of 59 x 59 bands:
// 239 us (16 blocks, one output per thread at a time) -> 14 us, and the separate addition of the parts (4 us) goes.
struct SpecRows {
  using A = float;
  static constexpr bool A_K = true;
  const float* coarse;
  int nparts;
  long long pstride;
  int mc, bc;
  const float2* gc;
  float2* u;
  __device__ __forceinline__ float a(int, int R, int sc) const {
    const float* p = coarse + (long long)R * mc + sc;
    float v = __ldg(p);
    for (int i = 1; i < nparts; ++i) v += __ldg(p + i * pstride);
    return v;
  }
  __device__ __forceinline__ float2 b(int, int sc, int qc) const { return __ldg(gc + (long long)sc * bc + qc); }
  __device__ __forceinline__ void put(int, int R, int qc, float2 v) const { u[(long long)R * bc + qc] = v; }
};
struct SpecCols {
  using A = float2;
  static constexpr bool A_K = false;
  const float2* u;
  int mr, nq, bc;
  const float2* gr;
  float norm;
  float2* ihat;
  __device__ __forceinline__ float2 a(int, int jr, int sr) const { return __ldg(gr + (long long)sr * nq + jr); }
  __device__ __forceinline__ float2 b(int img, int sr, int qc) const { return u[((long long)img * mr + sr) * bc + qc]; }
  __device__ __forceinline__ void put(int img, int jr, int qc, float2 v) const {
    const float s = qc == 0 ? norm : 2.f * norm;
    ihat[((long long)img * nq + jr) * bc + qc] = make_float2(v.x * s, v.y * s);
  }
};

// RB output rows per block (grid ceil(ny / RB), count): V of those rows into shared memory by 16-frequency steps, then
// the columns x and nx - x from the same products (sx[nx - x] = conj sx[x]): with A = sum Re V Re sx and B = sum Im V Im sx
// they are A - B and A + B.  A half of the block takes a half of the rows, a thread up to three columns 128 apart; V is read
// as pairs of frequencies, one broadcast 16-byte load per row for 4 to 12 multiply-adds.  Bound: the reads of sx (each
// block reads its half, from L2) and FP32 issue.  Four 1000 x 750 images, 59 columns: 61 -> 31.9 us (44.7 with every column
// computed).
template <int R, int XV>
__device__ __forceinline__ void synth_columns(const float4* vs, int pairs, const float2* __restrict__ sx, int bc, int nx,
                                              int x0, float* o, int rows) {
  float a[R][XV], b[R][XV];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int u = 0; u < XV; ++u) a[r][u] = b[r][u] = 0.f;
  const int half = nx / 2 + 1, x = x0 + threadIdx.x % 128;
#pragma unroll 2
  for (int q = 0; q < pairs; ++q) {
    float2 t0[XV], t1[XV];
#pragma unroll
    for (int u = 0; u < XV; ++u) {
      const bool in = x + 128 * u < half;
      const float2* p = sx + (long long)(2 * q) * nx + x + 128 * u;
      t0[u] = in ? __ldg(p) : make_float2(0.f, 0.f);
      t1[u] = in && 2 * q + 1 < bc ? __ldg(p + nx) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 v = vs[r * pairs + q];
#pragma unroll
      for (int u = 0; u < XV; ++u) {
        a[r][u] = fmaf(v.x, t0[u].x, fmaf(v.z, t1[u].x, a[r][u]));
        b[r][u] = fmaf(v.y, t0[u].y, fmaf(v.w, t1[u].y, b[r][u]));
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int u = 0; u < XV; ++u) {
      const int xu = x + 128 * u;
      if (r >= rows || xu >= half) continue;
      float* row = o + (long long)r * nx;
      row[xu] = a[r][u] - b[r][u];
      if (xu > 0 && 2 * xu < nx) row[nx - xu] = a[r][u] + b[r][u];
    }
}

template <int RB>
__global__ void __launch_bounds__(256, 2) synth_kernel(const float2* __restrict__ ihat, int br, int bc,
                                                       const float2* __restrict__ sy, const float2* __restrict__ sx,
                                                       int ny, int nx, float* __restrict__ out) {
  constexpr int CG = 256 / RB, NQ = RB / 4, KS = 16;   // column groups of a row, outputs per thread, frequencies per step
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* vs = (float2*)smem_raw;   // [RB][2 * pairs]
  __shared__ float2 ys[KS][RB + 1], hs[KS][64];
  const int tid = threadIdx.x, y0 = blockIdx.x * RB, rows = min(RB, ny - y0), nq = 2 * br - 1, pairs = (bc + 1) / 2;
  const long long img = blockIdx.y;
  const float2* ih = ihat + img * (long long)nq * bc;
  const int r = tid / CG, cq = tid % CG;
  for (int q0 = 0; q0 < 2 * pairs; q0 += 64) {
    float2 acc[NQ];
#pragma unroll
    for (int j = 0; j < NQ; ++j) acc[j] = make_float2(0.f, 0.f);
    for (int k0 = 0; k0 < nq; k0 += KS) {
      __syncthreads();
      for (int e = tid; e < KS * RB; e += 256) {
        const int k = e % KS, rr = e / KS;
        ys[k][rr] = rr < rows && k0 + k < nq ? __ldg(sy + (long long)(y0 + rr) * nq + k0 + k) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < KS * 64 / 256; ++i) {
        const int e = tid + 256 * i, q = e % 64, k = e / 64;
        hs[k][q] = k0 + k < nq && q0 + q < bc ? __ldg(ih + (long long)(k0 + k) * bc + q0 + q) : make_float2(0.f, 0.f);
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < KS; ++k) {
        const float2 y = ys[k][r];
#pragma unroll
        for (int j = 0; j < NQ; ++j) cfma(acc[j], y, hs[k][cq + CG * j]);
      }
    }
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
      const int q = q0 + cq + CG * j;
      if (q < 2 * pairs) vs[r * 2 * pairs + q] = acc[j];
    }
  }
  __syncthreads();
  const int g = tid / 128 * (RB / 2), left = rows - g;   // this half's first row, and the rows from there on
  const float4* vg = (const float4*)vs + g * pairs;
  float* o = out + (img * ny + y0 + g) * (long long)nx;
  for (int x0 = 0; x0 < nx / 2 + 1;) {
    const int groups = (nx / 2 + 1 - x0 + 127) / 128;   // four as two and two, else three at a time
    if (groups == 1) {
      synth_columns<RB / 2, 1>(vg, pairs, sx, bc, nx, x0, o, left);
      x0 += 128;
    } else if (groups == 2 || groups == 4) {
      synth_columns<RB / 2, 2>(vg, pairs, sx, bc, nx, x0, o, left);
      x0 += 256;
    } else {
      synth_columns<RB / 2, 3>(vg, pairs, sx, bc, nx, x0, o, left);
      x0 += 384;
    }
  }
}

// part[0][i] += part[1][i] + ... + part[nparts-1][i], in place (float4 lanes; n is a multiple of 4).
__global__ void sum_parts_kernel(float* __restrict__ coarse, int nparts, long long n) {
  long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i >= n) return;
  float4 acc = *(const float4*)(coarse + i);
  for (int p = 1; p < nparts; ++p) {
    const float4 v = __ldg((const float4*)(coarse + p * n + i));
    acc.x += v.x;
    acc.y += v.y;
    acc.z += v.z;
    acc.w += v.w;
  }
  *(float4*)(coarse + i) = acc;
}

static int check_parts(int nparts, long long n) {
  return nparts > 1 && n % 4 != 0 ? fail(OI_EINVAL, "partial sums of %lld floats are not float4 aligned", n) : (int)OI_OK;
}

int fold_parts(float* coarse, int nparts, long long n, cudaStream_t s) {
  if (int rc = check_parts(nparts, n)) return rc;
  if (nparts <= 1) return OI_OK;
  sum_parts_kernel<<<(unsigned)ceil_div(n / 4, 256), 256, 0, s>>>(coarse, nparts, n);
  oi::note_launch();
  return check_launch("coarse spectrum/sum parts");
}

int coarse_spectrum(float* coarse, int count, int mr, int mc, int br, int bc, const void* gc, const void* gr,
                    void* ihat, cudaStream_t s, int nparts, void* room, long long room_bytes) {
  if (mr < 2 * br - 1 || mc < 2 * bc - 1)
    return fail(OI_EINVAL, "coarse grid %dx%d too small for band %dx%d", mr, mc, br, bc);
  if (mr > 1024 || count > 65535) return fail(OI_ERANGE, "coarse grid mr=%d or count=%d out of range", mr, count);
  if (int rc = check_parts(nparts, (long long)count * mr * mc)) return rc;   // whichever form runs
  // (a caller's images may start at any float; the pairs of U may not)
  if ((long long)count * mr * bc * (long long)sizeof(float2) <= room_bytes && (uintptr_t)room % alignof(float2) == 0) {
    float2* u = (float2*)room;
    const int nq = 2 * br - 1;
    const SpecRows op{coarse, nparts, (long long)count * mr * mc, mc, bc, (const float2*)gc, u};
    // 32 x 32 tiles until the 64 x 64 ones alone fill the SMs (148): K is too short for a cluster to make up for it
    // (four 128 x 128 images: 14.7 us as 64 x 64 tiles, 8.9 as 32 x 32)
    int rc = (long long)ceil_div(count * mr, 64) * ceil_div(bc, 64) >= 148
                 ? dg::gemm<64, 64, 4, 4>(op, 1, count * mr, bc, mc, s, "coarse spectrum/rows")
                 : dg::gemm<32, 32, 2, 2>(op, 1, count * mr, bc, mc, s, "coarse spectrum/rows");
    if (rc) return rc;
    return dg::gemm<32, 32, 2, 2>(SpecCols{u, mr, nq, bc, (const float2*)gr, 1.0f / ((float)mr * (float)mc), (float2*)ihat},
                                  count, nq, bc, mr, s, "coarse spectrum/columns");
  }
  int rc = fold_parts(coarse, nparts, (long long)count * mr * mc, s);
  if (rc) return rc;
  size_t smem = sizeof(float2) * (size_t)mr * SP_QT;
  {
    int rc_smem = ensure_smem((const void*)coarse_spec_kernel, smem, "coarse spectrum");
    if (rc_smem) return rc_smem;
  }
  dim3 g1((unsigned)ceil_div(bc, SP_QT), (unsigned)count);
  coarse_spec_kernel<<<g1, 256, smem, s>>>(coarse, mr, mc, br, bc, (const float2*)gc, (const float2*)gr, (float2*)ihat);
  oi::note_launch();
  return check_launch("coarse spectrum");
}

template <int RB>
static void launch_synth_rb(const float2* ihat, int count, int br, int bc, const float2* sy, const float2* sx, int ny,
                            int nx, float* out, cudaStream_t s) {
  dim3 grid((unsigned)ceil_div(ny, RB), (unsigned)count);
  synth_kernel<RB><<<grid, 256, sizeof(float2) * RB * 2 * ((bc + 1) / 2), s>>>(ihat, br, bc, sy, sx, ny, nx, out);
  oi::note_launch();
}
// More rows per block reuse the sx values more; fewer fill the SMs when there are few rows (and 16 rows of more than 256
// frequencies pass the shared memory that needs no opt-in).
static void launch_synth(const float2* ihat, int count, int br, int bc, const float2* sy, const float2* sx, int ny, int nx,
                         float* out, cudaStream_t s) {
  auto enough = [&](int rb) { return (long long)ceil_div(ny, rb) * count >= 148; };
  if (enough(16) && bc <= 256)
    launch_synth_rb<16>(ihat, count, br, bc, sy, sx, ny, nx, out, s);
  else if (enough(8))
    launch_synth_rb<8>(ihat, count, br, bc, sy, sx, ny, nx, out, s);
  else
    launch_synth_rb<4>(ihat, count, br, bc, sy, sx, ny, nx, out, s);
}

}  // namespace oi

extern "C" int oi_coarse_to_image(float* coarse, int nparts, int count, int mr, int mc, int br, int bc,
                                  const void* gc, const void* gr, const void* sy, const void* sx, int ny, int nx,
                                  void* scratch, float* out, void* stream) {
  using namespace oi;
  if (!coarse || !gc || !gr || !sy || !sx || !scratch || !out || nparts <= 0 || count <= 0 || mr <= 0 || mc <= 0 ||
      br <= 0 || bc <= 0 || ny <= 0 || nx <= 0)
    return fail(OI_EINVAL, "oi_coarse_to_image: bad arguments");
  if (mr < 2 * br - 1 || mc < 2 * bc - 1)
    return fail(OI_EINVAL, "oi_coarse_to_image: coarse grid %dx%d too small for band %dx%d", mr, mc, br, bc);
  if (mr > 1024 || bc > 512 || nx > 2048 || count > 65535)
    return fail(OI_ERANGE, "oi_coarse_to_image: sizes out of range (mr=%d bc=%d nx=%d)", mr, bc, nx);
  cudaStream_t s = (cudaStream_t)stream;
  // U lives in `out` until the synthesis writes it
  int rc = coarse_spectrum(coarse, count, mr, mc, br, bc, gc, gr, scratch, s, nparts, out,
                           (long long)count * ny * nx * (long long)sizeof(float));
  if (rc) return rc;
  launch_synth((const float2*)scratch, count, br, bc, (const float2*)sy, (const float2*)sx, ny, nx, out, s);
  return check_launch("oi_coarse_to_image/synth");
}

extern "C" int oi_spectrum_to_image(const void* ihat, int count, int br, int bc, const void* sy, const void* sx,
                                    int ny, int nx, float* out, void* stream) {
  using namespace oi;
  if (!ihat || !sy || !sx || !out || count <= 0 || br <= 0 || bc <= 0 || ny <= 0 || nx <= 0)
    return fail(OI_EINVAL, "oi_spectrum_to_image: bad arguments");
  if (bc > 512 || nx > 2048 || count > 65535)
    return fail(OI_ERANGE, "oi_spectrum_to_image: sizes out of range (bc=%d nx=%d)", bc, nx);
  cudaStream_t s = (cudaStream_t)stream;
  launch_synth((const float2*)ihat, count, br, bc, (const float2*)sy, (const float2*)sx, ny, nx, out, s);
  return check_launch("oi_spectrum_to_image");
}
