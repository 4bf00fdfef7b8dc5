// Adjoint of the coherent sum, for inverse lithography (gradients of a loss L through the aerial image).
//
// Forward (coherent_fft.cu):  I(r) = sum_f w_f |E_f(r)|^2,  E_f(r) = sum_{m in band} A_f(m) exp(-2 pi i m.r/N),
// A_f = P_k .* c, c(m) = 1/(Ny Nx) sum_y t(y) exp(+2 pi i m.y/N).  Given g = dL/dI (real, Ny x Nx):
//   dL/dt(y) = 2/(Ny Nx) Re sum_{m in band} W(m) exp(-2 pi i m.y/N),   W(m) = sum_f w_f conj(P_f(m)) F_f(m),
//   F_f(m)   = sum_r g(r) E_f(r) exp(+2 pi i m.r/N).
// F_f is evaluated exactly on the coarse grid: with g^c(s) = 1/(Mr Mc) sum_{|q|<B} ghat(q) exp(-2 pi i q.s/M)
// (the band-limited coarse copy of g, ghat(q) = sum_r g(r) exp(+2 pi i q.r/N)),
//   F_f(m) = sum_s g^c(s) E_f^c(s) exp(+2 pi i m.s/M)      for M >= 2B - 1 (no alias of m - m' reaches the band).
// The same coarse quantities give <g, |E_f|^2> = sum_s g^c(s) |E_f^c(s)|^2, the per-field dot products from
// which the source-weight gradient of the Abbe image follows (dI/dw_j = (n I_j - I) / sum w).
//
// One block per (field split, plane, image): for each of its fields it recomputes E^c (row and column inverse FFTs, as the
// forward kernel, with the band wrapped: the phase of a shift cancels between E and the transform back),
// multiplies by g^c, and takes the product back to the band by column and row FFTs of which only the band's bins are
// formed, accumulating W in registers.  Nothing per field reaches global memory.
// Bound: FP32 and shared-memory issue (about 10k issue cycles a field on one SM).  With direct DFTs back to the band
// (128 terms a bin) a launch of 8 images of 16 fields took 124 us; now 18.6 us for the 8 packed fields an image that a
// real mask needs of those.  144 fields of 2 images: 113 -> 19 us.
#include "fft_common.cuh"

namespace oi {

using cg::brev5;
using X4 = cg::Axis<4>;

constexpr int ADJ_T = 512;                 // 128 columns x 4 threads each
constexpr int ADJ_M = X4::M, ADJ_LD = X4::FIELD_LD;

struct AdjointArgs {
  const float2* band;       // [batch][nch][br][bc]
  long long band_img_stride;
  int nch, br, bc, m0r, m0c;
  const float2* pupil;      // [nz][nk][br][bc]
  const float* weight;      // [nz][nk]
  const float* gcoarse;     // [batch][nz][mr][mc]
  int nz, nk, nsplit;
  const float2* wr;         // exp(+2 pi i j / mr)
  const float2* wc;         // exp(+2 pi i j / mc)
  float2* wout;             // [nsplit][batch][nz][nch][br][bc], or null: field dots alone
  float* field_dot;         // [batch][nz][nk*nch] or null
};

// 128-point transform X[m] = sum_s x[s] exp(+2 pi i m s / 128), -32 <= m < 32, by the four neighbouring lanes n1 = lane % 4,
// lane n1 holding x[n1 + 4 j] in v[j]: a 32-point transform each, then the two wanted outputs of every 4-point transform
// across the lanes, exchanged so that each lane ends with 16 of them: out[j] = X[m] of place band_bin(j, n1) (m mod 64).
__device__ __forceinline__ int band_bin(int j, int n1) { return brev5(j) + (n1 >> 1) + 32 * (n1 & 1); }
__device__ __forceinline__ void band_dft128(float2 (&v)[32], float2 (&out)[16], const float2* tw, int n1) {
  cg::dft32<+1>(v);
#pragma unroll
  for (int i = 1; i < 32; ++i) {
    const float2 t = tw[brev5(i) * 4 + n1];
    v[i] = cmul(v[i], make_float2(t.x, -t.y));
  }
  const bool hi = n1 & 2, odd = n1 & 1;
  // lanes n1 and n1 ^ 2 share the work on their pair: the lower takes even k2 (registers below 16), the upper odd k2
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float2 keep = hi ? v[16 + j] : v[j], give = hi ? v[j] : v[16 + j];
    const float2 got = make_float2(__shfl_xor_sync(0xffffffffu, give.x, 2), __shfl_xor_sync(0xffffffffu, give.y, 2));
    const float2 lo = hi ? got : keep, up = hi ? keep : got;   // lanes n1 and n1 + 2 of the pair
    const float2 s = make_float2(lo.x + up.x, lo.y + up.y), d = make_float2(lo.x - up.x, lo.y - up.y);
    // m = k2: s_0 + s_1 on the even lane; m = k2 - 32: d_0 - i d_1 on the odd one
    const float2 send = odd ? s : d;
    const float2 recv = make_float2(__shfl_xor_sync(0xffffffffu, send.x, 1), __shfl_xor_sync(0xffffffffu, send.y, 1));
    out[j] = odd ? make_float2(recv.x + d.y, recv.y - d.x) : make_float2(s.x + recv.x, s.y + recv.y);
  }
}

__global__ void __launch_bounds__(ADJ_T, 1) coherent_adjoint_kernel(AdjointArgs a) {
  constexpr int T = ADJ_T, WARPS = T / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* twr = (float2*)smem_raw;              // [32][4]
  float2* twc = twr + 128;                      // [32][4]
  float2* as = twc + 128;                       // [64][BAND_LD]: columns at their places, else zero
  float2* x = as + X4::B * X4::BAND_LD;         // [64][ADJ_LD]: rows transformed, then columns back, at their places
  float* red = (float*)(x + X4::B * ADJ_LD);    // [2][WARPS]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = blockIdx.x, z = blockIdx.y, br = a.br, bc = a.bc, plane = br * bc;
  const long long b = blockIdx.z;
  cg::build_twiddles<4>(twr, a.wr, tid, T);
  cg::build_twiddles<4>(twc, a.wc, tid, T);
  for (int j = tid; j < X4::B * (X4::BAND_LD + ADJ_LD); j += T) as[j] = make_float2(0.f, 0.f);
  const int pr = X4::place0(a.m0r, br), pc = X4::place0(a.m0c, bc);
  __syncthreads();
  const float* gc = a.gcoarse + (b * a.nz + z) * (long long)ADJ_M * ADJ_M;
  const int nfield = a.nk * a.nch;
  const float2* pup = a.pupil + (long long)z * a.nk * plane;
  const int n1 = tid & 3, sc = tid >> 2;        // column task (and, for rows below br, row task sc)
  for (int c = 0; c < a.nch; ++c) {
    float2 wacc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) wacc[j] = make_float2(0.f, 0.f);
    int parity = 0;
    for (int f = split; f < nfield; f += a.nsplit) {
      if (f % a.nch != c) continue;
      const int k = f / a.nch;
      const float w = __ldg(a.weight + (long long)z * a.nk + k);
      const float2* pk = pup + (long long)k * plane;
      const float2* hc = a.band + b * a.band_img_stride + (long long)c * plane;
#pragma unroll 2
      for (int ir = warp; ir < br; ir += WARPS) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int ic = lane + 32 * u;
          if (ic < bc) as[ir * X4::BAND_LD + ((pc + ic) & 63)] = cmul(__ldg(pk + ir * bc + ic), __ldg(hc + ir * bc + ic));
        }
      }
      __syncthreads();
      // E^c: row inverse FFTs of the band rows, then column inverse FFTs
      float2 v[32];
      if (sc < br) {
        cg::band_ifft<4>(v, as + sc * X4::BAND_LD, 1, twc, n1);
#pragma unroll
        for (int i = 0; i < 32; ++i) x[((pr + sc) & 63) * ADJ_LD + n1 + 4 * brev5(i)] = v[i];
      }
      __syncthreads();
      cg::band_ifft<4>(v, x + sc, ADJ_LD, twr, n1);
      float dot = 0.f;
      float2 y[32];   // Y = g^c E^c in row order: y[j] at row n1 + 4 j
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float g = __ldg(gc + (n1 + 4 * brev5(i)) * ADJ_M + sc);
        dot = fmaf(g, fmaf(v[i].x, v[i].x, v[i].y * v[i].y), dot);
        y[brev5(i)] = make_float2(g * v[i].x, g * v[i].y);
      }
      if (a.field_dot) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if (lane == 0) red[parity * WARPS + warp] = dot;
      }
      float2 out[16];
      if (a.wout) {
        band_dft128(y, out, twr, n1);
        __syncthreads();   // every column task has read its rows
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int place = band_bin(j, n1);
          if (((place - pr) & 63) < br) x[place * ADJ_LD + sc] = out[j];
        }
      }
      __syncthreads();
      if (a.field_dot && warp == 0) {
        float s = lane < WARPS ? red[parity * WARPS + lane] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) a.field_dot[(b * a.nz + z) * (long long)nfield + f] = s;
      }
      parity ^= 1;
      if (a.wout && (sc & ~7) < br) {   // whole warps: the exchange is among a row's four lanes
        const int row = sc < br ? sc : br - 1;
#pragma unroll
        for (int j = 0; j < 32; ++j) y[j] = x[((pr + row) & 63) * ADJ_LD + n1 + 4 * j];
        band_dft128(y, out, twc, n1);
        if (sc < br) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int ic = (band_bin(j, n1) - pc) & 63;
            if (ic < bc) {
              const float2 p = __ldg(pk + sc * bc + ic);
              cfma(wacc[j], make_float2(w * p.x, -w * p.y), out[j]);
            }
          }
        }
      }
      // the next field's products go to `as`, which no thread reads past the row pass; its rows overwrite x after the
      // barrier that follows them
    }
    if (a.wout && sc < br) {
      float2* o = a.wout + ((((long long)split * gridDim.z + b) * a.nz + z) * a.nch + c) * plane + sc * bc;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int ic = (band_bin(j, n1) - pc) & 63;
        if (ic < bc) o[ic] = wacc[j];
      }
    }
  }
}

static int launch_adjoint(const AdjointArgs& a, int batch, cudaStream_t s, const char* what) {
  const size_t smem = sizeof(float2) * (256 + (size_t)X4::B * (X4::BAND_LD + ADJ_LD)) + sizeof(float) * 2 * (ADJ_T / 32);
  int rc = ensure_smem((const void*)coherent_adjoint_kernel, smem, what);
  if (rc) return rc;
  dim3 grid((unsigned)a.nsplit, (unsigned)a.nz, (unsigned)batch);
  coherent_adjoint_kernel<<<grid, ADJ_T, smem, s>>>(a);
  oi::note_launch();
  return check_launch(what);
}

static int adjoint(const void* band, int batch, int nch, int m0r, int br, int m0c, int bc, const void* pupil, const float* weight, int nz,
                   int nk, const float* gcoarse, int mr, int mc, const void* wr, const void* wc, int nsplit, void* wout,
                   float* field_dot, cudaStream_t s, const char* what) {
  if (!band || !pupil || !weight || !gcoarse || !wr || !wc || batch <= 0 || nch <= 0 || br <= 0 || bc <= 0 || nz <= 0 ||
      nk <= 0 || nsplit <= 0)
    return fail(OI_EINVAL, "%s: bad arguments", what);
  if (!(mr == ADJ_M && mc == ADJ_M) || 2 * br - 1 > mr || 2 * bc - 1 > mc || nsplit > nk * nch || batch > 65535 || nz > 65535)
    return fail(OI_ERANGE, "%s: coarse %dx%d / band %dx%d / split %d unsupported (coarse grid must be 128x128, band at "
                "most 64x64)", what, mr, mc, br, bc, nsplit);
  AdjointArgs a{(const float2*)band, (long long)nch * br * bc, nch, br, bc, m0r, m0c, (const float2*)pupil, weight, gcoarse, nz,
                nk, nsplit, (const float2*)wr, (const float2*)wc, (float2*)wout, field_dot};
  return launch_adjoint(a, batch, s, what);
}

// half[b][qr + R][qc] = scale (qc ? 2 : 1) (W(q) + conj W(-q)) / 2, |qr| <= R, 0 <= qc <= C, from the adjoint's shares
// W = sum over nparts arrays of [batch][nz] bands (zero off the band): the Hermitian half-spectrum of Re sum W exp.
// 32 outputs per block, the shares dealt to 8 threads an output (an Abbe model has up to 144 of them): with one thread an
// output 72 shares took 50 us, now 5.5 us.
constexpr int HERM_Q = 8;
__global__ void __launch_bounds__(32 * HERM_Q) hermitian_half_kernel(const float2* __restrict__ w, int nparts, long long pstride,
                                                                     int nz, int br, int bc, int m0r, int m0c, int R, int C,
                                                                     float scale, float2* __restrict__ half) {
  __shared__ float4 sh[HERM_Q][32];
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5, wd = C + 1, e = blockIdx.x * 32 + lane;
  const bool in = e < (2 * R + 1) * wd;
  const int qr = e / wd - R, qc = e % wd;
  const long long b = blockIdx.y;
  auto place = [&](int r, int c) -> long long {   // offset in a share's band of plane 0, or -1 off the band
    const int ir = r - m0r, ic = c - m0c;
    return in && ir >= 0 && ir < br && ic >= 0 && ic < bc ? (b * nz * br + ir) * bc + ic : -1;
  };
  const long long p = place(qr, qc), m = place(-qr, -qc), plane = (long long)br * bc;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int i = q; i < nparts * nz; i += HERM_Q) {
    const float2* o = w + (i / nz) * pstride + (i % nz) * plane;
    const float2 u = p >= 0 ? __ldg(o + p) : make_float2(0.f, 0.f), v = m >= 0 ? __ldg(o + m) : make_float2(0.f, 0.f);
    s.x += u.x;
    s.y += u.y;
    s.z += v.x;
    s.w += v.y;
  }
  sh[q][lane] = s;
  __syncthreads();
  if (q != 0 || !in) return;
#pragma unroll
  for (int i = 1; i < HERM_Q; ++i) {
    const float4 t = sh[i][lane];
    s.x += t.x;
    s.y += t.y;
    s.z += t.z;
    s.w += t.w;
  }
  const float f = (qc ? 1.f : 0.5f) * scale;
  half[(b * (2 * R + 1) + qr + R) * wd + qc] = make_float2(f * (s.x + s.z), f * (s.y - s.w));
}

}  // namespace oi

extern "C" int oi_coherent_adjoint(const void* band, int batch, int nch, int m0r, int br, int m0c, int bc,
                                   const void* pupil, const float* weight, int nz, int nk, const float* gcoarse,
                                   int mr, int mc, const void* wr, const void* wc, int nsplit, void* wout,
                                   float* field_dot, void* stream) {
  using namespace oi;
  if (!wout) return fail(OI_EINVAL, "oi_coherent_adjoint: bad arguments");
  return adjoint(band, batch, nch, m0r, br, m0c, bc, pupil, weight, nz, nk, gcoarse, mr, mc, wr, wc, nsplit, wout, field_dot,
                 (cudaStream_t)stream, "oi_coherent_adjoint");
}

extern "C" int oi_coherent_field_dots(const void* band, int batch, int nch, int m0r, int br, int m0c, int bc,
                                      const void* pupil, const float* weight, int nz, int nk, const float* gcoarse, int mr, int mc,
                                      const void* wr, const void* wc, int nsplit, float* field_dot, void* stream) {
  using namespace oi;
  if (!field_dot) return fail(OI_EINVAL, "oi_coherent_field_dots: bad arguments");
  return adjoint(band, batch, nch, m0r, br, m0c, bc, pupil, weight, nz, nk, gcoarse, mr, mc, wr, wc, nsplit, nullptr, field_dot,
                 (cudaStream_t)stream, "oi_coherent_field_dots");
}

extern "C" int oi_hermitian_half(const void* w, int nparts, int batch, int nz, int m0r, int br, int m0c, int bc, float scale,
                                 void* half, void* stream) {
  using namespace oi;
  if (!w || !half || nparts <= 0 || batch <= 0 || nz <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_hermitian_half: bad arguments");
  const int R = max(abs(m0r), abs(m0r + br - 1)), C = max(abs(m0c), abs(m0c + bc - 1));
  const long long band = (long long)br * bc, size = (long long)(2 * R + 1) * (C + 1);
  constexpr int MOST = 65535;   // images per launch: the grid's second dimension
  for (int b = 0; b < batch; b += min(MOST, batch - b)) {
    dim3 grid((unsigned)ceil_div(size, 32), (unsigned)min(MOST, batch - b));
    hermitian_half_kernel<<<grid, 32 * HERM_Q, 0, (cudaStream_t)stream>>>((const float2*)w + (long long)b * nz * band, nparts,
                                                                          (long long)batch * nz * band, nz, br, bc, m0r, m0c, R, C,
                                                                          scale, (float2*)half + b * size);
    oi::note_launch();
    if (int rc = check_launch("oi_hermitian_half")) return rc;
  }
  return OI_OK;
}
