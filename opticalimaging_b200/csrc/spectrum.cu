// Band-limited forward spectrum of the mask near field (the numerical core of Scatter.CalculateSpectrum,
// Scatter.py:10-35, restricted to the frequencies the pupil can pass).
//
// Two separable passes, FP32 on the CUDA cores:
//   pass x: t[b][c][y][ic]    = sum_x h[b][y][x][c] * wx[x][ic]              (rows x Nx  by  Nx x Bc)
//   pass y: band[b][c][ir][ic] = scale * sum_y wy[y][ir] * t[b][c][y][ic]    (Br x Ny  by  Ny x Bc)
// The x pass streams the whole mask once; it is the HBM-facing part.  The y pass reads the small t.
#include "dft_gemm.cuh"
#include <cstdint>
#include <mutex>

namespace oi {

// Both passes are tile products (dft_gemm.cuh).  Four 1000 x 750 masks, 59 x 59 band: x pass 156 -> 35 us, y pass 122 ->
// 14 us (as tiles without a shared K loop they had 63 and 8 blocks for 148 SMs).
template <int KIND> struct FieldT { using A = float; };
template <> struct FieldT<OI_FIELD_COMPLEX_C64> { using A = float2; };

// pass x.  Row R of t is (b, c, y) with R = (b*nch + c)*ny + y; r0: the first row of a slice (below 2^30 rows each).
template <int KIND> struct BandX {
  using A = typename FieldT<KIND>::A;
  static constexpr bool A_K = true;
  const void* field;
  long long r0;
  int ny, nx, nch, bc;
  const float2* wx;
  float2* t;
  __device__ __forceinline__ A a(int, int R, int x) const {
    if constexpr (KIND == OI_FIELD_REAL_F32) return __ldg((const float*)field + (r0 + R) * nx + x);
    if constexpr (KIND == OI_FIELD_U8) return (float)__ldg((const uint8_t*)field + (r0 + R) * nx + x);
    if constexpr (KIND == OI_FIELD_COMPLEX_C64) {
      const int bcidx = r0 ? (int)((r0 + R) / ny) : R / ny, y = (int)(r0 + R - (long long)bcidx * ny);
      const int b = bcidx / nch, c = bcidx - b * nch;
      return __ldg((const float2*)field + (((long long)b * ny + y) * nx + x) * nch + c);
    }
  }
  __device__ __forceinline__ float2 b(int, int x, int ic) const { return __ldg(wx + (long long)x * bc + ic); }
  __device__ __forceinline__ void put(int, int R, int ic, float2 v) const { t[(r0 + R) * bc + ic] = v; }
};

// A real field's row transform on a band that holds frequency 0: t[-k] = conj t[k], so the x pass forms k = 0 .. kc-1 only
// (kc - 1 the largest |frequency|; a k beyond the band's own end is the conjugate of the column at -k) and the y pass reads
// the others mirrored.  Half the products of the x pass: four 1000 x 750 masks, 35 -> 19.7 us.
template <int KIND> struct BandXHalf {
  using A = float;
  static constexpr bool A_K = true;
  const void* field;
  long long r0;
  int nx, bc, m0c, kc;
  const float2* wx;
  float2* t;
  __device__ __forceinline__ float a(int, int R, int x) const {
    return KIND == OI_FIELD_U8 ? (float)__ldg((const uint8_t*)field + (r0 + R) * nx + x)
                               : __ldg((const float*)field + (r0 + R) * nx + x);
  }
  __device__ __forceinline__ float2 b(int, int x, int k) const {
    const bool own = k < m0c + bc;
    const float2 w = __ldg(wx + (long long)x * bc + (own ? k : -k) - m0c);
    return own ? w : make_float2(w.x, -w.y);
  }
  __device__ __forceinline__ void put(int, int R, int k, float2 v) const { t[(r0 + R) * kc + k] = v; }
};
struct BandYHalf {
  using A = float2;
  static constexpr bool A_K = false;
  const float2* t;
  int ny, br, bc, m0c, kc;
  const float2* wy;
  float scale;
  float2* band;
  __device__ __forceinline__ float2 a(int, int ir, int y) const { return __ldg(wy + (long long)y * br + ir); }
  __device__ __forceinline__ float2 b(int mat, int y, int ic) const {
    const int m = m0c + ic;
    const float2 v = t[((long long)mat * ny + y) * kc + (m < 0 ? -m : m)];
    return m < 0 ? make_float2(v.x, -v.y) : v;
  }
  __device__ __forceinline__ void put(int mat, int ir, int ic, float2 v) const {
    band[((long long)mat * br + ir) * bc + ic] = make_float2(v.x * scale, v.y * scale);
  }
};

// pass y: per image-channel matrix, band = scale * wy^T t.
struct BandY {
  using A = float2;
  static constexpr bool A_K = false;
  const float2* t;
  int ny, br, bc;
  const float2* wy;
  float scale;
  float2* band;
  __device__ __forceinline__ A a(int, int ir, int y) const { return __ldg(wy + (long long)y * br + ir); }
  __device__ __forceinline__ float2 b(int mat, int y, int ic) const { return t[((long long)mat * ny + y) * bc + ic]; }
  __device__ __forceinline__ void put(int mat, int ir, int ic, float2 v) const {
    band[((long long)mat * br + ir) * bc + ic] = make_float2(v.x * scale, v.y * scale);
  }
};

template <int KIND>
static int band_x(const void* field, int batch, int ny, int nx, int nch, int bc, const float2* wx, float2* t, cudaStream_t s) {
  const long long rows = (long long)batch * nch * ny, slice = 1LL << 30;
  for (long long r0 = 0; r0 < rows; r0 += slice) {
    const int n = (int)(rows - r0 < slice ? rows - r0 : slice);
    const int rc = dg::gemm<64, 64, 4, 4>(BandX<KIND>{field, r0, ny, nx, nch, bc, wx, t}, 1, n, bc, nx, s, "oi_band_spectrum/x");
    if (rc) return rc;
  }
  return OI_OK;
}

template <int KIND>
static int band_half(const void* field, int batch, int ny, int nx, int m0c, int br, int bc, const float2* wx, const float2* wy,
                     float scale, float2* t, float2* band, cudaStream_t s) {
  const int kc = max(-m0c, m0c + bc - 1) + 1;
  const long long rows = (long long)batch * ny, slice = 1LL << 30;
  for (long long r0 = 0; r0 < rows; r0 += slice) {
    const int n = (int)(rows - r0 < slice ? rows - r0 : slice);
    const BandXHalf<KIND> op{field, r0, nx, bc, m0c, kc, wx, t};
    const int rc = kc <= 32 ? dg::gemm<128, 32, 8, 2>(op, 1, n, kc, nx, s, "oi_band_spectrum_real/x")
                            : dg::gemm<64, 64, 4, 4>(op, 1, n, kc, nx, s, "oi_band_spectrum_real/x");
    if (rc) return rc;
  }
  return dg::gemm<32, 32, 2, 2>(BandYHalf{t, ny, br, bc, m0c, kc, wy, scale, band}, batch, br, bc, ny, s,
                                "oi_band_spectrum_real/y");
}

}  // namespace oi

extern "C" int oi_band_spectrum_real(const void* field, int kind, int batch, int ny, int nx, int br, int m0c, int bc,
                                     const void* wx, const void* wy, float scale, void* scratch, void* band,
                                     void* stream) {
  using namespace oi;
  if (!field || !wx || !wy || !scratch || !band || batch <= 0 || ny <= 0 || nx <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_band_spectrum_real: bad arguments (batch=%d ny=%d nx=%d br=%d bc=%d)", batch, ny, nx, br, bc);
  if (kind != OI_FIELD_REAL_F32 && kind != OI_FIELD_U8)
    return fail(OI_EINVAL, "oi_band_spectrum_real: real float32 or uint8 masks only (kind=%d)", kind);
  if (batch > 65535) return fail(OI_ERANGE, "oi_band_spectrum_real: batch too large");
  if (m0c > 0 || m0c + bc <= 0) return fail(OI_ERANGE, "oi_band_spectrum_real: band %d+%d does not hold frequency 0", m0c, bc);
  cudaStream_t s = (cudaStream_t)stream;
  return kind == OI_FIELD_U8 ? band_half<OI_FIELD_U8>(field, batch, ny, nx, m0c, br, bc, (const float2*)wx, (const float2*)wy,
                                                      scale, (float2*)scratch, (float2*)band, s)
                             : band_half<OI_FIELD_REAL_F32>(field, batch, ny, nx, m0c, br, bc, (const float2*)wx,
                                                            (const float2*)wy, scale, (float2*)scratch, (float2*)band, s);
}

extern "C" int oi_band_spectrum(const void* field, int kind, int batch, int ny, int nx, int nch, int br, int bc,
                                const void* wx, const void* wy, float scale, void* scratch, void* band,
                                void* stream) {
  using namespace oi;
  if (!field || !wx || !wy || !scratch || !band || batch <= 0 || ny <= 0 || nx <= 0 || nch <= 0 || br <= 0 ||
      bc <= 0)
    return fail(OI_EINVAL, "oi_band_spectrum: bad arguments (batch=%d ny=%d nx=%d nch=%d br=%d bc=%d)", batch, ny,
                nx, nch, br, bc);
  if (kind != OI_FIELD_COMPLEX_C64 && nch != 1)
    return fail(OI_EINVAL, "oi_band_spectrum: real and u8 fields have one channel (nch=%d)", nch);
  if ((long long)batch * nch > 65535) return fail(OI_ERANGE, "oi_band_spectrum: batch too large");
  cudaStream_t s = (cudaStream_t)stream;
  const float2* wxf = (const float2*)wx;
  float2* t = (float2*)scratch;
  int rc;
  switch (kind) {
    case OI_FIELD_REAL_F32: rc = band_x<OI_FIELD_REAL_F32>(field, batch, ny, nx, nch, bc, wxf, t, s); break;
    case OI_FIELD_U8: rc = band_x<OI_FIELD_U8>(field, batch, ny, nx, nch, bc, wxf, t, s); break;
    case OI_FIELD_COMPLEX_C64: rc = band_x<OI_FIELD_COMPLEX_C64>(field, batch, ny, nx, nch, bc, wxf, t, s); break;
    default: return fail(OI_EINVAL, "oi_band_spectrum: unknown field kind %d", kind);
  }
  if (rc) return rc;
  return dg::gemm<32, 32, 2, 2>(BandY{t, ny, br, bc, (const float2*)wy, scale, (float2*)band}, batch * nch, br, bc, ny, s,
                                "oi_band_spectrum/y");
}

// ---------------------------------------------------------------------------------------------------
// Band spectrum for callers that cannot allocate device memory.
//
// oi_band_spectrum needs a caller-provided scratch buffer for the intermediate row transform.  Some callers
// cannot provide one: code that only ever receives device pointers from a host application that owns every
// allocation (and forbids its plug-ins from calling cudaMalloc), or code running where an allocation would
// stall or fail (inside a fixed memory budget that is already fully handed out).  This entry point serves
// them: its scratch is a fixed-size array compiled into the library, one copy on each GPU that loads it,
// kept until the process exits.  Only the inputs and the output come from the caller.
namespace oi {

constexpr long long kStaticScratchF2 = OI_NOALLOC_SCRATCH_COMPLEX;  // complex values: 16 MiB per device
static __device__ __align__(256) float2 g_static_scratch[kStaticScratchF2];

// Device address of g_static_scratch on each device.  In host code the symbol itself is only a host-side handle,
// so the address comes from cudaGetSymbolAddress.  It is looked up again on every call whose stream is not
// capturing (a context torn down and created again -- cudaDeviceReset -- loads the module anew, possibly
// elsewhere, so an address kept from before would be stale); a call on a capturing stream makes no lookup and
// uses the address the last call on that device found.
static float2* g_static_scratch_ptr[64] = {nullptr};
static std::mutex g_static_scratch_mu;

static int static_scratch(cudaStream_t stream, float2** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(OI_ECUDA, "oi_band_spectrum_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return fail(OI_ERANGE, "oi_band_spectrum_noalloc: device %d out of range", dev);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  e = cudaStreamIsCapturing(stream, &cap);
  if (e != cudaSuccess)
    return fail(OI_ECUDA, "oi_band_spectrum_noalloc: cudaStreamIsCapturing: %s", cudaGetErrorString(e));
  std::lock_guard<std::mutex> lock(g_static_scratch_mu);
  if (cap == cudaStreamCaptureStatusNone) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess || !p)
      return fail(OI_ECUDA, "oi_band_spectrum_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    g_static_scratch_ptr[dev] = (float2*)p;
  } else if (!g_static_scratch_ptr[dev]) {
    return fail(OI_EINVAL, "oi_band_spectrum_noalloc: the first call on device %d is being captured into a "
                           "graph; make one call on that device before any stream capture", dev);
  }
  *out = g_static_scratch_ptr[dev];
  return OI_OK;
}

}  // namespace oi

extern "C" int oi_band_spectrum_noalloc(const void* field, int kind, int batch, int ny, int nx, int nch, int br,
                                        int bc, const void* wx, const void* wy, float scale, void* band,
                                        void* stream) {
  using namespace oi;
  if (!field || !wx || !wy || !band || batch <= 0 || ny <= 0 || nx <= 0 || nch <= 0 || br <= 0 || bc <= 0)
    return fail(OI_EINVAL, "oi_band_spectrum_noalloc: bad arguments (batch=%d ny=%d nx=%d nch=%d br=%d bc=%d)",
                batch, ny, nx, nch, br, bc);
  const long long need = (long long)batch * nch * ny * bc;
  if (need > kStaticScratchF2)
    return fail(OI_ERANGE,
                "oi_band_spectrum_noalloc: needs %lld complex scratch values (batch*nch*ny*bc) but the built-in "
                "scratch holds %lld; use oi_band_spectrum with a caller buffer or split the batch",
                need, kStaticScratchF2);
  float2* scratch = nullptr;
  int rc = static_scratch((cudaStream_t)stream, &scratch);
  if (rc) return rc;
  // every scratch entry the y pass reads is written by the x pass first: nothing needs clearing
  return oi_band_spectrum(field, kind, batch, ny, nx, nch, br, bc, wx, wy, scale, scratch, band, stream);
}
