// FP64 TCC assembly: TCC = sum_e h_e h_e^H with h[e][p][j] the weighted shifted pupils (GetTCCMatrix,
// CalculateTCCMatrix.py:58-75, with the diagonal source-weight matrix folded into h as sqrt(w)).
// The TCC is Hermitian: only lower-triangle 64x64 tiles are computed; each off-diagonal tile is written
// twice, once as is and once conjugate-transposed.
//
// Bound: FP64 issue.  A pupil sample outside the shifted disc is zero, and 64 consecutive samples against 16
// consecutive source points are mostly all inside or all outside: with the marks of the non-zero 16 x 16 blocks of h
// (one pass over it) a tile skips the chunks in which either side is zero and the other finite, which add nothing.
// 3481 x 3481 over 3 x 520 points: 6.3 -> 0.79 ms with marks.  Few tiles (961 x 961: 136 for 148 SMs, those of the low
// frequencies the longest) share their chunks among the blocks of a cluster, whose tiles meet in shared memory: 320 -> 124
// us.
#include "zgemm64.cuh"
#include <cooperative_groups.h>

namespace oi {

struct TccArgs {
  const double2* h;
  int ne, fg, nsrc;
  const unsigned char* flags;   // marks of h, or null: every chunk counts
  int fr, fc;
  double2* tcc;
};

__global__ void __launch_bounds__(256, 2) tcc_assemble_kernel(TccArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  // lower-triangle tile index -> (tp, tq), tp >= tq
  const long long t = blockIdx.x / S;
  int tp = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) / 2.0);
  while ((long long)tp * (tp + 1) / 2 > t) --tp;
  while ((long long)(tp + 1) * (tp + 2) / 2 <= t) ++tp;
  const int tq = (int)(t - (long long)tp * (tp + 1) / 2);
  const int p0 = tp * zg::T, q0 = tq * zg::T;
  const int per = (a.nsrc + zg::KC - 1) / zg::KC;
  const long long plane = (long long)a.fg * a.nsrc;
  zg::TileAcc acc;
  acc.clear();
  auto active = [&](int c) {
    if (!a.flags) return true;
    const int e = c / per, kc = c - e * per;
    const unsigned char* f = a.flags + (long long)e * a.fr * a.fc + kc;
    unsigned x = 0, y = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      x |= f[(4 * tp + u) * a.fc];
      y |= f[(4 * tq + u) * a.fc];
    }
    return ((x | y) & 2u) || ((x & y) & 1u);   // a value that is not finite makes 0 times it count
  };
  auto load = [&](int c, double2* As, double2* Bs) {
    const int e = c / per, k0 = (c - e * per) * zg::KC;
    zg::load_rows(As, a.h + e * plane, a.nsrc, p0, a.fg, k0, a.nsrc);
    zg::load_rows(Bs, a.h + e * plane, a.nsrc, q0, a.fg, k0, a.nsrc);
  };
  zg::tile_loop<zg::CONJ_B>(acc, smem, rank, S, per * a.ne, active, load);
  auto put = [&](int i, int j, double2 v) {
    const int p = p0 + i, q = q0 + j;
    if (p >= a.fg || q >= a.fg) return;
    a.tcc[(long long)p * a.fg + q] = v;
    if (tp != tq) a.tcc[(long long)q * a.fg + p] = make_double2(v.x, -v.y);
  };
  if (S == 1) {
    acc.each([&](int i, int j, double2 v) { put(zg::tile_row() + i, zg::tile_col() + j, v); });
    return;
  }
  double2* tile = (double2*)smem;   // [64][64], over the ring
  __syncthreads();
  acc.each([&](int i, int j, double2 v) { tile[(zg::tile_row() + i) * zg::T + zg::tile_col() + j] = v; });
  cluster.sync();
  for (int e = rank * 256 + threadIdx.x; e < zg::T * zg::T; e += S * 256) {
    double2 s = make_double2(0.0, 0.0);
    for (int r = 0; r < S; ++r) {   // in rank order
      const double2 v = *cluster.map_shared_rank(tile + e, r);
      s.x += v.x;
      s.y += v.y;
    }
    put(e / zg::T, e % zg::T, s);
  }
  cluster.sync();   // the others may still be reading this block's tile
}

static long long tcc_marks(int ne, int fg, int nsrc) { return (long long)ne * zg::flag_dim(fg) * zg::flag_dim(nsrc); }

static int tcc_assemble(const void* h, int ne, int fg, int nsrc, void* tcc, unsigned char* marks, cudaStream_t s,
                        const char* what) {
  if (!h || !tcc || (ne != 1 && ne != 3) || fg <= 0 || nsrc <= 0)
    return fail(OI_EINVAL, "%s: bad arguments (ne=%d fg=%d nsrc=%d)", what, ne, fg, nsrc);
  const long long nt = ceil_div(fg, zg::T), tiles = nt * (nt + 1) / 2;
  if (tiles > 0x7fffffffLL) return fail(OI_ERANGE, "%s: fg=%d too large", what, fg);
  if (int rc = ensure_smem((const void*)tcc_assemble_kernel, zg::SMEM, what)) return rc;
  if (marks)
    if (int rc = zg::mark_blocks((const double2*)h, ne, fg, nsrc, marks, s)) return rc;
  TccArgs a{(const double2*)h, ne, fg, nsrc, marks, zg::flag_dim(fg), zg::flag_dim(nsrc), (double2*)tcc};
  // blocks per tile: while that leaves fewer than two blocks per SM (148), at least 8 chunks each
  const int chunks = ne * ceil_div(nsrc, zg::KC);
  int S = 1;
  while (S < 8 && tiles * S < 148 * 2 && chunks >= 16 * S) S *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * S));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = zg::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, tcc_assemble_kernel, a);
  note_launch();
  return check_launch(what);
}

}  // namespace oi

extern "C" int oi_tcc_assemble64(const void* h, int ne, int fg, int nsrc, void* tcc, void* stream) {
  return oi::tcc_assemble(h, ne, fg, nsrc, tcc, nullptr, (cudaStream_t)stream, "oi_tcc_assemble64");
}

extern "C" int oi_tcc_assemble64_marked_workspace(int ne, int fg, int nsrc, long long* bytes) {
  using namespace oi;
  if (!bytes || ne <= 0 || fg <= 0 || nsrc <= 0) return fail(OI_EINVAL, "oi_tcc_assemble64_marked_workspace: bad arguments");
  *bytes = tcc_marks(ne, fg, nsrc);
  return OI_OK;
}

extern "C" int oi_tcc_assemble64_marked(const void* h, int ne, int fg, int nsrc, void* tcc, void* work,
                                        long long work_bytes, void* stream) {
  using namespace oi;
  if (!work || ne <= 0 || fg <= 0 || nsrc <= 0) return fail(OI_EINVAL, "oi_tcc_assemble64_marked: bad arguments");
  if (work_bytes < tcc_marks(ne, fg, nsrc))
    return fail(OI_ERANGE, "oi_tcc_assemble64_marked: %lld workspace bytes given, %lld needed", work_bytes,
                tcc_marks(ne, fg, nsrc));
  return tcc_assemble(h, ne, fg, nsrc, tcc, (unsigned char*)work, (cudaStream_t)stream, "oi_tcc_assemble64_marked");
}
