// FP64 top-K eigenpairs of a Hermitian positive semi-definite operator, for the SOCS decomposition
// (DecomposeTCC_SOCS.py:7-9, where the reference takes a full torch.svd of its complex64 TCC and keeps the
// leading K singular pairs).  Subspace iteration on a block of p vectors with Rayleigh-Ritz, on the GPU, in double
// precision:
//
//   X = random n x p;   EIG_START times:  X R = T X          (Cholesky QR twice: X^H X = I to rounding)
//   X R = f(T) X, f the Chebyshev polynomial that is small on [0, lambda_p], of the degree that should reach tol
//   repeat:   Z = T X, H = X^H Z (p x p), H = Q diag(w) Q^H (cyclic Jacobi), X = X Q, Z = Z Q, residuals
//             ||Z_i - w_i X_i|| of the leading k; stop when their maximum is below tol * w_0, else another filter
//   result:   the Ritz pairs (w_i, X_i), i < k, eigenvalues descending and clamped at zero.
//
// Plain subspace iteration gains lambda_{p+1} / lambda_k per product with T; the filter on the unwanted interval
// gains rho = x + sqrt(x^2 - 1), x = 2 lambda_k / lambda_p - 1, per product (configuration 3, k = 24, p = 64: 4.8
// against 18).  Both ends of the interval come from the last projection, or before the first one from the diagonal of
// R, which after EIG_START iterations holds the leading eigenvalues to some per cent: most operators then need one
// projection (configuration 3: 13 products with T and 6 orthonormalisations; 21 products, 17 orthonormalisations and
// 4 projections without the filter).  A filter is cut into pieces whose amplification of lambda_0 over lambda_k stays
// below EIG_AMP, with an orthonormalisation after each: the columns, ordered by eigenvalue, then stay independent to
// working precision.  Where the interval does not separate (lambda_p too near lambda_k) or a filter did not help,
// plain iterations run instead.
//
// T is a dense n x n matrix or the factored form T = sum_e h_e h_e^H (h [ne][n][s], the scaled pupil matrix of
// CalculateTCCMatrix.py:33-51), applied without forming T.  Both hold many zero blocks (pupil samples outside the
// shifted discs): a pass over the operand marks its non-zero 16 x 16 blocks once, and the products skip the rest.
#include "zgemm64.cuh"
#include <algorithm>
#include <cmath>
#include <vector>

namespace oi {

namespace zg {

__global__ void __launch_bounds__(256) mark_blocks_kernel(const double2* __restrict__ M, int rows, int cols,
                                                          unsigned char* __restrict__ flags, int fc,
                                                          const int* __restrict__ perm) {
  const int col = blockIdx.x * 256 + threadIdx.x, r16 = blockIdx.y;
  const double2* m = M + (long long)blockIdx.z * rows * cols;
  bool nz = false, bad = false;
  if (col < cols) {
    const int pc = perm ? __ldg(perm + col) : col;
#pragma unroll 4
    for (int i = 0; i < KC; ++i) {
      const int r = r16 * KC + i;
      if (r >= rows) break;
      const double2 v = __ldg(m + (long long)(perm ? __ldg(perm + r) : r) * cols + pc);
      nz |= v.x != 0.0 || v.y != 0.0;
      bad |= !isfinite(v.x) || !isfinite(v.y);
    }
  }
  const unsigned n = __ballot_sync(0xffffffffu, nz), b = __ballot_sync(0xffffffffu, bad);
  if ((threadIdx.x & 15) == 0) {
    const int c16 = col >> 4, sh = threadIdx.x & 16;
    if (c16 < fc)
      flags[((long long)blockIdx.z * gridDim.y + r16) * fc + c16] =
          (((n >> sh) & 0xffffu) ? 1 : 0) | (((b >> sh) & 0xffffu) ? 2 : 0);
  }
}

int mark_blocks(const double2* M, int batch, int rows, int cols, unsigned char* flags, cudaStream_t s, const int* perm) {
  dim3 grid((unsigned)ceil_div(cols, 256), (unsigned)flag_dim(rows), (unsigned)batch);
  if (grid.y > 65535 || grid.z > 65535) return fail(OI_ERANGE, "mark_blocks: %d x %d x %d too large", batch, rows, cols);
  mark_blocks_kernel<<<grid, 256, 0, s>>>(M, rows, cols, flags, flag_dim(cols), perm);
  note_launch();
  return check_launch("mark_blocks");
}

}  // namespace zg

namespace eg {

constexpr int PMAX = 64;                   // block size limit (one column tile, and the one-CTA steps)
constexpr int EIG_START = 3;               // plain iterations before the first filter
constexpr int EIG_DEGREE = 12;             // products with T between projections, at most
constexpr double EIG_AMP = 1e8;            // a filter piece's amplification of lambda_0 over lambda_k

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 conjd(double2 a) { return make_double2(a.x, -a.y); }

// Tile of block i of n: from the middle outwards.  The middle rows of a TCC (low frequencies) have the most non-zero
// blocks; started first, they do not end last.
__device__ __forceinline__ int heavy_first(int i, int n) {
  const int m = n / 2;
  return i & 1 ? m - 1 - i / 2 : m + i / 2;
}

// parts[(bat * splits + z)][m][p] = the share z of op(A_bat) B_bat: 64 rows per block (blockIdx.x), share blockIdx.y,
// batch blockIdx.z.  AH false: A = M [m][k], K over nseg segments of k (segment e at M + e * sm), B [nseg * k][p].
// AH true: A = conj(M_bat)^T, M_bat [k][m].  Share z takes the chunks z, z + splits, ... so that zero blocks spread
// over the shares.
struct GemmArgs {
  const double2* M;
  long long sm;                  // elements between segments / batches of M
  int m, k, nseg, p;
  const double2* B;
  double2* parts;
  const unsigned char* flags;    // of M (zg::mark_blocks)
  int fr, fc;
  const int* perm;               // the order of a dense T's rows and columns (null: its own)
};
template <bool AH>
__global__ void __launch_bounds__(256, 2) gemm_kernel(GemmArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  pdl_trigger();
  pdl_wait();
  const int mt = heavy_first(blockIdx.x, gridDim.x), m0 = mt * zg::T, splits = gridDim.y;
  const int per = (a.k + zg::KC - 1) / zg::KC;
  const double2* M = a.M + (AH ? blockIdx.z * a.sm : 0);
  const unsigned char* fl = a.flags + (AH ? (long long)blockIdx.z * a.fr * a.fc : 0);
  zg::TileAcc acc;
  acc.clear();
  auto active = [&](int c) {
    const int e = c / per, kc = c - e * per;
    unsigned f = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      f |= AH ? fl[(long long)kc * a.fc + 4 * mt + u] : fl[((long long)e * a.fr + 4 * mt + u) * a.fc + kc];
    return (f & 1u) != 0;
  };
  auto load = [&](int c, double2* As, double2* Bs) {
    const int e = c / per, k0 = (c - e * per) * zg::KC;
    if (AH)
      zg::load_cols(As, M, a.m, m0, a.m, k0, a.k);
    else if (a.perm)
      zg::load_rows_perm(As, M, a.k, m0, a.m, k0, a.k, a.perm);
    else
      zg::load_rows(As, M + e * a.sm, a.k, m0, a.m, k0, a.k);
    zg::load_cols(Bs, a.B + (long long)e * a.k * a.p, a.p, 0, a.p, k0, a.k);
  };
  zg::tile_loop<AH ? zg::CONJ_A : zg::NONE>(acc, smem, blockIdx.y, splits, per * a.nseg, active, load);
  double2* out = a.parts + ((long long)blockIdx.z * splits + blockIdx.y) * a.m * a.p;
  acc.each([&](int i, int j, double2 v) {
    const int r = m0 + zg::tile_row() + i, c = zg::tile_col() + j;
    if (r < a.m && c < a.p) out[(long long)r * a.p + c] = v;
  });
}

// The order of a dense T's indices: those with a zero on the diagonal (of a Hermitian, positive semi-definite T the
// ones whose whole row and column are zero: frequencies outside every shifted pupil) go to the two ends, so that the
// others fill whole tiles in the middle.  Any order gives the same eigenpairs, only the number of non-zero blocks
// differs: 0.62 -> 0.41 of the blocks of a 3481 x 3481 TCC, whose whole set-up takes 5.97 ms instead of 6.58.  One block;
// perm[place] = index.
__global__ void __launch_bounds__(1024) order_kernel(int n, const double2* __restrict__ T, int* __restrict__ perm) {
  __shared__ int wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, per = (n + 1023) / 1024, i0 = min(n, tid * per), i1 = min(n, i0 + per);
  auto on = [&](int i) {
    const double2 d = __ldg(T + (long long)i * n + i);
    return !(d.x == 0.0 && d.y == 0.0);
  };
  int c = 0;
  for (int i = i0; i < i1; ++i) c += on(i);
  int incl = c;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, s);
    if (lane >= s) incl += v;
  }
  if (lane == 31) wsum[tid >> 5] = incl;
  __syncthreads();
  int before = incl - c, total = 0;
  for (int w = 0; w < 32; ++w) {
    if (w < tid >> 5) before += wsum[w];
    total += wsum[w];
  }
  const int off = (n - total) / 2 / zg::T * zg::T;
  int zeros = i0 - before;   // zero indices before i0
  for (int i = i0; i < i1; ++i) {
    if (on(i)) {
      perm[off + before++] = i;
    } else {
      perm[zeros < off ? zeros : total + zeros] = i;
      ++zeros;
    }
  }
}

// Row-block kernels: each block takes groups of RB rows (g, g + gridDim.x, ...) of n x p arrays, held in shared memory
// with rows of PL values.  gram: the block's share of L^H Y (Hermitian: L = Y, or Y = T L), accumulated over its
// groups; its 16 x 16 blocks on and above the diagonal are stored.
constexpr int PL = zg::LD;
template <int RB>
__device__ __forceinline__ void gram_rows(zg::TileAcc& acc, const double2* L, const double2* Y) {
  zg::warp_mma<zg::CONJ_A, RB>(acc, L + zg::tile_row(), 1, PL, Y + zg::tile_col(), PL);
}
__device__ __forceinline__ void store_gram(const zg::TileAcc& acc, double2* gparts) {
  acc.each([&](int i, int j, double2 v) {
    const int r = zg::tile_row() + i, c = zg::tile_col() + j;
    if ((c >> 4) >= (r >> 4)) gparts[(long long)blockIdx.x * PMAX * PMAX + r * PMAX + c] = v;
  });
}

// out = alpha sum_z parts[z] + beta b1 + gamma b0 (rows of n x p; batch blockIdx.y of n rows), and, with gparts, the
// shares of left^H out (left null: out^H out).  out may be b0.
struct FoldArgs {
  const double2* parts;
  int nparts, n, p;
  double alpha, beta, gamma;
  const double2 *b1, *b0, *left;
  double2 *out, *gparts;
};
template <int RB>
__global__ void __launch_bounds__(256) fold_kernel(FoldArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* ys = (double2*)smem;                // [RB][PL]
  double2* ls = a.left ? ys + RB * PL : ys;    // left's rows, when given
  const int tid = threadIdx.x;
  pdl_trigger();
  pdl_wait();
  const long long np = (long long)a.n * a.p, boff = blockIdx.y * np;
  zg::TileAcc acc;
  acc.clear();
  for (int g = blockIdx.x; g * RB < a.n; g += gridDim.x) {
    double2 v[RB / 4];
#pragma unroll
    for (int i = 0; i < RB / 4; ++i) v[i] = make_double2(0, 0);
    const int c = tid & 63;
    auto at = [&](int i) { return (long long)(g * RB + (tid >> 6) + 4 * i) * a.p + c; };
    auto in = [&](int i) { return c < a.p && g * RB + (tid >> 6) + 4 * i < a.n; };
    for (int z = 0; z < a.nparts; ++z) {
      const double2* p = a.parts + boff * a.nparts + z * np;
#pragma unroll
      for (int i = 0; i < RB / 4; ++i)
        if (in(i)) v[i] = cadd(v[i], p[at(i)]);
    }
#pragma unroll
    for (int i = 0; i < RB / 4; ++i) {
      double2 y = make_double2(a.alpha * v[i].x, a.alpha * v[i].y), l = make_double2(0, 0);
      if (in(i)) {
        const long long e = at(i);
        if (a.b1) {
          const double2 b = a.b1[e];
          y.x = fma(a.beta, b.x, y.x);
          y.y = fma(a.beta, b.y, y.y);
        }
        if (a.b0) {
          const double2 b = a.b0[e];
          y.x = fma(a.gamma, b.x, y.x);
          y.y = fma(a.gamma, b.y, y.y);
        }
        a.out[boff + e] = y;
        if (a.left) l = a.left[e];
      }
      ys[((tid >> 6) + 4 * i) * PL + c] = y;
      if (a.left) ls[((tid >> 6) + 4 * i) * PL + c] = l;
    }
    if (a.gparts) {
      __syncthreads();
      gram_rows<RB>(acc, ls, ys);
      __syncthreads();
    }
  }
  if (a.gparts) store_gram(acc, a.gparts);
}

// G[r][c] = sum_b gparts[b][r][c] (p x p of the 64 x 64 shares), in a fixed order, for the stored 16 x 16 blocks, and
// their mirror images.
__global__ void __launch_bounds__(256) sum_gram_kernel(const double2* gparts, int nparts, int p, double2* G) {
  __shared__ double2 sh[4][64];
  pdl_trigger();
  pdl_wait();
  const int c = threadIdx.x & 63, q = threadIdx.x >> 6, r = blockIdx.x;
  if ((c >> 4) < (r >> 4)) nparts = 0;
  double2 s = make_double2(0, 0);
#pragma unroll 8
  for (int b = q; b < nparts; b += 4) s = cadd(s, gparts[(long long)b * PMAX * PMAX + r * PMAX + c]);
  sh[q][c] = s;
  __syncthreads();
  if (q != 0 || c >= p || (c >> 4) < (r >> 4)) return;
  s = cadd(cadd(sh[0][c], sh[1][c]), cadd(sh[2][c], sh[3][c]));
  G[r * p + c] = s;
  if ((c >> 4) > (r >> 4)) G[c * p + r] = conjd(s);
}

// One CTA: from the Gram matrix G of a block X, Rinv such that X Rinv has orthonormal columns:
// S scales the columns (first pass: to unit length, diag(G)^-1/2; second pass: not at all, so that columns which the
// first pass found dependent and left near zero stay there), shift is added to the diagonal against rank deficiency
// (a pivot below it is raised to it), S G S + shift = L D L^H with L unit lower triangular, Rinv = S L^-H D^-1/2.
// The elimination of the columns builds L^-1 in place: step j subtracts (A[a][j] / d_j) times row j from the rows
// a > j, where columns c > j still hold the trailing matrix, columns c < j hold L^-1 and column j becomes -A[a][j] / d_j.
// rdiag[c] = the diagonal of R = (X Rinv)^H X (the second pass multiplies the two passes' factors).
// Bound: the chain of 64 dependent steps.  Each thread keeps its 2 x 4 entries (ty + 32 i, tx + 16 j) in registers; a
// step is one barrier (row j and column j through a double-buffered line of shared memory, 1 / d_j by the entry's
// owner).  64 x 64: 39 us; with the matrix in shared memory, three barriers a step and a back substitution by one
// thread per column it was 277 us.
__global__ void __launch_bounds__(512) chol_inv_kernel(int p, const double2* G, double2* Rinv, double* rdiag,
                                                       double shift, bool first) {
  __shared__ double2 rowb[2][PMAX], colb[2][PMAX];
  __shared__ double invb[2], sc[PMAX], D[PMAX];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  pdl_trigger();
  pdl_wait();
  if (tid < PMAX) {
    const double g = tid < p ? G[tid * p + tid].x : 1.0;
    sc[tid] = !first ? 1.0 : g > 0 ? 1.0 / sqrt(g) : 0.0;
  }
  __syncthreads();
  double2 a[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = ty + 32 * i, c = tx + 16 * j;
      double2 v = make_double2(r == c ? 1.0 : 0.0, 0);
      if (r < p && c < p) v = G[r * p + c];
      const double s = sc[r] * sc[c];
      a[i][j] = r == c ? make_double2(v.x * s + shift, 0.0) : make_double2(v.x * s, v.y * s);
    }
#pragma unroll
  for (int jb = 0; jb < 4; ++jb) {
#pragma unroll 1
    for (int jj = 0; jj < 16; ++jj) {
      const int j = 16 * jb + jj, buf = j & 1;
      const bool col = tx == jj;   // this thread holds column j, as a[.][jb]
      if (ty == (j & 31)) {
#pragma unroll
        for (int k = 0; k < 4; ++k) rowb[buf][tx + 16 * k] = a[jb >> 1][k];
        if (col) {
          double d = a[jb >> 1][jb].x;
          if (!(d > shift)) d = shift;
          D[j] = d;
          invb[buf] = 1.0 / d;
        }
      }
      if (col) {
#pragma unroll
        for (int i = 0; i < 2; ++i) colb[buf][ty + 32 * i] = a[i][jb];
      }
      __syncthreads();
      const double inv = -invb[buf];
      double2 row[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) row[k] = rowb[buf][tx + 16 * k];
      if (col) row[jb] = make_double2(1.0, 0.0);   // column j becomes the multiplier itself
#pragma unroll
      for (int i = jb >> 1; i < 2; ++i) {   // rows of the block before are done
        const bool on = ty + 32 * i > j;
        double2 m = colb[buf][ty + 32 * i];
        m = on ? make_double2(m.x * inv, m.y * inv) : make_double2(0, 0);
        if (on && col) a[i][jb] = make_double2(0, 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (i > (jb >> 1) || on) cfma(a[i][k], m, row[k]);
        }
      }
    }
  }
  __syncthreads();   // D
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = ty + 32 * i, c = tx + 16 * j;   // L^-1[r][c] -> Rinv[c][r]
      if (r >= p || c >= p) continue;
      const double s = c <= r ? sc[c] / sqrt(D[r]) : 0.0;
      const double2 v = r == c ? make_double2(1, 0) : a[i][j];
      Rinv[c * p + r] = c <= r ? make_double2(v.x * s, -v.y * s) : make_double2(0, 0);
    }
  if (tid < p) {
    const double d = sqrt(D[tid]);
    rdiag[tid] = !first ? rdiag[tid] * d : sc[tid] > 0 ? d / sc[tid] : 0.0;
  }
}

// Loads a group of RB rows of an n x p array (zero beyond) into [RB][PL], and a p x p matrix into [64][PL].
template <int RB>
__device__ __forceinline__ void load_group(double2* s, const double2* src, int n, int p, int g) {
#pragma unroll
  for (int i = 0; i < RB / 4; ++i) {
    const int e = threadIdx.x + 256 * i, r = e >> 6, c = e & 63;
    s[r * PL + c] = g * RB + r < n && c < p ? src[(long long)(g * RB + r) * p + c] : make_double2(0, 0);
  }
}
__device__ __forceinline__ void load_square(double2* s, const double2* src, int p) {
#pragma unroll 4
  for (int e = threadIdx.x; e < PMAX * PMAX; e += 256) {
    const int r = e >> 6, c = e & 63;
    s[r * PL + c] = r < p && c < p ? src[r * p + c] : make_double2(0, 0);
  }
}
// xs q for a group: RB x 64 by 8 warps, 16 rows x 8 NI columns each (NI = RB / 16)
template <int RB> using GroupAcc = zg::Acc<2, RB / 16>;
template <int RB> __device__ __forceinline__ int group_row() { return RB == 32 ? 16 * (threadIdx.x >> 7) : 0; }
template <int RB> __device__ __forceinline__ int group_col() { return (RB / 2) * ((threadIdx.x >> 5) & (128 / RB - 1)); }
template <int RB>
__device__ __forceinline__ void times_square(GroupAcc<RB>& o, const double2* xs, const double2* q) {
  o.clear();
  zg::warp_mma<zg::NONE, PMAX>(o, xs + group_row<RB>() * PL, PL, 1, q + group_col<RB>(), PL);
}

// X <- X Rinv in place (groups of RB rows), and, with gparts, the shares of the result's Gram matrix.
template <int RB>
__global__ void __launch_bounds__(256) scale_kernel(int n, int p, double2* X, const double2* Rinv, double2* gparts) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* q = (double2*)smem;          // [64][PL]
  double2* xs = q + PMAX * PL;          // [RB][PL]
  pdl_trigger();
  pdl_wait();
  load_square(q, Rinv, p);
  zg::TileAcc acc;
  acc.clear();
  for (int g = blockIdx.x; g * RB < n; g += gridDim.x) {
    load_group<RB>(xs, X, n, p, g);
    __syncthreads();
    GroupAcc<RB> o;
    times_square<RB>(o, xs, q);
    __syncthreads();
    o.each([&](int i, int j, double2 v) {
      const int r = group_row<RB>() + i, c = group_col<RB>() + j;
      xs[r * PL + c] = v;
      if (g * RB + r < n && c < p) X[(long long)(g * RB + r) * p + c] = v;
    });
    __syncthreads();
    if (gparts) gram_rows<RB>(acc, xs, xs);
    __syncthreads();
  }
  if (gparts) store_gram(acc, gparts);
}

// X <- X Q, Z <- Z Q in place, and the shares rparts[block][64] of sum_rows |Z - w X|^2 per column.
template <int RB>
__global__ void __launch_bounds__(256) ritz_kernel(int n, int p, double2* X, double2* Z, const double2* Q, const double* w,
                                                   double* rparts) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* q = (double2*)smem;          // [64][PL]
  double2* xs = q + PMAX * PL;          // [RB][PL]
  double2* zs = xs + RB * PL;           // [RB][PL]
  const int tid = threadIdx.x;
  pdl_trigger();
  pdl_wait();
  load_square(q, Q, p);
  double res = 0;   // column tid / 4, rows tid % 4 + 4 i
  const int col = tid >> 2;
  const double wc = col < p ? w[col] : 0.0;
  for (int g = blockIdx.x; g * RB < n; g += gridDim.x) {
    load_group<RB>(xs, X, n, p, g);
    load_group<RB>(zs, Z, n, p, g);
    __syncthreads();
    GroupAcc<RB> ox, oz;
    times_square<RB>(ox, xs, q);
    times_square<RB>(oz, zs, q);
    __syncthreads();
    ox.each([&](int i, int j, double2 v) { xs[(group_row<RB>() + i) * PL + group_col<RB>() + j] = v; });
    oz.each([&](int i, int j, double2 v) { zs[(group_row<RB>() + i) * PL + group_col<RB>() + j] = v; });
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RB / 4; ++i) {
      const int e = tid + 256 * i, r = e >> 6, c = e & 63;
      if (g * RB + r < n && c < p) {
        X[(long long)(g * RB + r) * p + c] = xs[r * PL + c];
        Z[(long long)(g * RB + r) * p + c] = zs[r * PL + c];
      }
    }
#pragma unroll
    for (int i = 0; i < RB / 4; ++i) {
      const double2 x = xs[((tid & 3) + 4 * i) * PL + col], z = zs[((tid & 3) + 4 * i) * PL + col];
      const double dx = z.x - wc * x.x, dy = z.y - wc * x.y;
      res += dx * dx + dy * dy;
    }
    __syncthreads();
  }
  res += __shfl_xor_sync(0xffffffffu, res, 1);
  res += __shfl_xor_sync(0xffffffffu, res, 2);
  if ((tid & 3) == 0) rparts[blockIdx.x * PMAX + col] = res;
}

// res[c] = sqrt(sum_b rparts[b][c]).
__global__ void __launch_bounds__(1024) residual_kernel(const double* rparts, int nparts, int p, double* res) {
  __shared__ double sh[16][PMAX];
  const int c = threadIdx.x & 63, q = threadIdx.x >> 6;
  pdl_trigger();
  pdl_wait();
  double s = 0;
  for (int b = q; b < nparts; b += 16) s += rparts[b * PMAX + c];
  sh[q][c] = s;
  __syncthreads();
  if (q == 0 && c < p) {
    for (int i = 1; i < 16; ++i) s += sh[i][c];
    res[c] = sqrt(s);
  }
}

// Deterministic start block: entries uniform in [-1, 1] + i [-1, 1] from a 64-bit mix of their index.
__global__ void start_block_kernel(double2* X, long long count, unsigned long long seed) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= count) return;
  auto mix = [](unsigned long long x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
  };
  const unsigned long long a = mix(seed ^ (2ull * e)), b = mix(seed ^ (2ull * e + 1));
  X[e] = make_double2((double)(a >> 11) * 0x1.0p-52 - 1.0, (double)(b >> 11) * 0x1.0p-52 - 1.0);
}

// One CTA: eigendecomposition of a Hermitian p x p matrix (p <= 64; worked on as 64 x 64, zero beyond p) by cyclic
// Jacobi sweeps in the round-robin order (32 disjoint rotations per step).  w: eigenvalues descending; Q: row-major,
// column i the eigenvector of w[i].
// A step is two phases of FP64 work on one SM: the two-sided update of A, one 2 x 2 block J_k^H A J_l per thread for
// the 528 pairs (k, l) of one triangle (its mirror block is stored with it), and the update of V, during which one
// warp derives the next step's rotations (algebraically, from square roots and divisions).  Pairs are dealt as
// (k, k + d mod 32): neighbouring lanes touch neighbouring rows and columns, which with a row of 64 values falls on
// different banks.  Sweeps end when the off-diagonal part is at rounding level, or below 1e-12 and no longer falling.
// 64 x 64: 145 us a sweep, 2 to 7 sweeps; with separate column and row updates of the full matrix, trigonometric
// rotations and serial bookkeeping by one thread a decomposition took 2.8 ms.
struct Rot { double cs, sn, ex, ey; };
constexpr int JN = PMAX, JH = PMAX / 2;
constexpr size_t JACOBI_SMEM = 2 * sizeof(double2) * JN * JN;
__global__ void __launch_bounds__(1024, 1) heev_jacobi_kernel(int p, const double2* Hin, double* w, double2* Q, int max_sweeps) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* A = (double2*)smem_raw;
  double2* V = A + JN * JN;
  __shared__ Rot R[2][JH];
  __shared__ int place[JN];
  __shared__ double red[2][32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  pdl_trigger();
  pdl_wait();
  for (int e = t; e < JN * JN; e += 1024) {
    const int r = e / JN, c = e % JN;
    const bool in = r < p && c < p;
    const double2 u = in ? Hin[r * p + c] : make_double2(0, 0), v = in ? Hin[c * p + r] : make_double2(0, 0);
    A[e] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
    V[e] = make_double2(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  // the value in slot s at a step of the round robin: slot 0 stays, the others move one slot a step; pair k: slots k
  // and 63 - k
  auto elem = [](int s, int step) {
    const int q = s - 1 - step;
    return s == 0 ? 0 : 1 + (q < 0 ? q + JN - 1 : q);
  };
  auto rotate = [&](int k, int step, int buf) {
    const int i = elem(k, step), j = elem(JN - 1 - k, step);
    const double a = A[i * JN + i].x, b = A[j * JN + j].x;
    const double2 c = A[i * JN + j];
    const double g2 = c.x * c.x + c.y * c.y;
    Rot r = {1.0, 0.0, 1.0, 0.0};
    if (g2 > 1e-290) {   // (a smaller value is set to zero with its block)
      const double rg = rsqrt(g2), tau = 0.5 * (a - b) * rg;
      const double tn = copysign(1.0 / (fabs(tau) + sqrt(1.0 + tau * tau)), tau);
      r.cs = rsqrt(1.0 + tn * tn);
      r.sn = tn * r.cs;
      r.ex = c.x * rg;
      r.ey = -c.y * rg;   // conj(e^{i phi})
    }
    R[buf][k] = r;
  };
  if (warp == 0) rotate(t, 0, 0);
  int buf = 0;
  double last = 0;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    double o = 0, d = 0;
    for (int e = t; e < JN * JN; e += 1024) {
      const double2 x = A[e];
      const double v = x.x * x.x + x.y * x.y;
      if (e / JN == e % JN) d += v; else o += v;
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      o += __shfl_xor_sync(0xffffffffu, o, s);
      d += __shfl_xor_sync(0xffffffffu, d, s);
    }
    if (lane == 0) {
      red[0][warp] = o;
      red[1][warp] = d;
    }
    __syncthreads();
    o = 0;
    d = 0;
    for (int i = 0; i < 32; ++i) {   // the same sums in the same order in every thread
      o += red[0][i];
      d += red[1][i];
    }
    if (!(o > 1e-30 * (o + d)) || (sweep > 0 && o < 1e-24 * (o + d) && o > 0.25 * last)) break;
    last = o;
#pragma unroll 1
    for (int step = 0; step < JN - 1; ++step, buf ^= 1) {
      if (t < JH * (JH + 1) / 2) {
        const int dd = t / JH, k = t % JH, l = (k + dd) % JH;
        const Rot rk = R[buf][k], rl = R[buf][l];
        const int ik = elem(k, step), jk = elem(JN - 1 - k, step), il = elem(l, step), jl = elem(JN - 1 - l, step);
        double2 m[2][2] = {{A[ik * JN + il], A[ik * JN + jl]}, {A[jk * JN + il], A[jk * JN + jl]}};
#pragma unroll
        for (int u = 0; u < 2; ++u) {   // columns by J_l
          const double2 a = m[u][0], b = cmul(m[u][1], make_double2(rl.ex, rl.ey));
          m[u][0] = make_double2(rl.cs * a.x + rl.sn * b.x, rl.cs * a.y + rl.sn * b.y);
          m[u][1] = make_double2(rl.cs * b.x - rl.sn * a.x, rl.cs * b.y - rl.sn * a.y);
        }
#pragma unroll
        for (int v = 0; v < 2; ++v) {   // rows by J_k^H
          const double2 a = m[0][v], b = cmul(m[1][v], make_double2(rk.ex, -rk.ey));
          m[0][v] = make_double2(rk.cs * a.x + rk.sn * b.x, rk.cs * a.y + rk.sn * b.y);
          m[1][v] = make_double2(rk.cs * b.x - rk.sn * a.x, rk.cs * b.y - rk.sn * a.y);
        }
        if (dd == 0) {
          A[ik * JN + ik] = make_double2(m[0][0].x, 0.0);
          A[jk * JN + jk] = make_double2(m[1][1].x, 0.0);
          A[ik * JN + jk] = A[jk * JN + ik] = make_double2(0.0, 0.0);
        } else {
          A[ik * JN + il] = m[0][0];
          A[ik * JN + jl] = m[0][1];
          A[jk * JN + il] = m[1][0];
          A[jk * JN + jl] = m[1][1];
          A[il * JN + ik] = conjd(m[0][0]);
          A[jl * JN + ik] = conjd(m[0][1]);
          A[il * JN + jk] = conjd(m[1][0]);
          A[jl * JN + jk] = conjd(m[1][1]);
        }
      }
      __syncthreads();
      if (warp == 0) {
        rotate(t, step + 1 < JN - 1 ? step + 1 : 0, buf ^ 1);
      } else {
        const int i = elem(lane, step), j = elem(JN - 1 - lane, step);
        const Rot q = R[buf][lane];
        for (int r = warp - 1; r < JN; r += 31) {   // V <- V J
          const double2 a = V[r * JN + i], b = cmul(V[r * JN + j], make_double2(q.ex, q.ey));
          V[r * JN + i] = make_double2(q.cs * a.x + q.sn * b.x, q.cs * a.y + q.sn * b.y);
          V[r * JN + j] = make_double2(q.cs * b.x - q.sn * a.x, q.cs * b.y - q.sn * a.y);
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if (t < p) {   // eigenvalues descending: each value's place by counting (where one is NaN they keep their order)
    const double x = A[t * JN + t].x;
    bool bad = false;
    int at = 0;
    for (int i = 0; i < p; ++i) {
      const double y = A[i * JN + i].x;
      bad |= isnan(y);
      at += y > x || (y == x && i < t);
    }
    place[t] = bad ? t : at;
    w[place[t]] = x;
  }
  __syncthreads();
  for (int e = t; e < p * p; e += 1024) Q[(e / p) * p + place[e % p]] = V[(e / p) * JN + e % p];
}

// Output: vecs [n][k] = columns 0..k-1 of XQ (row-major n x p, rows in the order perm, if any), vals[i] = max(w[i], 0).
__global__ void output_kernel(int n, int p, int k, const double2* __restrict__ XQ, const double* __restrict__ w,
                              const int* __restrict__ perm, double2* vecs, double* vals) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < (long long)n * k) vecs[(perm ? perm[e / k] : e / k) * k + e % k] = XQ[(e / k) * p + e % k];
  if (e < k) vals[e] = w[e] > 0 ? w[e] : 0.0;
}

// ------------------------------------------------------------------------------------------- host side
constexpr int SMS = 148, GRAM_BLOCKS = 2 * SMS;

// Shares of the K loop for `tiles` output tiles and `chunks` chunks of K: four blocks per SM (two are resident; tiles
// differ in their non-zero blocks, and smaller shares even that out), at least eight chunks each (each share is an array the
// fold reads), at most 32 shares.
static int shares(int tiles, int chunks) {
  const int s = std::max(1, 4 * SMS / tiles);
  return std::max(1, std::min(std::min(s, 32), chunks / 8));
}

struct Sizes {
  long long np, pp, parts, flags, perm;
  int ne, s_;
  Sizes(int n, int p, int ne_, int s) : ne(ne_), s_(s) {
    perm = ne > 0 ? 0 : (long long)n * 4;
    np = (long long)n * p;
    pp = (long long)p * p;
    const int tn = ceil_div(n, zg::T);
    if (ne > 0) {
      const int ts = ceil_div(s, zg::T);
      const long long back = (long long)shares(ts * ne, ceil_div(n, zg::KC)) * ne * s * p;
      parts = std::max(back, shares(tn, ne * ceil_div(s, zg::KC)) * np);
      flags = (long long)ne * zg::flag_dim(n) * zg::flag_dim(s);
    } else {
      parts = shares(tn, ceil_div(n, zg::KC)) * np;
      flags = (long long)zg::flag_dim(n) * zg::flag_dim(n);
    }
    flags = (flags + 15) / 16 * 16;
  }
  long long wf() const { return (long long)ne * s_ * PMAX; }
  long long complex_values() const { return 2 * np + wf() + 3 * pp + parts + (long long)GRAM_BLOCKS * PMAX * PMAX; }
  long long bytes(int p) const { return 16 * complex_values() + 8 * ((long long)GRAM_BLOCKS * PMAX + 3 * p) + flags + perm + 256; }
};

struct Solver {
  cudaStream_t s;
  int n, p, ne, seg;           // T: dense (ne = 0, seg = n) or ne pupil matrices [n][seg]
  const double2* M;
  const unsigned char* flags;
  const int* perm;
  double2 *Wf, *parts, *gparts, *G, *Rinv;
  double* rdiag;
  int status = OI_OK;

  template <typename... KArgs, typename... Args>
  void run(const char* what, void (*kern)(KArgs...), dim3 grid, int block, size_t smem, Args... args) {
    if (status || (smem > 48 * 1024 && (status = ensure_smem((const void*)kern, smem, what)))) return;
    (void)launch_pdl(kern, grid, dim3(block), smem, s, args...);
    note_launch();
    status = check_launch(what);
  }
  bool fine() const { return n <= 16 * SMS; }   // 16-row groups fill the SMs better; 32-row ones reuse more
  int groups() const { return std::min(GRAM_BLOCKS, ceil_div(n, fine() ? 16 : 32)); }

  void fold(const FoldArgs& f, int batch = 1) {
    const int blocks = f.gparts ? groups() : ceil_div(f.n, 16);
    const size_t row = sizeof(double2) * PL * (f.left ? 2 : 1);
    if (!f.gparts || fine())
      run("oi_eig_topk64/fold", fold_kernel<16>, dim3(blocks, batch), 256, 16 * row, f);
    else
      run("oi_eig_topk64/fold", fold_kernel<32>, dim3(blocks, batch), 256, 32 * row, f);
  }
  // out = alpha T in + beta b1 + gamma b0; gram: the shares of left^H out (left null: out^H out) into gparts.
  void apply(const double2* in, double2* out, double alpha, double beta, const double2* b1, double gamma,
             const double2* b0, bool gram, const double2* left) {
    const double2* B = in;
    const int tn = ceil_div(n, zg::T);
    if (ne > 0) {
      const int ts = ceil_div(seg, zg::T), sh = shares(ts * ne, ceil_div(n, zg::KC));
      GemmArgs g{M, (long long)n * seg, seg, n, 1, p, in, parts, flags, zg::flag_dim(n), zg::flag_dim(seg), nullptr};
      run("oi_eig_topk64/gemm", gemm_kernel<true>, dim3(ts, sh, ne), 256, zg::SMEM, g);   // Wf_e = h_e^H in
      fold(FoldArgs{parts, sh, seg, p, 1.0, 0.0, 0.0, nullptr, nullptr, nullptr, Wf, nullptr}, ne);
      B = Wf;
    }
    const int nseg = ne > 0 ? ne : 1, sh = shares(tn, nseg * ceil_div(seg, zg::KC));
    GemmArgs g{M, (long long)n * seg, n, seg, nseg, p, B, parts, flags, zg::flag_dim(n), zg::flag_dim(seg), perm};
    run("oi_eig_topk64/gemm", gemm_kernel<false>, dim3(tn, sh, 1), 256, zg::SMEM, g);
    fold(FoldArgs{parts, sh, n, p, alpha, beta, gamma, b1, b0, left, out, gram ? gparts : nullptr});
  }
  void sum_gram() { run("oi_eig_topk64/gram", sum_gram_kernel, dim3(p), 256, 0, (const double2*)gparts, groups(), p, G); }
  // X R = X by Cholesky QR, the Gram shares of X in gparts: one pass keeps the columns independent, a second one
  // (wanted before a projection) makes them orthonormal to rounding.
  void orth(double2* X, int passes) {
    for (int pass = 0; pass < passes; ++pass) {
      sum_gram();
      run("oi_eig_topk64/chol", chol_inv_kernel, dim3(1), 512, 0, p, (const double2*)G, Rinv, rdiag,
          pass == 0 ? 1e-13 : 1e-15, pass == 0);
      double2* gp = pass + 1 < passes ? gparts : nullptr;
      if (fine())
        run("oi_eig_topk64/scale", scale_kernel<16>, dim3(groups()), 256, sizeof(double2) * PL * (PMAX + 16), n, p, X,
            (const double2*)Rinv, gp);
      else
        run("oi_eig_topk64/scale", scale_kernel<32>, dim3(groups()), 256, sizeof(double2) * PL * (PMAX + 32), n, p, X,
            (const double2*)Rinv, gp);
    }
  }
};

}  // namespace eg
}  // namespace oi

extern "C" int oi_eig_topk64_workspace(int n, int p, int ne, int s, long long* bytes) {
  using namespace oi;
  if (!bytes || n <= 0 || p <= 0) return fail(OI_EINVAL, "oi_eig_topk64_workspace: bad arguments");
  *bytes = eg::Sizes(n, p, std::max(ne, 0), std::max(s, 0)).bytes(p);
  return OI_OK;
}

extern "C" int oi_eig_topk64(const void* tcc, const void* h, int ne, int n, int s, int k, int p, int max_iter,
                             double tol, void* vecs, double* vals, void* work, long long work_bytes, int* iters,
                             void* stream) {
  using namespace oi;
  using namespace oi::eg;
  const bool dense = tcc != nullptr;
  if ((!tcc && !h) || (tcc && h) || !vecs || !vals || !work || n <= 0 || k <= 0 || p <= 0 || max_iter <= 0 ||
      (!dense && (ne <= 0 || s <= 0)))
    return fail(OI_EINVAL, "oi_eig_topk64: bad arguments");
  if (p > PMAX || p % 2 || k > p || p > n)
    return fail(OI_ERANGE, "oi_eig_topk64: need k <= p <= min(n, %d), p even (k=%d p=%d n=%d)", PMAX, k, p, n);
  if (dense) ne = 0, s = n;
  const Sizes sz(n, p, ne, s);
  const long long need = sz.bytes(p);
  if (work_bytes < need) return fail(OI_ERANGE, "oi_eig_topk64: %lld workspace bytes given, %lld needed", work_bytes, need);
  cudaStream_t st = (cudaStream_t)stream;
  double2* X = (double2*)(((uintptr_t)work + 255) & ~(uintptr_t)255);
  double2* Z = X + sz.np;
  double2* Wf = Z + sz.np;
  double2* G = Wf + sz.wf();
  double2* Rinv = G + sz.pp;
  double2* Q = Rinv + sz.pp;
  double2* parts = Q + sz.pp;
  double2* gparts = parts + sz.parts;
  double* rparts = (double*)(gparts + (long long)GRAM_BLOCKS * PMAX * PMAX);
  double* w = rparts + (long long)GRAM_BLOCKS * PMAX;   // [p], then the residuals [p] and the diagonal of R [p]
  double* res = w + p;
  double* rdiag = res + p;
  unsigned char* flags = (unsigned char*)(rdiag + p);
  const double2* M = (const double2*)(dense ? tcc : h);
  int* perm = dense ? (int*)(flags + sz.flags) : nullptr;   // flags: a multiple of 16 bytes
  if (dense) {
    order_kernel<<<1, 1024, 0, st>>>(n, M, perm);
    note_launch();
    if (int rc = check_launch("oi_eig_topk64/order")) return rc;
  }
  if (int rc = zg::mark_blocks(M, dense ? 1 : ne, n, s, flags, st, perm)) return rc;
  Solver sv{st, n, p, ne, s, M, flags, perm, Wf, parts, gparts, G, Rinv, rdiag};

  start_block_kernel<<<(unsigned)ceil_div(sz.np, 256), 256, 0, st>>>(Z, sz.np, 0x5eed0f71ull + (unsigned long long)n);
  note_launch();
  if (int rc = check_launch("oi_eig_topk64/start")) return rc;
  int it = 0, stalls = 0;   // products with T so far (a projection's own is not counted)
  double last = -1;
  bool converged = false;
  std::vector<double> host(2 * (size_t)p);
  auto fetch = [&](const double* src, size_t count) {
    if (!sv.status && (cudaMemcpyAsync(host.data(), src, 8 * count, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                       cudaStreamSynchronize(st) != cudaSuccess))
      sv.status = fail(OI_ECUDA, "oi_eig_topk64: %s", cudaGetErrorString(cudaGetLastError()));
    return sv.status == OI_OK;
  };
  auto plain = [&](int count, int last_passes) {   // X R = T X
    for (int i = 0; i < count && it < max_iter; ++i, ++it) {
      sv.apply(X, X, 1.0, 0.0, nullptr, 0.0, nullptr, true, nullptr);
      sv.orth(X, i + 1 < count && it + 1 < max_iter ? 1 : last_passes);
    }
  };
  // X R = f(T) X with f small on [0, b], for values w0 >= wk wanted and the residual `worst` (over w0)
  auto filter = [&](double w0, double wk, double b, double worst) {
    const double x = 2 * wk / b - 1, x0 = 2 * w0 / b - 1;
    if (!(x > 1.05)) return plain(4, 2);
    const double rho = x + std::sqrt(x * x - 1), rho0 = x0 + std::sqrt(x0 * x0 - 1);
    const double want = std::ceil(std::log(100.0 * worst / tol) / std::log(rho));
    int total = (int)std::max(1.0, std::min((double)std::min(EIG_DEGREE, max_iter - it), want));
    const double piece = std::log(EIG_AMP) / std::max(std::log(rho0 / rho), 1e-9);
    const int degree = (int)std::max(1.0, std::min((double)total, piece));
    const double c = 0.5 * b, e = 0.5 * b;
    while (total > 0 && !sv.status) {
      const int d = std::min(degree, total);
      total -= d;
      it += d;
      // Y_j = T_j((T - c) / e) X / T_j((w0 - c) / e) by the scaled three-term recurrence, Y_0 in X, Y_1 in Z
      const double s1 = e / (w0 - c);
      sv.apply(X, Z, s1 / e, -c * s1 / e, X, 0.0, nullptr, d == 1, nullptr);
      double sig = s1;
      for (int j = 2; j <= d; ++j) {
        const double s2 = 1.0 / (2.0 / s1 - sig);
        sv.apply(Z, X, 2 * s2 / e, -2 * s2 * c / e, Z, -sig * s2, X, j == d, nullptr);
        sig = s2;
        std::swap(X, Z);
      }
      std::swap(X, Z);   // the newest is in X
      sv.orth(X, total > 0 ? 1 : 2);
    }
  };

  std::swap(X, Z);   // the random block is the first X
  plain(EIG_START, 1);
  bool ready = false;   // X is orthonormal to rounding
  if (it < max_iter && fetch(rdiag, p)) {
    for (int i = 0; i < p; ++i)
      if (!(host[i] > 0)) host[i] = 0;
    std::sort(host.begin(), host.begin() + p, [](double a, double b) { return a > b; });
    const double w0 = host[0], wk = host[k - 1], wp = host[p - 1];
    // the error left after the plain iterations; a TCC that is not a number, or of a rank below k, goes on to the
    // projection as it is
    ready = w0 > 0 && wk > 1e-8 * w0;
    if (ready)
      filter(w0, wk, std::max(1.05 * wp, 1e-8 * w0), std::min(1.0, std::pow(wp / wk, EIG_START)) * wk / w0);
  }
  if (!ready) {
    sv.fold(FoldArgs{nullptr, 0, n, p, 0.0, 1.0, 0.0, X, nullptr, nullptr, X, gparts});
    sv.orth(X, 2);
  }
  while (!sv.status) {
    // Rayleigh-Ritz: Z = T X, H = X^H Z
    sv.apply(X, Z, 1.0, 0.0, nullptr, 0.0, nullptr, true, X);
    sv.sum_gram();
    sv.run("oi_eig_topk64/jacobi", heev_jacobi_kernel, dim3(1), 1024, JACOBI_SMEM, p, (const double2*)G, w, Q, 40);
    if (sv.fine())
      sv.run("oi_eig_topk64/ritz", ritz_kernel<16>, dim3(sv.groups()), 256, sizeof(double2) * PL * (PMAX + 32), n, p, X, Z,
             (const double2*)Q, (const double*)w, rparts);
    else
      sv.run("oi_eig_topk64/ritz", ritz_kernel<32>, dim3(sv.groups()), 256, sizeof(double2) * PL * (PMAX + 64), n, p, X, Z,
             (const double2*)Q, (const double*)w, rparts);
    sv.run("oi_eig_topk64/residual", residual_kernel, dim3(1), 1024, 0, (const double*)rparts, sv.groups(), p, res);
    if (!fetch(w, 2 * (size_t)p)) break;
    double worst = 0;   // (fmax passes NaN by: a TCC that is not a number ends here, with NaN pairs)
    for (int i = 0; i < k; ++i) worst = std::fmax(worst, host[p + i]);
    const double w0 = std::fabs(host[0]) > 0 ? std::fabs(host[0]) : 1.0;
    if (worst <= tol * w0) {
      converged = true;
      break;
    }
    if (it >= max_iter) break;
    if (last >= 0 && worst > 0.25 * last) ++stalls;
    last = worst;
    if (stalls)
      plain(4, 2);
    else
      filter(w0, host[k - 1], std::max(1.05 * host[p - 1], 1e-8 * w0), worst / w0);
  }
  if (sv.status) return sv.status;
  if (iters) *iters = converged ? it : -it;
  // X holds the Ritz vectors (columns by descending w)
  output_kernel<<<(unsigned)ceil_div((long long)n * k > p ? (long long)n * k : p, 256), 256, 0, st>>>(
      n, p, k, X, w, perm, (double2*)vecs, vals);
  note_launch();
  return check_launch("oi_eig_topk64/output");
}
