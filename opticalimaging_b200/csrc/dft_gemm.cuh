// FP32 tile products of the DFT forms (grids that are not powers of two, coarse grids of any multiple of 64): complex
// outputs C[m][n] = sum_k A[m][k] B[k][n], A real or complex.
//
// Bound: FP32 issue, and for the sizes of a few clips the number of blocks: a 59-wide band gives one tile per 64 rows.
// So the K loop of a tile is shared by a cluster of up to 8 blocks, whose partial tiles meet in shared memory (each
// block adds a slice of the tile over the cluster in rank order: deterministic, no partial sums in global memory).
// Each thread owns TM x TN outputs a tile-quarter apart (conflict-free reads of both operands); the next chunk of K is
// fetched into registers while the current one is multiplied.
#pragma once
#include "oi_common.cuh"
#include <cooperative_groups.h>

namespace oi {
namespace dg {

constexpr int KC = 16, THREADS = 256;

__device__ __forceinline__ void mac(float2& acc, float a, float2 b) {
  acc.x = fmaf(a, b.x, acc.x);
  acc.y = fmaf(a, b.y, acc.y);
}
__device__ __forceinline__ void mac(float2& acc, float2 a, float2 b) { cfma(acc, a, b); }

// Op: types A (float or float2); a(batch, m, k), b(batch, k, n) with m, k, n in range; put(batch, m, n, value);
// A_K: whether A is contiguous along k (else along m).  Grid: x tiles of m, y tiles of n, z = batch * cluster size.
template <int BM, int BN, int TM, int TN, typename Op>
__global__ void __launch_bounds__(THREADS, 2) gemm_kernel(Op op, int M, int N, int K) {
  using A = typename Op::A;
  static_assert((BM / TM) * (BN / TN) == THREADS, "one TM x TN output set per thread");
  constexpr int LA = BM * KC / THREADS, LB = BN * KC / THREADS, SY = BM / TM, SX = BN / TN;
  union Smem {
    struct {
      A a[2][KC][BM + 1];
      float2 b[2][KC][BN];
    } k;
    float2 tile[BM][BN];
  };
  __shared__ __align__(16) unsigned char raw[sizeof(Smem)];
  Smem& sm = *(Smem*)raw;
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, tx = tid % SX, ty = tid / SX;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN, batch = blockIdx.z / S;
  const int chunks = (K + KC - 1) / KC, c0 = (int)((long long)chunks * rank / S), c1 = (int)((long long)chunks * (rank + 1) / S);
  A ra[LA];
  float2 rb[LB];
  auto fetch = [&](int c) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int e = tid + THREADS * i, m = Op::A_K ? e / KC : e % BM, k = c * KC + (Op::A_K ? e % KC : e / BM);
      ra[i] = A();
      if (m0 + m < M && k < K) ra[i] = op.a(batch, m0 + m, k);
    }
#pragma unroll
    for (int i = 0; i < LB; ++i) {
      const int e = tid + THREADS * i, n = e % BN, k = c * KC + e / BN;
      rb[i] = n0 + n < N && k < K ? op.b(batch, k, n0 + n) : make_float2(0.f, 0.f);
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int e = tid + THREADS * i;
      sm.k.a[buf][Op::A_K ? e % KC : e / BM][Op::A_K ? e / KC : e % BM] = ra[i];
    }
#pragma unroll
    for (int i = 0; i < LB; ++i) {
      const int e = tid + THREADS * i;
      sm.k.b[buf][e / BN][e % BN] = rb[i];
    }
  };
  float2 acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
  if (c0 < c1) {
    fetch(c0);
    stage(0);
  }
  __syncthreads();
  for (int c = c0; c < c1; ++c) {
    const int buf = (c - c0) & 1;
    if (c + 1 < c1) fetch(c + 1);
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      A a[TM];
      float2 b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = sm.k.a[buf][k][ty + SY * i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = sm.k.b[buf][k][tx + SX * j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) mac(acc[i][j], a[i], b[j]);
    }
    if (c + 1 < c1) stage(buf ^ 1);
    __syncthreads();
  }
  if (S == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int m = m0 + ty + SY * i, n = n0 + tx + SX * j;
        if (m < M && n < N) op.put(batch, m, n, acc[i][j]);
      }
    return;
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sm.tile[ty + SY * i][tx + SX * j] = acc[i][j];
  cluster.sync();
  for (int e = rank * THREADS + tid; e < BM * BN; e += S * THREADS) {
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (m >= M || n >= N) continue;
    float2 s = make_float2(0.f, 0.f);
    for (int r = 0; r < S; ++r) {
      const float2 v = *cluster.map_shared_rank(&sm.tile[0][0] + e, r);
      s.x += v.x;
      s.y += v.y;
    }
    op.put(batch, m, n, s);
  }
  cluster.sync();   // the others may still be reading this block's tile
}

// Cluster size: as many blocks as bring two to every SM (148), at least two chunks of K each, at most 8.
template <int BM, int BN, int TM, int TN, typename Op>
int gemm(const Op& op, int batch, int M, int N, int K, cudaStream_t s, const char* what) {
  const long long tiles = (long long)ceil_div(M, BM) * ceil_div(N, BN) * batch;
  int S = 1;
  while (S < 8 && tiles * S < 2 * 148 && K >= 2 * S * 2 * KC) S *= 2;
  if (ceil_div(N, BN) > 65535 || (long long)batch * S > 65535)
    return fail(OI_ERANGE, "%s: %d matrices of %d columns are out of range", what, batch, N);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ceil_div(M, BM), (unsigned)ceil_div(N, BN), (unsigned)(batch * S));
  cfg.blockDim = dim3(THREADS);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = (unsigned)S;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, gemm_kernel<BM, BN, TM, TN, Op>, op, M, N, K);
  note_launch();
  return check_launch(what);
}

}  // namespace dg
}  // namespace oi
