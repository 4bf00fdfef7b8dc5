// Complex FP64 tile product shared by the eigensolver (eig64.cu) and the TCC assembly (tcc64.cu): a 64 x 64 output
// tile by 256 threads, K in chunks of 16 through a ring of shared-memory stages filled by 16-byte asynchronous
// copies (one complex value each, so either operand can be transposed on the way in).
//
// Bound: FP64 issue (64 DFMA per SM and cycle).  Each thread owns the 4 x 4 outputs (ty + 16 i, tx + 16 j): per k a
// warp reads 4 + 4 values as 12 conflict-free shared-memory wavefronts against 64 DFMA (128 issue cycles).  With the
// outputs 4 ty + i, 4 tx + j the column reads are 64 bytes apart, an 8-way bank conflict, and the TCC assembly ran at
// a third of the FP64 rate.
#pragma once
#include "oi_common.cuh"
#include <cstdint>

namespace oi {
namespace zg {

constexpr int T = 64, KC = 16;             // output tile, K chunk
constexpr int LD = T + 1;                  // stage row (odd: transposing copies touch every bank)
constexpr int STAGES = 3;
constexpr int STAGE_Z = 2 * KC * LD;       // complex values per stage: A and B
constexpr int LIST = 1024;                 // chunks looked at together
constexpr size_t SMEM = sizeof(double2) * STAGES * STAGE_Z + sizeof(unsigned short) * LIST + 64;

__device__ __forceinline__ void cp16(double2* dst, const double2* src, bool on) {
  const int bytes = on ? 16 : 0;   // 0: the destination is zero-filled, the source is not read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc (+)= a b, conj(a) b or a conj(b)
enum Conj { NONE, CONJ_A, CONJ_B };
template <int C> __device__ __forceinline__ void mac(double2& acc, double2 a, double2 b) {
  if (C == NONE) cfma(acc, a, b);
  if (C == CONJ_A) cfma_conj(acc, b, a);
  if (C == CONJ_B) cfma_conj(acc, a, b);
}

// Runs the K loop of one tile.  active(c): whether chunk c (first + i * step, c < chunks) contributes; load(c, As, Bs)
// issues the copies of chunk c into As[KC][LD], Bs[KC][LD] (k-major).  acc[i][j] is output (ty + 16 i, tx + 16 j).
template <int C, typename Active, typename Load>
__device__ __forceinline__ void tile_loop(double2 (&acc)[4][4], unsigned char* smem, int first, int step, int chunks,
                                          Active active, Load load) {
  double2* ring = (double2*)smem;
  unsigned short* list = (unsigned short*)(ring + STAGES * STAGE_Z);
  int* wsum = (int*)(list + LIST);   // [8] per-warp counts
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, warp = tid >> 5, lane = tid & 31;
  for (int base = 0; first + base * step < chunks; base += LIST) {
    int count = 0;
    __syncthreads();   // the previous window's list and stages are consumed
    for (int o = 0; o < LIST && first + (base + o) * step < chunks; o += 256) {
      const int c = first + (base + o + tid) * step;
      const bool on = o + tid < LIST && c < chunks && active(c);
      const unsigned m = __ballot_sync(0xffffffffu, on);
      if (lane == 0) wsum[warp] = __popc(m);
      __syncthreads();
      int at = count;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const int n = wsum[w];
        if (w < warp) at += n;
        count += n;
      }
      if (on) list[at + __popc(m & ((1u << lane) - 1))] = (unsigned short)(o + tid);
      __syncthreads();
    }
    auto fetch = [&](int i) {
      if (i < count) {
        double2* s = ring + (i % STAGES) * STAGE_Z;
        load(first + (base + list[i]) * step, s, s + KC * LD);
      }
      cp_commit();
    };
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) fetch(i);
    for (int i = 0; i < count; ++i) {
      cp_wait<STAGES - 2>();
      __syncthreads();                 // chunk i is in place; chunk i - 1's stage is free
      fetch(i + STAGES - 1);
      const double2* As = ring + (i % STAGES) * STAGE_Z;
      const double2* Bs = As + KC * LD;
#pragma unroll 4
      for (int k = 0; k < KC; ++k) {
        double2 a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = As[k * LD + ty + 16 * u];
#pragma unroll
        for (int u = 0; u < 4; ++u) b[u] = Bs[k * LD + tx + 16 * u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) mac<C>(acc[u][v], a[u], b[v]);
      }
    }
    cp_wait<0>();
  }
}

// Copies of a 16 (k) x 64 block into a stage.  rows: the block's 64-index is the source's row (k contiguous in
// memory); else k is the source's row (the 64-index contiguous).
__device__ __forceinline__ void load_rows(double2* s, const double2* src, long long ld, int r0, int nr, int k0, int nk) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = threadIdx.x + 256 * i, k = e & 15, r = e >> 4;
    const bool on = r0 + r < nr && k0 + k < nk;
    cp16(s + k * LD + r, on ? src + (long long)(r0 + r) * ld + k0 + k : src, on);
  }
}
__device__ __forceinline__ void load_cols(double2* s, const double2* src, long long ld, int c0, int nc, int k0, int nk) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = threadIdx.x + 256 * i, c = e & 63, k = e >> 6;
    const bool on = c0 + c < nc && k0 + k < nk;
    cp16(s + k * LD + c, on ? src + (long long)(k0 + k) * ld + c0 + c : src, on);
  }
}

// Marks of the 16 x 16 blocks of M [batch][rows][cols]: flags[b][r16][c16], pitches fr = flag_rows(rows) and
// fc = flag_cols(cols) (padded to whole 64-row / 64-column tiles); bit 0 a non-zero value, bit 1 a value that is not
// finite.  One block per 16 rows x 256 columns.
__host__ __device__ inline int flag_dim(int n) { return (n + T - 1) / T * (T / KC); }
int mark_blocks(const double2* M, int batch, int rows, int cols, unsigned char* flags, cudaStream_t s);

}  // namespace zg
}  // namespace oi
