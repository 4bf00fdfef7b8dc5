// Complex FP64 tile product shared by the eigensolver (eig64.cu) and the TCC assembly (tcc64.cu): a 64 x 64 output
// tile by 256 threads, K in chunks of 16 through a ring of shared-memory stages filled by 16-byte asynchronous
// copies (one complex value each, so either operand can be transposed on the way in).
//
// Bound: FP64 issue (64 multiply-adds per SM and cycle).  The products run on the FP64 matrix instruction
// (mma.sync m8n8k4): each of the 8 warps owns 32 x 16 outputs, and per four k a warp reads 4 + 2 shared-memory values a
// lane for 32 matrix instructions (8192 multiply-adds).  As scalar FMAs on 4 x 4 outputs a thread, the same work needs
// 32 such reads, and shared memory is as busy as the FP64 pipe: T X at 3481 x 3481 x 64, 0.62 of its blocks
// non-zero, 218 -> 169 us (126 with 0.41 of them, in the eigensolver's order of rows).
#pragma once
#include "oi_common.cuh"
#include <cstdint>

namespace oi {
namespace zg {

constexpr int T = 64, KC = 16;             // output tile, K chunk
constexpr int LD = T + 2;                  // stage row: 2 (mod 8), so that a fragment's 4 x 2 values fall on 8 banks
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

// Output tile of a warp, 8 MI x 8 NI complex values: lane l holds rows l / 4 + 8 i, columns 2 (l % 4) + {0, 1} + 8 j.
template <int MI, int NI> struct Acc {
  double re[MI][NI][2], im[MI][NI][2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  }
  // f(row, column, value) of this lane's values
  template <typename F> __device__ __forceinline__ void each(F f) const {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u)
          f((lane >> 2) + 8 * i, 2 * (lane & 3) + u + 8 * j, make_double2(re[i][j][u], im[i][j][u]));
  }
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// acc += a b, conj(a) b or a conj(b) over KN (a multiple of 4) values of k: a(i, k) = A[i * am + k * ak], row i of the
// warp's tile, b(k, j) = B[k * bk + j].
enum Conj { NONE, CONJ_A, CONJ_B };
template <int C, int KN, int MI, int NI>
__device__ __forceinline__ void warp_mma(Acc<MI, NI>& acc, const double2* A, int am, int ak, const double2* B, int bk) {
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
#pragma unroll
  for (int k = 0; k < KN; k += 4) {
    double2 a[MI], b[NI];
#pragma unroll
    for (int i = 0; i < MI; ++i) a[i] = A[(r + 8 * i) * am + (k + q) * ak];
#pragma unroll
    for (int j = 0; j < NI; ++j) b[j] = B[(k + q) * bk + r + 8 * j];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j) {
        dmma(acc.re[i][j], a[i].x, b[j].x);
        dmma(acc.re[i][j], C == NONE ? -a[i].y : a[i].y, b[j].y);
        dmma(acc.im[i][j], C == CONJ_B ? -a[i].x : a[i].x, b[j].y);
        dmma(acc.im[i][j], C == CONJ_A ? -a[i].y : a[i].y, b[j].x);
      }
  }
}

using TileAcc = Acc<4, 2>;   // 64 x 64 by 8 warps: warp w at rows 32 (w / 4), columns 16 (w % 4)
__device__ __forceinline__ int tile_row() { return 32 * (threadIdx.x >> 7); }
__device__ __forceinline__ int tile_col() { return 16 * ((threadIdx.x >> 5) & 3); }

// Runs the K loop of one tile.  active(c): whether chunk c (first + i * step, c < chunks) contributes; load(c, As, Bs)
// issues the copies of chunk c into As[KC][LD], Bs[KC][LD] (k-major).
template <int C, typename Active, typename Load>
__device__ __forceinline__ void tile_loop(TileAcc& acc, unsigned char* smem, int first, int step, int chunks,
                                          Active active, Load load) {
  double2* ring = (double2*)smem;
  unsigned short* list = (unsigned short*)(ring + STAGES * STAGE_Z);
  int* wsum = (int*)(list + LIST);   // [8] per-warp counts
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
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
      warp_mma<C, KC>(acc, As + tile_row(), 1, LD, Bs + tile_col(), LD);
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
// load_rows of the block of src with its rows and columns taken in the order perm.
__device__ __forceinline__ void load_rows_perm(double2* s, const double2* src, long long ld, int r0, int nr, int k0, int nk,
                                               const int* __restrict__ perm) {
  const int k = threadIdx.x & 15, col = k0 + k < nk ? __ldg(perm + k0 + k) : 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = (threadIdx.x >> 4) + 16 * i;
    const bool on = r0 + r < nr && k0 + k < nk;
    cp16(s + k * LD + r, on ? src + (long long)__ldg(perm + r0 + r) * ld + col : src, on);
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
// finite.  One block per 16 rows x 256 columns.  perm (may be null): the order in which M's rows and columns are taken.
__host__ __device__ inline int flag_dim(int n) { return (n + T - 1) / T * (T / KC); }
int mark_blocks(const double2* M, int batch, int rows, int cols, unsigned char* flags, cudaStream_t s,
                const int* perm = nullptr);

}  // namespace zg
}  // namespace oi
