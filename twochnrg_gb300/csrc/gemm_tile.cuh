// The FP64 tile product shared by the grouped GEMM kernels.
#pragma once

#include "nrg_device.cuh"

namespace nrg {

// One tile of C = A B, 4 RW rows x kGemmTile columns, per CTA of 128 threads: warp
// w holds rows RW w .. RW w + RW - 1, lane = column.  An SM does 1.7 FP64 FMA per
// clock, so neither shared memory nor the operands' traffic bounds a tile of this
// size (0.5 B per FMA); what counts is that the FP64 pipe of every SM is busy and
// on useful elements.  A warp's FMAs follow each other at 64 cycles however few
// there are, so a tile of 32 rows takes 32 us at K = 85 also alone on its SM.
// Blocks of an iteration are 10 to 300 states: a tile of 32 leaves fewer rows and
// columns past the edges than one of 64 and four times as many tiles for 152 SMs,
// four warps keep the four sub-partitions busy, rows past the edge are left out
// in pairs (a predicated FP64 operation costs as much as one that runs), and where
// the tiles of 32 rows leave SMs idle they are of 16 or 8 rows (gemm_rows).
// Operator rotations of the tangent sweep at 200 kept (blocks of about 85 states)
// 58 ms with 64 x 64 tiles of 256 threads, 15 ms with 32 x 32, 9.6 ms with the
// rows chosen; of a one-channel sweep at 500 kept 15.8, 7.0 and 4.5 ms; of a
// full-size two-channel iteration (blocks to 300 kept of 4400) 54, 40 and 39 ms.
constexpr int kGemmThreads = 128;
constexpr int kGemmK = 16;

template <int RW>
struct GemmSmem {
  double a[kGemmK][4 * RW + 1];
  double b[kGemmK][kGemmTile];
};

template <int RW, int R>
__device__ __forceinline__ void tile_fma(const GemmSmem<RW>& S, int kc, int row, double* acc) {
  const int lane = threadIdx.x & 31;
  for (int k = 0; k < kc; k += 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double b = S.b[k + q][lane];
#pragma unroll
      for (int i = 0; i < R; ++i) acc[i] = fma(S.a[k + q][row + i], b, acc[i]);
    }
  }
}

// acc[i] += sum_k A(row + i, k) B(k, lane) for this warp's rows of the tile.
// loadA(r, k) and loadB(k, c) give elements of the tile (0 past an edge);
// A_ROWS: consecutive threads read consecutive rows of A (a transposed
// operand), else consecutive k.  `rows`: rows of the tile inside the matrix.
template <int RW, bool A_ROWS, class LoadA, class LoadB>
__device__ __forceinline__ void gemm_tile(GemmSmem<RW>& S, int K, int rows, LoadA loadA, LoadB loadB, double* acc) {
  constexpr int kRows = 4 * RW, kPerA = kRows * kGemmK / kGemmThreads, kPerB = kGemmTile * kGemmK / kGemmThreads;
  const int tid = threadIdx.x, warp = tid >> 5, row = RW * warp;
  const int mine = min(RW, rows - row);  // <= 0: none
  double ra[kPerA], rb[kPerB];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < kPerA; ++q) {
      const int idx = tid + q * kGemmThreads;
      const int r = A_ROWS ? idx % kRows : idx / kGemmK, k = A_ROWS ? idx / kRows : idx % kGemmK;
      ra[q] = k0 + k < K ? loadA(r, k0 + k) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kPerB; ++q) {
      const int idx = tid + q * kGemmThreads, kb = idx / kGemmTile, c = idx % kGemmTile;
      rb[q] = k0 + kb < K ? loadB(k0 + kb, c) : 0.0;
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += kGemmK) {
    __syncthreads();  // also of the CTA's last call, whose tiles S holds
#pragma unroll
    for (int q = 0; q < kPerA; ++q) {
      const int idx = tid + q * kGemmThreads;
      const int r = A_ROWS ? idx % kRows : idx / kGemmK, k = A_ROWS ? idx / kRows : idx % kGemmK;
      S.a[k][r] = ra[q];
    }
#pragma unroll
    for (int q = 0; q < kPerB; ++q) {
      const int idx = tid + q * kGemmThreads;
      S.b[idx / kGemmTile][idx % kGemmTile] = rb[q];
    }
    __syncthreads();
    if (k0 + kGemmK < K) fetch(k0 + kGemmK);  // the next chunk, in flight during this one's FMAs
    const int kc = min(kGemmK, (K - k0 + 3) & ~3);
    if (RW >= 8 && mine > 6) tile_fma<RW, 8>(S, kc, row, acc);
    else if (RW >= 8 && mine > 4) tile_fma<RW, 6>(S, kc, row, acc);
    else if (RW >= 4 && mine > 2) tile_fma<RW, 4>(S, kc, row, acc);
    else if (mine > 0) tile_fma<RW, 2>(S, kc, row, acc);
  }
}

}  // namespace nrg
