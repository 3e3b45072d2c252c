// The FP64 tile product shared by the grouped GEMM kernels.
#pragma once

#include "nrg_device.cuh"

namespace nrg {

// One kGemmTile x kGemmTile tile of C = A B per CTA of 128 threads: warp w
// holds rows 8 w .. 8 w + 7, lane = column.  An SM does 1.7 FP64 FMA per clock,
// so neither shared memory nor the operands' traffic bounds a tile of this
// size (0.5 B per FMA); what counts is that the FP64 pipe of every SM is busy
// and on useful elements.  Blocks of an iteration are 10 to 300 states: a tile
// of 32 leaves fewer rows and columns past the edges than one of 64 and four
// times as many tiles for 152 SMs, four warps keep the four sub-partitions
// busy, and rows past the edge are left out in pairs (a predicated FP64
// operation costs as much as one that runs).  Operator rotations of the
// tangent sweep at 200 kept (blocks of about 85 states) 58 ms with 64 x 64
// tiles of 256 threads, 15 ms so; of a one-channel sweep at 500 kept 15.8 and
// 7.0 ms; of a full-size two-channel iteration (blocks to 300 kept of 4400)
// 54 and 40 ms.
constexpr int kGemmThreads = 128;
constexpr int kGemmK = 16;

struct GemmSmem {
  double a[kGemmK][kGemmTile + 1];
  double b[kGemmK][kGemmTile];
};

template <int R>
__device__ __forceinline__ void tile_fma(const GemmSmem& S, int kc, int row, double* acc) {
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
template <bool A_ROWS, class LoadA, class LoadB>
__device__ __forceinline__ void gemm_tile(GemmSmem& S, int K, int rows, LoadA loadA, LoadB loadB, double* acc) {
  constexpr int kPer = kGemmTile * kGemmK / kGemmThreads;
  const int tid = threadIdx.x, warp = tid >> 5, row = 8 * warp;
  const int mine = min(8, rows - row);  // <= 0: none
  double ra[kPer], rb[kPer];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int idx = tid + q * kGemmThreads;
      const int r = A_ROWS ? idx % kGemmTile : idx / kGemmK, k = A_ROWS ? idx / kGemmTile : idx % kGemmK;
      ra[q] = k0 + k < K ? loadA(r, k0 + k) : 0.0;
      const int kb = idx / kGemmTile, c = idx % kGemmTile;
      rb[q] = k0 + kb < K ? loadB(k0 + kb, c) : 0.0;
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += kGemmK) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int idx = tid + q * kGemmThreads;
      const int r = A_ROWS ? idx % kGemmTile : idx / kGemmK, k = A_ROWS ? idx / kGemmTile : idx % kGemmK;
      S.a[k][r] = ra[q];
      S.b[idx / kGemmTile][idx % kGemmTile] = rb[q];
    }
    __syncthreads();
    if (k0 + kGemmK < K) fetch(k0 + kGemmK);  // the next chunk, in flight during this one's FMAs
    const int kc = min(kGemmK, (K - k0 + 3) & ~3);
    if (mine > 6) tile_fma<8>(S, kc, row, acc);
    else if (mine > 4) tile_fma<6>(S, kc, row, acc);
    else if (mine > 2) tile_fma<4>(S, kc, row, acc);
    else if (mine > 0) tile_fma<2>(S, kc, row, acc);
  }
}

}  // namespace nrg
