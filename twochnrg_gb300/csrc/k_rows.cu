// Householder tridiagonalization of blocks whose rows fit in the shared memory
// of a thread-block cluster (FP64): the blocks of the one-channel sweeps and
// the small sectors of the two-channel ones.
//
// What bounds it.  A warp-wide FP64 operation occupies an SM sub-partition for
// 64 cycles whatever its active lanes (76 with all four busy), a division or
// square root for 350-600, so on a block of a few hundred states it is neither
// the trailing update nor the matrix's traffic that counts but the chain of
// reductions and scalars of every column, and every scalar that all warps
// compute redundantly.  Hence:
//  * every CTA keeps complete rows (row r in CTA r mod CL), so that y = A u
//    needs no sum over the CTAs: 3 FMA per element of the full matrix instead
//    of 4 per element of one triangle, but one all-gather per column where
//    the triangle needs a reduction and a gather;
//  * the reflector u = x - beta e_1 stays unnormalized (H = I - tau u u^T), and
//    A u = A x - beta (A e_1), so that the sweep starts from x while a warp of
//    its own forms |x|, beta and tau;
//  * the pending update is kept as A - p y^T - q u^T with p_r = tau u_r and q_r =
//    tau y_r - 2 h u_r of the own rows, so that no w is formed over the columns;
//  * the gather carries the column of the next step beside y, so that every
//    CTA forms the next x for itself; it goes by st.async to the CTAs' own
//    mbarriers (about 400 cycles), where a cluster barrier after remote stores
//    takes 700-1200 and also waits for the reflector's stores to memory.
// Four sweep warps, one per sub-partition, keep the FP64 pipe busy (its latency
// equals its issue interval); the fifth does the scalars.  An FP64 operation
// that is predicated off in every lane costs as much as one that runs, so the
// loops below have warp-uniform bounds (the vectors end in kPad zeros), are not
// unrolled where they may end early, and compare doubles as integers.
// One block alone (kernel with its launch, GB300): 64 / 128 / 256 / 400 / 600
// states in 0.119 / 0.275 / 0.878 / 2.24 / 6.04 ms on 16 CTAs (0.125 / 0.289 /
// 0.914 / 2.31 / 6.14 with w formed over the columns), where the lower-triangle
// cluster kernel (k_tridiag.cu) took 0.674 / 1.51 / 3.25 / 6.07 / 11.6 ms.  The
// FP64 work of the sweep, 3 FMA per element at 1.7 per cycle and SM, is 0.33 of
// the 0.878 ms at 256 and 4.2 of the 6.04 at 600; the rest is the chain of one
// column, 1.9 us at any size.
//
// Waits: an mbarrier wait per step, bounded; cluster barriers per block.
//
// Outputs as tridiag_kernel's: d, e, tau, and u_j in row j, columns j+1..n-1
// (u_j[j+1] is not 1 here; the back-transformation reads it from the row).
#include <cooperative_groups.h>

#include "nrg_device.cuh"

namespace cg = cooperative_groups;

namespace nrg {

namespace {

constexpr int kSweep = 4;                       // sweep warps
constexpr int kRowsThreads = (kSweep + 1) * 32; // + the scalar warp
constexpr int kMaxCl = 16;
constexpr int kPad = 32;                        // zeros past the vectors' ends

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t map_rank(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// Asynchronous stores into a CTA of the cluster, counted on that CTA's mbarrier.
__device__ __forceinline__ void put2(uint32_t dst, double a, double b, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst), "d"(a),
               "d"(b), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void put1(uint32_t dst, double a, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(dst), "d"(a), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void expect_bytes(uint32_t bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Barrier of the whole cluster (the forms that need no converged warp).
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

struct RowsSm {
  double* x;      // 2 x ldv: u of the last step, x of this one
  double* y;      // y of the last step
  double2* ya;    // 2 x ldv: gathered (y, next column), by step parity
  double* tot;    // own rows: products, then -p_r of the update they lead to
  double* acol;   // own rows: next-column elements, then -q_r
  double* part;   // norm partials of the sweep threads
  double* dp;     // 2 x kMaxCl partial dots
  double* sc;     // scalars of the step
  double* rows;
  uint64_t* bar;  // one mbarrier per step parity
  int* dead;      // a wait gave up
  int ldv, ld;
};

enum { SC_BETA, SC_TU1, SC_B, SC_COUNT = 4 };

__host__ __device__ inline size_t rows_smem_doubles(int maxn, int cl) {
  const size_t ldv = (size_t)maxn + (maxn & 1) + kPad, own = ((size_t)maxn + cl - 1) / cl;
  return 7 * ldv + 2 * own + kSweep * 32 + 2 * kMaxCl + SC_COUNT + own * (size_t)(maxn | 1) + 4;
}

__device__ inline RowsSm rows_carve(double* sm, int maxn, int cl) {
  RowsSm S;
  S.ldv = maxn + (maxn & 1) + kPad;
  S.ld = maxn | 1;
  const int own = (maxn + cl - 1) / cl;
  double* p = sm;
  S.ya = (double2*)p; p += 4 * S.ldv;
  S.x = p; p += 2 * S.ldv;
  S.y = p; p += S.ldv;
  S.tot = p; p += own;
  S.acol = p; p += own;
  S.part = p; p += kSweep * 32;
  S.dp = p; p += 2 * kMaxCl;
  S.sc = p; p += SC_COUNT;
  S.bar = (uint64_t*)p; p += 2;
  S.dead = (int*)p; p += 2;
  S.rows = p;
  return S;
}

// RT of the CTA's rows: the pending update A - p y^T - q u^T and the product with
// x over columns j+1..n-1.
template <int RT>
__device__ __forceinline__ void sweep_rows(const RowsSm& S, int n, int j, int i0, const double* xc, const double* uo) {
  const int lane = threadIdx.x & 31;
  double* row = S.rows + i0 * S.ld;
  const int step = kSweep * S.ld;
  double pr[RT], qr[RT], acc[RT];
#pragma unroll
  for (int q = 0; q < RT; ++q) {
    pr[q] = S.tot[i0 + q * kSweep];
    qr[q] = S.acol[i0 + q * kSweep];
    acc[q] = 0.0;
  }
  const int ns = (n - j - 1 + 31) >> 5;
  int c = j + 1 + lane;
  auto col = [n](int k) { return min(k, n - 1); };  // past the row's end the vectors are 0
  // A sub-partition runs one sweep warp, so the next strip is loaded before
  // this one's FMAs (90 cycles per FMA without, 74 with; 72 is the pipe's).
  double u = uo[c], y = S.y[c], x = xc[c], r[RT];
#pragma unroll
  for (int q = 0; q < RT; ++q) r[q] = row[q * step + col(c)];
  for (int k = 0; k < ns; ++k, c += 32) {
    double un = 0.0, yn = 0.0, xn = 0.0, rn[RT];
    if (k + 1 < ns) {
      un = uo[c + 32]; yn = S.y[c + 32]; xn = xc[c + 32];
#pragma unroll
      for (int q = 0; q < RT; ++q) rn[q] = row[q * step + col(c + 32)];
    }
#pragma unroll
    for (int q = 0; q < RT; ++q) r[q] = fma(qr[q], u, r[q]);
#pragma unroll
    for (int q = 0; q < RT; ++q) r[q] = fma(pr[q], y, r[q]);
#pragma unroll
    for (int q = 0; q < RT; ++q) acc[q] = fma(r[q], x, acc[q]);
#pragma unroll
    for (int q = 0; q < RT; ++q) {
      if (c < n) row[q * step + c] = r[q];
      r[q] = rn[q];
    }
    u = un; y = yn; x = xn;
  }
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < RT; ++q) S.acol[i0 + q * kSweep] = row[q * step + j + 1];
  }
  if (RT <= 2) {
#pragma unroll
    for (int q = 0; q < RT; ++q) acc[q] = warp_sum_fixed(acc[q]);
    if (lane == 0) {
#pragma unroll
      for (int q = 0; q < RT; ++q) S.tot[i0 + q * kSweep] = acc[q];
    }
  } else {
    const double v = reduce_rows<RT>(acc);
    constexpr int kStep = 32 / RT;
    if (lane % kStep == 0) S.tot[i0 + (lane / kStep) * kSweep] = v;
  }
}

__device__ __forceinline__ bool split_dot_at(int m, int CL) { return m > 192 && CL > 1; }
// Bytes a CTA receives in a step with m trailing rows: 16 per row, the CTAs'
// shares of u.y where they are sent, and a token from each CTA that has no row
// left.  Every CTA so waits for every other in every step: a store for step
// g + 2 goes out after its target has finished step g, whose buffer and mbarrier
// it uses again.
__device__ __forceinline__ int step_bytes(int m, int CL) {
  return 16 * m + (split_dot_at(m, CL) ? 8 * CL : 8 * max(0, CL - m));
}

constexpr long long kWaitCycles = 4000000000ll;  // about two seconds

__global__ void __launch_bounds__(kRowsThreads, 3) tridiag_rows_kernel(TridiagArgs A) {
  extern __shared__ __align__(16) double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const RowsSm S = rows_carve(sm, A.maxn, CL);
  volatile int* dead = S.dead;
  if (tid == 0) {
    for (int p = 0; p < 2; ++p)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(S.bar + p)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *dead = 0;
  }
  cluster_sync();  // every CTA runs and its mbarriers are ready before any store to it
  // Steps done over all blocks: step g uses mbarrier g & 1 in its phase g >> 1.
  uint32_t g = 0;

  // Every cluster has its list of blocks, so that its CTAs need not ask another
  // for the next one.
  const int me = (int)blockIdx.x / CL, q1 = A.first ? A.first[me + 1] : A.nblocks;
  for (int qi = A.first ? A.first[me] : 0; qi < q1; ++qi) {
    const int b = A.order[qi];
    const int n = A.bsize[b];
    double* H = A.H + A.hoff[b];
    const int so = A.soff[b];
    if (n > A.maxn) {
      if (rank == 0 && tid == 0) atomicOr(A.flag, DEV_SIZE);
      continue;
    }
    if (n == 1) {
      if (rank == 0 && tid == 0) { A.d[so] = H[0]; A.e[so] = 0.0; A.tau[so] = 0.0; }
      continue;
    }
    __syncthreads();  // the last block's final reads are done
    // The CTA's rows, and row 0 (the first x).
    const int own = (n - rank + CL - 1) / CL;
    for (int i = warp; i < own; i += kSweep + 1) {
      const double* src = H + (int64_t)(rank + CL * i) * n;
      double* dst = S.rows + (size_t)i * S.ld;
      for (int c = lane; c < n; c += 32) dst[c] = __ldcg(src + c);
    }
    for (int c = tid; c < n + kPad; c += kRowsThreads) {
      S.x[c] = c < n ? __ldcg(H + c) : 0.0;
      S.x[S.ldv + c] = 0.0;  // no update pending
      S.y[c] = 0.0;
    }
    for (int i = tid; i < own; i += kRowsThreads) S.tot[i] = S.acol[i] = 0.0;
    if (tid == 0 && n > 2 && !*dead) expect_bytes(smem_u32(S.bar + (g & 1)), step_bytes(n - 1, CL));
    cluster_sync();  // every row is read before any is overwritten, every mbarrier armed
    if (warp < kSweep) {  // norm partials of the first x (elements 2..n-1)
      double s = 0.0;
      for (int c = 2 + tid; c < n; c += kSweep * 32) s = fma(S.x[c], S.x[c], s);
      S.part[tid] = s;
    }
    __syncthreads();

    double* xc = S.x;          // column j of A^(j); x[j] = d_j
    double* uo = S.x + S.ldv;  // u_{j-1}, its update pending with S.y
    for (int j = 0; j + 2 < n; ++j, ++g) {
      const int m = n - j - 1;
      double2* ya = S.ya + (g & 1) * S.ldv;
      double* dp = S.dp + (g & 1) * kMaxCl;
      const uint32_t bar = smem_u32(S.bar + (g & 1));
      // u.y by the scalar warp alone from the gathered y (m/32 FMA after the
      // gather), or for longer columns as one share per CTA sent along (a
      // reduction over the own rows before it and one over the CTAs after it).
      const bool split_dot = split_dot_at(m, CL);
      const int i0 = j + 1 <= rank ? 0 : (j + 1 - rank + CL - 1) / CL;  // first own row of the trailing matrix
      double tau = 0.0, beta, u1, tu1 = 0.0, rs = 0.0, sum = 1.0, h2 = 0.0;
      if (warp == kSweep) {
        // The next step's mbarrier is armed before this step's stores go out, so
        // that no store for that step can come before it.
        if (lane == 0 && j + 3 < n && !*dead) expect_bytes(smem_u32(S.bar + ((g + 1) & 1)), step_bytes(m - 1, CL));
        // |x|, beta, u_1 = alpha - beta, tau u_1
        double s = S.part[lane];
#pragma unroll 1
        for (int q = 1; q < kSweep && 32 * q <= m; ++q) s += S.part[lane + 32 * q];
        s = warp_sum_fixed(s);
        const double alpha = xc[j + 1];
        beta = alpha;
        u1 = alpha;
        const double sig2 = fma(alpha, alpha, s);
        // s != 0, and |x|^2 a normal number (2^-960 or more) whose reciprocal is one too
        if (__double_as_longlong(s) != 0 && __double2hiint(sig2) >= ((1023 - 960) << 20)) {
          rs = fast_rsqrt(sig2);
          const double sig = sig2 * rs;
          beta = -copysign(sig, alpha);
          sum = sig + fabs(alpha);
          u1 = copysign(sum, alpha);
          tu1 = copysign(rs, alpha);  // tau u_1
        }
        if (lane == 0) {
          S.sc[SC_BETA] = beta;
          S.sc[SC_TU1] = tu1;
        }
      } else {
        int i = i0 + warp;
#pragma unroll 1
        for (; i + 3 * kSweep < own; i += 4 * kSweep) sweep_rows<4>(S, n, j, i, xc, uo);
        if (i + kSweep < own) { sweep_rows<2>(S, n, j, i, xc, uo); i += 2 * kSweep; }
        if (i < own) sweep_rows<1>(S, n, j, i, xc, uo);
      }
      __syncthreads();
      // (y, next column) of the own rows to every CTA; tau meanwhile.
      if (warp == kSweep) {
        if (split_dot) {
          double dv = 0.0;
#pragma unroll 1
          for (int i = i0 + lane; i < own; i += 32) {
            const int r = rank + CL * i;
            dv = fma(r == j + 1 ? u1 : xc[r], fma(-beta, S.acol[i], S.tot[i]), dv);
          }
          dv = warp_sum_fixed(dv);
          if (lane < CL && !*dead) put1(map_rank(smem_u32(dp + rank), lane), dv, map_rank(bar, lane));
        } else if (i0 >= own && lane < CL && !*dead) {
          put1(map_rank(smem_u32(dp + rank), lane), 0.0, map_rank(bar, lane));  // the token
        }
        tau = rs * fast_rcp(sum);  // 2 / u.u = 1 / (|x| (|x| + |alpha|))
        if (rank == j % CL) {
          if (lane == 0) { A.d[so + j] = xc[j]; A.e[so + j] = beta; A.tau[so + j] = tau; H[(int64_t)j * n + j + 1] = u1; }
        }
      } else {
        beta = S.sc[SC_BETA];
        tu1 = S.sc[SC_TU1];
#pragma unroll 1
        for (int i = i0 + lane; i < own; i += 32) {
          const double a = S.acol[i], y = fma(-beta, a, S.tot[i]);
          const uint32_t dst = smem_u32(ya + rank + CL * i);
          for (int q = *dead ? CL : warp; q < CL; q += kSweep) put2(map_rank(dst, q), y, a, map_rank(bar, q));
        }
        if (rank == j % CL)  // u_j into row j, which no CTA reads any more (the scalar warp writes u_1)
          for (int c = j + 2 + tid; c < n; c += kSweep * 32) H[(int64_t)j * n + c] = xc[c];
      }
      // Bounded.  A CTA whose wait gives up raises the flag, stops storing to
      // the others and arming its mbarriers, and runs on (its numbers void) to
      // the cluster barriers, so that no CTA leaves while another stores to it.
      if (!*dead) {
        const long long t0 = clock64();
        while (!try_wait(bar, (g >> 1) & 1u))
          if (clock64() - t0 > kWaitCycles) {
            atomicOr(A.flag, DEV_TIMEOUT);
            *dead = 1;
            break;
          }
      }
      __syncwarp();
      // x of the next step: column j+1 of A - u w^T - w u^T with w = tau y - h u,
      // h = tau^2 (u.y) / 2, is a - (tau u_1) y - (w_1 - h u_1) u.
      if (warp == kSweep) {
        double dv = 0.0;
        if (split_dot) {
          dv = lane < CL ? dp[lane] : 0.0;
        } else {
#pragma unroll 1
          for (int c = j + 1 + lane; c < n; c += 32) dv = fma(c == j + 1 ? u1 : xc[c], ya[c].x, dv);
          __syncwarp();
        }
        dv = warp_sum_fixed(dv);
        const double t = tau * dv;  // of the block's scale, where tau^2 may leave the range
        const double b = fma(-tu1, t, tau * ya[j + 1].x);
        h2 = tau * t;
        if (lane == 0) {
          S.sc[SC_B] = b;
          xc[j + 1] = u1;
        }
      } else {
#pragma unroll 1
        for (int c = j + 1 + tid; c < n; c += kSweep * 32) {
          const double2 v = ya[c];
          uo[c] = fma(-tu1, v.x, v.y);
          S.y[c] = v.x;
        }
      }
      __syncthreads();
      if (warp < kSweep) {
        const double bb = S.sc[SC_B];
        double s = 0.0;
#pragma unroll 1
        for (int c = j + 1 + tid; c < n; c += kSweep * 32) {
          const double x = fma(-bb, xc[c], uo[c]);
          uo[c] = x;
          s = fma(x, c >= j + 3 ? x : 0.0, s);
        }
        S.part[tid] = s;
      } else {  // the own rows' part of the update, one lane each
#pragma unroll 1
        for (int i = i0 + lane; i < own; i += 32) {
          const double u = xc[rank + CL * i], y = fma(-beta, S.acol[i], S.tot[i]);
          S.tot[i] = -tau * u;
          S.acol[i] = fma(h2, u, -tau * y);
        }
      }
      __syncthreads();
      double* t = xc; xc = uo; uo = t;
    }
    // The last 2 x 2 block: row n-2 is the last x; the corner has its update pending.
    if (rank == (n - 1) % CL && tid == 0) {
      const int i = (n - 1) / CL;
      const double a = fma(S.tot[i], S.y[n - 1], fma(S.acol[i], uo[n - 1], S.rows[(size_t)i * S.ld + n - 1]));
      A.d[so + n - 2] = xc[n - 2];
      A.e[so + n - 2] = xc[n - 1];
      A.d[so + n - 1] = a;
      A.e[so + n - 1] = 0.0;
      A.tau[so + n - 2] = 0.0;
      A.tau[so + n - 1] = 0.0;
    }
  }
  cluster_sync();
}

cudaLaunchConfig_t rows_config(int cluster, int nclusters, size_t smem, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(cluster * nclusters), 1, 1);
  cfg.blockDim = dim3(kRowsThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

cudaError_t rows_attributes(int cluster) {
  cudaError_t err =
      cudaFuncSetAttribute(tridiag_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem());
  if (err == cudaSuccess && cluster > 8)
    err = cudaFuncSetAttribute(tridiag_rows_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return err;
}

bool rows_cluster_ok(int cluster) { return cluster >= 1 && cluster <= kMaxCl && (cluster & (cluster - 1)) == 0; }

}  // namespace

size_t tridiag_rows_smem_bytes(int maxn, int cluster) { return sizeof(double) * rows_smem_doubles(maxn, cluster); }

int tridiag_rows_max_clusters(int cluster, int maxn) {
  if (!rows_cluster_ok(cluster)) return 0;
  const size_t smem = tridiag_rows_smem_bytes(maxn, cluster);
  if (smem > (size_t)max_dyn_smem() || rows_attributes(cluster) != cudaSuccess) return 0;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = rows_config(cluster, 1, smem, attr);
  int nc = 0;
  if (cudaOccupancyMaxActiveClusters(&nc, tridiag_rows_kernel, &cfg) != cudaSuccess) return 0;
  return nc;
}

cudaError_t launch_tridiag_rows(const TridiagArgs& a, int cluster, int nclusters, cudaStream_t s) {
  if (!rows_cluster_ok(cluster) || nclusters < 1) return cudaErrorInvalidValue;
  const size_t smem = tridiag_rows_smem_bytes(a.maxn, cluster);
  if (smem > (size_t)max_dyn_smem()) return cudaErrorInvalidValue;
  cudaError_t err = rows_attributes(cluster);
  if (err != cudaSuccess) return err;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = rows_config(cluster, nclusters, smem, attr);
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, tridiag_rows_kernel, a);
}

}  // namespace nrg
