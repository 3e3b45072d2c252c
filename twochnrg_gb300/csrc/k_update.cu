// Operator rotation into the new kept basis (FP64).
//
// Replaces the per-pair element loop and the two cblas_dgemm calls of
// UpdateMatrices (UpdateMatrices.cpp:333-560): O_new(i,j) = Z_i . F(i,j) . Z_j^T.
// F is never formed: it is a sum of site-structured terms (an f-type operator
// acts on the new site only, so F couples states that came from the same old
// state; an impurity operator acts on the old part only, so F is the old
// operator block between states of the same site type).  gather_kernel
// builds T = F . Z_j^T row group by row group from those terms (no atomics:
// each CTA owns one destination row group), then gemm_kernel forms
// O = Z_i . T for every (operator, block pair) job of the iteration in one
// grouped launch.
#include "gemm_tile.cuh"
#include "nrg_device.cuh"

namespace nrg {

namespace {

// The site-operator terms (the old operators' are imp_gemm_kernel's).  TAN:
// direction blockIdx.y of the tangent pass, with Zt's tangent into T's.
template <bool TAN>
__global__ void __launch_bounds__(256) gather_kernel(UpdateArgs A) {
  const int g = blockIdx.x;
  double* const Tall = TAN ? A.dT + A.t_stride * blockIdx.y : A.T;
  const double* const Zall = TAN ? A.dZt + A.z_stride * blockIdx.y : A.Zt;
  const int t0 = A.group_first[g], nt = A.group_count[g];
  for (int t = t0; t < t0 + nt; ++t) {
    const GatherTerm G = A.terms[t];
    const RotJob J = A.jobs[G.job];
    const int kj = J.kj;
    double* T = Tall + J.t_off;
    const double* Zt = Zall + J.zt_off;
    for (int idx = threadIdx.x; idx < G.rows * kj; idx += blockDim.x) {
      const int a = idx / kj, c = idx - a * kj;
      double* dst = T + (int64_t)(G.dst_base + a * G.dst_stride) * kj + c;
      *dst = fma(G.coef, Zt[(int64_t)(G.src_base + a * G.src_stride) * J.ldz + c], *dst);
    }
    __syncthreads();
  }
}

// O (ki x kj) = Z_I (ki x nI) . T (nI x kj), one tile per CTA; TAN: Z' T + Z T'.
template <int RW, bool TAN>
__global__ void __launch_bounds__(kGemmThreads, 6) gemm_kernel(UpdateArgs A) {
  __shared__ GemmSmem<RW> S;
  const RotJob J = A.jobs[A.tile_job[blockIdx.x]];
  const int mn = A.tile_mn[blockIdx.x], p = TAN ? blockIdx.y : 0;
  const int m0 = (mn >> 16) * 4 * RW, n0 = (mn & 0xffff) * kGemmTile;
  const int rows = J.ki - m0, K = J.nI, N = J.kj;
  double acc[RW] = {};
  auto product = [&](const double* Am, const double* Bm) {
    Am += J.z_off + (int64_t)m0 * K;
    Bm += J.t_off;
    gemm_tile<RW, false>(S, K, rows, [&](int r, int k) { return r < rows ? Am[(int64_t)r * K + k] : 0.0; },
                         [&](int k, int c) { return n0 + c < N ? Bm[(int64_t)k * N + n0 + c] : 0.0; }, acc);
  };
  if (TAN) product(A.dZ + A.z_stride * p, A.T);
  product(A.Z, TAN ? A.dT + A.t_stride * p : A.T);
  const int c = n0 + (threadIdx.x & 31), r0 = m0 + RW * (threadIdx.x >> 5);
  double* O = (TAN ? A.dnew_ops[16 * p + J.op] : A.new_ops[J.op]) + J.o_off;
  if (c >= N) return;
#pragma unroll
  for (int i = 0; i < RW; ++i)
    if (r0 + i < J.ki) O[(int64_t)(r0 + i) * J.ldo + c] = acc[i];
}

// Impurity-operator terms (old block x rows of Zt) as GEMM tiles:
// T[dst(a)] += sum_terms coef * sum_b M[a][b] Zt[src(b)].  The terms of one
// group share their destination rows (one row group of one job) and are
// summed inside the tile, so tiles of different groups never overlap.  TAN: M
// with Zt's tangent and M's tangent with Zt, into T's.
template <int RW, bool TAN>
__global__ void __launch_bounds__(kGemmThreads, 6) imp_gemm_kernel(UpdateArgs A) {
  __shared__ GemmSmem<RW> S;
  const int grp = A.tile1_group[blockIdx.x], p = TAN ? blockIdx.y : 0;
  const int t0 = A.group1_first[grp], nt = A.group1_count[grp];
  const int mn = A.tile1_mn[blockIdx.x];
  const GatherTerm G0 = A.terms1[t0];
  const RotJob J = A.jobs[G0.job];
  const int m0 = (mn >> 16) * 4 * RW, n0 = (mn & 0xffff) * kGemmTile;
  const int rows = G0.rows - m0, N = J.kj;
  double* T = (TAN ? A.dT + A.t_stride * p : A.T) + J.t_off;
  double acc[RW] = {};
  for (int t = t0; t < t0 + nt; ++t) {
    const GatherTerm G = A.terms1[t];
    auto product = [&](const double* M, const double* Zt) {
      const double* Am = M + G.old_off + (int64_t)m0 * G.old_ld;  // rows x srows, row stride old_ld
      Zt += J.zt_off;
      gemm_tile<RW, false>(S, G.srows, rows,
                           [&](int r, int k) { return r < rows ? G.coef * Am[(int64_t)r * G.old_ld + k] : 0.0; },
                           [&](int k, int c) {
                             return n0 + c < N ? Zt[(int64_t)(G.src_base + k * G.src_stride) * J.ldz + n0 + c] : 0.0;
                           },
                           acc);
    };
    product(A.old_ops[G.op], TAN ? A.dZt + A.z_stride * p : A.Zt);
    if (TAN) product(A.dold_ops[16 * p + G.op], A.Zt);
  }
  const int c = n0 + (threadIdx.x & 31), r0 = m0 + RW * (threadIdx.x >> 5);
  if (c >= N) return;
#pragma unroll
  for (int i = 0; i < RW; ++i)
    if (r0 + i < G0.rows) T[(int64_t)(G0.dst_base + (r0 + i) * G0.dst_stride) * N + c] += acc[i];
}

template <bool TAN>
void launch_all(const UpdateArgs& a, cudaStream_t s) {
  const unsigned nd = TAN ? a.ndir : 1;
  if (a.ngroups > 0) gather_kernel<TAN><<<dim3(a.ngroups, nd), 256, 0, s>>>(a);
  if (a.ntiles1 > 0) {
    const dim3 g(a.ntiles1, nd);
    if (a.rows1 == 8) imp_gemm_kernel<8, TAN><<<g, kGemmThreads, 0, s>>>(a);
    else if (a.rows1 == 4) imp_gemm_kernel<4, TAN><<<g, kGemmThreads, 0, s>>>(a);
    else imp_gemm_kernel<2, TAN><<<g, kGemmThreads, 0, s>>>(a);
  }
  if (a.ntiles > 0) {
    const dim3 g(a.ntiles, nd);
    if (a.rows == 8) gemm_kernel<8, TAN><<<g, kGemmThreads, 0, s>>>(a);
    else if (a.rows == 4) gemm_kernel<4, TAN><<<g, kGemmThreads, 0, s>>>(a);
    else gemm_kernel<2, TAN><<<g, kGemmThreads, 0, s>>>(a);
  }
}

}  // namespace

void launch_update(const UpdateArgs& a, cudaStream_t s) {
  if (a.ndir > 0) launch_all<true>(a, s);
  else launch_all<false>(a, s);
}

}  // namespace nrg
