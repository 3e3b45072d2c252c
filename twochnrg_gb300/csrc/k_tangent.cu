// Tangents of the NRG sweep with respect to the model parameters (the
// derivative pass behind nrg_grad_forward / nrg_grad_backward).
//
// The reference has no derivative code; its Hellmann-Feynman averages
// (CalcOpAvg of n_d, n_d^2 and S_z, CalcOpAvg.cpp:13-84, set up in
// CodeHandler_ModelSwitch.cpp:748-780) are what these derivatives are checked
// against, besides finite differences.  At a fixed kept-state set the sweep is
// a smooth map parameters -> observables, and one tangent direction dp is
// carried through every step:
//
//   dH_N            the assembly kernel on (dE_old, dO_old) (H_N is linear in them)
//   dH~ = Z^T dH Z  two grouped GEMMs with every eigenvector of the block
//   dlambda_k       = dH~_kk
//   dz_l            = sum_k z_k dH~_kl / (lambda_l - lambda_k)     (kept l)
//                     with no coupling inside a degenerate level (|gap| below
//                     a tolerance), where the eigenvectors are not determined
//   dO_new          = dZ_I (F Z_J^T) + Z_I (F dZ_J^T + dF Z_J^T)   (the update plan's tangent form)
//   d<O>, dTchi     weighted sums below
//
// The four directions go through every step together (a grid dimension of each
// kernel, or jobs of one grouped launch): at 200 kept one direction leaves most SMs
// idle and its kernels last 3 to 30 us.  A sweep with all four 40.5 ms one after the
// other with F Z^T formed three times, 22 ms so.
//
// This file holds the small kernels of that pass; the GEMMs and the
// rotation reuse the sweep's own kernels.
#include <algorithm>

#include "nrg_device.cuh"

namespace nrg {

namespace {

constexpr int kThreads = 256;
constexpr int kBlocks = 304;  // two CTAs of one warp per SM for the reductions
constexpr int kMaxAvg = 5;    // averaged operators (two sums each between the 12 thermodynamic and the last)
constexpr int kEigParts = 4;  // CTAs per block of the division pass

// kEigParts CTAs per block: dlambda and the coupling matrix C (n x kept, row-major)
// of the block's kept eigenvectors.
__global__ void __launch_bounds__(kThreads) tan_eig_kernel(TanEigArgs A) {
  const int b = blockIdx.x;
  const int n = A.bsize[b], k = A.nkeep[b];
  const int p = blockIdx.z;
  const double* D = A.dHt + A.h_stride * p + A.hoff[b];
  double* dlam = A.dlam + (int64_t)A.nstates * p + A.soff[b];
  const double* lam = A.ev + A.soff[b];
  double lmax = 0.0;
  for (int i = 0; i < n; ++i) lmax = fmax(lmax, fabs(lam[i]));
  const double tol = A.degen_tol * fmax(1.0, lmax);
  const int first = blockIdx.y * blockDim.x + threadIdx.x, stride = gridDim.y * blockDim.x;
  for (int x = first; x < n; x += stride) dlam[x] = D[(int64_t)x * n + x];
  double* C = A.C + A.c_stride * p + A.coff[b];
  for (int idx = first; idx < n * k; idx += stride) {
    const int r = idx / k, l = idx - r * k;
    const double gap = lam[l] - lam[r];
    C[idx] = (r == l || fabs(gap) <= tol) ? 0.0 : D[(int64_t)r * n + l] / gap;
  }
}

// dE of every state (shifted: dlambda - dlambda of the ground state) into
// dE_all, and the kept states' dE in the kept order into dE_kept.
__global__ void tan_shift_kernel(const double* dlam, int nstates, int gs, double* dE_all, const int* kept_state,
                                 int nkept, double* dE_kept, double* gs_out) {
  const int p = blockIdx.y;
  dlam += (int64_t)nstates * p; dE_all += (int64_t)nstates * p; dE_kept += (int64_t)nkept * p;
  const double g = dlam[gs];
  if (blockIdx.x == 0 && threadIdx.x == 0) gs_out[p] = g;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nstates; i += gridDim.x * blockDim.x)
    dE_all[i] = dlam[i] - g;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nkept; i += gridDim.x * blockDim.x)
    dE_kept[i] = dlam[kept_state[i]] - g;
}

// Per new-basis state g, the tangent of the old energy it came from.
__global__ void tan_gather_kernel(const double* dE_kept_old, int nold, const int* stcf, int n, double* out) {
  const int p = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[(int64_t)n * p + i] = dE_kept_old[(int64_t)nold * p + stcf[i]];
}

__global__ void tan_scale_kernel(const double* a, double s, int64_t n, double* out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = s * a[i];
}

// Partial sums over states, in a fixed order per CTA (deterministic):
// per temperature t: sum deg w dE, sum SzSq w dE, sum deg E w dE, with w = e^{-beta_t E};
// then per averaged operator o over the kept states at betabar:
// sum deg w dO_ii, sum deg w O_ii dE, and sum deg w dE.
__global__ void __launch_bounds__(32) tan_sums_kernel(TanSumArgs A, double* partial) {
  constexpr int W = TanSumArgs::kMaxOut;
  const int p = blockIdx.y;
  const double* dEs = A.dE + (int64_t)A.nstates * p;
  const double* dEks = A.dEk + (int64_t)A.nkept * p;
  const double* const* dops = A.dops + 8 * p;
  partial += (size_t)gridDim.x * W * p;
  double acc[W];
#pragma unroll
  for (int t = 0; t < W; ++t) acc[t] = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.nstates; i += gridDim.x * blockDim.x) {
    const int b = A.state_block[i];
    const double S = A.bq[2 * b + 1];
    const double deg = A.totalS ? 2.0 * S + 1.0 : 1.0;
    const double szsq = A.totalS ? (1.0 / 12.0) * deg * (deg * deg - 1.0) : S * S;
    const double E = A.en[i], dE = dEs[i];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const double w = exp(-A.beta[t] * E);
      acc[3 * t] += deg * w * dE;
      acc[3 * t + 1] += szsq * w * dE;
      acc[3 * t + 2] += deg * E * w * dE;
    }
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.nkept; i += gridDim.x * blockDim.x) {
    const int kb = A.kstate_block[i];
    const int x = i - A.koff[kb];
    const double deg = A.totalS ? 2.0 * A.kbq[2 * kb + 1] + 1.0 : 1.0;
    const double E = A.ken[i], dE = dEks[i];
    const double w = deg * exp(-A.betabar * E);
#pragma unroll
    for (int o = 0; o < kMaxAvg; ++o) {
      if (o >= A.nops) break;
      const int64_t off = A.diag_off[o * A.nkblocks + kb];
      const int64_t e = off >= 0 ? off + (int64_t)x * A.kld[kb] + x : -1;
      const double O = e >= 0 ? A.ops[o][e] : 0.0, dO = e >= 0 ? dops[o][e] : 0.0;
      acc[12 + 2 * o] += w * dO;
      acc[12 + 2 * o + 1] += w * O * dE;
    }
    acc[W - 1] += w * dE;
  }
#pragma unroll
  for (int t = 0; t < W; ++t) {
    const double v = warp_sum_fixed(acc[t]);
    if (threadIdx.x == 0) partial[(size_t)blockIdx.x * W + t] = v;
  }
}

// One warp per output, lanes over the partials.
__global__ void __launch_bounds__(32) tan_fold_kernel(const double* partial, int nparts, double* out) {
  constexpr int W = TanSumArgs::kMaxOut;
  partial += (size_t)nparts * W * blockIdx.y;
  double v = 0.0;
  for (int p = threadIdx.x; p < nparts; p += 32) v += partial[(size_t)p * W + blockIdx.x];
  v = warp_sum_fixed(v);
  if (threadIdx.x == 0) out[W * blockIdx.y + blockIdx.x] = v;
}

int grid_for(int64_t n) { return (int)std::min<int64_t>(std::max<int64_t>((n + 255) / 256, 1), 1184); }

}  // namespace

void launch_tan_eig(const TanEigArgs& a, int nblocks, cudaStream_t s) {
  if (nblocks > 0) tan_eig_kernel<<<dim3(nblocks, kEigParts, kTanDirs), kThreads, 0, s>>>(a);
}
void launch_tan_shift(const double* dlam, int nstates, int gs, double* dE_all, const int* kept_state, int nkept,
                      double* dE_kept, double* gs_out, cudaStream_t s) {
  tan_shift_kernel<<<dim3(grid_for(std::max(nstates, nkept)), kTanDirs), 256, 0, s>>>(dlam, nstates, gs, dE_all,
                                                                                     kept_state, nkept, dE_kept, gs_out);
}
void launch_tan_gather(const double* dE_kept_old, int nold, const int* stcf, int n, double* out, cudaStream_t s) {
  if (n > 0) tan_gather_kernel<<<dim3(grid_for(n), kTanDirs), 256, 0, s>>>(dE_kept_old, nold, stcf, n, out);
}
void launch_tan_scale(const double* a, double scale, int64_t n, double* out, cudaStream_t s) {
  if (n > 0) tan_scale_kernel<<<grid_for(n), 256, 0, s>>>(a, scale, n, out);
}
size_t tan_partial_doubles() { return (size_t)kBlocks * TanSumArgs::kMaxOut * kTanDirs; }
void launch_tan_sums(const TanSumArgs& a, double* partial, double* out, cudaStream_t s) {
  tan_sums_kernel<<<dim3(kBlocks, kTanDirs), 32, 0, s>>>(a, partial);
  tan_fold_kernel<<<dim3(TanSumArgs::kMaxOut, kTanDirs), 32, 0, s>>>(partial, kBlocks, out);
}

}  // namespace nrg
