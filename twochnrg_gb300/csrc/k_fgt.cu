// Lehmann sums of one shell by expansion about bins of the records' keys.
//
// A(omega) needs sum_i w_i exp(-(t - key_i)^2) at every frequency's t.  Summed
// directly (lehmann_kernel, k_dm.cu) a record costs three FP64 operations per
// frequency and an exponential per sixteen: 5.8e9 terms and 194 ms for a
// one-channel spectral function of 13 million records and 2000 frequencies.
// Here the records of a list are put into bins of width 2 r in their key, and
// with s = key - centre, tau = t - centre,
//   exp(-(tau - s)^2) = sum_n (s/r)^n b_n(tau),  b_n = r^n H_n(tau) exp(-tau^2) / n!
// (the generating function of the Hermite polynomials H_n), so that a bin
// is its kTerms moments sum_i w_i (s_i/r)^n and a record costs two operations
// per moment, once: 10.7 ms for the same sums, most of it the moments (about 6.5)
// and their evaluation (2.0).  Lists of the tangents use
// (tau - s) exp(-(tau - s)^2) = sum_n (s/r)^n (n+1)/(2r) b_{n+1}(tau).
//
// What is dropped, and what is rounded.  With r = 1/16 and 28 terms the first
// one dropped is below (2 r |tau|)^28 / 28! of the Gaussian: 3e-15 of it at
// |tau| = 27.4, beyond which exp(-tau^2) is 0, and below 1e-17 up to 22.  One
// rounding of tau or tau^2 serves a whole bin here, where the direct sum's
// average out over the records, so both are carried with their error
// (exp(-tau^2) moves by 2 tau times that of tau): against long double, relative
// to the sum, at most 6e-16 within a width, 2e-15 at 18 widths and 1e-14 at 26
// (direct sum 3e-16, 6e-14, 9e-14; by its recurrence over even frequencies
// 1e-14, 4e-13, 2e-6).
//
// The records are sorted by bin with a stable counting sort (counts per chunk,
// one scan, ranks by warp matching), so every sum has a fixed order.
#include "nrg_device.cuh"

namespace nrg {

namespace {

constexpr int kTerms = kFgtTerms;
constexpr double kR = 1.0 / 16;
constexpr int kWarps = 8;

__device__ __forceinline__ bool is_finite(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

// -1: the record's term is 0 at every frequency of the list.  A weight that is
// not finite makes its term NaN there too, so it is put into a bin.
__device__ __forceinline__ int bin_of(const FgtList& L, int64_t i) {
  const int b = (int)floor((L.key[i] - L.origin) * (1.0 / (2.0 * kR)));
  if (b >= 0 && b < L.nbins) return b;
  return is_finite(L.w[i]) ? -1 : 0;
}

// Records of chunk c of the list: [begin, end); warp w of the CTA takes a
// contiguous eighth (a multiple of 32 records).
__device__ __forceinline__ void chunk_range(const FgtList& L, int c, int64_t* begin, int64_t* end) {
  *begin = (int64_t)c * L.chunk;
  *end = min(*begin + L.chunk, L.nrec);
}

// Counts per bin of the CTA's chunk.
__global__ void __launch_bounds__(kWarps * 32) fgt_count_kernel(const FgtList* lists, const int* chunk_list) {
  __shared__ int hist[kFgtMaxBins];
  const int li = chunk_list[blockIdx.x];
  const FgtList L = lists[li];
  for (int b = threadIdx.x; b < L.nbins; b += blockDim.x) hist[b] = 0;
  __syncthreads();
  int64_t r0, r1;
  chunk_range(L, (int)blockIdx.x - L.chunk0, &r0, &r1);
  for (int64_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
    const int b = bin_of(L, i);
    if (b >= 0) atomicAdd(&hist[b], 1);
  }
  __syncthreads();
  int* out = L.counts + (int64_t)((int)blockIdx.x - L.chunk0) * L.nbins;
  for (int b = threadIdx.x; b < L.nbins; b += blockDim.x) out[b] = hist[b];
}

// One CTA per list: counts -> positions of every (chunk, bin), and the bins' starts.
__global__ void __launch_bounds__(1024) fgt_scan_kernel(const FgtList* lists) {
  __shared__ int sum[kFgtMaxBins];
  const FgtList L = lists[blockIdx.x];
  const int b = threadIdx.x;
  int run = 0;
  if (b < L.nbins)
    for (int c = 0; c < L.nchunks; ++c) {
      int* p = L.counts + (int64_t)c * L.nbins + b;
      const int v = *p;
      *p = run;
      run += v;
    }
  sum[b] = run;
  __syncthreads();
  for (int o = 1; o < kFgtMaxBins; o <<= 1) {
    const int v = b >= o ? sum[b - o] : 0;
    __syncthreads();
    sum[b] += v;
    __syncthreads();
  }
  if (b < L.nbins) L.start[b] = sum[b] - run;
  if (b == L.nbins - 1) L.start[L.nbins] = sum[b];
}

// Record indices in bin order, those of a bin in list order.
__global__ void __launch_bounds__(kWarps * 32) fgt_sort_kernel(const FgtList* lists, const int* chunk_list) {
  __shared__ int pos[kWarps][kFgtMaxBins];
  const FgtList L = lists[chunk_list[blockIdx.x]];
  const int c = (int)blockIdx.x - L.chunk0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t r0, r1;
  chunk_range(L, c, &r0, &r1);
  const int64_t per = L.chunk / kWarps;
  const int64_t w0 = r0 + warp * per, w1 = min(w0 + per, r1);
  for (int b = lane; b < L.nbins; b += 32) pos[warp][b] = 0;
  __syncwarp();
  for (int64_t i = w0 + lane; i < w1; i += 32) {
    const int b = bin_of(L, i);
    if (b >= 0) atomicAdd(&pos[warp][b], 1);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < L.nbins; b += blockDim.x) {
    int run = L.start[b] + L.counts[(int64_t)c * L.nbins + b];
    for (int w = 0; w < kWarps; ++w) {
      const int v = pos[w][b];
      pos[w][b] = run;
      run += v;
    }
  }
  __syncthreads();
  for (int64_t i0 = w0; i0 < w1; i0 += 32) {
    const int64_t i = i0 + lane;
    const int b = i < w1 ? bin_of(L, i) : -1;
    const unsigned same = __match_any_sync(0xffffffffu, b);
    const int rank = __popc(same & ((1u << lane) - 1u));
    int at = 0;
    if (b >= 0) at = pos[warp][b];
    __syncwarp();
    if (b >= 0) {
      L.perm[at + rank] = (int)i;
      if (rank == 0) pos[warp][b] = at + __popc(same);
    }
    __syncwarp();
  }
}

// The moments of one bin and weight array: thread t sums the bin's records t,
// t + 256, ..., then the lanes and the warps in a fixed order.  Weight array 0
// is the primal one; 1 + 2 p and 2 + 2 p are d w and g of direction p, the
// latter's moments scaled by (n + 1) / (2 r).
__global__ void __launch_bounds__(kWarps * 32) fgt_moments_kernel(const FgtList* lists, const int* bin_list) {
  __shared__ double part[kWarps][kTerms];
  const int li = bin_list[blockIdx.x];
  const FgtList L = lists[li];
  const int b = (int)blockIdx.x - L.bin0, set = blockIdx.y;
  const int s0 = L.start[b], s1 = L.start[b + 1];
  if (s0 == s1) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double* w = set == 0 ? L.w : (set & 1) ? L.tw + (int64_t)(set >> 1) * L.tstride
                                               : L.tg + (int64_t)((set >> 1) - 1) * L.tstride;
  const double centre = L.origin + (2 * b + 1) * kR;
  double m[kTerms];
#pragma unroll
  for (int n = 0; n < kTerms; ++n) m[n] = 0.0;
  for (int q = s0 + (int)threadIdx.x; q < s1; q += kWarps * 32) {
    const int i = L.perm[q];
    const double u = (L.key[i] - centre) * (1.0 / kR);
    double v = w[i];
#pragma unroll
    for (int n = 0; n < kTerms; ++n) {
      m[n] += v;
      v *= u;
    }
  }
#pragma unroll
  for (int n = 0; n < kTerms; ++n) {
    const double v = warp_sum_fixed(m[n]);
    if (lane == 0) part[warp][n] = v;
  }
  __syncthreads();
  if (threadIdx.x < kTerms) {
    double v = 0.0;
    for (int q = 0; q < kWarps; ++q) v += part[q][threadIdx.x];
    if (set > 0 && !(set & 1)) v *= (threadIdx.x + 1) * (1.0 / (2.0 * kR));
    L.moments[((int64_t)set * kTerms + threadIdx.x) * L.nbins + b] = v;
  }
}

// Whether n terms do at this |tau| (its upper 32 bits): the next one is below
// 1e-16 of the smallest term of the bin, (|tau|/8)^n / n! exp(|tau|/8).
__device__ __forceinline__ bool enough(int n, int hi) {
  return (n == 12 && hi < 0x3ffe0000) ||   // 1.875
         (n == 16 && hi < 0x40140000) ||   // 5
         (n == 20 && hi < 0x40238000) ||   // 9.75
         (n == 24 && hi < 0x402e8000);     // 15.25
}

// One warp per (list, output, frequency): lanes over the bins.
__global__ void __launch_bounds__(kWarps * 32) fgt_eval_kernel(LehmannArgs A, const FgtList* lists, int nlists,
                                                              const int* first_warp, int nwarps) {
  const int wid = (int)(blockIdx.x * kWarps + (threadIdx.x >> 5)), lane = threadIdx.x & 31, out = blockIdx.y;
  if (wid >= nwarps) return;
  int li = 0;
  while (li + 1 < nlists && first_warp[li + 1] <= wid) ++li;
  const FgtList L = lists[li];
  const int j = wid - first_warp[li];
  const int k = A.omega_idx[L.omega_first + j];
  const double t = L.gauss ? (A.omega[k] / A.dn[L.shell]) * A.inv_bt
                           : (A.log_omega[k] - A.log_dn[L.shell]) * A.inv_b - A.b_quarter;
  // weight arrays of this output: the primal, or d w and g of a direction
  const double* M0 = L.moments + (int64_t)(out == 0 ? 0 : 2 * out - 1) * kTerms * L.nbins;
  const double* M1 = M0 + (int64_t)kTerms * L.nbins;
  double acc = 0.0;
  for (int b = lane; b < L.nbins; b += 32) {
    if (L.start[b] == L.start[b + 1]) continue;
    const double centre = L.origin + (2 * b + 1) * kR;  // exact: the origin is a multiple of 2 r
    const double tau = t - centre;
    if (fabs(tau) > 27.4) {  // exp(-(|tau| - r)^2) is 0, and so is the term of a finite weight
      if (!is_finite(M0[b])) acc = __longlong_as_double(0x7ff8000000000000ll);
      continue;
    }
    const double back = tau - t, err = (t - (tau - back)) - (centre + back);  // t - centre = tau + err
    const double sq = tau * tau, g = exp(-sq);
    double bm = 0.0, bn = fma(-g, fma(2.0 * tau, err, fma(tau, tau, -sq)), g), sum = 0.0;
    const double x = 2.0 * kR * tau;
    const int at = __double2hiint(fabs(tau));
    if (out == 0) {
#pragma unroll
      for (int n = 0; n < kTerms; ++n) {
        if (enough(n, at)) break;
        sum = fma(M0[(int64_t)n * L.nbins + b], bn, sum);
        const double bp = fma(x, bn, -2.0 * kR * kR * bm) * (1.0 / (n + 1));
        bm = bn;
        bn = bp;
      }
    } else {
#pragma unroll
      for (int n = 0; n < kTerms; ++n) {
        if (enough(n, at)) break;
        sum = fma(M0[(int64_t)n * L.nbins + b], bn, sum);
        const double bp = fma(x, bn, -2.0 * kR * kR * bm) * (1.0 / (n + 1));
        sum = fma(M1[(int64_t)n * L.nbins + b], bp, sum);
        bm = bn;
        bn = bp;
      }
    }
    acc += sum;
  }
  acc = warp_sum_fixed(acc);
  if (lane == 0) (out == 0 ? L.part : L.tpart + (int64_t)(out - 1) * L.tpart_stride)[j] = acc;
}

}  // namespace

void launch_fgt(const LehmannArgs& a, const FgtList* lists, int nlists, const int* chunk_list, int nchunks,
                const int* bin_list, int nbins, const int* first_warp, int nwarps, int ntan, cudaStream_t s) {
  if (nlists <= 0) return;
  fgt_count_kernel<<<nchunks, kWarps * 32, 0, s>>>(lists, chunk_list);
  fgt_scan_kernel<<<nlists, kFgtMaxBins, 0, s>>>(lists);
  fgt_sort_kernel<<<nchunks, kWarps * 32, 0, s>>>(lists, chunk_list);
  fgt_moments_kernel<<<dim3(nbins, 1 + 2 * ntan), kWarps * 32, 0, s>>>(lists, bin_list);
  fgt_eval_kernel<<<dim3((nwarps + kWarps - 1) / kWarps, 1 + ntan), kWarps * 32, 0, s>>>(a, lists, nlists, first_warp,
                                                                                    nwarps);
}

}  // namespace nrg
