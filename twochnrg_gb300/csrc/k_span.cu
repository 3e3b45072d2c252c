// Householder tridiagonalization of one block by a group of many SMs (FP64):
// the blocks whose rows do not fit in a cluster's shared memory.
//
// The scheme is the row kernel's (k_rows.cu): complete rows dealt to the CTAs
// (row r in CTA r mod G), the unnormalized reflector u = x - beta e_1, the sweep
// over the rows started from x while a warp of its own forms the scalars, one
// all-gather of (y, next column) per column.  What differs:
//  * the group is any number of CTAs of a cooperative grid, so the gather goes
//    through L2.  Its pairs carry their own readiness: an entry holds kEmpty
//    until its value is there, and the reader polls the entry itself, which
//    saves the fence, the counter and the second round trip of a grid barrier
//    (two of which per column were a third of tridiag_grid_kernel's time on one
//    block of 1900 states).  Three buffers in turn; a CTA empties its entries of
//    a buffer two steps after they were read.
//  * rows beyond the shared memory stay in place in the matrix (L2): the first
//    ones, which are finished first.
//  * rows that do not make up one per warp are split over the four warps by
//    columns.
//  * the pending update is kept as A - p y^T - q u^T with p_r = tau u_r and
//    q_r = tau y_r - 2 h u_r per row, so that no w is formed over the columns:
//    three instead of five FP64 operations per column and CTA beside the sweep.
//
// What bounds it: per column the gather through L2 (2 us), the scalars after it and
// the replicated vector operations, 4 to 6 us, beside the sweep's FP64 work, 3 FMA
// per element at 1.7 per cycle and SM.  One block (kernel with its launch): 640
// states in 8.8 / 5.2 / 3.6 / 3.5 ms on 16 / 32 / 96 / 152 CTAs, by the cluster
// kernel of k_tridiag.cu 12.9; 1300 states in 14 ms on 152 CTAs; 1901 states in 26.7
// ms, 24.9 with the gather as it is now (13 us per column), by tridiag_grid_kernel
// 52.7 (27.7).
//
// Waits: a poll per entry and share, bounded by the clock; every CTA runs before
// the first one (a barrier of the cooperative grid).
//
// Outputs as tridiag_kernel's: d, e, tau, and u_j in row j, columns j+1..n-1.
#include <cooperative_groups.h>

#include "nrg_device.cuh"

namespace cg = cooperative_groups;

namespace nrg {

namespace {

constexpr int kSweep = 4;                        // sweep warps, one per sub-partition
constexpr int kSpanThreads = (kSweep + 2) * 32;  // + the scalar warp + one that empties the exchange entries
constexpr int kPad = 32;                         // zeros past the vectors' ends
constexpr int kSplitCols = 128;                  // at least a strip of columns per warp
constexpr int kPollCols = 768;                   // from here on the gather waits for the shares
constexpr int kBufs = 3;
constexpr long long kEmpty = -1;                 // a NaN that no FP64 operation gives

__device__ __forceinline__ double2 load_pair(const double2* p) {
  double2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_pair(double2* p, double a, double b) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ double load_share(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_share(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool is_full(double v) { return __double_as_longlong(v) != kEmpty; }
// What is sent never looks empty, whatever NaN came in with the block.
__device__ __forceinline__ double filled(double v) { return is_full(v) ? v : __longlong_as_double(0x7ff8000000000000ll); }
__device__ __forceinline__ bool is_full(double2 v) { return is_full(v.x) && is_full(v.y); }

// A group's exchange area in global memory.
struct SpanEx {
  double2* pair;    // copies x kBufs x maxn
  double* share;    // copies x kBufs x G
  unsigned* count;  // barrier of the group
};

__host__ __device__ inline size_t span_ex_doubles(int maxn, int G, int R) {
  return (2 * kBufs * (size_t)maxn + kBufs * (size_t)G) * R + 2 + (G & R & 1);
}
// Shared memory besides the rows.
__host__ __device__ inline size_t span_fixed_doubles(int n, int G) {
  return 3 * ((size_t)n + (n & 1) + kPad) + 4 * (((size_t)n + G - 1) / G) + kSweep * 32 + kSweep * kSweep + 6 + 2;
}

struct SpanSm {
  double* x;     // 2 x ldv: u of the last step, x of this one
  double* y;     // y of the last step
  double* tot;   // row products and next-column elements of the CTA's own rows
  double* acol;
  double* p;     // -p_r and -q_r of the own rows
  double* q;
  double* part;  // norm partials of the sweep threads
  double* quart; // row products of the split rows, by warp
  double* sc;    // scalars of the step
  double* rows;
  int ldv, ld;
};

enum { SC_BETA, SC_TU1, SC_B, SC_H2 };

// RT of the CTA's rows at `row` (own rows i0, i0 + di, ...): the pending update
// and the product with x over strips s0 .. s1-1 of columns j+1..n-1, whose sums
// go to out[k * od].
template <int RT>
__device__ __forceinline__ void span_rows(const SpanSm& S, double* row, int64_t ld, int n, int j, int i0, int di, int s0,
                                          int s1, double* out, int od, const double* xc, const double* uo) {
  const int lane = threadIdx.x & 31, step = (int)(di * ld);
  double p[RT], q[RT], acc[RT];
#pragma unroll
  for (int k = 0; k < RT; ++k) {
    p[k] = S.p[i0 + k * di];
    q[k] = S.q[i0 + k * di];
    acc[k] = 0.0;
  }
  int c = j + 1 + 32 * s0 + lane;
  auto col = [n](int k) { return min(k, n - 1); };  // past the row's end the vectors are 0
  double u = uo[c], y = S.y[c], x = xc[c], r[RT];
#pragma unroll
  for (int k = 0; k < RT; ++k) r[k] = row[k * step + col(c)];
  for (int s = s0; s < s1; ++s, c += 32) {
    double un = 0.0, yn = 0.0, xn = 0.0, rn[RT];
    if (s + 1 < s1) {  // the next strip is loaded before this one's FMAs
      un = uo[c + 32]; yn = S.y[c + 32]; xn = xc[c + 32];
#pragma unroll
      for (int k = 0; k < RT; ++k) rn[k] = row[k * step + col(c + 32)];
    }
#pragma unroll
    for (int k = 0; k < RT; ++k) r[k] = fma(q[k], u, r[k]);
#pragma unroll
    for (int k = 0; k < RT; ++k) r[k] = fma(p[k], y, r[k]);
#pragma unroll
    for (int k = 0; k < RT; ++k) acc[k] = fma(r[k], x, acc[k]);
#pragma unroll
    for (int k = 0; k < RT; ++k) {
      if (c < n) row[k * step + c] = r[k];
      if (s == 0 && lane == 0) S.acol[i0 + k * di] = r[k];
      r[k] = rn[k];
    }
    u = un; y = yn; x = xn;
  }
  if (RT <= 2) {
#pragma unroll
    for (int k = 0; k < RT; ++k) acc[k] = warp_sum_fixed(acc[k]);
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < RT; ++k) out[k * od] = acc[k];
    }
  } else {
    const double v = reduce_rows<RT>(acc);
    constexpr int kStep = 32 / RT;
    if (lane % kStep == 0) out[(lane / kStep) * od] = v;
  }
}

// The warp's rows among own rows [first, end): `base` is own row i = 0's place.
__device__ __forceinline__ void span_sweep(const SpanSm& S, double* base, int64_t ld, int first, int end, int n, int j,
                                           const double* xc, const double* uo) {
  const int warp = threadIdx.x >> 5, ns = (n - j - 1 + 31) >> 5;
  int i = first + warp;
#pragma unroll 1
  for (; i + 3 * kSweep < end; i += 4 * kSweep)
    span_rows<4>(S, base + i * ld, ld, n, j, i, kSweep, 0, ns, S.tot + i, kSweep, xc, uo);
  if (i + kSweep < end) {
    span_rows<2>(S, base + i * ld, ld, n, j, i, kSweep, 0, ns, S.tot + i, kSweep, xc, uo);
    i += 2 * kSweep;
  }
  if (i < end) span_rows<1>(S, base + i * ld, ld, n, j, i, kSweep, 0, ns, S.tot + i, kSweep, xc, uo);
}
// Own rows [first, end), at most kSweep - 1: every warp takes a quarter of the
// columns.
__device__ __forceinline__ void span_split(const SpanSm& S, double* base, int64_t ld, int first, int end, int n, int j,
                                           const double* xc, const double* uo) {
  const int warp = threadIdx.x >> 5, ns = (n - j - 1 + 31) >> 5;
  const int s0 = ns * warp / kSweep, s1 = ns * (warp + 1) / kSweep;
  int i = first;
  if (i + 1 < end) {
    span_rows<2>(S, base + i * ld, ld, n, j, i, 1, s0, s1, S.quart + warp, kSweep, xc, uo);
    i += 2;
  }
  if (i < end) span_rows<1>(S, base + i * ld, ld, n, j, i, 1, s0, s1, S.quart + (i - first) * kSweep + warp, kSweep, xc, uo);
}

// The gathered y and the first part of the next x, L entries per thread in flight
// (a round trip through L2 each).
template <int L>
__device__ __forceinline__ void gather(const SpanSm& S, const double2* pair, int j, int n, double tu1, double* uo,
                                       volatile int* dead, int* flag, long long limit) {
#pragma unroll 1
  for (int c = j + 1 + (int)threadIdx.x; c < n; c += L * kSweep * 32) {
    double2 v[L];
#pragma unroll
    for (int k = 0; k < L; ++k) v[k] = load_pair(pair + min(c + k * kSweep * 32, n - 1));
#pragma unroll
    for (int k = 0; k < L; ++k) {
      const int ck = c + k * kSweep * 32;
      if (ck >= n) break;
      if (!is_full(v[k]) && !*dead) {
        const long long t0 = clock64();
        do {
          if (clock64() - t0 > limit) { *dead = 1; atomicOr(flag, DEV_TIMEOUT); }
          v[k] = load_pair(pair + ck);
        } while (!is_full(v[k]) && !*dead);
      }
      uo[ck] = fma(-tu1, v[k].x, v[k].y);
      S.y[ck] = v[k].x;
    }
  }
}

// Barrier of the group: every CTA arrives once per call.
__device__ __forceinline__ void group_barrier(const SpanEx& E, unsigned target, volatile int* dead, int* flag,
                                              long long limit) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(E.count, 1u);
    const long long t0 = clock64();
    while (!*dead) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(E.count) : "memory");
      if (v >= target) break;
      if (clock64() - t0 > limit) { *dead = 1; atomicOr(flag, DEV_TIMEOUT); }
    }
    __threadfence();
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kSpanThreads, 1) tridiag_span_kernel(TridiagArgs A, SpanArgs P) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int dead_s;
  const int R = P.copies, G = P.G, group = (int)blockIdx.x / G, rank = (int)blockIdx.x % G;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  volatile int* dead = &dead_s;
  SpanEx E;
  {
    double* w = P.work + (size_t)group * span_ex_doubles(A.maxn, G, R);
    E.pair = (double2*)w;
    E.share = w + 2 * kBufs * (size_t)A.maxn * R;
    E.count = (unsigned*)(E.share + (size_t)kBufs * G * R + (G & R & 1));
    const double empty = __longlong_as_double(kEmpty);
    for (int k = rank * kSpanThreads + tid; k < kBufs * A.maxn * R; k += G * kSpanThreads) store_pair(E.pair + k, empty, empty);
    for (int k = rank * kSpanThreads + tid; k < kBufs * G * R; k += G * kSpanThreads) store_share(E.share + k, empty);
    if (rank == 0 && tid == 0) *E.count = 0;
    if (tid == 0) *dead = 0;
  }
  cg::this_grid().sync();  // every CTA runs; the exchange areas are empty

  uint32_t g = 0;         // steps done over all blocks: step g uses buffer g % kBufs
  unsigned arrived = 0;   // target of the group's barrier
  for (int qi = P.first[group]; qi < P.first[group + 1]; ++qi) {
    const int b = P.list[qi];
    const int n = A.bsize[b];
    double* H = A.H + A.hoff[b];
    const int so = A.soff[b];
    if (n > A.maxn || n < 3 || span_fixed_doubles(n, G) > (size_t)P.smem_doubles) {
      if (rank == 0 && tid == 0) atomicOr(A.flag, DEV_SIZE);
      continue;
    }
    const int own = (n - rank + G - 1) / G;
    SpanSm S;
    S.ldv = n + (n & 1) + kPad;
    S.ld = n | 1;
    {
      const int om = (n + G - 1) / G;
      double* p = sm;
      S.x = p; p += 2 * S.ldv;
      S.y = p; p += S.ldv;
      S.tot = p; p += om;
      S.acol = p; p += om;
      S.p = p; p += om;
      S.q = p; p += om;
      S.part = p; p += kSweep * 32;
      S.quart = p; p += kSweep * kSweep;
      S.sc = p; p += 6;
      S.rows = p;
    }
    const int room = (P.smem_doubles - (int)span_fixed_doubles(n, G)) / S.ld;
    const int ng = max(0, own - room);  // own rows [0, ng) stay in the matrix
    double* gbase = H + (int64_t)rank * n;
    const int64_t gld = (int64_t)G * n;
    double* sbase = S.rows - (int64_t)ng * S.ld;
    for (int i = ng + warp; i < own; i += kSpanThreads / 32) {
      const double* src = gbase + i * gld;
      double* dst = sbase + i * S.ld;
      for (int c = lane; c < n; c += 32) dst[c] = __ldcg(src + c);
    }
    for (int c = tid; c < S.ldv; c += kSpanThreads) {
      S.x[c] = c < n ? __ldcg(H + c) : 0.0;  // row 0: the first x
      S.x[S.ldv + c] = 0.0;                  // no update pending
      S.y[c] = 0.0;
    }
    for (int i = tid; i < own; i += kSpanThreads) S.p[i] = S.q[i] = 0.0;
    group_barrier(E, arrived += G, dead, A.flag, P.wait_cycles);  // row 0 is read before it is overwritten
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
      // this step's buffer of copy 0, and the copy that this CTA reads
      double2* pair0 = E.pair + (size_t)(g % kBufs) * A.maxn;
      double* share0 = E.share + (size_t)(g % kBufs) * G;
      const double2* pair = pair0 + (size_t)(rank % R) * kBufs * A.maxn;
      const double* share = share0 + (size_t)(rank % R) * kBufs * G;
      const int i0 = j + 1 <= rank ? 0 : (j + 1 - rank + G - 1) / G;  // first own row of the trailing matrix
      // Rows that do not make up one per warp are split by columns: with 12 rows
      // per CTA and fewer as the matrix shrinks the warps' shares are otherwise
      // up to a third apart.
      const int isplit = m >= kSplitCols ? own - (own - max(i0, min(ng, own))) % kSweep : own;
      auto total = [&](int i) {
        if (i < isplit) return S.tot[i];
        const double* q = S.quart + (i - isplit) * kSweep;
        return (q[0] + q[1]) + (q[2] + q[3]);
      };
      double tau = 0.0, beta, u1, tu1 = 0.0, rs = 0.0, sum = 1.0;
      if (warp == kSweep) {
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
        __syncwarp();
      } else if (warp == kSweep + 1) {
        // The next step's entries, read by every CTA before it sent the entries
        // that this one gathered last, become empty again, before this step's
        // share goes out.  The fence costs 2000 cycles or more, beside the sweep;
        // it also orders the shares read in the last step before this step's polls.
        const double empty = __longlong_as_double(kEmpty);
        double2* np = E.pair + (size_t)((g + 1) % kBufs) * A.maxn;
        for (int k = 0; k < R; ++k, np += kBufs * A.maxn)
          for (int i = lane; i < own; i += 32)
            if (rank + G * i + 1 >= j) store_pair(np + rank + G * i, empty, empty);
        if (lane < R) store_share(E.share + (size_t)((g + 1) % kBufs + kBufs * lane) * G + rank, empty);
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
      } else {
        if (i0 < ng) span_sweep(S, gbase, gld, i0, ng, n, j, xc, uo);
        span_sweep(S, sbase, S.ld, max(i0, ng), isplit, n, j, xc, uo);
        if (isplit < own) span_split(S, sbase, S.ld, isplit, own, n, j, xc, uo);
      }
      __syncthreads();
      if (warp == kSweep) {
        // The own rows' share of u.y, also from a CTA without rows: every CTA
        // so waits for every other in every step.
        double dv = 0.0;
#pragma unroll 1
        for (int i = i0 + lane; i < own; i += 32) {
          const int r = rank + G * i;
          dv = fma(r == j + 1 ? u1 : xc[r], fma(-beta, S.acol[i], total(i)), dv);
        }
        dv = warp_sum_fixed(dv);
        if (lane < R) store_share(share0 + (size_t)kBufs * lane * G + rank, dv);
        tau = rs * fast_rcp(sum);  // 2 / u.u = 1 / (|x| (|x| + |alpha|))
        if (rank == j % G && lane == 0) {
          A.d[so + j] = xc[j]; A.e[so + j] = beta; A.tau[so + j] = tau;
          H[(int64_t)j * n + j + 1] = u1;
        }
        double2 v1 = load_pair(pair + j + 1);
        dv = 0.0;
#pragma unroll 1
        for (int q0 = 0; q0 < G; q0 += 64) {  // two loads in flight
          const int qa = min(q0 + lane, G - 1), qb = min(q0 + lane + 32, G - 1);
          double va = load_share(share + qa), vb = load_share(share + qb);
          const long long t0 = clock64();
          while (!(is_full(va) && is_full(vb)) && !*dead) {
            if (clock64() - t0 > P.wait_cycles) { *dead = 1; atomicOr(A.flag, DEV_TIMEOUT); }
            va = load_share(share + qa);
            vb = load_share(share + qb);
          }
          dv += (q0 + lane < G ? va : 0.0) + (q0 + lane + 32 < G ? vb : 0.0);
        }
        __syncwarp();
        if (m > kPollCols) asm volatile("barrier.cta.arrive 1, %0;" ::"n"((kSweep + 1) * 32) : "memory");
        dv = warp_sum_fixed(dv);
        if (!is_full(v1) && !*dead) {
          const long long t0 = clock64();
          do {
            if (clock64() - t0 > P.wait_cycles) { *dead = 1; atomicOr(A.flag, DEV_TIMEOUT); }
            v1 = load_pair(pair + j + 1);
          } while (!is_full(v1) && !*dead);
        }
        __syncwarp();
        const double t = tau * dv;  // of the block's scale, where tau^2 may leave the range
        if (lane == 0) {
          S.sc[SC_B] = fma(-tu1, t, tau * v1.x);
          S.sc[SC_H2] = tau * t;
          xc[j + 1] = u1;
        }
      } else if (warp < kSweep) {
        beta = S.sc[SC_BETA];
        tu1 = S.sc[SC_TU1];
#pragma unroll 1
        for (int i = i0 + lane; i < own; i += 32) {
          const double a = filled(S.acol[i]), y = filled(fma(-beta, a, total(i)));
          for (int k = warp; k < R; k += kSweep) store_pair(pair0 + (size_t)k * kBufs * A.maxn + rank + G * i, y, a);
        }
        if (rank == j % G)  // u_j into row j, which no CTA reads any more (the scalar warp writes u_1)
          for (int c = j + 2 + tid; c < n; c += kSweep * 32) H[(int64_t)j * n + c] = xc[c];
        // x of the next step: column j+1 of A - p y^T - q u^T, in two parts.
        // Few entries per thread are polled as they come.  Many would crowd the L2
        // lines that are still to be written: they are read once the scalar warp
        // has every share, when all are there or about to be.  One block of 1901 /
        // 1000 / 600 states: polled 2, 4, 8 deep 25.8, 26.0, 35.5 / 6.70, 6.96, 8.67
        // / 3.03, 3.14, 3.20 ms; after the shares 8 deep 25.0 / 6.85 / 3.11 ms.
        if (m > kPollCols) {
          asm volatile("barrier.cta.sync 1, %0;" ::"n"((kSweep + 1) * 32) : "memory");
          gather<8>(S, pair, j, n, tu1, uo, dead, A.flag, P.wait_cycles);
        } else {
          gather<2>(S, pair, j, n, tu1, uo, dead, A.flag, P.wait_cycles);
        }
      }
      __syncthreads();
      if (warp == kSweep) {  // the own rows' part of the update, one lane each
        const double h2 = S.sc[SC_H2];
#pragma unroll 1
        for (int i = i0 + lane; i < own; i += 32) {
          const int r = rank + G * i;
          const double u = xc[r];
          S.p[i] = -tau * u;
          S.q[i] = fma(h2, u, -tau * fma(-beta, S.acol[i], total(i)));
        }
      }
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
      }
      __syncthreads();
      double* t = xc; xc = uo; uo = t;
    }
    // The last 2 x 2 block: row n-2 is the last x; the corner has its update pending.
    if (rank == (n - 1) % G && tid == 0) {
      const int i = (n - 1) / G;
      double a = i < ng ? gbase[i * gld + n - 1] : sbase[i * S.ld + n - 1];
      a = fma(S.p[i], S.y[n - 1], fma(S.q[i], uo[n - 1], a));
      A.d[so + n - 2] = xc[n - 2];
      A.e[so + n - 2] = xc[n - 1];
      A.d[so + n - 1] = a;
      A.e[so + n - 1] = 0.0;
      A.tau[so + n - 2] = 0.0;
      A.tau[so + n - 1] = 0.0;
    }
    // All gathers are done: empty the own entries for the next block.
    group_barrier(E, arrived += G, dead, A.flag, P.wait_cycles);
    const double empty = __longlong_as_double(kEmpty);
    for (int k = tid; k < kBufs * R * own; k += kSpanThreads)
      store_pair(E.pair + (size_t)(k / own) * A.maxn + rank + G * (k % own), empty, empty);
    if (tid < kBufs * R) store_share(E.share + (size_t)tid * G + rank, empty);
  }
}

cudaError_t span_attributes() {
  return cudaFuncSetAttribute(tridiag_span_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem() - 1024);
}

// Room for the rows of the largest block, as far as there is any.
size_t span_smem_bytes(int maxn, int G) {
  const size_t all = sizeof(double) * (span_fixed_doubles(maxn, G) + ((size_t)maxn + G - 1) / G * (size_t)(maxn | 1));
  return std::min(all, (size_t)max_dyn_smem() - 1024);
}

}  // namespace

size_t tridiag_span_work(int maxn, int groups, int G, int copies) { return groups * span_ex_doubles(maxn, G, copies); }

bool tridiag_span_fits(int n) { return sizeof(double) * span_fixed_doubles(n, 16) <= (size_t)max_dyn_smem() - 1024; }

cudaError_t launch_tridiag_span(const TridiagArgs& a, SpanArgs p, int groups, cudaStream_t s) {
  if (p.G < 1 || groups < 1 || p.copies < 1 || p.copies > 32) return cudaErrorInvalidValue;
  cudaError_t err = span_attributes();
  if (err != cudaSuccess) return err;
  const size_t smem = span_smem_bytes(a.maxn, p.G);
  p.smem_doubles = (int)(smem / sizeof(double));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.G * groups), 1, 1);
  cfg.blockDim = dim3(kSpanThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, tridiag_span_kernel, a, p);
}

}  // namespace nrg
