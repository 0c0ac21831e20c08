// Rank-revealing factor of a density matrix: P = C C^T by Cholesky with
// diagonal pivoting.
//
// K(P) is cheapest from r columns with P = C C^T, r the rank (the occupied
// orbitals of a closed-shell density). An eigendecomposition gives them, but
// its tridiagonalization is a chain of n grid-wide steps (1.1 ms for n = 180,
// 2.3 ms for n = 318, 11 ms for n = 960). A density is positive semidefinite,
// so Cholesky with the largest remaining diagonal as pivot gives them in r
// steps and stops by itself: Higham, "Analysis of the Cholesky decomposition
// of a semi-definite matrix" (1990), bounds its error by a small multiple of
// r eps |P|. Whether P was positive semidefinite is read off the residual
// P - C C^T, every element of which is checked; the caller takes the
// eigensolver when it is not small.
#include "internal.h"

#include <algorithm>
#include <cstring>

namespace dfjk {
namespace {

constexpr int kCta = 8;         // CTAs per cluster, one cluster per spin channel
constexpr int kLanes = 8;       // k lanes (warps) per block
constexpr int kPer = 4;         // rows per lane and pass
constexpr int kRows = 32 * kPer;

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct Pivot {
  double v;
  long long i;
};

// the larger value, the lower index among equal ones
__device__ __forceinline__ Pivot better(Pivot a, Pivot b) {
  return b.v > a.v || (b.v == a.v && b.i < a.i) ? b : a;
}

// Columns Ct[k][i] (k < rank) of P[spin] for the cluster of blockIdx.x / 8;
// the rank out. Left-looking: step k forms column p of the residual from P
// and the k columns so far, C[i][k] = (P[p][i] - sum_q C[i][q] C[p][q]) /
// sqrt(d_p), and updates the residual diagonal d. Each CTA owns a run of rows
// (its part of d in shared memory); a warp per k lane sums every eighth q
// over up to 128 rows at a time. One cluster barrier per step carries the CTAs' pivot
// candidates (distributed shared memory, two sets of slots) and makes the new
// column visible. Bound by that barrier and the L2 latency of the pivot row,
// about 2 us a step, and past some hundred columns by the reads of the former
// ones, n r^2 / 2 values in all on eight SMs.
// A residual diagonal only falls, so one below -accept times the largest diagonal
// shows that the factor would be refused: its CTA sends an infinite candidate, and
// every CTA stops with rank -1 (a difference of densities after the columns of its
// positive part).
__global__ void __cluster_dims__(kCta, 1, 1) __launch_bounds__(kLanes * 32)
    pivoted_cholesky_kernel(const double* __restrict__ Pall, int64_t n, int64_t max_rank,
                            double rel_tol, double accept, double* Ctall,
                            LowRankInfo* __restrict__ info) {
  extern __shared__ double sm[];
  __shared__ double red[kLanes][kRows];
  __shared__ Pivot slot[2][kCta];
  const int spin = blockIdx.x / kCta, cta = blockIdx.x % kCta;
  const double* P = Pall + (int64_t)spin * n * n;
  double* Ct = Ctall + (int64_t)spin * n * n;
  const int64_t per = (n + kCta - 1) / kCta;
  const int64_t lo = cta * per, hi = lo + per < n ? lo + per : n;
  double* d = sm;            // residual diagonal of rows lo .. hi - 1 (-1: pivoted)
  double* crow = sm + per;   // C[p][0 .. k - 1]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  cluster_barrier();   // every CTA runs before anything is written into it
  Pivot best{-1.0, 0};
  if (warp == 0)
    for (int64_t i = lo + lane; i < hi; i += 32) {
      d[i - lo] = P[i * n + i];
      best = better(best, Pivot{d[i - lo], i});
    }
  double first = 0.0;
  int64_t k = 0;
  for (;; ++k) {
    if (warp == 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        Pivot q{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
        best = better(best, q);
      }
      if (lane < kCta) {
        // this CTA's candidate into slot [k & 1][cta] of CTA `lane`
        uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(&slot[k & 1][cta])), r;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(lane));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(best.v) : "memory");
        asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(r + 8), "l"(best.i) : "memory");
      }
      __syncwarp();
    }
    cluster_barrier();
    Pivot p = slot[k & 1][0];
#pragma unroll
    for (int c = 1; c < kCta; ++c) p = better(p, slot[k & 1][c]);
    if (k == 0) first = p.v;
    if (p.v == INFINITY) {
      k = -1;
      break;
    }
    // the same decision in every CTA: all read the same eight candidates
    if (k == max_rank || !(p.v > rel_tol * first) || !(p.v > 0.0)) break;
    for (int64_t q = threadIdx.x; q < k; q += kLanes * 32) crow[q] = __ldcg(Ct + q * n + p.i);
    __syncthreads();
    const double inv = 1.0 / sqrt(p.v);
    best = Pivot{-1.0, 0};
    for (int64_t r0 = lo; r0 < hi; r0 += kRows) {
      double sum[kPer] = {};
#pragma unroll 4
      for (int64_t q = warp; q < k; q += kLanes) {
        const double c = crow[q];
        const double* col = Ct + q * n + r0 + lane;
#pragma unroll
        for (int u = 0; u < kPer; ++u)
          if (r0 + lane + 32 * u < hi) sum[u] += col[32 * u] * c;
      }
#pragma unroll
      for (int u = 0; u < kPer; ++u) red[warp][lane + 32 * u] = sum[u];
      __syncthreads();
      if (warp == 0) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          const int64_t i = r0 + lane + 32 * u;
          if (i >= hi) break;
          double t = 0.0;
#pragma unroll
          for (int w = 0; w < kLanes; ++w) t += red[w][lane + 32 * u];
          double di = d[i - lo], c = 0.0;
          bool below = k == 0 && di < -accept * first;
          if (i == p.i) {
            c = sqrt(p.v);
            di = -1.0;
          } else if (di >= 0.0) {
            // (rounding can leave a residual diagonal just below zero: its row
            // is finished then, as a pivoted one is)
            c = (P[p.i * n + i] - t) * inv;
            di -= c * c;
            below = di < -accept * first;
          }
          d[i - lo] = di;
          Ct[k * n + i] = c;
          if (below) best = Pivot{INFINITY, i};
          else if (di >= 0.0) best = better(best, Pivot{di, i});
        }
      }
      __syncthreads();
    }
  }
  // (the last barrier of the loop: no CTA still writes into another's slots)
  if (cta == 0 && threadIdx.x == 0) info->rank[spin] = (int)k;
}

// worst[spin] = max |P - C C^T| over every element, and scale[spin] = max |P|
// (bits of non-negative doubles order as integers); 32 x 32 tiles, the rank
// read on the device
__global__ void __launch_bounds__(256) residual_kernel(const double* __restrict__ Pall, int64_t n,
                                                       const double* __restrict__ Ctall,
                                                       LowRankInfo* __restrict__ info) {
  __shared__ double A[32][33], B[32][33];
  const int spin = blockIdx.z;
  const double* P = Pall + (int64_t)spin * n * n;
  const double* Ct = Ctall + (int64_t)spin * n * n;
  const int r = info->rank[spin];
  const int64_t i0 = blockIdx.y * 32, j0 = blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int q0 = 0; q0 < r; q0 += 32) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int q = q0 + ty + 8 * u;
      A[ty + 8 * u][tx] = q < r && i0 + tx < n ? Ct[(int64_t)q * n + i0 + tx] : 0.0;
      B[ty + 8 * u][tx] = q < r && j0 + tx < n ? Ct[(int64_t)q * n + j0 + tx] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int q = 0; q < 32; ++q) {
      const double b = B[q][tx];
#pragma unroll
      for (int u = 0; u < 4; ++u) s[u] += A[q][ty + 8 * u] * b;
    }
    __syncthreads();
  }
  double w = 0.0, m = 0.0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int64_t i = i0 + ty + 8 * u, j = j0 + tx;
    if (i < n && j < n) {
      const double v = P[i * n + j];
      w = fmax(w, fabs(v - s[u]));
      m = fmax(m, fabs(v));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    w = fmax(w, __shfl_xor_sync(0xffffffffu, w, o));
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  if (tx == 0) {
    atomicMax(&info->worst[spin], (unsigned long long)__double_as_longlong(w));
    atomicMax(&info->scale[spin], (unsigned long long)__double_as_longlong(m));
  }
}

// sum_q Ct[q][i] H[q][j], H[q][j] = (cos + sin)(2 pi q j / r) / sqrt r (Hartley's
// matrix, orthogonal and symmetric for every r), at out[i][j] (rows of r rounded up
// to even, zero there) or out[j][i]. The r values that H consists of, by q j mod r,
// in shared memory. A block has 32 rows and eight columns, so that a few dozen
// orbitals already give some forty blocks (those past r leave at once); bound by
// the latency of the loads of Ct.
constexpr int kSpRows = 32, kSpCols = 8;
__global__ void __launch_bounds__(kSpRows * kSpCols) spread_kernel(const double* __restrict__ Ct,
                                                                   int64_t n, const int* __restrict__ rank,
                                                                   bool rows, double* __restrict__ out) {
  extern __shared__ double cas[];
  const int r = *rank, ncp = rows ? r + (r & 1) : r;
  if ((int)blockIdx.y * kSpCols >= ncp) return;   // (r may be -1)
  for (int t = threadIdx.x; t < r; t += kSpRows * kSpCols) {
    double sn, cs;
    sincospi(2.0 * t / r, &sn, &cs);
    cas[t] = (cs + sn) / sqrt((double)r);
  }
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)kSpRows + threadIdx.x % kSpRows;
  const int j = blockIdx.y * kSpCols + threadIdx.x / kSpRows;
  if (i >= n || j >= ncp) return;
  double acc = 0.0;
  if (j < r) {
    int t = 0;
#pragma unroll 8
    for (int q = 0; q < r; ++q) {
      acc += Ct[q * n + i] * cas[t];
      t += j;
      if (t >= r) t -= r;
    }
  }
  out[rows ? i * ncp + j : j * n + i] = acc;
}

size_t chol_smem(int64_t n) { return (size_t)((n + kCta - 1) / kCta + n) * sizeof(double); }

}  // namespace

bool low_rank_supported(int64_t n) { return chol_smem(n) <= (size_t)200 << 10; }

bool LowRankInfo::within(int sp, double tol) const {
  double w, m;
  std::memcpy(&w, &worst[sp], sizeof w);
  std::memcpy(&m, &scale[sp], sizeof m);
  return w <= tol * m;
}

void launch_low_rank(const double* P, int64_t n, int nspin, int64_t max_rank, double* Ct,
                     double accept, LowRankInfo* info, cudaStream_t s) {
  const size_t smem = chol_smem(n);
  allow_shared(pivoted_cholesky_kernel);
  pivoted_cholesky_kernel<<<kCta * nspin, kLanes * 32, smem, s>>>(P, n, std::min(max_rank, n), kLowRankTol,
                                                                   accept, Ct, info);
  DFJK_LAUNCHED();
  const unsigned t = (unsigned)((n + 31) / 32);
  residual_kernel<<<dim3(t, t, (unsigned)nspin), 256, 0, s>>>(P, n, Ct, info);
  DFJK_LAUNCHED();
}

void spread_columns(const double* Ct, int64_t n, int64_t max_rank, const int* rank, bool rows,
                    double* out, cudaStream_t s) {
  max_rank = std::max<int64_t>(1, std::min(max_rank, n));
  allow_shared(spread_kernel);
  const dim3 grid((unsigned)((n + kSpRows - 1) / kSpRows), (unsigned)((max_rank + kSpCols) / kSpCols));
  spread_kernel<<<grid, kSpRows * kSpCols, (size_t)max_rank * sizeof(double), s>>>(Ct, n, rank, rows, out);
  DFJK_LAUNCHED();
}

}  // namespace dfjk
