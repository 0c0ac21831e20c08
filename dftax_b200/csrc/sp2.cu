// The SP2 projection of a small Fock matrix in one launch (scf.h).
//
// The projection's steps are a chain: X -> X^2 or 2X - X^2, the branch picked
// by the traces. Launched step by step (a GEMM and an update kernel each) a
// step of m = 90 costs 13 us of which the arithmetic is a fraction, and an SCF
// iteration takes some 34 steps. Here a cluster of eight CTAs keeps a full copy
// of X in each shared memory and runs every step: 8 x 8 tiles of the lower
// triangle of X^2 on the float64 tensor cores (X is symmetric, so rows serve
// as columns), spread over the 64 warps; the owners write the new tile and its
// mirror image to memory, laid out as in shared memory, and every CTA copies the
// new X back from L2 in one sweep of 16-byte asynchronous copies (stored
// straight into all eight shared memories, 16 scattered 8-byte remote stores per
// value, a step of m = 150 took 20 us). Two cluster barriers per step.
// Bound by those barriers and the L2 round trip.
#include "dmma.cuh"
#include "scf.h"

namespace dfjk {
namespace {

constexpr int kCta = 8, kWarps = 8;
constexpr int kTilesPerWarp = (kSp2ClusterMax / 8 * (kSp2ClusterMax / 8 + 1) / 2 + kCta * kWarps - 1) / (kCta * kWarps);
constexpr int kMaxTiles = kSp2ClusterMax / 8;

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// the address of this CTA's shared location `p` in CTA `cta` of the cluster
__device__ __forceinline__ uint32_t remote(const void* p, int cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(r)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(cta));
  return r;
}

__device__ __forceinline__ void remote_store(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// A: m x m symmetric (the lower triangle is read); Xout: the projector; rec:
// {steps, Tr X before the last step, 1 when converged}; Xg: scratch of mp rows of
// mp + 4 (mp = m rounded up to 8). The stopping rule is that of the stepwise
// path: the idempotency error Tr X - Tr X^2 below 1e-15 m, or below 1e-9 and not
// below its value two steps before. By then the traces no longer tell the
// branches apart, so X^2 and then 2X - X^2 follow, which square the errors of
// both ends of the spectrum (kSp2Extra steps).
__global__ void __cluster_dims__(kCta, 1, 1) __launch_bounds__(kWarps * 32)
    sp2_cluster_kernel(const double* __restrict__ A, int m, int nocc, int max_steps,
                       double* Xg, double* __restrict__ Xout, double* __restrict__ rec) {
  extern __shared__ __align__(16) double X[];   // [mp][P]
  __shared__ double tz[2][kMaxTiles];           // diagonal tiles' traces of X^2
  __shared__ double rlo[kWarps], rhi[kWarps];
  const int mt = (m + 7) / 8, mp = mt * 8, P = mp + 4;   // 4 past a multiple of 8: no bank conflicts
  const int cta = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int fr = lane >> 2, fk = lane & 3;
  for (int q = tid; q < mp * P; q += kWarps * 32) {
    const int i = q / P, j = q % P;
    double v = 0.0;
    if (i < m && j < m) v = i >= j ? A[(int64_t)j * m + i] : A[(int64_t)i * m + j];
    X[q] = v;
  }
  __syncthreads();
  // Gershgorin bounds of A (row r through column r)
  double lo = INFINITY, hi = -INFINITY;
  for (int r = tid; r < m; r += kWarps * 32) {
    double off = 0.0;
    for (int c = 0; c < m; ++c)
      if (c != r) off += fabs(X[c * P + r]);
    lo = fmin(lo, X[r * P + r] - off);
    hi = fmax(hi, X[r * P + r] + off);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) {
    rlo[warp] = lo;
    rhi[warp] = hi;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    lo = fmin(lo, rlo[w]);
    hi = fmax(hi, rhi[w]);
  }
  const double width = hi - lo;
  for (int q = tid; q < mp * P; q += kWarps * 32) {
    const int i = q / P, j = q % P;
    if (i < m && j < m) X[q] = width > 0.0 ? ((i == j ? hi : 0.0) - X[q]) / width : 0.0;
  }
  __syncthreads();
  cluster_barrier();   // every CTA runs before anything is written into it
  // this warp's tiles (ti >= tj) of the lower triangle
  const int nt = mt * (mt + 1) / 2, gw = cta * kWarps + warp;
  int ti[kTilesPerWarp], tj[kTilesPerWarp];
#pragma unroll
  for (int q = 0; q < kTilesPerWarp; ++q) {
    const int t = gw + q * kCta * kWarps;
    int a = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
    while ((a + 1) * (a + 2) / 2 <= t) ++a;
    while (a * (a + 1) / 2 > t) --a;
    ti[q] = t < nt ? a : -1;
    tj[q] = t - a * (a + 1) / 2;
  }
  double e1 = INFINITY, e2 = INFINITY, t1 = 0.0;
  const double N = (double)nocc;
  int it = 0, last = max_steps;
  bool done = false;
  for (; it < last; ++it) {
    double z[kTilesPerWarp][2];
#pragma unroll
    for (int q = 0; q < kTilesPerWarp; ++q) {
      if (ti[q] < 0) break;
      double c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
      const double* a = X + (8 * ti[q] + fr) * P + fk;
      const double* b = X + (8 * tj[q] + fr) * P + fk;
#pragma unroll 4
      for (int k = 0; k < mp; k += 8) {
        dmma_8x8x4(c0, a[k], b[k]);
        dmma_8x8x4(c1, a[k + 4], b[k + 4]);
      }
      z[q][0] = c0[0] + c1[0];
      z[q][1] = c0[1] + c1[1];
      if (ti[q] == tj[q]) {
        const double d = warp_sum((2 * fk == fr ? z[q][0] : 0.0) + (2 * fk + 1 == fr ? z[q][1] : 0.0));
        if (lane < kCta) remote_store(remote(&tz[it & 1][ti[q]], lane), d);
      }
    }
    double d = 0.0;
    for (int r = lane; r < m; r += 32) d += X[r * P + r];
    t1 = warp_sum(d);
    cluster_barrier();   // no CTA reads the old X any more; the traces have arrived
    const double t2 = warp_sum(lane < mt ? tz[it & 1][lane] : 0.0);
    const bool sq = done ? it == last - 2 : fabs(t2 - N) < fabs(2.0 * t1 - t2 - N);
    const double e = fabs(t1 - t2);
    if (!done && (e < 1e-15 * m || (e < 1e-9 && e >= e2))) {
      done = true;
      last = it + 1 + kSp2Extra;
    }
    e2 = e1;
    e1 = e;
    const bool bad = !(e < INFINITY);
#pragma unroll
    for (int q = 0; q < kTilesPerWarp; ++q) {
      if (ti[q] < 0) break;
      const int i = 8 * ti[q] + fr, j0 = 8 * tj[q] + 2 * fk;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int j = j0 + r;
        if (i < j) continue;   // a diagonal tile writes its lower half and the mirror image
        const double v = sq ? z[q][r] : 2.0 * X[i * P + j] - z[q][r];
        Xg[i * P + j] = v;
        Xg[j * P + i] = v;
      }
    }
    cluster_barrier();   // the new X is complete in memory (and visible: release, acquire)
    for (int q = tid; q < mp * P / 2; q += kWarps * 32) {
      // (the four doubles past a row's mp are never read)
      cp_async16(X + 2 * q, Xg + 2 * q, true);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (bad) break;      // (the same in every CTA: all see the same traces)
  }
  if (cta != 0) return;
  for (int q = tid; q < m * m; q += kWarps * 32) Xout[q] = X[q / m * P + q % m];
  if (tid == 0) {
    rec[0] = it;
    rec[1] = t1;
    rec[2] = done ? 1.0 : 0.0;
  }
}

}  // namespace

size_t sp2_cluster_bytes(int m) {
  const int mp = (m + 7) / 8 * 8;
  return (size_t)mp * (mp + 4) * sizeof(double);
}

void launch_sp2_cluster(const double* A, int m, int nocc, int max_steps, double* Xg, double* X,
                        double* rec, cudaStream_t s) {
  const size_t smem = sp2_cluster_bytes(m);
  allow_shared(sp2_cluster_kernel);
  sp2_cluster_kernel<<<kCta, kWarps * 32, smem, s>>>(A, m, nocc, max_steps, Xg, X, rec);
  DFJK_LAUNCHED();
}

}  // namespace dfjk
