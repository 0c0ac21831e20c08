// Hermite R integrals built by a group of lanes, for the kernels that give a
// warp (or part of one) to a shell pair or triple: the 2-center metric (md.cu)
// and the derivative integrals (grad3c.cuh, grad.cu).
#pragma once

#include "eri3c.cuh"

namespace dfjk {

// The Hermite R ladder of order M by a group of TL lanes: lane gl holds the
// entries h = gl + TL j, each with what its recursion reads packed into a word
// (order, axis, the second term's factor, the two entries).
template <int M, int TL>
struct HermiteGroup {
  static constexpr int NR = hcount(M), RJ = (NR + TL - 1) / TL;
  static_assert(M < 15 && NR <= 512, "packed table fields");
  uint32_t tab[RJ];

  __device__ __forceinline__ void init(int gl) {
#pragma unroll
    for (int j = 0; j < RJ; ++j) {
      const int h = gl + TL * j;
      tab[j] = 15u;   // past every order
      if (h < NR) {
        int t, u, v;
        hdecode(h, t, u, v);
        const int ax = v > 0 ? 2 : (u > 0 ? 1 : 0), k = v > 0 ? v : (u > 0 ? u : t);
        const int dt = ax == 0, du = ax == 1, dv = ax == 2;
        const int e1 = k > 0 ? hidx(t - dt, u - du, v - dv) : 0;
        const int e2 = k > 1 ? hidx(t - 2 * dt, u - 2 * du, v - 2 * dv) : 0;
        const int mul = k > 1 ? k - 1 : 0;
        tab[j] = (uint32_t)(t + u + v) | (uint32_t)ax << 4 | (uint32_t)mul << 6 |
                 (uint32_t)e1 << 10 | (uint32_t)e2 << 19;
      }
    }
  }

  // R_{tuv} (t + u + v <= M, packed by hidx) at (X, Y, Z), T = rho r^2, of the
  // Coulomb (omega = 0) or erf(omega r)/r operator, in sRa or sRb (the one
  // returned; NR doubles each, sB: M + 1). Whole warps call it together; it
  // ends with the lanes in step.
  __device__ __forceinline__ const double* run(double T, double rho, double omega, double X,
                                               double Y, double Z, const double* __restrict__ boys,
                                               const double* __restrict__ asym, double* sB,
                                               double* sRa, double* sRb, int gl) const {
    double sat = 1.0, rs = 1.0;
    if (omega > 0.0) {
      sat = omega * omega / (omega * omega + rho);
      rs = sqrt(sat);
    }
    const double x = -2.0 * rho * sat;
    for (int o = gl; o <= M; o += TL) {
      double f = rs * boys_order(o, sat * T, boys, asym);
      for (int k = 0; k < o; ++k) f *= x;
      sB[o] = f;
    }
    __syncwarp();
    double* src = sRa;
    double* dst = sRb;
    if (gl == 0) src[0] = sB[M];
    __syncwarp();
#pragma unroll 1
    for (int n = M - 1; n >= 0; --n) {
#pragma unroll
      for (int j = 0; j < RJ; ++j) {
        const uint32_t e = tab[j];
        const int ord = e & 15, ax = e >> 4 & 3, mul = e >> 6 & 15;
        if (ord > M - n) continue;
        double val;
        if (ord == 0) {
          val = sB[n];
        } else {
          val = (ax == 0 ? X : (ax == 1 ? Y : Z)) * src[e >> 10 & 511];
          if (mul) val += mul * src[e >> 19];
        }
        dst[gl + TL * j] = val;
      }
      __syncwarp();
      double* tmp = src;
      src = dst;
      dst = tmp;
    }
    return src;
  }
};

}  // namespace dfjk
