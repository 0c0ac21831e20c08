// Geometry derivative of the 3-center integrals (ab|c), contracted on the fly
// with a weight G of the 3-center row layout (rows = bra function pairs of
// the kept shell pairs, columns = auxiliary functions in sorted order).
//
// For one kept shell pair (a, b) (a has the larger l, center A; b center B)
// and one auxiliary shell c (center C) a group of lanes forms
//   fA = sum_{i,m} G[i][m] d(ab|c)[i][m]/dA,  fC = sum_{i,m} G[i][m] d(ab|c)[i][m]/dC,
// and fB = -fA - fC (the integral is unchanged when all three centers move
// together). In the McMurchie-Davidson form of eri3c.cuh,
//   (ab|c)[i][m] = pref sum_h Esph[i][h] W_m[h],  W_m[h] = sum_c T[c][m] R_{h+c}(P - C),
// only R depends on C: dR_{tuv}/dC_x = -R_{t+1,u,v}. d/dA acts on the bra
// Gaussian, d/dA_x x_A^k e^{-a x_A^2} = 2a x_A^{k+1} e^{..} - k x_A^{k-1} e^{..},
// so its Hermite expansion uses D^x = 2a E^{k+1,j} - k E^{k-1,j} (one order
// higher in t + u + v; pair_deriv_kernel, in spherical components).
// dftax obtains the same derivatives by differentiating its integral build
// (dftax/ks/forces.py:245-270 through dftax/integrals/eri3c_bucketed.py:376-426).
#pragma once

#include "hermite_group.cuh"

namespace dfjk {

struct PairDerivArgs {
  const int* pp_pair;
  const int* pp_pa;
  const int* pp_pb;
  const int* pair_s1;
  const int* pair_s2;
  ShellView orb;
  const double* c2s;
  int off1, off2;
  int64_t pp_begin, pp_count;
  double* dsph;         // [pp - pp_begin][3][na*nb][hcount(l1 + l2 + 1)]
};

// A primitive pair's tables by one warp (LAB <= 2) or one block: the three
// axes' E tables (shared, by three lanes), the derivative axis' coefficients,
// then one output (direction, function pair, Hermite entry) per lane. A thread
// per function pair and direction left (dd) at 750 threads on four waters and
// its Hermite sums in local memory: 149 us.
template <int L1, int L2>
__global__ void __launch_bounds__(128) pair_deriv_kernel(PairDerivArgs a) {
  constexpr int NA = 2 * L1 + 1, NB = 2 * L2 + 1, NAB = NA * NB, NH1 = hcount(L1 + L2 + 1);
  constexpr int CA = nc_(L1), CB = nc_(L2), T1 = L1 + L2 + 2;
  constexpr int TPP = L1 + L2 <= 2 ? 32 : 128, PPB = 128 / TPP;
  // [0]: E of the axis, [1]: 2 al E[li + 1] - li E[li - 1] (zero past their orders)
  __shared__ double sE[PPB][2][3][L1 + 1][L2 + 1][T1];
  const int g = threadIdx.x / TPP, gl = threadIdx.x % TPP;
  const int64_t local = blockIdx.x * (int64_t)PPB + g;
  const bool on = local < a.pp_count;
  const int64_t pp = a.pp_begin + (on ? local : 0);
  if (gl < 3) {
    const int pr = a.pp_pair[pp], s1 = a.pair_s1[pr], s2 = a.pair_s2[pr];
    const double al = a.orb.pexp[a.orb.prim0[s1] + a.pp_pa[pp]];
    const double be = a.orb.pexp[a.orb.prim0[s2] + a.pp_pb[pp]];
    double E[L1 + 2][L2 + 1][T1];
    e_axis<L1 + 1, L2>(al, be, a.orb.cen[3 * s1 + gl] - a.orb.cen[3 * s2 + gl], E);
#pragma unroll
    for (int i = 0; i <= L1; ++i)
#pragma unroll
      for (int j = 0; j <= L2; ++j)
#pragma unroll
        for (int t = 0; t < T1; ++t) {
          sE[g][0][gl][i][j][t] = E[i][j][t];
          double v = 2.0 * al * E[i + 1][j][t];
          if (i > 0) v -= i * E[i - 1][j][t];
          sE[g][1][gl][i][j][t] = v;
        }
  }
  __syncthreads();
  if (!on) return;
  const double* TA = a.c2s + a.off1;
  const double* TB = a.c2s + a.off2;
  double* dst = a.dsph + local * (3 * NAB * NH1);
#pragma unroll 1
  for (int q = gl; q < 3 * NAB * NH1; q += TPP) {
    const int h = q % NH1, ab = q / NH1 % NAB, dir = q / (NH1 * NAB);
    const int ia = ab / NB, ib = ab % NB;
    int t, u, v;
    hdecode(h, t, u, v);
    double sum = 0.0;
#pragma unroll 1
    for (int ca = 0; ca < CA; ++ca) {
      const double ta = TA[ca * NA + ia];
      if (ta == 0.0) continue;
      const int ax = comp_x(L1, ca), ay = comp_y(L1, ca), az = L1 - ax - ay;
#pragma unroll 1
      for (int cb = 0; cb < CB; ++cb) {
        const double tab = ta * TB[cb * NB + ib];
        if (tab == 0.0) continue;
        const int bx = comp_x(L2, cb), by = comp_y(L2, cb), bz = L2 - bx - by;
        // orders past an axis' own are zero in the tables
        sum += tab * sE[g][dir == 0][0][ax][bx][t] * sE[g][dir == 1][1][ay][by][u] *
               sE[g][dir == 2][2][az][bz][v];
      }
    }
    dst[q] = sum;
  }
}

struct Grad3cArgs {
  const int64_t* pair_row0;
  const int64_t* pair_pp0;
  const int* pair_npp;
  const int* pair_s1;
  const int* pair_s2;
  const double* pp_P;
  const double* pp_g;
  const double* pp_pref;
  const double* esph;        // class block base: [pp - esph_pp0][na*nb][nh]
  int64_t esph_pp0;
  const double* dsph;        // [pp - dsph_pp0][3][na*nb][nh1]
  int64_t dsph_pp0;
  const int* aux_sorted;
  ShellView aux;
  const double* c2s_aux;     // (ncart x 2lc+1) block of the LC group
  const double* boys;
  const double* boys_asym;
  int64_t pair_begin;        // global pair index of blockIdx.x == 0
  int aux_begin, aux_count, col_base;
  int64_t row_base;          // global row of G[0]
  int64_t ld;
  const double* G;
  int sms;                   // of the device (the launch reads it)
  double omega;
  double* grad_orb;          // [orbital shell][3]
  double* grad_aux;          // [aux shell][3]
};

// A group of lanes (a warp, or 8 lanes when LAB <= 1) per (pair, auxiliary
// shell):
//   * the Boys values, one order per lane;
//   * the Hermite R ladder of order LAB + LC + 1, level by level in two shared
//     buffers, each lane updating a fixed set of (t, u, v) entries;
//   * W_m[h] = pref sum_c T[c][m] R[h + c], h of order <= LAB + 1, the lane's h
//     in registers and in shared memory;
//   * for each bra row i: gh_m[h] += G[i][m] Esph[i][h] and, unless the pair is
//     one shell with itself, fA_d += D_d[i][h] sum_m G[i][m] W_m[h];
//   * fC_d = -sum_{m,h} gh_m[h] W_m[h + e_d].
// Bound by latency at few triples and by the G contraction, NAB (2 NC + 3) NH1
// products, at many. One thread per triple (R, W, gh and the derivative sums,
// up to 1000 doubles, in local memory) took 7.9 ms for (H2O)_4, where (dd|d)
// has 280 triples.
template <int LA, int LB, int LC>
struct GradShape {
  static constexpr int NC = 2 * LC + 1, NCC = nc_(LC), LAB = LA + LB;
  static constexpr int NAB = (2 * LA + 1) * (2 * LB + 1);
  static constexpr int NH = hcount(LAB), NH1 = hcount(LAB + 1), M1 = LAB + LC + 1, NR = hcount(M1);
  static constexpr int TL = LAB <= 1 ? 8 : 32, GPB = 128 / TL;   // lanes per group, groups per block
  // Hermite entries per lane, and components m held at a time: at most 15 sums
  // of each kind per lane (27 or 36 at once spilled kilobytes)
  static constexpr int HJ = (NH1 + TL - 1) / TL;
  static constexpr int MP = (NC * HJ + 14) / 15, MC = (NC + MP - 1) / MP;
  static constexpr int GROUP = 2 * NR + MC * NH1 + NAB * NC + (M1 + 1);   // doubles
  static constexpr size_t smem = (size_t)(NCC * NC + GPB * GROUP) * sizeof(double) +
                                 (size_t)NH1 * NCC * sizeof(short);
};

template <int LA, int LB, int LC>
__global__ void __launch_bounds__(128) grad3c_kernel(Grad3cArgs a) {
  using S = GradShape<LA, LB, LC>;
  constexpr int NC = S::NC, NCC = S::NCC, NAB = S::NAB, NH = S::NH, NH1 = S::NH1, M1 = S::M1;
  constexpr int NR = S::NR, TL = S::TL, GPB = S::GPB;
  constexpr int HJ = S::HJ, MC = S::MC;
  extern __shared__ double gsm[];
  __shared__ double red[4][6];
  const int grp = threadIdx.x / TL, gl = threadIdx.x % TL;
  double* sT = gsm;
  double* sRa = sT + NCC * NC + grp * S::GROUP;
  double* sRb = sRa + NR;
  double* sW = sRb + NR;
  double* sG = sW + MC * NH1;
  double* sB = sG + NAB * NC;
  short* sI = reinterpret_cast<short*>(gsm + NCC * NC + GPB * S::GROUP);   // hidx(h + c)
  for (int q = threadIdx.x; q < NCC * NC; q += 128) sT[q] = a.c2s_aux[q];
  for (int q = threadIdx.x; q < NH1 * NCC; q += 128) {
    int t, u, v;
    hdecode(q / NCC, t, u, v);
    const int c = q % NCC;
    sI[q] = (short)hidx(t + comp_x(LC, c), u + comp_y(LC, c), v + comp_z(LC, c));
  }
  HermiteGroup<M1, TL> ladder;
  ladder.init(gl);
  // h + e_d of the lane's Hermite entries
  int up[HJ][3];
#pragma unroll
  for (int j = 0; j < HJ; ++j) {
    int t = 0, u = 0, v = 0;
    if (gl + TL * j < NH) hdecode(gl + TL * j, t, u, v);
    up[j][0] = hidx(t + 1, u, v);
    up[j][1] = hidx(t, u + 1, v);
    up[j][2] = hidx(t, u, v + 1);
  }
  __syncthreads();
  const int64_t pr = a.pair_begin + blockIdx.x;
  const int s1 = a.pair_s1[pr], s2 = a.pair_s2[pr];
  const bool same = s1 == s2;   // fA + fB = -fC lands on one shell: no d/dA needed
  const int64_t pp0 = a.pair_pp0[pr];
  const int npp = a.pair_npp[pr];
  const double* Gp = a.G + (a.pair_row0[pr] - a.row_base) * a.ld + a.col_base;
  double fab[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};   // this lane's part of fA and fB
  for (int base = blockIdx.y * GPB; base < a.aux_count; base += gridDim.y * GPB) {
    // groups past the last shell run along with zero weights
    const bool on = base + grp < a.aux_count;
    const int slot = on ? base + grp : a.aux_count - 1;
    const int kc = a.aux_sorted[a.aux_begin + slot];
    const double C0 = a.aux.cen[3 * kc], C1 = a.aux.cen[3 * kc + 1], C2 = a.aux.cen[3 * kc + 2];
    const int cp0 = a.aux.prim0[kc], cnp = a.aux.nprim[kc];
    const int cmax = TL == 32 ? cnp : __reduce_max_sync(0xffffffffu, cnp);
    for (int q = gl; q < NAB * NC; q += TL)
      sG[q] = on ? Gp[(int64_t)(q / NC) * a.ld + slot * NC + q % NC] : 0.0;
    double fA[3] = {0.0, 0.0, 0.0}, fC[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int q = 0; q < npp; ++q) {
      const int64_t pp = pp0 + q;
      const double X = a.pp_P[3 * pp] - C0, Y = a.pp_P[3 * pp + 1] - C1, Z = a.pp_P[3 * pp + 2] - C2;
      const double g = a.pp_g[pp], pab = a.pp_pref[pp];
      const double* E = a.esph + (pp - a.esph_pp0) * (NAB * NH);
      const double* D = a.dsph + (pp - a.dsph_pp0) * (3 * NAB * NH1);
#pragma unroll 1
      for (int ic = 0; ic < cmax; ++ic) {
        // (a group with fewer primitives repeats its last with a zero factor)
        const int pc = cp0 + (ic < cnp ? ic : cnp - 1);
        const double gc = a.aux.pexp[pc], cc = ic < cnp ? a.aux.pcoef[pc] : 0.0;
        const double rho = g * gc / (g + gc);
        const double T = rho * (X * X + Y * Y + Z * Z);
        const double* src = ladder.run(T, rho, a.omega, X, Y, Z, a.boys, a.boys_asym, sB, sRa, sRb, gl);
        double hob = 1.0;
#pragma unroll
        for (int k = 0; k < LC; ++k) hob *= -0.5 / gc;
        const double pref = pab * cc * kTwoPi25 / (g * gc * sqrt(g + gc)) * hob;
        // MC components m at a time, so that w and gh stay in registers
#pragma unroll 1
        for (int m0 = 0; m0 < NC; m0 += MC) {
          double w[HJ][MC], gh[HJ][MC];
#pragma unroll
          for (int j = 0; j < HJ; ++j) {
            const int h = gl + TL * j;
#pragma unroll
            for (int m = 0; m < MC; ++m) w[j][m] = gh[j][m] = 0.0;
            if (h >= NH1) continue;
#pragma unroll 1
            for (int c = 0; c < NCC; ++c) {
              const double r = src[sI[h * NCC + c]];
#pragma unroll
              for (int m = 0; m < MC; ++m)
                if (m0 + m < NC) w[j][m] += sT[c * NC + m0 + m] * r;
            }
#pragma unroll
            for (int m = 0; m < MC; ++m) {
              w[j][m] *= pref;
              sW[m * NH1 + h] = w[j][m];
            }
          }
          __syncwarp();
#pragma unroll 1
          for (int i = 0; i < NAB; ++i) {
            double gi[MC];
#pragma unroll
            for (int m = 0; m < MC; ++m) gi[m] = m0 + m < NC ? sG[i * NC + m0 + m] : 0.0;
#pragma unroll
            for (int j = 0; j < HJ; ++j) {
              const int h = gl + TL * j;
              if (h < NH) {
                const double e = __ldg(E + i * NH + h);
#pragma unroll
                for (int m = 0; m < MC; ++m) gh[j][m] += gi[m] * e;
              }
              if (!same && h < NH1) {
                double v = 0.0;
#pragma unroll
                for (int m = 0; m < MC; ++m) v += gi[m] * w[j][m];
#pragma unroll
                for (int d = 0; d < 3; ++d) fA[d] += v * __ldg(D + (d * NAB + i) * NH1 + h);
              }
            }
          }
#pragma unroll
          for (int j = 0; j < HJ; ++j) {
            if (gl + TL * j >= NH) continue;
#pragma unroll
            for (int m = 0; m < MC; ++m)
#pragma unroll
              for (int d = 0; d < 3; ++d) fC[d] -= gh[j][m] * sW[m * NH1 + up[j][d]];
          }
          __syncwarp();   // sW is rewritten by the next components
        }
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      fab[d] += fA[d];
      fab[3 + d] -= fA[d] + fC[d];
#pragma unroll
      for (int o = TL / 2; o > 0; o >>= 1) fC[d] += __shfl_xor_sync(0xffffffffu, fC[d], o);
    }
    if (on && gl < 3) atomicAdd(a.grad_aux + 3 * kc + gl, gl == 0 ? fC[0] : (gl == 1 ? fC[1] : fC[2]));
    __syncwarp();   // sG is rewritten by the next shell
  }
  // fA and fB = -fA - fC summed over the block (one shell pair)
#pragma unroll
  for (int k = 0; k < 6; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) fab[k] += __shfl_xor_sync(0xffffffffu, fab[k], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < 6; ++k) red[threadIdx.x >> 5][k] = fab[k];
  __syncthreads();
  if (threadIdx.x < 6) {
    double sum = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) sum += red[q][threadIdx.x];
    const int sh = threadIdx.x < 3 ? s1 : s2;
    atomicAdd(a.grad_orb + 3 * sh + threadIdx.x % 3, sum);
  }
}

// npair shell pairs; each block walks about four auxiliary shells per group
// once the pairs alone fill the device
template <int LA, int LB, int LC>
inline void launch_grad3c_one(unsigned npair, cudaStream_t s, const Grad3cArgs& a) {
  using S = GradShape<LA, LB, LC>;
  if (S::smem > (size_t)48 << 10)
    cudaFuncSetAttribute(grad3c_kernel<LA, LB, LC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)S::smem);
  const unsigned full = (unsigned)((a.aux_count + S::GPB - 1) / S::GPB);
  const unsigned gy = (uint64_t)npair * full > 8 * (uint64_t)a.sms ? (full + 3) / 4 : full;
  grad3c_kernel<LA, LB, LC><<<dim3(npair, gy), 128, S::smem, s>>>(a);
}

template <int LA, int LB>
inline bool launch_grad3c_lc(int lc, unsigned npair, cudaStream_t s, const Grad3cArgs& a) {
  switch (lc) {
    case 0: launch_grad3c_one<LA, LB, 0>(npair, s, a); return true;
    case 1: launch_grad3c_one<LA, LB, 1>(npair, s, a); return true;
    case 2: launch_grad3c_one<LA, LB, 2>(npair, s, a); return true;
    case 3: launch_grad3c_one<LA, LB, 3>(npair, s, a); return true;
    case 4: launch_grad3c_one<LA, LB, 4>(npair, s, a); return true;
    default: return false;
  }
}

// npp primitive pairs
template <int LA, int LB>
inline void launch_pair_deriv_t(int64_t npp, cudaStream_t s, const PairDerivArgs& a) {
  constexpr int per = LA + LB <= 2 ? 4 : 1;
  pair_deriv_kernel<LA, LB><<<(unsigned)((npp + per - 1) / per), 128, 0, s>>>(a);
}

#define DFJK_GRAD3C_DECL(A, B)                                                              \
  bool launch_grad3c_##A##B(int lc, unsigned npair, cudaStream_t s, const Grad3cArgs& a);  \
  void launch_pair_deriv_##A##B(int64_t npp, cudaStream_t s, const PairDerivArgs& a);
DFJK_GRAD3C_DECL(0, 0)
DFJK_GRAD3C_DECL(1, 0)
DFJK_GRAD3C_DECL(1, 1)
DFJK_GRAD3C_DECL(2, 0)
DFJK_GRAD3C_DECL(2, 1)
DFJK_GRAD3C_DECL(2, 2)
DFJK_GRAD3C_DECL(3, 0)
DFJK_GRAD3C_DECL(3, 1)
DFJK_GRAD3C_DECL(3, 2)
DFJK_GRAD3C_DECL(3, 3)
#undef DFJK_GRAD3C_DECL

}  // namespace dfjk
