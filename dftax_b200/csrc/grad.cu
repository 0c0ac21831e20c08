// Nuclear gradient of the DF energy at a fixed density.
//
// dftax's forces() differentiate the energy through the integral build
// (dftax/ks/forces.py:245-270), with the metric pseudo-inverse differentiated
// by d(V+) = -V+ dV V+ (_metric_pinv_jvp, dftax/ks/terms.py:196-204). For
// E = 1/2 c^T V+ c + sum_s k_s sum_PQ V+_PQ tr(P_s T_P P_s T_Q) (c_P =
// tr(P_tot T_P), T_P = (..|P), k_s = -a_x/4 closed shell, -a_x/2 per spin)
// that derivative is
//   dE = sum_{mn,P} G[mn][P] d(mn|P) - 1/2 sum_PQ W[P][Q] d(P|Q),
// and in terms of the plan's B = T L (V+ = L L^T) and g = B^T vec(P_tot):
//   H[r][x] = w_r (g_x P_tot[r] + sum_s 2 k_s (P_s B_x P_s)[r])   (w_r = 2 for
//             off-diagonal bra pairs: they stand for (m,n) and (n,m)),
//   M = H^T B = g g^T + sum_s 2 k_s tr(P_s B_x P_s B_y),  E = 1/2 tr(M),
//   G = H L^T (3-center row layout),  W = L M L^T.
// G and W are contracted with the integral derivatives on the fly
// (grad3c.cuh; grad2c_kernel below); nothing of size rows x naux beyond one
// chunk of G is kept.
#include "dmma.cuh"
#include "grad3c.cuh"
#include "internal.h"

#include <algorithm>

namespace dfjk {

namespace {

ShellView view(const Shells& s) {
  return ShellView{s.d_l.as<int>(), s.d_nprim.as<int>(), s.d_prim0.as<int>(),
                   s.d_cen.as<double>(), s.d_pexp.as<double>(), s.d_pcoef.as<double>()};
}

bool launch_grad3c(int l1, int l2, int lc, unsigned npair, cudaStream_t s, const Grad3cArgs& a) {
  switch (l1 * 4 + l2) {
    case 0: return launch_grad3c_00(lc, npair, s, a);
    case 4: return launch_grad3c_10(lc, npair, s, a);
    case 5: return launch_grad3c_11(lc, npair, s, a);
    case 8: return launch_grad3c_20(lc, npair, s, a);
    case 9: return launch_grad3c_21(lc, npair, s, a);
    case 10: return launch_grad3c_22(lc, npair, s, a);
    case 12: return launch_grad3c_30(lc, npair, s, a);
    case 13: return launch_grad3c_31(lc, npair, s, a);
    case 14: return launch_grad3c_32(lc, npair, s, a);
    case 15: return launch_grad3c_33(lc, npair, s, a);
    default: return false;
  }
}

bool launch_pair_deriv(int l1, int l2, int64_t npp, cudaStream_t s, const PairDerivArgs& a) {
  switch (l1 * 4 + l2) {
    case 0: launch_pair_deriv_00(npp, s, a); return true;
    case 4: launch_pair_deriv_10(npp, s, a); return true;
    case 5: launch_pair_deriv_11(npp, s, a); return true;
    case 8: launch_pair_deriv_20(npp, s, a); return true;
    case 9: launch_pair_deriv_21(npp, s, a); return true;
    case 10: launch_pair_deriv_22(npp, s, a); return true;
    case 12: launch_pair_deriv_30(npp, s, a); return true;
    case 13: launch_pair_deriv_31(npp, s, a); return true;
    case 14: launch_pair_deriv_32(npp, s, a); return true;
    case 15: launch_pair_deriv_33(npp, s, a); return true;
    default: return false;
  }
}

// H[r][x] = w_r g[x] Ptot[m][n]   (x < ldb; g is zero past the kept directions)
__global__ void h_init_kernel(const double* __restrict__ g, const double* __restrict__ Ptot,
                              int64_t nao, const int* __restrict__ rm, const int* __restrict__ rn,
                              const int8_t* __restrict__ kind, int64_t nrows, int64_t ldb,
                              double* __restrict__ H) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nrows * ldb) return;
  const int64_t r = i / ldb, x = i % ldb;
  const double wr = kind[r] == 2 ? 2.0 : 1.0;
  H[i] = wr * g[x] * Ptot[(int64_t)rm[r] * nao + rn[r]];
}

// Bd[x][m][n] = B[r][x0 + x] for every row r = (m, n); off-diagonal rows also
// fill [n][m] (the rows of a diagonal shell pair hold both orders already)
__global__ void unpack_b_kernel(const double* __restrict__ B, int64_t ldb, int64_t nrows,
                                const int* __restrict__ rm, const int* __restrict__ rn,
                                const int8_t* __restrict__ kind, int64_t nao, int64_t x0,
                                int64_t nx, double* __restrict__ Bd) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nrows * nx) return;
  const int64_t r = i / nx, x = i % nx;
  const double v = B[r * ldb + x0 + x];
  const int m = rm[r], n = rn[r];
  double* plane = Bd + x * nao * nao;
  plane[(int64_t)m * nao + n] = v;
  if (kind[r] == 2) plane[(int64_t)n * nao + m] = v;
}

// H[r][x0 + x] += w_r a T[x][m][n]
__global__ void h_add_kernel(const double* __restrict__ T, int64_t nao, const int* __restrict__ rm,
                             const int* __restrict__ rn, const int8_t* __restrict__ kind,
                             int64_t nrows, int64_t ldb, int64_t x0, int64_t nx, double a,
                             double* __restrict__ H) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nrows * nx) return;
  const int64_t r = i / nx, x = i % nx;
  const double wr = kind[r] == 2 ? 2.0 : 1.0;
  H[r * ldb + x0 + x] += wr * a * T[x * nao * nao + (int64_t)rm[r] * nao + rn[r]];
}

// H[r][x0 + x] += w_r a sum_j U[m][x][j] C'[n][j] for every row r = (m, n) of B:
// block (m, 64 directions, 64 entries of m's list; rows are taken under their
// first function) on the float64 tensor cores. Rows of U and C' are staged as
// they lie, 16 j per step (16-byte pieces, index xor 4 (row % 2): a load phase of
// two rows x four pieces falls in distinct banks; the j order inside a step is
// free). The sum over j is short (the density's rank), so two stages suffice.
constexpr int kBtT = 64, kBtK = 16;

__global__ void __launch_bounds__(256) back_transform_kernel(
    const double* __restrict__ U, const double* __restrict__ Cp, int64_t ncp, int64_t nx,
    const int* __restrict__ kptr, const int* __restrict__ krow, const int* __restrict__ kn,
    const int* __restrict__ rm, const int8_t* __restrict__ kind, int64_t ldb, int64_t x0, double a,
    double* __restrict__ H) {
  __shared__ __align__(16) double sm[2][2][kBtT * kBtK];   // [stage][entries, directions]
  __shared__ int srow[kBtT], sn[kBtT];
  const int m = blockIdx.x;
  const int64_t xt = (int64_t)blockIdx.y * kBtT;
  const int e0 = kptr[m] + blockIdx.z * kBtT, e1 = kptr[m + 1];
  if (e0 >= e1) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  bool any = false;
  if (tid < kBtT) {
    const int e = e0 + tid;
    int r = -1, n = 0;
    if (e < e1 && rm[krow[e]] == m) {
      r = krow[e];
      n = kn[e];
    }
    srow[tid] = r;
    sn[tid] = n;
    any = r >= 0;
  }
  if (!__syncthreads_or(any)) return;
  const int wr = (warp & 3) * 16, wc = (warp >> 2) * 32;
  const int fr = lane >> 2, fk = lane & 3;
  double acc[2][4][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[i][b][0] = acc[i][b][1] = 0.0;
  const int nst = (int)((ncp + kBtK - 1) / kBtK);
  const int sr = tid >> 3, sp = tid & 7;
  auto stage = [&](int q) {
    const int64_t k = (int64_t)q * kBtK + 2 * sp;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = sr + 32 * j, o = r * kBtK + 2 * (sp ^ (4 * (r & 1)));
      const bool oe = k < ncp && srow[r] >= 0, ox = k < ncp && xt + r < nx;
      cp_async16(&sm[q & 1][0][o], oe ? Cp + (int64_t)sn[r] * ncp + k : Cp, oe);
      cp_async16(&sm[q & 1][1][o], ox ? U + ((int64_t)m * nx + xt + r) * ncp + k : U, ox);
    }
    cp_async_commit();
  };
  stage(0);
  for (int q = 0; q < nst; ++q) {
    if (q + 1 < nst) {
      stage(q + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int piece = 2 * ((4 * h + fk) ^ (4 * (fr & 1)));
      double2 af[2], bf[4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        af[i] = *reinterpret_cast<const double2*>(&sm[q & 1][0][(wr + 8 * i + fr) * kBtK + piece]);
#pragma unroll
      for (int b = 0; b < 4; ++b)
        bf[b] = *reinterpret_cast<const double2*>(&sm[q & 1][1][(wc + 8 * b + fr) * kBtK + piece]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          dmma_8x8x4(acc[i][b], af[i].x, bf[b].x);
          dmma_8x8x4(acc[i][b], af[i].y, bf[b].y);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = srow[wr + 8 * i + fr];
    if (r < 0) continue;
    const double f = (kind[r] == 2 ? 2.0 : 1.0) * a;
    double* row = H + (int64_t)r * ldb + x0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int64_t x = xt + wc + 8 * b + 2 * fk + q;
        if (x < nx) row[x] += f * acc[i][b][q];
      }
  }
}

__global__ void add2_kernel(const double* __restrict__ a, const double* __restrict__ b, int64_t n,
                            double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = a[i] + b[i];
}

// out[0] = sum_i M[i][i] (one block, fixed order)
__global__ void trace_kernel(const double* __restrict__ M, int64_t n, int64_t ld,
                             double* __restrict__ out) {
  __shared__ double part[256];
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += M[i * ld + i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = part[0];
}

// ---------------------------------------------------------------------------
// 2-center derivative: (P|Q) depends on A - B only, so
//   d(P|Q)/dA_x = hob sum_{c1,c2} T_P[c1][p] T_Q[c2][q] R_{c1 + c2 + e_x}(A - B) = -d/dB_x.
// One warp per unordered pair of shells of the (LP, LQ) groups; the
// contribution -1/2 sum_{p,q} W[p][q] d(p|q) counts both orders of a pair. The
// warp projects W onto cartesian components through shared memory, builds R
// with the 3-center kernel's ladder and spreads the (c1, c2) products over its
// lanes. (A thread per pair kept all of it in local memory: 66 threads for
// (f|f) on four waters took 177 us.)
// ---------------------------------------------------------------------------

struct Grad2cArgs {
  const int* aux_sorted;
  ShellView aux;
  const double* c2s;
  int offP, offQ;
  const double* boys;
  const double* boys_asym;
  int beginP, countP, beginQ, countQ;
  int colP, colQ;
  int64_t ld;
  const double* W;       // naux x naux, sorted columns (symmetric)
  double omega;
  double* grad_aux;      // [aux shell][3]
};

template <int LP, int LQ>
__global__ void __launch_bounds__(128) grad2c_kernel(Grad2cArgs a) {
  constexpr int NP = 2 * LP + 1, NQ = 2 * LQ + 1, CP = nc_(LP), CQ = nc_(LQ);
  constexpr int M1 = LP + LQ + 1, NR = hcount(M1);
  __shared__ double sW[4][NP * NQ], sH[4][CP * NQ], sC[4][CP * CQ];
  __shared__ double sR[4][2][NR], sB[4][M1 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t gid = blockIdx.x * (int64_t)4 + warp;
  if (gid >= (int64_t)a.countP * a.countQ) return;
  const int ip = (int)(gid / a.countQ), iq = (int)(gid % a.countQ);
  if (LP == LQ && ip >= iq) return;   // same group: each unordered pair once; a shell with itself has no derivative
  const int sp = a.aux_sorted[a.beginP + ip], sq = a.aux_sorted[a.beginQ + iq];
  const double X = a.aux.cen[3 * sp] - a.aux.cen[3 * sq];
  const double Y = a.aux.cen[3 * sp + 1] - a.aux.cen[3 * sq + 1];
  const double Z = a.aux.cen[3 * sp + 2] - a.aux.cen[3 * sq + 2];
  const double* TP = a.c2s + a.offP;
  const double* TQ = a.c2s + a.offQ;
  // W projected on the cartesian components: sum_{p,q} T_P[c1][p] W[p][q] T_Q[c2][q]
  const int r0 = a.colP + ip * NP, c0 = a.colQ + iq * NQ;
  for (int q = lane; q < NP * NQ; q += 32)
    sW[warp][q] = a.W[(int64_t)(r0 + q / NQ) * a.ld + c0 + q % NQ];
  __syncwarp();
  for (int q = lane; q < CP * NQ; q += 32) {
    double s = 0.0;
    for (int k = 0; k < NP; ++k) s += __ldg(TP + q / NQ * NP + k) * sW[warp][k * NQ + q % NQ];
    sH[warp][q] = s;
  }
  __syncwarp();
  for (int q = lane; q < CP * CQ; q += 32) {
    double s = 0.0;
    for (int k = 0; k < NQ; ++k) s += sH[warp][q / CQ * NQ + k] * __ldg(TQ + q % CQ * NQ + k);
    sC[warp][q] = s;
  }
  HermiteGroup<M1, 32> ladder;
  ladder.init(lane);
  double f[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
  for (int i = 0; i < a.aux.nprim[sp]; ++i) {
    const double al = a.aux.pexp[a.aux.prim0[sp] + i], ca = a.aux.pcoef[a.aux.prim0[sp] + i];
#pragma unroll 1
    for (int j = 0; j < a.aux.nprim[sq]; ++j) {
      const double be = a.aux.pexp[a.aux.prim0[sq] + j], cb = a.aux.pcoef[a.aux.prim0[sq] + j];
      const double rho = al * be / (al + be);
      const double* R = ladder.run(rho * (X * X + Y * Y + Z * Z), rho, a.omega, X, Y, Z, a.boys,
                                   a.boys_asym, sB[warp], sR[warp][0], sR[warp][1], lane);
      double hob = kTwoPi25 * ca * cb / (al * be * sqrt(al + be));
#pragma unroll
      for (int k = 0; k < LP; ++k) hob *= 0.5 / al;
#pragma unroll
      for (int k = 0; k < LQ; ++k) hob *= -0.5 / be;
      for (int q = lane; q < CP * CQ; q += 32) {
        const int c1 = q / CQ, c2 = q % CQ;
        const double wc = hob * sC[warp][q];
        const int x1 = comp_x(LP, c1), y1 = comp_y(LP, c1), x2 = comp_x(LQ, c2), y2 = comp_y(LQ, c2);
        const int x = x1 + x2, y = y1 + y2, z = LP + LQ - x - y;
        f[0] += wc * R[hidx(x + 1, y, z)];
        f[1] += wc * R[hidx(x, y + 1, z)];
        f[2] += wc * R[hidx(x, y, z + 1)];
      }
      __syncwarp();   // sB and R are rewritten by the next primitives
    }
  }
  // -1/2 (W_pq + W_qp) d(p|q)/dA = -f on P's center, +f on Q's (dB = -dA)
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) f[d] += __shfl_xor_sync(0xffffffffu, f[d], o);
    if (lane == d) {
      atomicAdd(a.grad_aux + 3 * sp + d, -f[d]);
      atomicAdd(a.grad_aux + 3 * sq + d, f[d]);
    }
  }
}

#define DFJK_G2_CASES(X)                                                      \
  X(0, 0) X(1, 0) X(1, 1) X(2, 0) X(2, 1) X(2, 2) X(3, 0) X(3, 1) X(3, 2) X(3, 3) \
  X(4, 0) X(4, 1) X(4, 2) X(4, 3) X(4, 4)

void launch_grad2c(Plan& p, const double* W, double* grad_aux, cudaStream_t s) {
  const Context& c = *p.ctx;
  for (int lp = 0; lp <= p.aux.lmax; ++lp) {
    if (!p.aux_lcount[lp]) continue;
    for (int lq = 0; lq <= lp; ++lq) {
      if (!p.aux_lcount[lq]) continue;
      Grad2cArgs a;
      a.aux_sorted = p.d_aux_sorted.as<int>();
      a.aux = view(p.aux);
      a.c2s = p.c2s_aux.dev.as<double>();
      a.offP = p.c2s_aux.off[lp];
      a.offQ = p.c2s_aux.off[lq];
      a.boys = c.boys.as<double>();
      a.boys_asym = c.boys_asym.as<double>();
      a.beginP = p.aux_lbegin[lp];
      a.countP = p.aux_lcount[lp];
      a.beginQ = p.aux_lbegin[lq];
      a.countQ = p.aux_lcount[lq];
      a.colP = p.aux_col0[p.aux_order[a.beginP]];
      a.colQ = p.aux_col0[p.aux_order[a.beginQ]];
      a.ld = p.naux;
      a.W = W;
      a.omega = p.atten;
      a.grad_aux = grad_aux;
      const int64_t n = (int64_t)a.countP * a.countQ;
      const unsigned blocks = (unsigned)((n + 3) / 4);
      bool done = false;
#define X(A, B)                                              \
  if (lp == A && lq == B) {                                  \
    grad2c_kernel<A, B><<<blocks, 128, 0, s>>>(a);           \
    done = true;                                             \
  }
      DFJK_G2_CASES(X)
#undef X
      if (!done) fail(DFJK_ERR_UNSUPPORTED, "aux derivative class (%d,%d) not compiled", lp, lq);
      DFJK_LAUNCHED();
    }
  }
}

// derivative tables of the pairs [b, e) of class cr into dsph, then the
// 3-center derivative contraction of those pairs with G (rows from row_base)
void launch_grad3c_pairs(Plan& p, const ClassRange& cr, int64_t b, int64_t e, double* dsph,
                         const double* G, int64_t row_base, double* grad_orb, double* grad_aux,
                         cudaStream_t s) {
  const Context& c = *p.ctx;
  const int64_t pp_b = p.pair_pp0[b];
  const int64_t pp_e = p.pair_pp0[e - 1] + p.pair_npp[e - 1];
  {
    PairDerivArgs a;
    a.pp_pair = p.d_pp_pair.as<int>();
    a.pp_pa = p.d_pp_pa.as<int>();
    a.pp_pb = p.d_pp_pb.as<int>();
    a.pair_s1 = p.d_pair_s1.as<int>();
    a.pair_s2 = p.d_pair_s2.as<int>();
    a.orb = view(p.orb);
    a.c2s = p.c2s_orb.dev.as<double>();
    a.off1 = p.c2s_orb.off[cr.l1];
    a.off2 = p.c2s_orb.off[cr.l2];
    a.pp_begin = pp_b;
    a.pp_count = pp_e - pp_b;
    a.dsph = dsph;
    if (!launch_pair_deriv(cr.l1, cr.l2, a.pp_count, s, a))
      fail(DFJK_ERR_UNSUPPORTED, "pair derivative class (%d,%d) not compiled", cr.l1, cr.l2);
    DFJK_LAUNCHED();
  }
  for (int lc = 0; lc <= p.aux.lmax; ++lc) {
    if (p.aux_lcount[lc] == 0) continue;
    Grad3cArgs a;
    a.pair_row0 = p.d_pair_row0.as<int64_t>();
    a.pair_pp0 = p.d_pair_pp0.as<int64_t>();
    a.pair_npp = p.d_pair_npp.as<int>();
    a.pair_s1 = p.d_pair_s1.as<int>();
    a.pair_s2 = p.d_pair_s2.as<int>();
    a.pp_P = p.d_pp_P.as<double>();
    a.pp_g = p.d_pp_g.as<double>();
    a.pp_pref = p.d_pp_pref.as<double>();
    a.esph = p.d_esph.as<double>() + cr.esph_off;
    a.esph_pp0 = cr.pp_begin;
    a.dsph = dsph;
    a.dsph_pp0 = pp_b;
    a.aux_sorted = p.d_aux_sorted.as<int>();
    a.aux = view(p.aux);
    a.c2s_aux = p.c2s_aux.dev.as<double>() + p.c2s_aux.off[lc];
    a.boys = c.boys.as<double>();
    a.boys_asym = c.boys_asym.as<double>();
    a.pair_begin = b;
    a.aux_begin = p.aux_lbegin[lc];
    a.aux_count = p.aux_lcount[lc];
    a.col_base = p.aux_col0[p.aux_order[p.aux_lbegin[lc]]];
    a.row_base = row_base;
    a.ld = p.naux;
    a.G = G;
    a.sms = num_sms(c.device);
    a.omega = p.atten;
    a.grad_orb = grad_orb;
    a.grad_aux = grad_aux;
    if (!launch_grad3c(cr.l1, cr.l2, lc, (unsigned)(e - b), s, a))
      fail(DFJK_ERR_UNSUPPORTED, "3-center derivative class (%d,%d|%d) not compiled", cr.l1, cr.l2, lc);
    DFJK_LAUNCHED();
  }
}

}  // namespace

double energy_gradient(Plan& p, const double* P, int nspin, double hf, double* grad_orb,
                       double* grad_aux, cudaStream_t s) {
  Context& c = *p.ctx;
  const int64_t n = p.nao, nn = n * n, ldb = p.ldb, naux = p.naux, rows = p.nrows;
  check_finite(p, P, nn * nspin, s, "the density");
  DFJK_CUDA(cudaMemsetAsync(grad_orb, 0, (size_t)p.orb.n * 3 * sizeof(double), s));
  DFJK_CUDA(cudaMemsetAsync(grad_aux, 0, (size_t)p.aux.n * 3 * sizeof(double), s));
  DevBuf Ptot_b, g, H, M, T, W;
  const double* Ptot = P;
  if (nspin == 2) {
    Ptot_b.alloc(nn * sizeof(double));
    add2_kernel<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(P, P + nn, nn, Ptot_b.as<double>());
    DFJK_LAUNCHED();
    Ptot = Ptot_b.as<double>();
  }
  g.alloc(ldb * sizeof(double));
  gamma_from_density(p, Ptot, g.as<double>(), s);
  // H = w (g P_tot + sum_s 2 k_s P_s B_x P_s)
  H.alloc((size_t)std::max<int64_t>(rows, 1) * ldb * sizeof(double));
  if (rows > 0) {
    h_init_kernel<<<(unsigned)((rows * ldb + 255) / 256), 256, 0, s>>>(
        g.as<double>(), Ptot, n, p.d_row_m.as<int>(), p.d_row_n.as<int>(), p.d_row_w.as<int8_t>(),
        rows, ldb, H.as<double>());
    DFJK_LAUNCHED();
  }
  DFJK_CUBLAS(cublasSetStream(c.cublas, s));
  if (hf != 0.0 && rows > 0) {
    const double k = (nspin == 1 ? -0.25 : -0.5) * hf;
    const int64_t xc = std::max<int64_t>(1, std::min<int64_t>(p.nfit, ((int64_t)1 << 30) / (16 * nn)));
    DevBuf Bd, T1;
    // the densities' factors P_s = C C^T (lowrank.cu): with r = rank, B_x C
    // (half transform), C^T B_x C, C (C^T B_x C) and its product with C^T at the
    // kept pairs cost 2 n^2 r + 4 n r^2 + n^2 r per direction instead of 4 n^3; past
    // half the functions the dense form is no dearer, and the factor stops there
    LowRankInfo fh{};
    const bool low = low_rank_supported(n);
    if (low) {
      p.ws_lowrank.ensure((size_t)nn * nspin * sizeof(double));
      DevBuf fd;
      fd.alloc(sizeof fh);
      DFJK_CUDA(cudaMemsetAsync(fd.p, 0, sizeof fh, s));
      launch_low_rank(P, n, nspin, n / 2, p.ws_lowrank.as<double>(), kLowRankAccept,
                      fd.as<LowRankInfo>(), s);
      DFJK_CUDA(cudaMemcpyAsync(&fh, fd.p, sizeof fh, cudaMemcpyDeviceToHost, s));
      DFJK_CUDA(cudaStreamSynchronize(s));
    }
    const double one = 1.0, zero = 0.0;
    for (int sp = 0; sp < nspin; ++sp) {
      const double* Ps = P + sp * nn;
      if (low && fh.within(sp, kLowRankAccept)) {
        const int64_t ncp = fh.rank[sp] + (fh.rank[sp] & 1);
        if (ncp == 0) continue;
        DevBuf Cp, X, Y;
        Cp.alloc((size_t)n * ncp * sizeof(double));
        pack_columns(p.ws_lowrank.as<double>() + sp * nn, n, fh.rank[sp], ncp, Cp.as<double>(), s);
        // 64 directions at a time (the half transform's tile), up to 1 GB of X
        int64_t xl = ((int64_t)1 << 30) / (n * ncp * (int64_t)sizeof(double)) / 64 * 64;
        xl = std::min<int64_t>(std::max<int64_t>(xl, 64), p.nfit);
        X.alloc((size_t)n * xl * ncp * sizeof(double));
        Y.alloc((size_t)ncp * xl * ncp * sizeof(double));
        for (int64_t x0 = 0; x0 < p.nfit; x0 += xl) {
          const int64_t nx = std::min(xl, p.nfit - x0);
          half_transform(p, Cp.as<double>(), ncp, x0, nx, X.as<double>(), s);
          const int xj = (int)(nx * ncp);
          DFJK_CUBLAS(cublasDgemm(c.cublas, CUBLAS_OP_N, CUBLAS_OP_T, xj, (int)ncp, (int)n, &one,
                                  X.as<double>(), xj, Cp.as<double>(), (int)ncp, &zero,
                                  Y.as<double>(), xj));
          DFJK_CUBLAS(cublasDgemm(c.cublas, CUBLAS_OP_N, CUBLAS_OP_N, xj, (int)n, (int)ncp, &one,
                                  Y.as<double>(), xj, Cp.as<double>(), (int)ncp, &zero,
                                  X.as<double>(), xj));
          const dim3 grid((unsigned)n, (unsigned)((nx + kBtT - 1) / kBtT), (unsigned)((n + kBtT - 1) / kBtT));
          back_transform_kernel<<<grid, 256, 0, s>>>(
              X.as<double>(), Cp.as<double>(), ncp, nx, p.d_kptr.as<int>(), p.d_krow.as<int>(),
              p.d_kn.as<int>(), p.d_row_m.as<int>(), p.d_row_w.as<int8_t>(), ldb, x0, 2.0 * k,
              H.as<double>());
          DFJK_LAUNCHED();
        }
        continue;
      }
      Bd.ensure((size_t)xc * nn * sizeof(double));
      T1.ensure((size_t)xc * nn * sizeof(double));
      for (int64_t x0 = 0; x0 < p.nfit; x0 += xc) {
        const int64_t nx = std::min(xc, p.nfit - x0);
        DFJK_CUDA(cudaMemsetAsync(Bd.p, 0, (size_t)nx * nn * sizeof(double), s));
        unpack_b_kernel<<<(unsigned)((rows * nx + 255) / 256), 256, 0, s>>>(
            p.d_B.as<double>(), ldb, rows, p.d_row_m.as<int>(), p.d_row_n.as<int>(),
            p.d_row_w.as<int8_t>(), n, x0, nx, Bd.as<double>());
        DFJK_LAUNCHED();
        // T1_x = B_x P_s, Bd_x = P_s T1_x (all symmetric but T1)
        DFJK_CUBLAS(cublasDgemmStridedBatched(c.cublas, CUBLAS_OP_N, CUBLAS_OP_N, (int)n, (int)n,
                                              (int)n, &one, Bd.as<double>(), (int)n, nn, Ps, (int)n,
                                              0, &zero, T1.as<double>(), (int)n, nn, (int)nx));
        DFJK_CUBLAS(cublasDgemmStridedBatched(c.cublas, CUBLAS_OP_N, CUBLAS_OP_N, (int)n, (int)n,
                                              (int)n, &one, Ps, (int)n, 0, T1.as<double>(), (int)n,
                                              nn, &zero, Bd.as<double>(), (int)n, nn, (int)nx));
        h_add_kernel<<<(unsigned)((rows * nx + 255) / 256), 256, 0, s>>>(
            Bd.as<double>(), n, p.d_row_m.as<int>(), p.d_row_n.as<int>(), p.d_row_w.as<int8_t>(),
            rows, ldb, x0, nx, 2.0 * k, H.as<double>());
        DFJK_LAUNCHED();
      }
    }
  }
  // M = H^T B (ldb x ldb); E = 1/2 tr(M)
  const double one = 1.0, zero = 0.0;
  M.alloc((size_t)ldb * ldb * sizeof(double));
  if (rows > 0) {
    DFJK_CUBLAS(cublasDgemm(c.cublas, CUBLAS_OP_N, CUBLAS_OP_T, (int)ldb, (int)ldb, (int)rows, &one,
                            H.as<double>(), (int)ldb, p.d_B.as<double>(), (int)ldb, &zero,
                            M.as<double>(), (int)ldb));
  } else {
    DFJK_CUDA(cudaMemsetAsync(M.p, 0, (size_t)ldb * ldb * sizeof(double), s));
  }
  DevBuf tr;
  tr.alloc(sizeof(double));
  trace_kernel<<<1, 256, 0, s>>>(M.as<double>(), ldb, ldb, tr.as<double>());
  DFJK_LAUNCHED();
  // W = L M L^T
  T.alloc((size_t)naux * ldb * sizeof(double));
  W.alloc((size_t)naux * naux * sizeof(double));
  DFJK_CUBLAS(cublasDgemm(c.cublas, CUBLAS_OP_N, CUBLAS_OP_N, (int)naux, (int)ldb, (int)ldb, &one,
                          p.d_L.as<double>(), (int)naux, M.as<double>(), (int)ldb, &zero,
                          T.as<double>(), (int)naux));
  DFJK_CUBLAS(cublasDgemm(c.cublas, CUBLAS_OP_N, CUBLAS_OP_T, (int)naux, (int)naux, (int)ldb,
                          &one, T.as<double>(), (int)naux, p.d_L.as<double>(), (int)naux,
                          &zero, W.as<double>(), (int)naux));
  M.free();
  T.free();
  launch_grad2c(p, W.as<double>(), grad_aux, s);
  // G = H L^T chunk by chunk, contracted with the 3-center derivatives
  if (rows > 0) {
    auto chunks = pair_chunks(p, naux, chunk_budget(p));
    int64_t maxrows = 1;
    for (auto& ch : chunks) maxrows = std::max(maxrows, rows_of(p, ch.first, ch.second));
    DevBuf G, dsph;
    G.alloc((size_t)maxrows * naux * sizeof(double));
    const int64_t dsph_budget = (int64_t)512 << 20;   // bytes of derivative tables per launch
    dsph.alloc((size_t)dsph_budget);
    auto per_pp = [](const ClassRange& cr) {
      const int nab = (2 * cr.l1 + 1) * (2 * cr.l2 + 1);
      return 3 * (int64_t)nab * hcount(cr.l1 + cr.l2 + 1) * (int64_t)sizeof(double);
    };
    for (auto& ch : chunks) {
      const int64_t r0 = p.pair_row0[ch.first], nr = rows_of(p, ch.first, ch.second);
      DFJK_CUBLAS(cublasDgemm(c.cublas, CUBLAS_OP_N, CUBLAS_OP_N, (int)naux, (int)nr, (int)ldb, &one,
                              p.d_L.as<double>(), (int)naux, H.as<double>() + r0 * ldb, (int)ldb,
                              &zero, G.as<double>(), (int)naux));
      struct Run { const ClassRange* cr; int64_t b, e, bytes; };
      std::vector<Run> runs;
      int64_t total = 0;
      for (const ClassRange& cr : p.classes) {
        const int64_t b = std::max(ch.first, cr.begin), e = std::min(ch.second, cr.begin + cr.count);
        if (b >= e) continue;
        int64_t npp = 0;
        for (int64_t q = b; q < e; ++q) npp += p.pair_npp[q];
        runs.push_back({&cr, b, e, npp * per_pp(cr)});
        total += runs.back().bytes;
      }
      if (total <= dsph_budget) {
        // all classes' tables fit side by side: the classes, independent and
        // mostly too small to fill the device, run on streams of their own
        SideFork side(c, kXcBranches, s);
        double* d = dsph.as<double>();
        for (size_t k = 0; k < runs.size(); ++k) {
          launch_grad3c_pairs(p, *runs[k].cr, runs[k].b, runs[k].e, d, G.as<double>(), r0, grad_orb,
                              grad_aux, side.stream((int)(k % kXcBranches)));
          d += runs[k].bytes / (int64_t)sizeof(double);
        }
        side.join();
        continue;
      }
      for (const Run& run : runs) {
        const ClassRange& cr = *run.cr;
        const int64_t per = per_pp(cr);
        // sub-runs whose primitive pairs' derivative tables fit in dsph
        int64_t q = run.b;
        while (q < run.e) {
          int64_t qe = q, npp = 0;
          while (qe < run.e && (qe == q || (npp + p.pair_npp[qe]) * per <= dsph_budget)) npp += p.pair_npp[qe++];
          if (npp * per > dsph_budget)
            fail(DFJK_ERR_MEMORY, "derivative tables of one shell pair exceed %lld bytes",
                 (long long)dsph_budget);
          launch_grad3c_pairs(p, cr, q, qe, dsph.as<double>(), G.as<double>(), r0, grad_orb,
                              grad_aux, s);
          q = qe;
        }
      }
    }
  }
  double e = 0.0;
  DFJK_CUDA(cudaMemcpyAsync(&e, tr.p, sizeof(double), cudaMemcpyDeviceToHost, s));
  DFJK_CUDA(cudaStreamSynchronize(s));
  return 0.5 * e;
}

}  // namespace dfjk
