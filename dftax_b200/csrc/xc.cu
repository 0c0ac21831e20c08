// Exchange-correlation energy and Fock matrix of a closed-shell density on a
// point grid, and the Becke partition of an atom-centered grid.
//
// Per chunk of G points (dftax/ks/terms.py:776-828, GridXC; energy/grid.py:10-45):
//   Phi[mu][g], dPhi[x][mu][g]   AO values and gradients (ao_kernel: one thread
//                                per point and shell, points fastest, so the
//                                stores of a warp are contiguous), as
//                                dftax/energy/gto.py:371-412 evaluates them;
//   X = Phi P on the float64 tensor cores, kept in registers;
//   rho_g = sum_mu X Phi, grad rho_g = 2 sum_mu X dPhi;
//   e_g = w rho eps_xc(rho, grad rho) and its derivatives v_rho, v_grad by
//   forward-mode dual numbers over the same expression as dftax's PBE
//   (xc.py:87-252, PBE0 :584-601; points with rho <= 1e-10 contribute nothing,
//   as the double-where of grid.py:31-44 makes them);
//   W = v_rho/2 Phi + v_grad . dPhi;
//   V += Phi^T W on the float64 tensor cores;
// and at the end Vxc = V + V^T, the symmetrized P-gradient of E_xc
// (scf.py:42-46). Small chunks keep few functions each and so cost the fewest
// products, but one chunk's kernels fill a fraction of the device: runs of
// chunks (groups) share their launches, and the groups run on two or more
// concurrent streams (group k on branch k % branches, one V accumulator each,
// summed in branch order at the end). The energy is summed per block in a fixed
// order and then over blocks on the host, so the result is reproducible. The
// SCF calls this with the same buffers every iteration: the second call
// captures its launches (nine or ten per group, the branches forked and
// joined by events) in a CUDA graph and later calls replay it.
#include "dmma.cuh"
#include "md_device.cuh"
#include "scf.h"

#include <algorithm>
#include <cmath>
#include <utility>

namespace dfjk {
namespace {

constexpr int kAoThreads = 128;

// ---------------------------------------------------------------------------
// Becke partition
// ---------------------------------------------------------------------------

// one thread per point; the point's distances to the atoms in shared memory
__global__ void becke_kernel(const double* __restrict__ pts, const int* __restrict__ owner,
                             const double* __restrict__ raw, int64_t n,
                             const double* __restrict__ xyz, const double* __restrict__ inv_rab,
                             const double* __restrict__ aab, int natom, double* __restrict__ w) {
  extern __shared__ double sr[];   // [natom][blockDim.x]
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int lt = threadIdx.x, nt = blockDim.x;
  if (i >= n) return;
  const double px = pts[3 * i], py = pts[3 * i + 1], pz = pts[3 * i + 2];
  for (int a = 0; a < natom; ++a) {
    const double dx = px - xyz[3 * a], dy = py - xyz[3 * a + 1], dz = pz - xyz[3 * a + 2];
    sr[a * nt + lt] = sqrt(dx * dx + dy * dy + dz * dz + 1e-30);
  }
  const int own = owner[i];
  double total = 0.0, mine = 0.0;
  for (int a = 0; a < natom; ++a) {
    const double ra = sr[a * nt + lt];
    double cell = 1.0;
    for (int b = 0; b < natom; ++b) {
      if (b == a) continue;
      const double mu = (ra - sr[b * nt + lt]) * inv_rab[a * natom + b];
      double f = mu + aab[a * natom + b] * (1.0 - mu * mu);
      f = 1.5 * f - 0.5 * f * f * f;
      f = 1.5 * f - 0.5 * f * f * f;
      f = 1.5 * f - 0.5 * f * f * f;
      cell *= 0.5 * (1.0 - f);
    }
    total += cell;
    if (a == own) mine = cell;
  }
  w[i] = raw[i] * mine / total;
}

// ---------------------------------------------------------------------------
// AO values and gradients
// ---------------------------------------------------------------------------

// p[n] for 0 <= n <= L (p[0] for n < 0) by selects, so p stays in registers
// whether or not n folds to a constant
template <int L>
__device__ __forceinline__ double pick(const double (&p)[L + 1], int n) {
  double r = p[0];
#pragma unroll
  for (int i = 1; i <= L; ++i) r = n == i ? p[i] : r;
  return r;
}

// values and gradients of one shell's NC cartesian components at (dx, dy,
// dz), in dftax's order (lx descending, then ly), transformed by the shell's
// block T (NC x nout) and stored at o, o + plane, ...; L is a template
// parameter so the component arrays stay in registers
template <int L>
__device__ __forceinline__ void ao_shell(const OrbView& ov, int s, double dx, double dy,
                                         double dz, bool live, int64_t o, int64_t G,
                                         int64_t plane, double* __restrict__ phi,
                                         double* __restrict__ dphi) {
  constexpr int NC = (L + 1) * (L + 2) / 2;
  const ShellView& sh = ov.sh;
  const int nout = ov.nout[L];                 // constant index: no local copy of ov
  const double* __restrict__ T = ov.c2s + ov.c2s_off[L];
  double val[NC], gx[NC], gy[NC], gz[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) val[k] = gx[k] = gy[k] = gz[k] = 0.0;
  if (live) {
    const double r2 = dx * dx + dy * dy + dz * dz;
    double rad = 0.0, drad = 0.0;
    for (int k = 0; k < sh.nprim[s]; ++k) {
      const double a = sh.pexp[sh.prim0[s] + k], c = sh.pcoef[sh.prim0[s] + k];
      const double e = c * exp(-a * r2);
      rad += e;
      drad += -2.0 * a * e;
    }
    double px[L + 1], py[L + 1], pz[L + 1];
    px[0] = py[0] = pz[0] = 1.0;
#pragma unroll
    for (int k = 1; k <= L; ++k) {
      px[k] = px[k - 1] * dx;
      py[k] = py[k - 1] * dy;
      pz[k] = pz[k - 1] * dz;
    }
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const int lx = comp_x(L, k), ly = comp_y(L, k), lz = L - lx - ly;
      const double xl = pick<L>(px, lx), yl = pick<L>(py, ly), zl = pick<L>(pz, lz);
      const double ang = xl * yl * zl;
      val[k] = ang * rad;
      const double dpx = lx * pick<L>(px, lx - 1);
      const double dpy = ly * pick<L>(py, ly - 1);
      const double dpz = lz * pick<L>(pz, lz - 1);
      gx[k] = dpx * yl * zl * rad + ang * drad * dx;
      gy[k] = xl * dpy * zl * rad + ang * drad * dy;
      gz[k] = xl * yl * dpz * rad + ang * drad * dz;
    }
  }
  for (int m = 0; m < nout; ++m) {
    double v = 0.0, a = 0.0, b = 0.0, c = 0.0;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const double t = T[q * nout + m];
      v += val[q] * t;
      a += gx[q] * t;
      b += gy[q] * t;
      c += gz[q] * t;
    }
    const int64_t om = o + (int64_t)m * G;
    phi[om] = v;
    dphi[om] = a;
    dphi[plane + om] = b;
    dphi[2 * plane + om] = c;
  }
}

// Phi[k][g] (ld G), dPhi[x][k][g] of a group's shell entries of angular
// momentum L: entry j is shell e_sh[j] of chunk e_chunk[j] with compact AOs k =
// e_out0[j] .. ; grid (G / 128, entries / kAoPer), kAoPer entries per block (one
// each made the launch of 90 000 blocks of 128 threads the bound). One instance
// per L, so the s and p shells, most of the work, do not carry the registers of
// the d and f cases.
constexpr int kAoPer = 4;
template <int L>
__global__ void __launch_bounds__(kAoThreads) ao_kernel(OrbView ov, const int* __restrict__ e_sh,
                                                        const int* __restrict__ e_out0,
                                                        const int* __restrict__ e_chunk, int nent,
                                                        const XcChunkInfo* __restrict__ info,
                                                        const double* __restrict__ pts, int64_t G,
                                                        double* __restrict__ phi,
                                                        double* __restrict__ dphi) {
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const ShellView& sh = ov.sh;
#pragma unroll 1
  for (int q = 0; q < kAoPer; ++q) {
    const int j = blockIdx.y * kAoPer + q;
    if (j >= nent) return;
    const int s = e_sh[j];
    const XcChunkInfo& ci = info[e_chunk[j]];
    const bool live = g < ci.ng;
    double dx = 0.0, dy = 0.0, dz = 0.0;
    if (live) {
      const double* p = pts + 3 * (ci.g0 + g);
      dx = p[0] - sh.cen[3 * s];
      dy = p[1] - sh.cen[3 * s + 1];
      dz = p[2] - sh.cen[3 * s + 2];
    }
    ao_shell<L>(ov, s, dx, dy, dz, live, (int64_t)e_out0[j] * G + g, G, (int64_t)ci.nsig * G,
                phi + ci.phi, dphi + 3 * ci.phi);
  }
}

// Pc[k1][k2] = P[map[k1]][map[k2]] of chunk blockIdx.y of a group, rows of ldp
// (nsig rounded up to even: the copies of rho_kernel are 16 bytes wide), zero
// in the padding
__global__ void gather_p_kernel(const double* __restrict__ P, int nao, const int* __restrict__ map,
                                const XcChunkInfo* __restrict__ info, double* __restrict__ Pc) {
  const XcChunkInfo& ci = info[blockIdx.y];
  const int64_t n = (int64_t)ci.nsig * ci.ldp;
  const int* mp = map + ci.ao;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = i / ci.ldp, b = i % ci.ldp;
    Pc[ci.pc + i] = b < ci.nsig ? P[(int64_t)mp[a] * nao + mp[b]] : 0.0;
  }
}

// V_y[m][n] += the group's chunks y, y + parts, ... (y = blockIdx.y) that hold
// both functions, chunk by chunk and slice by slice (V + V^T is taken at the end,
// so the products' order does not matter). nao^2 threads alone walk a small
// molecule's 50 chunks in a chain (72 us a group for (H2O)_6): several
// accumulators share it there.
__global__ void reduce_v_kernel(const double* __restrict__ part, int nslice, int count,
                                const XcChunkInfo* __restrict__ info, const int* __restrict__ pos,
                                int nao, double* __restrict__ V) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)nao * nao) return;
  const int m = (int)(i / nao), n = (int)(i % nao);
  double s = 0.0;
  for (int k = blockIdx.y; k < count; k += gridDim.y) {
    const int a = pos[(int64_t)k * nao + m], b = pos[(int64_t)k * nao + n];
    if (a < 0 || b < 0) continue;
    const XcChunkInfo& ci = info[k];
    const int64_t nn = (int64_t)ci.nsig * ci.nsig;
    const double* p = part + ci.part + (int64_t)a * ci.nsig + b;
    for (int z = 0; z < nslice; ++z) s += p[z * nn];
  }
  V[blockIdx.y * (int64_t)nao * nao + i] += s;
}

// ---------------------------------------------------------------------------
// PBE by forward-mode dual numbers. Exchange depends on the density and the norm
// of its gradient, correlation on the density and its own (differently guarded)
// norm: two derivatives carried through each, and the norms' derivatives by hand,
// instead of four (rho, gx, gy, gz) through both.
// ---------------------------------------------------------------------------

struct D2 {
  double v, d[2];
};
__device__ __forceinline__ D2 dc(double c) { return {c, {0.0, 0.0}}; }
__device__ __forceinline__ D2 operator+(D2 a, D2 b) {
  return {a.v + b.v, {a.d[0] + b.d[0], a.d[1] + b.d[1]}};
}
__device__ __forceinline__ D2 operator*(D2 a, D2 b) {
  D2 r;
  r.v = a.v * b.v;
#pragma unroll
  for (int k = 0; k < 2; ++k) r.d[k] = a.d[k] * b.v + a.v * b.d[k];
  return r;
}
// quotient rule as (a' - (a/b) b') / b: one division
__device__ __forceinline__ D2 operator/(D2 a, D2 b) {
  D2 r;
  const double ib = 1.0 / b.v;
  r.v = a.v * ib;
#pragma unroll
  for (int k = 0; k < 2; ++k) r.d[k] = (a.d[k] - r.v * b.d[k]) * ib;
  return r;
}
__device__ __forceinline__ D2 operator+(D2 a, double c) { a.v += c; return a; }
__device__ __forceinline__ D2 operator+(double c, D2 a) { a.v += c; return a; }
__device__ __forceinline__ D2 operator-(double c, D2 a) {
  return {c - a.v, {-a.d[0], -a.d[1]}};
}
__device__ __forceinline__ D2 operator*(D2 a, double c) {
  return {a.v * c, {a.d[0] * c, a.d[1] * c}};
}
__device__ __forceinline__ D2 operator*(double c, D2 a) { return a * c; }
__device__ __forceinline__ D2 operator/(D2 a, double c) { return a * (1.0 / c); }
__device__ __forceinline__ D2 operator/(double c, D2 a) { return dc(c) / a; }
__device__ __forceinline__ D2 dscale(D2 a, double f) {   // chain rule with df/dx = f
  D2 r;
#pragma unroll
  for (int k = 0; k < 2; ++k) r.d[k] = a.d[k] * f;
  return r;
}
__device__ __forceinline__ D2 dsqrt(D2 a) {
  const double q = sqrt(a.v);
  D2 r = dscale(a, 0.5 / q);
  r.v = q;
  return r;
}
// a^(1/3) for a > 0, with d/da = a^(1/3) / (3 a)
__device__ __forceinline__ D2 dcbrt(D2 a) {
  const double q = cbrt(a.v);
  D2 r = dscale(a, q / (3.0 * a.v));
  r.v = q;
  return r;
}
__device__ __forceinline__ D2 dlog1p(D2 a) {
  D2 r = dscale(a, 1.0 / (1.0 + a.v));
  r.v = log1p(a.v);
  return r;
}
__device__ __forceinline__ D2 dexpm1(D2 a) {
  const double q = expm1(a.v);
  D2 r = dscale(a, a.v > -0.5 ? q + 1.0 : exp(a.v));   // e^a = expm1(a) + 1 without cancellation
  r.v = q;
  return r;
}
// jnp.clip(x, lo): the bound itself (derivative 0) below lo
__device__ __forceinline__ D2 dclip(D2 a, double lo) { return a.v < lo ? dc(lo) : a; }

// eps per particle of PBE exchange, unpolarized (xc.py: PBEExchange._unpolarized);
// gnorm = |grad rho + 1e-30|
__device__ __forceinline__ D2 pbe_x(D2 rho, D2 gnorm) {
  constexpr double pi = 3.141592653589793;
  const D2 kF = dcbrt(3 * pi * pi * rho + 1e-30);
  const D2 s = gnorm / dclip(2 * kF * rho, 1e-30);
  const double kappa = 0.804, mu = 0.2195149727645171;
  const D2 ex_unif = -3 * kF / (4 * pi);
  const D2 fx = 1 + kappa - kappa / (1 + mu * s * s / kappa);
  return ex_unif * fx;
}

// eps per particle of PBE correlation with zeta = 0 (xc.py: PBECorrelation): PW92
// paramagnetic channel + PBE H with phi = 1; gn = sqrt(|grad rho|^2 + 1e-30)
__device__ __forceinline__ D2 pbe_c(D2 rho, D2 gn) {
  constexpr double pi = 3.141592653589793;
  const double gamma = (1.0 - 0.6931471805599453) / (pi * pi);
  const double beta = 0.06672455060314922;
  const double A = 0.0310907, a1 = 0.21370, b1 = 7.5957, b2 = 3.5876, b3 = 1.6382, b4 = 0.49294;
  const D2 rt = dclip(rho, 1e-20);
  const D2 rs = dcbrt(3 / (4 * pi * rt) + 1e-20);
  const D2 rss = dsqrt(rs);
  const D2 den = 2.0 * A * (b1 * rss + b2 * rs + b3 * rs * rss + b4 * rs * rs);
  const D2 eps_pw = -2.0 * A * (1.0 + a1 * rs) * dlog1p(1.0 / dclip(den, 1e-20));
  const D2 kf = dcbrt(3 * pi * pi * rt + 1e-20);
  const D2 ks = dsqrt(4 * kf / pi);
  const D2 t = gn / dclip(2 * ks * rt, 1e-20);
  const D2 dA = gamma * dexpm1(-1.0 * eps_pw / gamma);
  const D2 Ac = beta / dclip(dA, 1e-20);
  const D2 t2 = t * t;
  const D2 f1 = t2 + Ac * (t2 * t2);
  const D2 frac = beta * f1 / dclip(gamma * (1.0 + Ac * f1), 1e-20);
  return eps_pw + gamma * dlog1p(frac);
}

// per point of chunk blockIdx.y: rho, grad in, v_rho / 2, v_grad (weighted) out in
// place (vals [4][G] per chunk); e per block
constexpr int kPtThreads = 128;
__global__ void __launch_bounds__(kPtThreads) pbe_kernel(double* __restrict__ vals,
                                                         const XcChunkInfo* __restrict__ info,
                                                         int64_t G, const double* __restrict__ wts,
                                                         double xs, double cs, double thresh,
                                                         double* __restrict__ eg) {
  __shared__ double red[kPtThreads / 32];
  const XcChunkInfo ci = info[blockIdx.y];
  const int64_t g = blockIdx.x * (int64_t)kPtThreads + threadIdx.x;
  double* v = vals + blockIdx.y * 4 * G + g;
  double e = 0.0, vr = 0.0, v0 = 0.0, v1 = 0.0, v2 = 0.0;
  const double r = g < ci.ng ? v[0] : 0.0;
  if (r > thresh) {
    const double w = wts[ci.g0 + g], gx = v[G], gy = v[2 * G], gz = v[3 * G];
    const double ax = gx + 1e-30, ay = gy + 1e-30, az = gz + 1e-30;
    const double na = sqrt(ax * ax + ay * ay + az * az);
    const double nb = sqrt(gx * gx + gy * gy + gz * gz + 1e-30);
    const D2 R = {r, {1.0, 0.0}};
    const D2 fx = R * (xs * pbe_x(R, D2{na, {0.0, 1.0}}));
    const D2 fc = R * (cs * pbe_c(R, D2{nb, {0.0, 1.0}}));
    e = w * (fx.v + fc.v);
    vr = 0.5 * w * (fx.d[0] + fc.d[0]);
    const double qa = w * fx.d[1] / na, qb = w * fc.d[1] / nb;
    v0 = qa * ax + qb * gx;
    v1 = qa * ay + qb * gy;
    v2 = qa * az + qb * gz;
  }
  v[0] = vr;
  v[G] = v0;
  v[2 * G] = v1;
  v[3 * G] = v2;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 1; q < kPtThreads / 32; ++q) e += red[q];
    eg[blockIdx.y * (int64_t)gridDim.x + blockIdx.x] = e;
  }
}

// W[mu][g] = v_rho/2 Phi + v_grad . dPhi of chunk blockIdx.z: two points per
// thread (16-byte accesses), kWPer functions per block. Bound by memory: 40 bytes
// per function and point.
constexpr int kWThreads = 128, kWPer = 8;
__global__ void __launch_bounds__(kWThreads) w_kernel(const double* __restrict__ phig,
                                                      const double* __restrict__ dphig,
                                                      const double* __restrict__ vals,
                                                      const XcChunkInfo* __restrict__ info, int64_t G,
                                                      double* __restrict__ Wg) {
  const XcChunkInfo ci = info[blockIdx.z];
  const int c0 = blockIdx.y * kWPer;
  if (c0 >= ci.nsig) return;
  const int64_t g = 2 * (blockIdx.x * (int64_t)kWThreads + threadIdx.x);   // G is a multiple of 256
  const int64_t plane = (int64_t)ci.nsig * G;
  const double* phi = phig + ci.phi + g;
  const double* dphi = dphig + 3 * ci.phi + g;
  double* W = Wg + ci.phi + g;
  double2 v[4];
#pragma unroll
  for (int d = 0; d < 4; ++d)
    v[d] = *reinterpret_cast<const double2*>(vals + (blockIdx.z * 4 + d) * G + g);
#pragma unroll
  for (int q = 0; q < kWPer; ++q) {
    const int c = c0 + q;
    if (c >= ci.nsig) break;
    const int64_t o = c * G;
    const double2 f = __ldg(reinterpret_cast<const double2*>(phi + o));
    double2 s = make_double2(v[0].x * f.x, v[0].y * f.y);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double2 t = __ldg(reinterpret_cast<const double2*>(dphi + d * plane + o));
      s.x += v[1 + d].x * t.x;
      s.y += v[1 + d].y * t.y;
    }
    *reinterpret_cast<double2*>(W + o) = s;
  }
}

// rho and grad rho of 64 points of a chunk per block (grid (G / 64, chunks of the
// group)), without X in memory:
//   * X = Phi Pc for all nsig functions, 64 columns at a time, on the float64
//     tensor cores: 16 functions per step through a four-stage cp.async ring
//     that runs on across the column blocks (the order of points and columns
//     inside a fragment is free: a lane's pair of fragments is one 16-byte load);
//   * after each column block the lane's X meets Phi and dPhi of the same
//     (point, function) pairs and adds to rho and grad rho;
//   * the partial sums of a point's lanes are added in a fixed order.
// As a cuBLAS DGEMM and a density kernel per chunk (H2O)_6 took 800 us. (With the
// functional and W in the same block, 64 of 256 threads on the former, a block
// took twice as long: 689 us per evaluation against the split kernels' sum.)
constexpr int kRpPts = 64, kRpCols = 64, kRpK = 16, kRpPitch = 68, kRpStages = 4;
constexpr int kRpStage = 2 * kRpK * kRpPitch;   // doubles
constexpr size_t kRpSmem = (size_t)kRpStages * kRpStage * sizeof(double);

__global__ void __launch_bounds__(256, 3) rho_kernel(
    const double* __restrict__ Pg, const double* __restrict__ phig, const double* __restrict__ dphig,
    const XcChunkInfo* __restrict__ info, int64_t G, double* __restrict__ vals) {
  const XcChunkInfo ci = info[blockIdx.y];
  const int nsig = ci.nsig, ldp = ci.ldp;
  const double* Pc = Pg + ci.pc;
  const double* phi = phig + ci.phi;
  const double* dphi = dphig + 3 * ci.phi;
  extern __shared__ __align__(16) double rsm[];
  __shared__ double red[2][4][kRpPts];   // per column half: rho, grad
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wx = (warp & 3) * 16, wi = (warp >> 2) * 32;
  const int fr = lane >> 2, fk = lane & 3;
  const int64_t g0 = blockIdx.x * (int64_t)kRpPts;
  const int64_t plane = (int64_t)nsig * G;
  const int nk = (nsig + kRpK - 1) / kRpK, ncb = (nsig + kRpCols - 1) / kRpCols;
  const int steps = nk * ncb;
  const int bk = tid >> 5, bx = 2 * (tid & 31);
  auto stage = [&](int q) {
    double* As = rsm + (q % kRpStages) * kRpStage;
    double* Bs = As + kRpK * kRpPitch;
    const int k0 = q % nk * kRpK, c = q / nk * kRpCols + bx;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int k = k0 + bk + 8 * j;
      const bool in = k < nsig, inc = in && c < ldp;
      cp_async16(As + (bk + 8 * j) * kRpPitch + bx, in ? phi + k * G + g0 + bx : phi, in);
      cp_async16(Bs + (bk + 8 * j) * kRpPitch + bx, inc ? Pc + (int64_t)k * ldp + c : Pc, inc);
    }
  };
  for (int q = 0; q < kRpStages - 1; ++q) {
    if (q < steps) stage(q);
    cp_async_commit();
  }
  // a column block's dPhi, 512 bytes of 3 x 64 rows, on its way to L2 while the
  // block's products run: its epilogue reads it ((H2O)_6, 512-point chunks: 1040 ->
  // 1013 us an evaluation)
  auto ahead = [&](int cb) {
    const int d = tid >> 6, c = cb * kRpCols + (tid & 63);
    if (d < 3 && c < nsig) prefetch_l2(dphi + d * plane + c * G + g0, kRpPts * sizeof(double));
  };
  double acc[2][4][2], sum[4][2];   // sum: rho, grad of the lane's two points
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll
  for (int d = 0; d < 4; ++d) sum[d][0] = sum[d][1] = 0.0;
  for (int q = 0; q < steps; ++q) {
    cp_async_wait<kRpStages - 2>();
    __syncthreads();
    if (q + kRpStages - 1 < steps) stage(q + kRpStages - 1);
    cp_async_commit();
    const double* As = rsm + (q % kRpStages) * kRpStage;
    const double* Bs = As + kRpK * kRpPitch;
    if (q % nk == 0) ahead(q / nk);
    if (q / nk * kRpCols + wi < nsig) {   // else the warp's columns lie past the functions
#pragma unroll
      for (int kk = 0; kk < kRpK; kk += 4) {
        const double2 av = *reinterpret_cast<const double2*>(As + (kk + fk) * kRpPitch + wx + 2 * fr);
        const double af[2] = {av.x, av.y};
        double bf[4];
#pragma unroll
        for (int b = 0; b < 4; b += 2) {
          const double2 v =
              *reinterpret_cast<const double2*>(Bs + (kk + fk) * kRpPitch + wi + 8 * b + 2 * fr);
          bf[b] = v.x;
          bf[b + 1] = v.y;
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) dmma_8x8x4(acc[a][b], af[a], bf[b]);
      }
    }
    if (q % nk == nk - 1) {
      // fragment (a, b), register r: point wx + 2 (lane / 4) + a, column
      // wi + 8 (b & ~1) + 4 (lane % 4) + 2 r + (b & 1)
      const int c0 = q / nk * kRpCols + wi;
      const double* at = phi + g0 + wx + 2 * fr;
      const double* dat = dphi + g0 + wx + 2 * fr;
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int c = c0 + 8 * (b & ~1) + 4 * fk + 2 * r + (b & 1);
          if (c < nsig) {
            const double x0 = acc[0][b][r], x1 = acc[1][b][r];
            const double2 f = __ldg(reinterpret_cast<const double2*>(at + c * G));
            sum[0][0] += x0 * f.x;
            sum[0][1] += x1 * f.y;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const double2 v = __ldg(reinterpret_cast<const double2*>(dat + d * plane + c * G));
              sum[1 + d][0] += x0 * v.x;
              sum[1 + d][1] += x1 * v.y;
            }
          }
          acc[0][b][r] = acc[1][b][r] = 0.0;
        }
    }
  }
  // the four lanes of a point, then the two column halves
#pragma unroll
  for (int d = 0; d < 4; ++d)
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      double s = sum[d][a];
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (fk == 0) red[warp >> 2][d][wx + 2 * fr + a] = s;
    }
  __syncthreads();
  {
    const int d = tid / kRpPts, g = tid % kRpPts;   // 256 threads: four sums of 64 points
    vals[(blockIdx.y * 4 + d) * G + g0 + g] = (d == 0 ? 1.0 : 2.0) * (red[0][d][g] + red[1][d][g]);
  }
}

// part[z][mu][nu] = sum_g Phi[mu][g] W[nu][g] over slice z = blockIdx.y of
// kVSlice points of chunk blockIdx.z (tile blockIdx.x, of the chunk's own count):
// 64 x 64 tiles on the float64 tensor cores, both operands staged as they lie
// (16 points a step, the 16-byte piece index xor 4 (row % 2): load phases of
// two rows x four pieces fall in distinct banks; the point order inside a step
// is free) through a four-stage cp.async ring with one barrier per step. The
// output is small and the sum long, so slices fill the device; 512 points keep
// a block's prologue and partial store near a tenth of its products.
constexpr int kVT = 64, kVK = 16, kVStages = 4, kVSlice = 512;
constexpr size_t kVSmem = (size_t)kVStages * 2 * kVT * kVK * sizeof(double);

__global__ void __launch_bounds__(256, 3) v_kernel(const double* __restrict__ phig,
                                                   const double* __restrict__ Wg,
                                                   const XcChunkInfo* __restrict__ info, int64_t G,
                                                   double* __restrict__ part) {
  extern __shared__ __align__(16) double vsm[];
  const XcChunkInfo ci = info[blockIdx.z];
  const int nsig = ci.nsig, nt = (nsig + kVT - 1) / kVT;
  if ((int)blockIdx.x >= nt * nt) return;
  const double* phi = phig + ci.phi;
  const double* W = Wg + ci.phi;
  const int r0 = (int)blockIdx.x / nt * kVT, c0 = (int)blockIdx.x % nt * kVT;
  const int64_t k0 = blockIdx.y * (int64_t)kVSlice;
  const int64_t k1 = k0 + kVSlice < G ? k0 + kVSlice : G;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // rows turned by block and column half: the warps past nsig then leave different
  // quarters of the SM, with their tensor pipes, idle ((H2O)_6: 1013 -> 1005 us)
  const int wr = ((warp + (warp >> 1 & 2) + (int)(blockIdx.x + blockIdx.y + blockIdx.z)) & 3) * 16;
  const int wc = (warp >> 2) * 32;
  const int fr = lane >> 2, fk = lane & 3;
  const bool work = r0 + wr < nsig && c0 + wc < nsig;
  double acc[2][4][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  const int nst = (int)((k1 - k0) / kVK);   // G and the slices are multiples of 16
  const int sr = tid >> 3, sp = tid & 7;
  auto stage = [&](int q) {
    double* As = vsm + (size_t)(q % kVStages) * (2 * kVT * kVK);
    const int64_t k = k0 + (int64_t)q * kVK + 2 * sp;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = sr + 32 * j, o = r * kVK + 2 * (sp ^ (4 * (r & 1)));
      const bool oa = r0 + r < nsig, ob = c0 + r < nsig;
      cp_async16(As + o, oa ? phi + (int64_t)(r0 + r) * G + k : phi, oa);
      cp_async16(As + kVT * kVK + o, ob ? W + (int64_t)(c0 + r) * G + k : W, ob);
    }
  };
  for (int q = 0; q < kVStages - 1; ++q) {
    if (q < nst) stage(q);
    cp_async_commit();
  }
  for (int q = 0; q < nst; ++q) {
    cp_async_wait<kVStages - 2>();
    __syncthreads();
    if (q + kVStages - 1 < nst) stage(q + kVStages - 1);
    cp_async_commit();
    if (!work) continue;
    const double* As = vsm + (size_t)(q % kVStages) * (2 * kVT * kVK);
    const double* Bs = As + kVT * kVK;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int piece = 2 * ((4 * h + fk) ^ (4 * (fr & 1)));
      double2 af[2], bf[4];
#pragma unroll
      for (int a = 0; a < 2; ++a)
        af[a] = *reinterpret_cast<const double2*>(As + (wr + 8 * a + fr) * kVK + piece);
#pragma unroll
      for (int b = 0; b < 4; ++b)
        bf[b] = *reinterpret_cast<const double2*>(Bs + (wc + 8 * b + fr) * kVK + piece);
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) dmma_8x8x4(acc[a][b], af[a].x, bf[b].x);
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) dmma_8x8x4(acc[a][b], af[a].y, bf[b].y);
    }
  }
  if (!work) return;
  double* out = part + ci.part + blockIdx.y * (int64_t)nsig * nsig;
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const int r = r0 + wr + 8 * a + fr;
    if (r >= nsig) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = c0 + wc + 8 * b + 2 * fk + q;
        if (c < nsig) out[(int64_t)r * nsig + c] = acc[a][b][q];
      }
  }
}

// out = sum over the nb branch accumulators V_b (n x n, stride n*n) of
// V_b + V_b^T, in branch order
__global__ void symmetrize_sum_kernel(const double* __restrict__ V, int nb, int n,
                                      double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nn = (int64_t)n * n;
  if (i >= nn) return;
  const int64_t r = i / n, c = i % n;
  double s = 0.0;
  for (int b = 0; b < nb; ++b) s += V[b * nn + i] + V[b * nn + c * n + r];
  out[i] = s;
}

}  // namespace

void launch_becke_partition(const double* pts, const int* owner, const double* raw, int64_t n,
                            const double* atom_xyz, const double* bragg, int natom, double* w,
                            cudaStream_t s) {
  if (n <= 0) return;
  // pair tables: 1 / R_AB and the size adjustment a_AB (becke.py: becke_partition)
  std::vector<double> inv((size_t)natom * natom, 0.0), aab((size_t)natom * natom, 0.0);
  for (int a = 0; a < natom; ++a)
    for (int b = 0; b < natom; ++b) {
      if (a == b) continue;
      const double dx = atom_xyz[3 * a] - atom_xyz[3 * b], dy = atom_xyz[3 * a + 1] - atom_xyz[3 * b + 1],
                   dz = atom_xyz[3 * a + 2] - atom_xyz[3 * b + 2];
      inv[(size_t)a * natom + b] = 1.0 / std::sqrt(dx * dx + dy * dy + dz * dz);
      const double chi = bragg[a] / bragg[b];
      const double u = (chi - 1.0) / (chi + 1.0);
      aab[(size_t)a * natom + b] = std::min(0.45, std::max(-0.45, u / (u * u - 1.0)));
    }
  std::vector<double> xyz(atom_xyz, atom_xyz + 3 * natom);
  DevBuf dxyz, dinv, daab;
  upload(dxyz, xyz);
  upload(dinv, inv);
  upload(daab, aab);
  int threads = 64;
  const size_t smem = (size_t)natom * threads * sizeof(double);
  if (smem > 200 * 1024) fail(DFJK_ERR_UNSUPPORTED, "Becke partition supports at most 400 atoms");
  allow_shared(becke_kernel);
  becke_kernel<<<(unsigned)((n + threads - 1) / threads), threads, smem, s>>>(
      pts, owner, raw, n, dxyz.as<double>(), dinv.as<double>(), daab.as<double>(), natom, w);
  DFJK_LAUNCHED();
  DFJK_CUDA(cudaStreamSynchronize(s));   // the pair tables are freed on return
}

// slices of a chunk's V product
static_assert(kXcMaxChunk / kVSlice < 65536, "slices: a grid dimension");
static int64_t xc_slices(int64_t G) { return (G + kVSlice - 1) / kVSlice; }

// V accumulators per branch: enough that their nao^2 threads each come to about
// 2^18
static int64_t v_parts(int64_t nao) {
  return std::min<int64_t>(8, std::max<int64_t>(1, ((int64_t)1 << 18) / (nao * nao)));
}

// A chunk of nsig functions takes 40 nsig G bytes of its group's, and beside them
// 8 nsig (nsig + 1) for its P block and 8 nsig^2 per slice of V: most, as a share of
// the group, with all nao functions. Four values a point, a function a point at least.
// A small grid does not fill a group.
int64_t xc_branch_bytes(int64_t nao, int64_t G, int64_t npoint) {
  const int64_t all = 40 * nao * ((npoint + G - 1) / G * G);
  const int64_t group = std::max(std::min(kXcGroupBytes, all), 40 * nao * G);
  const double share = (double)(nao + 1 + xc_slices(G) * nao) / (5.0 * (double)G);
  return group + (int64_t)(share * (double)group) + 32 * std::min(npoint + G, group / 40) +
         v_parts(nao) * nao * nao * 8;
}

void xc_chunk(const Shells& sh, const int (&nout)[8], int64_t n, const std::vector<double>& boxes,
              int64_t G, double thresh, XcWork& ws) {
  XcChunks& out = ws.ch;
  out.info.clear();
  out.groups.clear();
  out.max_phi = out.max_pc = out.max_part = out.max_points = 0;
  out.gemm_flop = 0.0;
  out.G = G;
  if (ws.exec) cudaGraphExecDestroy(ws.exec);
  ws.exec = nullptr;
  for (auto& a : ws.g_args) a = nullptr;
  ws.calls = 0;
  if (n == 0) return;
  // per shell: |phi| + |grad phi| <= sum_k |c_k| (1 + r^l + l r^(l-1) + 2 a_k r^(l+1)) e^(-a_k r^2)
  // for r beyond the distance d from the shell to a box, the polynomial taken
  // at max(d, its peak) (it decreases past sqrt((l+1)/(2 a_k))) and the
  // Gaussian at d
  auto bound = [&](int s, double d) {
    const int l = sh.l[s];
    double b = 0.0;
    for (int k = 0; k < sh.nprim[s]; ++k) {
      const double a = sh.pexp[sh.prim0[s] + k], c = std::fabs(sh.pcoef[sh.prim0[s] + k]);
      const double r = std::max(d, std::sqrt((l + 1) / (2.0 * a)));
      const double rl = std::pow(r, l);
      b += c * (1.0 + rl + (l > 0 ? l * rl / r : 0.0) + 2.0 * a * rl * r) * std::exp(-a * d * d);
    }
    return b;
  };
  const int nao = sh.nout;
  std::vector<int> aomap, pos;
  struct Entry {
    int sh, out0, chunk;
  };
  std::vector<Entry> ents[kXcMaxL + 1];   // of the open group, by l
  std::vector<int> e_sh, e_out0, e_chunk;
  XcGroup grp;
  int64_t phi = 0, pc = 0, part = 0;
  const int64_t nslice = xc_slices(G);
  auto close = [&] {
    if (grp.count == 0) return;
    grp.e_off = (int)e_sh.size();
    for (int l = 0; l <= kXcMaxL; ++l) {
      grp.e_cnt[l] = (int)ents[l].size();
      for (const Entry& e : ents[l]) {
        e_sh.push_back(e.sh);
        e_out0.push_back(e.out0);
        e_chunk.push_back(e.chunk);
      }
      ents[l].clear();
    }
    out.max_phi = std::max(out.max_phi, phi);
    out.max_pc = std::max(out.max_pc, pc);
    out.max_part = std::max(out.max_part, part);
    out.max_points = std::max(out.max_points, grp.count * G);
    out.groups.push_back(grp);
    grp = XcGroup{};
    phi = pc = part = 0;
  };
  // each chunk's shells
  struct Chunk {
    int64_t g0, ng;
    int nsig;
    std::vector<int> shells;
  };
  std::vector<Chunk> chunks;
  for (int64_t g0 = 0; g0 < n; g0 += G) {
    Chunk ch{g0, std::min(G, n - g0), 0, {}};
    double bl[3] = {INFINITY, INFINITY, INFINITY}, bh[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t b = g0 / kXcBox; b < (g0 + ch.ng + kXcBox - 1) / kXcBox; ++b)
      for (int d = 0; d < 3; ++d) {
        bl[d] = std::min(bl[d], boxes[6 * b + d]);
        bh[d] = std::max(bh[d], boxes[6 * b + 3 + d]);
      }
    for (int s = 0; s < sh.n; ++s) {
      double d2 = 0.0;
      for (int d = 0; d < 3; ++d) {
        const double c = sh.cen[3 * s + d];
        const double e = c < bl[d] ? bl[d] - c : (c > bh[d] ? c - bh[d] : 0.0);
        d2 += e * e;
      }
      if (bound(s, std::sqrt(d2)) <= thresh) continue;
      ch.shells.push_back(s);
      ch.nsig += nout[sh.l[s]];
    }
    // (without functions a chunk adds nothing: it stays out of the launches, which
    // take a group's chunks in a grid dimension of at most 65535)
    if (ch.nsig > 0) chunks.push_back(std::move(ch));
  }
  // the chunks with the most functions first: a group's chunks are then alike,
  // and a launch ends on its shortest blocks ((H2O)_6: 1052 -> 1040 us, (H2O)_8:
  // 1690 -> 1654)
  std::stable_sort(chunks.begin(), chunks.end(),
                   [](const Chunk& a, const Chunk& b) { return a.nsig > b.nsig; });
  for (const Chunk& ch : chunks) {
    const int nsig = ch.nsig;
    const int64_t ao = (int64_t)aomap.size();
    pos.resize(pos.size() + nao, -1);
    int* ps = pos.data() + pos.size() - nao;
    int c = 0;
    std::vector<Entry> mine;
    for (int s : ch.shells) {
      mine.push_back({s, c, 0});
      const int no = nout[sh.l[s]];
      for (int m = 0; m < no; ++m) {
        aomap.push_back(sh.out0[s] + m);
        ps[sh.out0[s] + m] = c + m;
      }
      c += no;
    }
    // AO values, three gradients and the weighted AOs: 40 bytes per function and point
    if (grp.count > 0 && (phi + (int64_t)nsig * G) * 40 > kXcGroupBytes) close();
    XcChunkInfo ci{nsig, nsig + (nsig & 1), ch.g0, ch.ng, phi, pc, part, ao};
    if (grp.count == 0) grp.first = (int)out.info.size();
    for (Entry e : mine) {
      e.chunk = grp.count;
      ents[std::min<int>(sh.l[e.sh], kXcMaxL)].push_back(e);
    }
    ++grp.count;
    grp.max_nsig = std::max(grp.max_nsig, nsig);
    phi += (int64_t)nsig * G;
    pc += (int64_t)nsig * ci.ldp;
    part += nslice * nsig * nsig;
    out.info.push_back(ci);
    out.gemm_flop += 4.0 * (double)G * nsig * nsig;   // X = Phi P and Phi^T W
  }
  close();
  upload(out.d_e_sh, e_sh);
  upload(out.d_e_out0, e_out0);
  upload(out.d_e_chunk, e_chunk);
  upload(out.d_ao_map, aomap);
  upload(out.d_pos, pos);
  upload(out.d_info, out.info);
}

// enqueues one evaluation's device work on s (buffers already sized)
static void xc_enqueue(const Context& c, const OrbView& ov, const double* pts, const double* w,
                       const double* P, double* Vxc, const XcParams& xp, XcWork& ws,
                       cudaStream_t s) {
  const int nao = ov.nao;
  const int64_t nn = (int64_t)nao * nao;
  const XcChunks& ch = ws.ch;
  const int64_t G = ch.G;
  const int64_t nblk = G / kPtThreads;
  const int nslice = (int)xc_slices(G);
  const int64_t parts = v_parts(nao);
  const int nb = std::min(std::max(ws.nbr, 1), kXcBranches);
  // fork: every branch starts after the caller's prior work on s
  DFJK_CUDA(cudaEventRecord(c.side_fork, s));
  for (int q = 0; q < nb; ++q) DFJK_CUDA(cudaStreamWaitEvent(c.side_stream[q], c.side_fork, 0));
  if (Vxc)
    for (int q = 0; q < nb; ++q)
      DFJK_CUDA(cudaMemsetAsync(ws.Vacc.as<double>() + q * parts * nn, 0, parts * nn * sizeof(double),
                                c.side_stream[q]));
  for (size_t k = 0; k < ch.groups.size(); ++k) {
    const XcGroup& gr = ch.groups[k];
    XcBranch& b = ws.br[k % nb];
    cudaStream_t bs = c.side_stream[k % nb];
    double* Vacc = ws.Vacc.as<double>() + (k % nb) * parts * nn;
    const XcChunkInfo* info = ch.d_info.as<XcChunkInfo>() + gr.first;
    double* phi = b.phi.as<double>();
    double* dphi = b.dphi.as<double>();
    // the group's shell entries lie by l: one launch per l present
    int j0 = gr.e_off;
    for (int l = 0; l < kXcMaxL + 1; ++l) {
      const int cnt = gr.e_cnt[l];
      if (cnt == 0) continue;
      const dim3 grid((unsigned)((G + kAoThreads - 1) / kAoThreads), (unsigned)((cnt + kAoPer - 1) / kAoPer));
      const int* es = ch.d_e_sh.as<int>() + j0;
      const int* eo = ch.d_e_out0.as<int>() + j0;
      const int* ec = ch.d_e_chunk.as<int>() + j0;
      switch (l) {
        case 0: ao_kernel<0><<<grid, kAoThreads, 0, bs>>>(ov, es, eo, ec, cnt, info, pts, G, phi, dphi); break;
        case 1: ao_kernel<1><<<grid, kAoThreads, 0, bs>>>(ov, es, eo, ec, cnt, info, pts, G, phi, dphi); break;
        case 2: ao_kernel<2><<<grid, kAoThreads, 0, bs>>>(ov, es, eo, ec, cnt, info, pts, G, phi, dphi); break;
        default: ao_kernel<3><<<grid, kAoThreads, 0, bs>>>(ov, es, eo, ec, cnt, info, pts, G, phi, dphi); break;
      }
      DFJK_LAUNCHED();
      j0 += cnt;
    }
    if (gr.max_nsig > 0) {
      const int64_t pn = (int64_t)gr.max_nsig * (gr.max_nsig + 1);
      gather_p_kernel<<<dim3((unsigned)std::min<int64_t>(64, (pn + 255) / 256), (unsigned)gr.count), 256, 0, bs>>>(
          P, nao, ch.d_ao_map.as<int>(), info, b.Pc.as<double>());
      DFJK_LAUNCHED();
    }
    rho_kernel<<<dim3((unsigned)(G / kRpPts), (unsigned)gr.count), 256, kRpSmem, bs>>>(
        b.Pc.as<double>(), phi, dphi, info, G, b.vals.as<double>());
    DFJK_LAUNCHED();
    pbe_kernel<<<dim3((unsigned)nblk, (unsigned)gr.count), kPtThreads, 0, bs>>>(
        b.vals.as<double>(), info, G, w, xp.x_scale, xp.c_scale, xp.rho_thresh,
        ws.ered.as<double>() + gr.first * nblk);
    DFJK_LAUNCHED();
    if (Vxc && gr.max_nsig > 0) {
      w_kernel<<<dim3((unsigned)(G / (2 * kWThreads)), (unsigned)((gr.max_nsig + kWPer - 1) / kWPer),
                      (unsigned)gr.count), kWThreads, 0, bs>>>(phi, dphi, b.vals.as<double>(), info, G,
                                                               b.W.as<double>());
      DFJK_LAUNCHED();
      const unsigned nt = (unsigned)((gr.max_nsig + kVT - 1) / kVT);
      v_kernel<<<dim3(nt * nt, (unsigned)nslice, (unsigned)gr.count), 256, kVSmem, bs>>>(
          phi, b.W.as<double>(), info, G, b.Vc.as<double>());
      DFJK_LAUNCHED();
      reduce_v_kernel<<<dim3((unsigned)((nn + 255) / 256), (unsigned)parts), 256, 0, bs>>>(
          b.Vc.as<double>(), nslice, gr.count, info, ch.d_pos.as<int>() + (int64_t)gr.first * nao,
          nao, Vacc);
      DFJK_LAUNCHED();
    }
  }
  // join: s waits for every branch
  for (int q = 0; q < nb; ++q) {
    DFJK_CUDA(cudaEventRecord(c.side_done[q], c.side_stream[q]));
    DFJK_CUDA(cudaStreamWaitEvent(s, c.side_done[q], 0));
  }
  if (Vxc) {
    symmetrize_sum_kernel<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(ws.Vacc.as<double>(),
                                                                        (int)(nb * parts), nao, Vxc);
    DFJK_LAUNCHED();
  }
}

double xc_energy_fock(const Context& c, const OrbView& ov, const double* pts, const double* w,
                      const double* P, double* Vxc, const XcParams& xp, XcWork& ws,
                      cudaStream_t s, double* Vcopy) {
  const int nao = ov.nao;
  const XcChunks& ch = ws.ch;
  const int64_t G = ch.G;
  const int64_t nchunk = (int64_t)ch.info.size();
  const int64_t nblk = G / kPtThreads;   // G is a multiple of 256
  for (int q = 0; q < std::min(std::max(ws.nbr, 1), kXcBranches); ++q) {
    XcBranch& b = ws.br[q];
    b.phi.ensure(ch.max_phi * sizeof(double));
    b.dphi.ensure(3 * ch.max_phi * sizeof(double));
    b.W.ensure(ch.max_phi * sizeof(double));
    b.vals.ensure(4 * ch.max_points * sizeof(double));
    b.Pc.ensure(ch.max_pc * sizeof(double));
    if (Vxc) b.Vc.ensure(ch.max_part * sizeof(double));
  }
  DFJK_CUDA(cudaFuncSetAttribute(rho_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRpSmem));
  DFJK_CUDA(cudaFuncSetAttribute(v_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVSmem));
  // the side streams and events are made here on first use, never during a capture
  side_streams(const_cast<Context&>(c));
  ws.ered.ensure((size_t)std::max<int64_t>(nchunk, 1) * nblk * sizeof(double));
  if (Vxc) ws.Vacc.ensure((size_t)std::max(ws.nbr, 1) * v_parts(nao) * nao * nao * sizeof(double));
  const void* args[4] = {P, Vxc, pts, w};
  const bool same = std::equal(args, args + 4, ws.g_args);
  if (ws.exec && same) {
    DFJK_CUDA(cudaGraphLaunch(ws.exec, s));
    count_launch(ws.graph_kernels);
  } else if (!ws.graph_off && ws.calls > 0 && Vxc) {
    // capture this call's work (the buffers above are already sized)
    if (ws.exec) {
      DFJK_CUDA(cudaGraphExecDestroy(ws.exec));
      ws.exec = nullptr;
    }
    if (!ws.cap) DFJK_CUDA(cudaStreamCreateWithFlags(&ws.cap, cudaStreamNonBlocking));
    const int64_t k0 = dfjk_kernel_launches();
    cudaGraph_t graph = nullptr;
    bool ok;
    {
      // no other thread of the library synchronizes the device meanwhile
      std::lock_guard<std::recursive_mutex> cap(capture_mutex());
      ok = cudaStreamBeginCapture(ws.cap, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
      if (ok) {
        try {
          xc_enqueue(c, ov, pts, w, P, Vxc, xp, ws, ws.cap);
        } catch (...) {
          ok = false;
        }
        const cudaError_t ec = cudaStreamEndCapture(ws.cap, &graph);
        ok = ok && ec == cudaSuccess && graph;
      }
    }
    if (ok) ok = cudaGraphInstantiate(&ws.exec, graph, 0) == cudaSuccess;
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    if (ok) {
      ws.graph_kernels = dfjk_kernel_launches() - k0;
      std::copy(args, args + 4, ws.g_args);
      DFJK_CUDA(cudaGraphLaunch(ws.exec, s));
    } else {
      // the same kernels, launched directly
      ws.exec = nullptr;
      ws.graph_off = true;
      xc_enqueue(c, ov, pts, w, P, Vxc, xp, ws, s);
    }
  } else {
    xc_enqueue(c, ov, pts, w, P, Vxc, xp, ws, s);
  }
  ++ws.calls;
  if (Vcopy && Vxc)
    DFJK_CUDA(cudaMemcpyAsync(Vcopy, Vxc, (size_t)nao * nao * sizeof(double),
                              cudaMemcpyDeviceToDevice, s));
  std::vector<double> e((size_t)nchunk * nblk);
  if (!e.empty())
    DFJK_CUDA(cudaMemcpyAsync(e.data(), ws.ered.p, e.size() * sizeof(double),
                              cudaMemcpyDeviceToHost, s));
  DFJK_CUDA(cudaStreamSynchronize(s));
  double sum = 0.0;
  for (double v : e) sum += v;
  return sum;
}

}  // namespace dfjk
