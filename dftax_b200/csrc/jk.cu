// J and K contractions over the fitted tensor B.
//
// B is row-major [nrows][ldb]: one row per AO pair (m, n) of a kept shell
// pair, one column per kept metric direction (B = (mn|P) L, L L^T = V+).
//
//   J: d[r] = w_r D[m, n]                (w_r = 2 off-diagonal pair, else 1)
//      gamma = B^T d                      (stream B once; CTA partials + reduce)
//      J[m, n] = J[n, m] = B[r] . gamma   (stream B again; warp per row)
//   K: X[m][x][i] = sum_{(r, n) in list(m)} B[r][x] C'[n][i]   (half transform)
//      K = X X^T over the (x, i) index, C' = C sqrt|w|
// Float64 plans run both K products on the float64 tensor cores (mma.sync
// m8n8k4 f64: the gathered half transform, then a split-k X X^T); mixed plans
// run them on the int8 tensor cores (ozaki.cu). J is float64 in both. J and K
// are the P-gradients of dftax's DFCoulomb.energy (terms.py:592-613):
// J = int3c (V+ gamma), K = einsum("mlP,PQ,nsQ,ls->mn") (hybrid.py:23-41).
#include "dmma.cuh"
#include "internal.h"

#include <algorithm>
#include <cmath>

namespace dfjk {

// ---------------------------------------------------------------------------
// J
// ---------------------------------------------------------------------------

// 32 bytes of B, read once: no L1 allocation (p 32-byte aligned)
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
  asm volatile("ld.global.nc.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
               : "l"(p));
}

// The density whose J is taken: sum_i w_i C[m][i] C[n][i] of ncol orbitals (w
// null: ones), or the matrix D when C is null.
struct DensitySource {
  const double* C;
  const double* w;
  int64_t ncol;
  const double* D;
};

// gamma partials: CTA (bx, by) sums rows [r0, r1) for columns [by*2048, +2048).
// The rows' weights d[r] = w_r D[m, n] are formed 32 at a time by the block
// itself (a warp takes four), so no launch and no array come before it. Bound by
// memory: 32-byte loads, four rows in flight per thread, four blocks per SM read
// 7.2 TB/s of a 14.5 GB B (16-byte loads of two rows: 6.7).
constexpr int kGtThreads = 256;
constexpr int kGtCols = kGtThreads * 8;
constexpr int kGtRows = 32;

__global__ void __launch_bounds__(kGtThreads) gamma_partial_kernel(
    const double* __restrict__ B, int64_t ldb, int64_t nrows, DensitySource src, int64_t nao,
    const int* __restrict__ rm, const int* __restrict__ rn, const int8_t* __restrict__ kind,
    int64_t rows_per_cta, double* __restrict__ part) {
  __shared__ double sd[kGtRows];
  const int64_t r0 = blockIdx.x * rows_per_cta;
  const int64_t r1 = min(nrows, r0 + rows_per_cta);
  // columns c0 .. + 3 and c0 + 1024 .. + 3 (ldb is a multiple of 8)
  const int64_t c0 = (int64_t)blockIdx.y * kGtCols + 4 * threadIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double acc[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[j][u] = 0.0;
  for (int64_t t0 = r0; t0 < r1; t0 += kGtRows) {
    if (src.C) {
#pragma unroll
      for (int q = 0; q < kGtRows / 8; ++q) {
        const int64_t r = t0 + warp + 8 * q;
        double s = 0.0;
        if (r < r1) {
          const double* cm = src.C + (int64_t)rm[r] * src.ncol;
          const double* cn = src.C + (int64_t)rn[r] * src.ncol;
          for (int64_t i = lane; i < src.ncol; i += 32)
            s += (src.w ? src.w[i] : 1.0) * cm[i] * cn[i];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        // off-diagonal pairs stand for both (m, n) and (n, m)
        if (lane == 0 && r < r1) sd[warp + 8 * q] = kind[r] == 2 ? 2.0 * s : s;
      }
    } else if (threadIdx.x < kGtRows && t0 + threadIdx.x < r1) {
      const int64_t r = t0 + threadIdx.x;
      const int64_t m = rm[r], n = rn[r];
      sd[threadIdx.x] = kind[r] == 2 ? src.D[m * nao + n] + src.D[n * nao + m] : src.D[m * nao + n];
    }
    __syncthreads();
    const int nr = (int)min(r1 - t0, (int64_t)kGtRows);
#pragma unroll 4
    for (int q = 0; q < nr; ++q) {
      const double d = sd[q];
      const double* row = B + (t0 + q) * ldb;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int64_t c = c0 + j * 4 * kGtThreads;
        if (c < ldb) {
          double v[4];
          load4(row + c, v);
#pragma unroll
          for (int u = 0; u < 4; ++u) acc[j][u] += d * v[u];
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int64_t c = c0 + j * 4 * kGtThreads;
    if (c < ldb)
#pragma unroll
      for (int u = 0; u < 4; ++u) part[blockIdx.x * ldb + c + u] = acc[j][u];
  }
}

// out[c] = sum_p part[p][c], bound by the latency of its dependent adds: one
// thread per column left them serial (592 partials: 61-81 us at every size, on
// 1-15 blocks). A block takes 32 columns; thread (y, x) sums the partials y,
// y + 32, ... of column x (a warp reads 256 contiguous bytes), and 32 sums are
// added in a fixed order: 3-5 us, reproducible.
constexpr int kRrCols = 32, kRrLanes = 32;
__global__ void __launch_bounds__(kRrCols * kRrLanes) reduce_rows_kernel(
    const double* __restrict__ part, int64_t nparts, int64_t ldb, double* __restrict__ out) {
  __shared__ double red[kRrLanes][kRrCols + 1];
  const int x = threadIdx.x % kRrCols, y = threadIdx.x / kRrCols;
  const int64_t c = blockIdx.x * (int64_t)kRrCols + x;
  double s = 0.0;
  if (c < ldb) {
#pragma unroll 4
    for (int64_t p = y; p < nparts; p += kRrLanes) s += part[p * ldb + c];
  }
  red[y][x] = s;
  __syncthreads();
  // warp y adds the lanes of column y by a shuffle tree (a fixed order)
  double t = red[x][y];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  const int64_t cc = blockIdx.x * (int64_t)kRrCols + y;
  if (x == 0 && cc < ldb) out[cc] = t;
}

static void launch_reduce_rows(const double* part, int64_t nparts, int64_t ldb, double* out,
                               cudaStream_t s) {
  reduce_rows_kernel<<<(unsigned)((ldb + kRrCols - 1) / kRrCols), kRrCols * kRrLanes, 0, s>>>(
      part, nparts, ldb, out);
  DFJK_LAUNCHED();
}

// J rows: one warp per row, J[m, n] and J[n, m]. Bound by memory: two 32-byte
// loads per lane in flight, 64 warps per SM (6.8 TB/s of a 14.5 GB B; four
// 16-byte loads: 5.7).
__global__ void __launch_bounds__(256) j_rows_kernel(
    const double* __restrict__ B, int64_t ldb, int64_t nrows, const double* __restrict__ gamma,
    const int* __restrict__ rm, const int* __restrict__ rn, const int8_t* __restrict__ kind,
    int64_t nao, double* __restrict__ J) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = (gridDim.x * (int64_t)blockDim.x) >> 5;
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < nrows; r += nwarps) {
    const double* row = B + r * ldb;
    // ldb is a multiple of 8 and c of 4: a load that starts inside the row ends there
    double s2[2] = {0.0, 0.0};
    auto add = [&](const double (&b)[4], int64_t c, double& s) {
      const double2 g0 = __ldg(reinterpret_cast<const double2*>(gamma + c));
      const double2 g1 = __ldg(reinterpret_cast<const double2*>(gamma + c + 2));
      s += b[0] * g0.x + b[1] * g0.y + b[2] * g1.x + b[3] * g1.y;
    };
    int64_t c = 4 * lane;
    for (; c + 128 < ldb; c += 256) {
      double b0[4], b1[4];
      load4(row + c, b0);
      load4(row + c + 128, b1);
      add(b0, c, s2[0]);
      add(b1, c + 128, s2[1]);
    }
    if (c < ldb) {
      double b0[4];
      load4(row + c, b0);
      add(b0, c, s2[0]);
    }
    double s = s2[0] + s2[1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const int k = kind[r];
      if (k == 0) continue;
      const int m = rm[r], n = rn[r];
      J[(int64_t)m * nao + n] = s;
      J[(int64_t)n * nao + m] = s;
    }
  }
}

int num_sms(int dev) {
  int n = 0;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 148;
}

__global__ void add_to_kernel(const double* __restrict__ x, int64_t n, double* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] += x[i];
}

// gamma (+)= Bc^T d over nrows rows of Bc (rows from row0 of the plan): fixed-
// order partial sums. At least eight rows per block, so that a small B leaves
// few partials to add.
static void gamma_rows(Plan& p, const double* Bc, int64_t row0, int64_t nrows,
                       const DensitySource& src, double* out, bool add, cudaStream_t s) {
  const int sms = num_sms(p.ctx->device);
  const int64_t ycols = (p.ldb + kGtCols - 1) / kGtCols;
  int64_t xparts = std::max<int64_t>(1, (int64_t)sms * 4 / ycols);
  xparts = std::min<int64_t>(xparts, (nrows + 7) / 8);
  const int64_t rows_per = (nrows + xparts - 1) / xparts;
  xparts = (nrows + rows_per - 1) / rows_per;
  DevBuf& part = p.ws_part;
  part.ensure((size_t)(xparts + (add ? 1 : 0)) * p.ldb * sizeof(double));
  double* sum = part.as<double>() + xparts * p.ldb;   // the chunk's gamma when adding
  gamma_partial_kernel<<<dim3((unsigned)xparts, (unsigned)ycols), kGtThreads, 0, s>>>(
      Bc, p.ldb, nrows, src, p.nao, p.d_row_m.as<int>() + row0, p.d_row_n.as<int>() + row0,
      p.d_row_w.as<int8_t>() + row0, rows_per, part.as<double>());
  DFJK_LAUNCHED();
  launch_reduce_rows(part.as<double>(), xparts, p.ldb, add ? sum : out, s);
  if (add) {
    add_to_kernel<<<(unsigned)((p.ldb + 255) / 256), 256, 0, s>>>(sum, p.ldb, out);
    DFJK_LAUNCHED();
  }
}

// gamma = B^T d into `gamma` (ldb doubles)
static void gamma_of(Plan& p, const DensitySource& src, double* gamma, cudaStream_t s) {
  if (p.opts.streamed || p.nrows == 0) {
    DFJK_CUDA(cudaMemsetAsync(gamma, 0, p.ldb * sizeof(double), s));
    if (p.nrows == 0) return;
    for_each_b_chunk(p, s, [&](int64_t r0, int64_t nr, const double* Bc) {
      if (nr > 0) gamma_rows(p, Bc, r0, nr, src, gamma, true, s);
    });
    return;
  }
  gamma_rows(p, p.d_B.as<double>(), 0, p.nrows, src, gamma, false, s);
}

static void j_from_gamma(Plan& p, const double* gamma, double* J, cudaStream_t s) {
  // without screening every element belongs to a row
  if (p.opts.screen > 0.0 || p.nrows == 0)
    DFJK_CUDA(cudaMemsetAsync(J, 0, (size_t)p.nao * p.nao * sizeof(double), s));
  if (p.nrows == 0) return;
  const int sms = num_sms(p.ctx->device);
  if (p.opts.streamed) {
    for_each_b_chunk(p, s, [&](int64_t r0, int64_t nr, const double* Bc) {
      if (nr == 0) return;
      const int64_t warps = std::min<int64_t>(nr, (int64_t)sms * 64);
      j_rows_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, s>>>(
          Bc, p.ldb, nr, gamma, p.d_row_m.as<int>() + r0, p.d_row_n.as<int>() + r0,
          p.d_row_w.as<int8_t>() + r0, p.nao, J);
      DFJK_LAUNCHED();
    });
    return;
  }
  const int64_t warps = std::min<int64_t>(p.nrows, (int64_t)sms * 64);
  j_rows_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, s>>>(
      p.d_B.as<double>(), p.ldb, p.nrows, gamma, p.d_row_m.as<int>(), p.d_row_n.as<int>(),
      p.d_row_w.as<int8_t>(), p.nao, J);
  DFJK_LAUNCHED();
}

// ---------------------------------------------------------------------------
// K: half transform X[m][x][i] = sum_{(r, n) in list(m)} B[r][x0 + x] C'[n][i]
// ---------------------------------------------------------------------------

// On the float64 tensor cores (mma.sync m8n8k4 f64: tcgen05 has no float64
// kind). A block of eight warps computes 64 directions x HtTile::I columns of
// one m, 16 list entries per k chunk, through a ring of three or four stages of
// 16-byte copies (three blocks per SM) with one barrier per chunk. Bound by the DMMA pipe once nocc
// is above ~20 columns: the tile's width follows the columns (half_tile), since
// columns of padding cost as much as real ones.
//   * Warps: WI of them side by side over the columns, 8 / WI over the
//     directions; a warp holds XF x IF fragments of 8 x 8.
//   * The order of rows and columns inside a fragment is free, so neighbouring
//     fragments interleave: a lane's elements of a pair of fragments are
//     adjacent and come with one 16-byte load. Rows of 64 + 4 and I + 4 doubles
//     put the 8 lanes of a load phase (4 k, 2 rows) in distinct banks.
// (H2O)_12 (nocc 60): 1353 us with 80-column tiles, 8-byte copies and two
// stages; see half_tile for the widths.
constexpr int kHtX = 64, kHtK = 16, kHtPX = kHtX + 4;

template <int IF_, int WI_>
struct HtTile {
  static constexpr int IF = IF_, WI = WI_, WX = 8 / WI, XF = kHtX / (8 * WX);
  static constexpr int I = 8 * IF * WI, PI = I + 4;
  static constexpr int kStage = kHtK * (kHtPX + PI);   // doubles
  static constexpr int kStages = 3 * 4 * kStage * 8 <= 224 * 1024 ? 4 : 3;
  static constexpr size_t smem = (size_t)kStages * kStage * sizeof(double);
};

// The list of m is entries [kbeg[m], kend[m]) (kend == nullptr: up to
// kbeg[m + 1]); entry e reads B row krow[e] - row0. accumulate: X += instead
// of X = (a streamed plan sums the chunks of B rows). ldb and ncol are even,
// B and Cp 16-byte aligned and x0 a multiple of 64, so every copy and store is
// aligned.
template <class T>
__global__ void __launch_bounds__(256, 3) half_transform_kernel(
    const double* __restrict__ B, int64_t ldb, int64_t x0, int64_t xc, const double* __restrict__ Cp,
    int64_t ncol, const int* __restrict__ kbeg, const int* __restrict__ kend,
    const int* __restrict__ krow, const int* __restrict__ kn, int64_t row0, int accumulate,
    double* __restrict__ X) {
  constexpr int XF = T::XF, IF = T::IF, PI = T::PI, kHtStages = T::kStages;
  constexpr int kCg = kHtK * T::I / 2, kCper = (kCg + 255) / 256;   // 16-byte copies of C' rows
  extern __shared__ __align__(16) double ht_smem[];
  const int m = blockIdx.x;
  const int64_t xt = (int64_t)blockIdx.y * kHtX;   // within the chunk
  const int64_t it = (int64_t)blockIdx.z * T::I;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wx = (warp % T::WX) * 8 * XF, wi = (warp / T::WX) * 8 * IF;
  const int fr = lane >> 2, fk = lane & 3;   // fragment row / k of this lane
  double acc[XF][IF][2];
#pragma unroll
  for (int a = 0; a < XF; ++a)
#pragma unroll
    for (int b = 0; b < IF; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  const int e0 = kbeg[m], e1 = kend ? kend[m] : kbeg[m + 1];
  const int nch = (e1 - e0 + kHtK - 1) / kHtK;
  // this thread's copies of a chunk: B rows tid / 32 and tid / 32 + 8 (one
  // 16-byte piece of each), kCper pieces of C' rows. Their list entries are
  // read one chunk ahead, so a copy never waits for its index.
  const int bk = tid >> 5, bx = 2 * (tid & 31);
  const bool bin = x0 + xt + bx < ldb;
  int nr[2], nn[kCper];
  auto fetch = [&](int c) {
    const int e = e0 + c * kHtK;
#pragma unroll
    for (int j = 0; j < 2; ++j) nr[j] = e + bk + 8 * j < e1 ? krow[e + bk + 8 * j] : -1;
#pragma unroll
    for (int j = 0; j < kCper; ++j) {
      const int k = (tid + 256 * j) / (T::I / 2);
      nn[j] = k < kHtK && e + k < e1 ? kn[e + k] : -1;
    }
  };
  auto stage = [&](int c) {
    double* Bs = ht_smem + (c % kHtStages) * T::kStage;
    double* Cs = Bs + kHtK * kHtPX;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const bool ok = nr[j] >= 0 && bin;
      cp_async16(Bs + (bk + 8 * j) * kHtPX + bx,
                 ok ? B + ((int64_t)nr[j] - row0) * ldb + x0 + xt + bx : B, ok);
    }
#pragma unroll
    for (int j = 0; j < kCper; ++j) {
      const int q = tid + 256 * j, k = q / (T::I / 2), i = 2 * (q % (T::I / 2));
      if (q >= kCg) break;
      const bool ok = nn[j] >= 0 && it + i < ncol;
      cp_async16(Cs + k * PI + i, ok ? Cp + (int64_t)nn[j] * ncol + it + i : Cp, ok);
    }
  };
  if (nch > 0) fetch(0);
  for (int c = 0; c < kHtStages - 1; ++c) {
    if (c < nch) {
      stage(c);
      if (c + 1 < nch) fetch(c + 1);
    }
    cp_async_commit();
  }
  for (int c = 0; c < nch; ++c) {
    // chunk c has landed, and every warp is done with the buffer of chunk c - 1
    cp_async_wait<kHtStages - 2>();
    __syncthreads();
    if (c + kHtStages - 1 < nch) {
      stage(c + kHtStages - 1);
      if (c + kHtStages < nch) fetch(c + kHtStages);
    }
    cp_async_commit();
    const double* Bs = ht_smem + (c % kHtStages) * T::kStage;
    const double* Cs = Bs + kHtK * kHtPX;
#pragma unroll
    for (int kk = 0; kk < kHtK; kk += 4) {
      double af[XF], bf[IF];
      if constexpr (XF == 2) {
        const double2 v = *reinterpret_cast<const double2*>(Bs + (kk + fk) * kHtPX + wx + 2 * fr);
        af[0] = v.x;
        af[1] = v.y;
      } else {
        af[0] = Bs[(kk + fk) * kHtPX + wx + fr];
      }
#pragma unroll
      for (int b = 0; b + 1 < IF; b += 2) {
        const double2 v =
            *reinterpret_cast<const double2*>(Cs + (kk + fk) * PI + wi + 8 * b + 2 * fr);
        bf[b] = v.x;
        bf[b + 1] = v.y;
      }
      if constexpr (IF % 2) bf[IF - 1] = Cs[(kk + fk) * PI + wi + 8 * (IF - 1) + fr];
#pragma unroll
      for (int a = 0; a < XF; ++a)
#pragma unroll
        for (int b = 0; b < IF; ++b) dmma_8x8x4(acc[a][b], af[a], bf[b]);
    }
  }
  // fragment (a, b), register r of this lane: direction wx + XF (lane / 4) + a;
  // column 8 b + 2 (2 (lane % 4) + r) + {0, 1} over a pair b, b + 1, and
  // 8 b + 2 (lane % 4) + r in an unpaired last fragment
  auto put = [&](double* o, double u, double v) {
    if (accumulate) {
      const double2 p = *reinterpret_cast<const double2*>(o);
      u += p.x;
      v += p.y;
    }
    *reinterpret_cast<double2*>(o) = make_double2(u, v);
  };
#pragma unroll
  for (int a = 0; a < XF; ++a) {
    const int64_t x = xt + wx + XF * fr + a;
    if (x >= xc) continue;
    double* row = X + ((int64_t)m * xc + x) * ncol;
#pragma unroll
    for (int b = 0; b + 1 < IF; b += 2)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int64_t i = it + wi + 8 * b + 4 * fk + 2 * r;
        if (i < ncol) put(row + i, acc[a][b][r], acc[a][b + 1][r]);
      }
    if constexpr (IF % 2) {
      const int64_t i = it + wi + 8 * (IF - 1) + 2 * fk;
      if (i < ncol) put(row + i, acc[a][IF - 1][0], acc[a][IF - 1][1]);
    }
  }
}

template <class T>
static void launch_half(const double* B, int64_t ldb, int64_t x0, int64_t xc, const double* Cp,
                        int64_t ncol, const int* kbeg, const int* kend, const int* krow,
                        const int* kn, int64_t row0, int accumulate, int64_t nao, double* X,
                        cudaStream_t s) {
  DFJK_CUDA(cudaFuncSetAttribute(half_transform_kernel<T>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem));
  const dim3 grid((unsigned)nao, (unsigned)((xc + kHtX - 1) / kHtX),
                  (unsigned)((ncol + T::I - 1) / T::I));
  half_transform_kernel<T><<<grid, 256, T::smem, s>>>(B, ldb, x0, xc, Cp, ncol, kbeg, kend, krow,
                                                      kn, row0, accumulate, X);
  DFJK_LAUNCHED();
}

// Column tile of the half transform: every tile streams the rows of B again
// and pays a prologue and an epilogue, worth about 12 columns, so the width
// with the smallest tiles x (width + 12) is taken (60 columns: one tile of 64,
// 160: two of 80, 82: two of 48).
static int half_tile(int64_t ncol) {
  int best = 80;
  int64_t cost = INT64_MAX;
  for (int w : {80, 64, 48, 40, 32, 24, 16, 8}) {
    const int64_t c = (ncol + w - 1) / w * (w + 12);
    if (c < cost) {
      cost = c;
      best = w;
    }
  }
  return best;
}

template <class... A>
static void launch_half_any(int64_t ncol, A... a) {
  switch (half_tile(ncol)) {
    case 8: launch_half<HtTile<1, 1>>(a...); return;
    case 16: launch_half<HtTile<2, 1>>(a...); return;
    case 24: launch_half<HtTile<3, 1>>(a...); return;
    case 32: launch_half<HtTile<4, 1>>(a...); return;
    case 40: launch_half<HtTile<5, 1>>(a...); return;
    case 48: launch_half<HtTile<3, 2>>(a...); return;
    case 64: launch_half<HtTile<4, 2>>(a...); return;
    default: launch_half<HtTile<5, 2>>(a...); return;
  }
}

// [kb[m], ke[m]): the entries of m's K list whose rows lie in [r0, r1) (each
// list is in ascending row order)
__global__ void list_bounds_kernel(const int* __restrict__ kptr, const int* __restrict__ krow,
                                   int64_t nao, int64_t r0, int64_t r1, int* __restrict__ kb,
                                   int* __restrict__ ke) {
  const int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (m >= nao) return;
  auto lower = [&](int lo, int hi, int64_t v) {
    while (lo < hi) {
      const int mid = lo + (hi - lo) / 2;
      if (krow[mid] < v) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  const int lo = kptr[m], hi = kptr[m + 1];
  kb[m] = lower(lo, hi, r0);
  ke[m] = lower(lo, hi, r1);
}

// K partials on the float64 tensor cores: for lower-triangle tile pair number
// blockIdx.x (tm >= tn, 64 x 64) and the k slice blockIdx.y,
// part[slice][tm*64 + r][tn*64 + c] = sum_k X[tm*64 + r][k] X[tn*64 + c][k]
// over the slice (X row-major, nao x kt, kt even). Bound by the DMMA pipe.
// Rows are staged as they lie, 16 k (eight 16-byte pieces, the piece index
// xor 4 (row % 2)) per chunk through a four-stage cp.async ring with one barrier
// per chunk; the k order inside a chunk is free, so a lane takes k pairs
// 2 (lane % 4) and its two k steps come with one 16-byte load, whose phases of
// two rows x four pieces fall in distinct banks. Tiles on the diagonal stage
// their rows once, and warps whose part lies above the diagonal or past nao
// skip their products.
constexpr int kSyT = 64, kSyK = 16, kSyStages = 4;
constexpr size_t kSySmem = (size_t)kSyStages * 2 * kSyT * kSyK * sizeof(double);

__global__ void __launch_bounds__(256, 3) syrk_part_kernel(const double* __restrict__ X, int64_t nao,
                                                           int64_t kt, int64_t kslice,
                                                           double* __restrict__ part) {
  extern __shared__ __align__(16) double sy_smem[];
  int tm = (int)((sqrt(8.0 * blockIdx.x + 1.0) - 1.0) * 0.5);
  while ((tm + 1) * (tm + 2) / 2 <= (int)blockIdx.x) ++tm;
  while (tm * (tm + 1) / 2 > (int)blockIdx.x) --tm;
  const int tn = (int)blockIdx.x - tm * (tm + 1) / 2;
  const bool diag = tm == tn;
  const int64_t r0 = (int64_t)tm * kSyT, c0 = (int64_t)tn * kSyT;
  const int64_t k0 = (int64_t)blockIdx.y * kslice;
  const int64_t k1 = k0 + kslice < kt ? k0 + kslice : kt;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // 16 rows x 32 columns a warp. Warps with nothing to do (above the diagonal, past
  // nao) leave the tensor pipe of their quarter of the SM idle, so the rows go to
  // the warps turned by block and column half ((H2O)_12: 572 -> 562 us).
  const int wr = ((warp + (warp >> 1 & 2) + (int)(blockIdx.x + blockIdx.y)) & 3) * 16;
  const int wc = (warp >> 2) * 32;
  const int fr = lane >> 2, fk = lane & 3;
  const bool work = r0 + wr < nao && c0 + wc < nao && !(diag && wc > wr + 15);
  double acc[2][4][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  const int nch = (int)((k1 - k0 + kSyK - 1) / kSyK);
  // this thread's copies of a chunk: rows tid / 8 and tid / 8 + 32, piece tid % 8
  const int sr = tid >> 3, sp = tid & 7;
  auto stage = [&](int c) {
    double* As = sy_smem + (size_t)(c % kSyStages) * (2 * kSyT * kSyK);
    const int64_t k = k0 + (int64_t)c * kSyK + 2 * sp;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = sr + 32 * j, o = r * kSyK + 2 * (sp ^ (4 * (r & 1)));
      const bool oa = k < k1 && r0 + r < nao;
      cp_async16(As + o, oa ? X + (r0 + r) * kt + k : X, oa);
      if (!diag) {
        const bool ob = k < k1 && c0 + r < nao;
        cp_async16(As + kSyT * kSyK + o, ob ? X + (c0 + r) * kt + k : X, ob);
      }
    }
  };
  for (int c = 0; c < kSyStages - 1; ++c) {
    if (c < nch) stage(c);
    cp_async_commit();
  }
  for (int c = 0; c < nch; ++c) {
    cp_async_wait<kSyStages - 2>();
    __syncthreads();
    if (c + kSyStages - 1 < nch) stage(c + kSyStages - 1);
    cp_async_commit();
    if (!work) continue;
    const double* As = sy_smem + (size_t)(c % kSyStages) * (2 * kSyT * kSyK);
    const double* Bs = diag ? As : As + kSyT * kSyK;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // k pairs 8 h + 2 fk, + 1 of this lane (rows differ by 8: the same parity)
      const int piece = 2 * ((4 * h + fk) ^ (4 * (fr & 1)));
      double2 af[2], bf[4];
#pragma unroll
      for (int a = 0; a < 2; ++a)
        af[a] = *reinterpret_cast<const double2*>(As + (wr + 8 * a + fr) * kSyK + piece);
#pragma unroll
      for (int b = 0; b < 4; ++b)
        bf[b] = *reinterpret_cast<const double2*>(Bs + (wc + 8 * b + fr) * kSyK + piece);
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
  double* out = part + (int64_t)blockIdx.y * nao * nao;
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const int64_t r = r0 + wr + 8 * a + fr;
    if (r >= nao) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int64_t c = c0 + wc + 8 * b + 2 * fk + q;
        if (c < nao) out[r * nao + c] = acc[a][b][q];
      }
  }
}

// K[i][j] = (beta0 ? 0 : K[i][j]) + sign * sum_s part[s][max(i,j)][min(i,j)], s in order
__global__ void syrk_reduce_kernel(const double* __restrict__ part, int64_t nsplit, int64_t nao,
                                   double sign, int beta0, double* __restrict__ K) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nao * nao) return;
  const int64_t i = t / nao, j = t % nao;
  const int64_t src = i >= j ? i * nao + j : j * nao + i;
  double acc = 0.0;
  for (int64_t s = 0; s < nsplit; ++s) acc += part[s * nao * nao + src];
  K[t] = beta0 ? sign * acc : K[t] + sign * acc;
}

// C'[m][j] = sqrt|w| C[m][sel[j]] for j < nsel (sel == nullptr: column j), zero
// in the padding columns up to ncp; C[m][j] lies at C[m * sm + j * sc]
__global__ void scale_cols_kernel(const double* __restrict__ C, const double* __restrict__ w,
                                  int64_t nao, int64_t sm, int64_t sc, const int* __restrict__ sel,
                                  int64_t nsel, int64_t ncp, double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nao * ncp) return;
  const int64_t m = i / ncp, j = i % ncp;
  double v = 0.0;
  if (j < nsel) {
    const int64_t col = sel ? sel[j] : j;
    v = C[m * sm + col * sc] * (w ? sqrt(fabs(w[col])) : 1.0);
  }
  out[i] = v;
}

void pack_columns(const double* Ct, int64_t nao, int64_t rank, int64_t ncp, double* Cp, cudaStream_t s) {
  scale_cols_kernel<<<(unsigned)((nao * ncp + 255) / 256), 256, 0, s>>>(Ct, nullptr, nao, 1, nao, nullptr,
                                                                       rank, ncp, Cp);
  DFJK_LAUNCHED();
}

void half_transform(Plan& p, const double* Cp, int64_t ncp, int64_t x0, int64_t n, double* X,
                    cudaStream_t s) {
  launch_half_any(ncp, (const double*)p.d_B.as<double>(), p.ldb, x0, n, Cp, ncp,
                  (const int*)p.d_kptr.as<int>(), (const int*)nullptr,
                  (const int*)p.d_krow.as<int>(), (const int*)p.d_kn.as<int>(), (int64_t)0, 0,
                  (int64_t)p.nao, X, s);
}

// K (+)= sign * X X^T (float64, full square) for X nao x kt row-major: lower
// 64 x 64 tile pairs times k slices, then a fixed-order sum of the slices
// (bit-reproducible). Three blocks run per SM; the slice count is the one whose
// waves x (slice length + 128: a block's prologue and partial stores in units
// of k) is smallest. One slice per 1024 k left a single block at small sizes
// ((H2O)_1: 46 us) and 1.4 waves at (H2O)_12 (719 us).
static void syrk_fp64(Plan& p, const double* X, int64_t kt, double sign, bool beta0, double* K,
                      cudaStream_t s) {
  const int64_t nao = p.nao;
  const int64_t nt = (nao + kSyT - 1) / kSyT, tiles = nt * (nt + 1) / 2;
  const int64_t slots = 3 * (int64_t)num_sms(p.ctx->device);
  const int64_t most = std::min<int64_t>(64, std::max<int64_t>(1, kt / 64));
  int64_t nsplit = 1;
  int64_t best = INT64_MAX;
  for (int64_t q = 1; q <= most; ++q) {
    const int64_t t = (tiles * q + slots - 1) / slots * ((kt + q - 1) / q + 128);
    if (best == INT64_MAX || 100 * t < 98 * best) {   // (a slice costs a partial of K)
      best = t;
      nsplit = q;
    }
  }
  const int64_t kslice = ((kt + nsplit - 1) / nsplit + kSyK - 1) / kSyK * kSyK;
  nsplit = (kt + kslice - 1) / kslice;
  p.ws_syrk.ensure((size_t)nsplit * nao * nao * sizeof(double));
  DFJK_CUDA(cudaFuncSetAttribute(syrk_part_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSySmem));
  syrk_part_kernel<<<dim3((unsigned)tiles, (unsigned)nsplit), 256, kSySmem, s>>>(
      X, nao, kt, kslice, p.ws_syrk.as<double>());
  DFJK_LAUNCHED();
  syrk_reduce_kernel<<<(unsigned)((nao * nao + 255) / 256), 256, 0, s>>>(
      p.ws_syrk.as<double>(), nsplit, nao, sign, beta0 ? 1 : 0, K);
  DFJK_LAUNCHED();
}

// Streamed plans: gamma = B^T d summed in the K half transform's first pass over
// B's chunks (one rebuild of B fewer per J/K call).
struct GammaFuse {
  DensitySource src;
  double* gamma = nullptr;
  bool done = false;
};

// K (+)= sign * X X^T for nsel columns of C (scaled by sqrt|w|): those of `sel`
// (host indices), or the first nsel when null; C[m][j] lies at C[m * sm + j * sc].
// fuse (streamed plans only) may be null
static void k_accumulate(Plan& p, const double* C, int64_t sm, int64_t sc, const double* w,
                         const std::vector<int>* sel, int64_t nsel, double sign, bool first,
                         double* K, cudaStream_t s, GammaFuse* fuse = nullptr) {
  const int64_t nao = p.nao;
  if (nsel == 0) return;
  DevBuf& dsel = p.ws_sel;
  DevBuf& Cp = p.ws_Cp;
  if (sel) {
    dsel.ensure(nsel * sizeof(int));
    DFJK_CUDA(cudaMemcpyAsync(dsel.p, sel->data(), nsel * sizeof(int), cudaMemcpyHostToDevice, s));
  }
  // an even number of columns (a zero one added) keeps the rows of C' and X
  // 16-byte aligned for the wide copies and the TMA stores of both forms;
  // unweighted columns that already lie so are used where they are
  const int64_t ncp = nsel + (nsel & 1);
  const double* Cc = C;
  if (w || sel || sc != 1 || sm != ncp || (reinterpret_cast<uintptr_t>(C) & 15)) {
    Cp.ensure((size_t)nao * ncp * sizeof(double));
    Cc = Cp.as<double>();
    scale_cols_kernel<<<(unsigned)((nao * ncp + 255) / 256), 256, 0, s>>>(
        C, w, nao, sm, sc, sel ? dsel.as<int>() : nullptr, nsel, ncp, Cp.as<double>());
    DFJK_LAUNCHED();
  }
  // x chunking so that X (nao * xc * ncp doubles) stays within budget; a
  // streamed plan rebuilds B once per x chunk, so it takes up to half the
  // free device memory
  int64_t budget = (int64_t)6 << 30;
  if (p.opts.streamed) {
    size_t fr = 0, tot = 0;
    DFJK_CUDA(cudaMemGetInfo(&fr, &tot));
    budget = std::max<int64_t>(budget, (int64_t)(fr / 2));
  }
  int64_t xc = budget / (nao * ncp * (int64_t)sizeof(double));
  xc = std::max<int64_t>(kHtX, xc / kHtX * kHtX);
  xc = std::min<int64_t>(xc, (p.nfit + kHtX - 1) / kHtX * kHtX);
  DevBuf& X = p.ws_X;
  X.ensure((size_t)nao * xc * ncp * sizeof(double));
  bool beta0 = first;
  for (int64_t x0 = 0; x0 < p.nfit; x0 += xc) {
    const int64_t n = std::min(xc, p.nfit - x0);
    p.timer.mark(kPhKhalf, s);
    const bool oz = p.opts.precision == DFJK_MIXED && !p.opts.streamed;
    if (p.opts.streamed) {
      // X = sum over chunks of B rows of the half transform of each chunk
      DFJK_CUDA(cudaMemsetAsync(X.p, 0, (size_t)nao * n * ncp * sizeof(double), s));
      p.ws_kb.ensure(nao * sizeof(int));
      p.ws_ke.ensure(nao * sizeof(int));
      const bool with_gamma = fuse && !fuse->done;
      if (with_gamma) DFJK_CUDA(cudaMemsetAsync(fuse->gamma, 0, p.ldb * sizeof(double), s));
      for_each_b_chunk(p, s, [&](int64_t r0, int64_t nr, const double* Bc) {
        if (with_gamma && nr > 0) gamma_rows(p, Bc, r0, nr, fuse->src, fuse->gamma, true, s);
        list_bounds_kernel<<<(unsigned)((nao + 255) / 256), 256, 0, s>>>(
            p.d_kptr.as<int>(), p.d_krow.as<int>(), nao, r0, r0 + nr, p.ws_kb.as<int>(),
            p.ws_ke.as<int>());
        DFJK_LAUNCHED();
        launch_half_any(ncp, Bc, p.ldb, x0, n, Cc, ncp,
                        (const int*)p.ws_kb.as<int>(), (const int*)p.ws_ke.as<int>(),
                        (const int*)p.d_krow.as<int>(), (const int*)p.d_kn.as<int>(), r0, 1, nao,
                        X.as<double>(), s);
      });
      if (with_gamma) fuse->done = true;
    } else if (oz) {
      if (x0 == 0) ozaki_prepare_c(p, Cc, ncp, s);
      ozaki_k1(p, ncp, x0, n, X.as<double>(), s);   // int8 tensor cores, exact accumulation
    } else {
      half_transform(p, Cc, ncp, x0, n, X.as<double>(), s);
    }
    p.timer.mark(kPhKhalf, s);
    p.timer.mark(kPhKsyrk, s);
    if (oz) {
      ozaki_syrk(p, X.as<double>(), n * ncp, sign, beta0, K, s);   // int8 tensor cores
    } else {
      syrk_fp64(p, X.as<double>(), n * ncp, sign, beta0, K, s);
    }
    p.timer.mark(kPhKsyrk, s);
    beta0 = false;
  }
  if (p.opts.precision == DFJK_MIXED && !p.opts.streamed) ozaki_check_k(p, s);
}

static void k_compute(Plan& p, const double* C, const double* w, int64_t ncol, double* K,
                      cudaStream_t s, GammaFuse* fuse = nullptr) {
  // every K path below leaves the full square, exactly symmetric
  if (!w) {
    k_accumulate(p, C, ncol, 1, nullptr, nullptr, ncol, 1.0, true, K, s, fuse);
    return;
  }
  std::vector<int> pos, neg;
  {
    std::vector<double> hw(ncol);
    DFJK_CUDA(cudaMemcpyAsync(hw.data(), w, ncol * sizeof(double), cudaMemcpyDeviceToHost, s));
    DFJK_CUDA(cudaStreamSynchronize(s));
    for (int64_t i = 0; i < ncol; ++i) {
      if (!std::isfinite(hw[i])) fail(DFJK_ERR_NUMERIC, "non-finite weight");
      if (hw[i] > 0) pos.push_back((int)i);
      else if (hw[i] < 0) neg.push_back((int)i);
    }
  }
  if (pos.empty() && neg.empty()) {
    DFJK_CUDA(cudaMemsetAsync(K, 0, (size_t)p.nao * p.nao * sizeof(double), s));
    return;
  }
  k_accumulate(p, C, ncol, 1, w, &pos, (int64_t)pos.size(), 1.0, true, K, s, fuse);
  k_accumulate(p, C, ncol, 1, w, &neg, (int64_t)neg.size(), -1.0, pos.empty(), K, s, fuse);
}

static void reset_jk_phases(Plan& p) {
  for (int ph = kPhJ; ph <= kPhKsyrk; ++ph) p.timer.reset(ph);
}

void jk_compute(Plan& p, const double* C, const double* w, int64_t ncol, double* J, double* K,
                cudaStream_t s) {
  reset_jk_phases(p);
  if (J) {
    p.timer.mark(kPhJ, s);
    DevBuf& gamma = p.ws_gamma;
    gamma.ensure(p.ldb * sizeof(double));
    const DensitySource src{C, w, ncol, nullptr};
    if (p.opts.streamed && K) {
      // one pass over B's chunks gives gamma and the K half transform; J
      // takes a second
      GammaFuse fuse{src, gamma.as<double>(), false};
      k_compute(p, C, w, ncol, K, s, &fuse);
      if (!fuse.done) gamma_of(p, src, gamma.as<double>(), s);
      j_from_gamma(p, gamma.as<double>(), J, s);
      p.timer.mark(kPhJ, s);
      return;
    }
    gamma_of(p, src, gamma.as<double>(), s);
    j_from_gamma(p, gamma.as<double>(), J, s);
    p.timer.mark(kPhJ, s);
  }
  if (K) k_compute(p, C, w, ncol, K, s);
}

// ---------------------------------------------------------------------------
// DFCoulomb.energy and its gradient
// ---------------------------------------------------------------------------

__global__ void add_kernel(const double* __restrict__ a, const double* __restrict__ b, int64_t n,
                           double* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = a[i] + b[i];
}

// The dots of an energy: block partials (sum of a[i] b[i], and F += c a when F
// is given), added by the last block to finish in block order, so the result
// does not depend on the schedule. One block of 256 threads left the trace of
// P K a chain of n^2 / 256 loads (14 us at n = 180, 45 us at n = 318).
constexpr int kDotBlocks = 128;

__global__ void __launch_bounds__(256) dot_axpy_kernel(const double* __restrict__ a,
                                                       const double* __restrict__ b, double c,
                                                       int64_t n, double* F, double* part,
                                                       unsigned* count, double* __restrict__ out) {
  __shared__ double sh[256];
  __shared__ bool last;
  auto block_sum = [&](double s) {
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    return sh[0];
  };
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const double v = a[i];
    s += v * b[i];
    if (F) F[i] += c * v;
  }
  s = block_sum(s);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s;
    __threadfence();
    last = atomicInc(count, gridDim.x - 1) == gridDim.x - 1;   // wraps to 0 for the next call
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  s = block_sum(threadIdx.x < gridDim.x ? __ldcg(part + threadIdx.x) : 0.0);
  if (threadIdx.x == 0) *out = s;
}

// what an energy reads back from the device (ws_scal)
struct EnergyScalars {
  double dot[5];                      // gamma . gamma, then Tr(P_s K) per spin and operator
  LowRankInfo low;
  int nonfinite;
  unsigned count;                     // of dot_axpy_kernel
};

__global__ void nonfinite_kernel(const double* __restrict__ x, int64_t n, int* __restrict__ bad) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n && !isfinite(x[i])) atomicExch(bad, 1);
}

static void dot_axpy(Plan& p, const double* a, const double* b, double c, int64_t n, double* F,
                     double* out, cudaStream_t s) {
  p.ws_dots.ensure(kDotBlocks * sizeof(double));
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(kDotBlocks, (n + 1023) / 1024));
  dot_axpy_kernel<<<blocks, 256, 0, s>>>(a, b, c, n, F, p.ws_dots.as<double>(),
                                         &p.ws_scal.as<EnergyScalars>()->count, out);
  DFJK_LAUNCHED();
}

// Eigen-factor of a symmetric Q (nao x nao): Ct row-major with Q = Ct diag(dw) Ct^T,
// eigenvalues below 1e-14 of the largest set to zero, so K(Q) = k_compute(Ct, dw).
static void density_factor(Plan& p, const double* Q, DevBuf& Ct, DevBuf& dw, cudaStream_t s) {
  Context& c = *p.ctx;
  const int64_t n = p.nao;
  DevBuf V, wv, work, info;
  V.alloc((size_t)n * n * sizeof(double));
  wv.alloc(n * sizeof(double));
  DFJK_CUDA(cudaMemcpyAsync(V.p, Q, (size_t)n * n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  DFJK_CUSOLVER(cusolverDnSetStream(c.cusolver, s));
  int lwork = 0;
  DFJK_CUSOLVER(cusolverDnDsyevd_bufferSize(c.cusolver, CUSOLVER_EIG_MODE_VECTOR,
                                            CUBLAS_FILL_MODE_LOWER, (int)n, V.as<double>(), (int)n,
                                            wv.as<double>(), &lwork));
  work.alloc((size_t)std::max(lwork, 1) * sizeof(double));
  info.alloc(sizeof(int));
  DFJK_CUSOLVER(cusolverDnDsyevd(c.cusolver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER,
                                 (int)n, V.as<double>(), (int)n, wv.as<double>(), work.as<double>(),
                                 lwork, info.as<int>()));
  std::vector<double> hw(n);
  int hinfo = 0;
  DFJK_CUDA(cudaMemcpyAsync(hw.data(), wv.p, n * sizeof(double), cudaMemcpyDeviceToHost, s));
  DFJK_CUDA(cudaMemcpyAsync(&hinfo, info.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  DFJK_CUDA(cudaStreamSynchronize(s));
  if (hinfo != 0) fail(DFJK_ERR_NUMERIC, "density eigensolver failed (info=%d)", hinfo);
  double big = 0.0;
  for (double v : hw) big = std::max(big, std::fabs(v));
  // eigenvectors are the columns of the column-major V, i.e. rows of the
  // row-major view: C[m][k] = V[k*n + m]; transpose into a row-major C
  Ct.alloc((size_t)n * n * sizeof(double));
  DFJK_CUBLAS(cublasSetStream(c.cublas, s));
  const double one = 1.0, zero = 0.0;
  DFJK_CUBLAS(cublasDgeam(c.cublas, CUBLAS_OP_T, CUBLAS_OP_N, (int)n, (int)n, &one, V.as<double>(),
                          (int)n, &zero, V.as<double>(), (int)n, Ct.as<double>(), (int)n));
  std::vector<double> wsel(n, 0.0);
  for (int64_t k = 0; k < n; ++k)
    if (std::fabs(hw[k]) > 1e-14 * big) wsel[k] = hw[k];
  upload(dw, wsel);
}

void gamma_from_density(Plan& p, const double* Ptot, double* gamma, cudaStream_t s) {
  gamma_of(p, DensitySource{nullptr, nullptr, 0, Ptot}, gamma, s);
}

// hf_lr: the long-range exchange of range-separated hybrids through the plan's
// long-range fit (terms.py:604-612). Two host synchronizations: the ranks (with
// the density check), and the scalars at the end.
double energy(Plan& p, const double* P, int nspin, double hf, double hf_lr, double* F,
              cudaStream_t s) {
  const int64_t n = p.nao, nn = n * n;
  const bool exch = hf != 0.0 || hf_lr != 0.0;
  reset_jk_phases(p);
  if (hf_lr != 0.0) reset_jk_phases(p.lr->p);
  p.ws_scal.ensure(sizeof(EnergyScalars));
  EnergyScalars* sc = p.ws_scal.as<EnergyScalars>();
  DFJK_CUDA(cudaMemsetAsync(sc, 0, sizeof(EnergyScalars), s));
  nonfinite_kernel<<<(unsigned)((nn * nspin + 255) / 256), 256, 0, s>>>(P, nn * nspin, &sc->nonfinite);
  DFJK_LAUNCHED();
  const bool low = exch && low_rank_supported(n);
  // mixed products take the factor's columns spread out and laid out as they are read
  const bool spread = low && p.opts.precision == DFJK_MIXED && !p.opts.streamed;
  const int64_t cap = low_rank_cap(n), ns = n * (cap + (cap & 1));
  if (low) p.ws_lowrank.ensure((size_t)nn * nspin * sizeof(double));
  if (spread) p.ws_spread.ensure((size_t)ns * nspin * sizeof(double));
  // the density's factor, a chain of small steps on a few SMs, runs beside J
  SideFork side(*p.ctx, low ? 1 : 0, s);
  if (low) {
    launch_low_rank(P, n, nspin, cap, p.ws_lowrank.as<double>(), kLowRankAccept, &sc->low, side.stream(0));
    for (int sp = 0; spread && sp < nspin; ++sp)
      spread_columns(p.ws_lowrank.as<double>() + sp * nn, n, cap, &sc->low.rank[sp], true,
                     p.ws_spread.as<double>() + sp * ns, side.stream(0));
  }
  const double* Pt = P;
  if (nspin == 2) {
    p.ws_Ptot.ensure(nn * sizeof(double));
    add_kernel<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(P, P + nn, nn, p.ws_Ptot.as<double>());
    DFJK_LAUNCHED();
    Pt = p.ws_Ptot.as<double>();
  }
  p.ws_gamma.ensure(p.ldb * sizeof(double));
  double* gamma = p.ws_gamma.as<double>();
  gamma_from_density(p, Pt, gamma, s);
  dot_axpy(p, gamma, gamma, 0.0, p.ldb, nullptr, &sc->dot[0], s);
  if (F) {
    j_from_gamma(p, gamma, F, s);
    if (nspin == 2)
      DFJK_CUDA(cudaMemcpyAsync(F + nn, F, nn * sizeof(double), cudaMemcpyDeviceToDevice, s));
  }
  side.join();
  EnergyScalars h;
  DFJK_CUDA(cudaMemcpyAsync(&h, sc, sizeof h, cudaMemcpyDeviceToHost, s));
  DFJK_CUDA(cudaStreamSynchronize(s));
  if (h.nonfinite) fail(DFJK_ERR_NUMERIC, "non-finite values in the density");
  if (!exch) return 0.5 * h.dot[0];
  p.ws_K.ensure(nn * sizeof(double));
  double* K = p.ws_K.as<double>();
  for (int sp = 0; sp < nspin; ++sp) {
    const double* Ps = P + sp * nn;
    const bool factored = low && h.low.within(sp, kLowRankAccept);
    DevBuf Ct, dw;
    if (!factored) density_factor(p, Ps, Ct, dw, s);   // indefinite, or too rough a factor
    // the factor's columns: C[m][k] at Cf[m * sm + k * sk]
    const int64_t rank = factored ? h.low.rank[sp] : 0;
    const double* Cf = (spread ? p.ws_spread : p.ws_lowrank).as<double>() + sp * (spread ? ns : nn);
    const int64_t sm = spread ? rank + (rank & 1) : 1, sk = spread ? 1 : n;
    const struct { Plan* plan; double coeff; } terms[2] = {{&p, hf},
                                                           {p.lr ? &p.lr->p : nullptr, hf_lr}};
    for (int t = 0; t < 2; ++t) {
      if (terms[t].coeff == 0.0) continue;
      Plan& q = *terms[t].plan;
      if (!factored) {
        k_compute(q, Ct.as<double>(), dw.as<double>(), n, K, s);
      } else if (rank > 0) {
        k_accumulate(q, Cf, sm, sk, nullptr, nullptr, rank, 1.0, true, K, s);
      } else {
        DFJK_CUDA(cudaMemsetAsync(K, 0, nn * sizeof(double), s));
      }
      // the trace of the exchange quadratic (terms.py:500-509), and F += a K
      const double a = (nspin == 1 ? -0.5 : -1.0) * terms[t].coeff;
      dot_axpy(p, K, Ps, a, nn, F ? F + sp * nn : nullptr, &sc->dot[1 + 2 * t + sp], s);
    }
  }
  DFJK_CUDA(cudaMemcpyAsync(h.dot, sc->dot, sizeof h.dot, cudaMemcpyDeviceToHost, s));
  DFJK_CUDA(cudaStreamSynchronize(s));
  double e = 0.5 * h.dot[0];
  for (int sp = 0; sp < nspin; ++sp)
    e += (nspin == 1 ? -0.25 : -0.5) * (hf * h.dot[1 + sp] + hf_lr * h.dot[3 + sp]);
  return e;
}

}  // namespace dfjk
