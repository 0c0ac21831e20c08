// Grid points along a Morton curve over 1-Bohr cells, on the device: keys, a
// stable radix sort by (key, index), the gathered points and their bounding
// boxes. Bound by launches at the usual sizes (a dozen kernels of a few us for
// 10^5 points). The threaded host sort that stood here took 4.0 ms for the 109 k
// points of (H2O)_3, most of it first touches of its arrays.
#include "common.h"
#include "scf.h"

#include <algorithm>
#include <cmath>
#include <vector>

namespace dfjk {
namespace {

constexpr int kThreads = 256;
constexpr int kDigits = 256;             // 8 bits a pass
constexpr int kWarps = kThreads / 32, kPerLane = 8;
constexpr int kTile = kThreads * kPerLane;   // points of a block; a warp has a contiguous run

// bit i of the low 21 bits of v to bit 3 i: a Morton key has x, y, z in turn
__device__ __forceinline__ uint64_t spread(uint64_t v) {
  v &= 0x1fffffULL;
  v = (v | v << 32) & 0x1f00000000ffffULL;
  v = (v | v << 16) & 0x1f0000ff0000ffULL;
  v = (v | v << 8) & 0x100f00f00f00f00fULL;
  v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
  v = (v | v << 2) & 0x1249249249249249ULL;
  return v;
}

// the least and greatest of a block's v per dimension: out[0..2], out[3..5]
__device__ void block_box(const double (&v)[3], bool in, double* __restrict__ out) {
  __shared__ double red[kWarps][6];
  double b[6];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    b[d] = in ? v[d] : INFINITY;
    b[3 + d] = in ? v[d] : -INFINITY;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      b[d] = fmin(b[d], __shfl_xor_sync(0xffffffffu, b[d], o));
      b[3 + d] = fmax(b[3 + d], __shfl_xor_sync(0xffffffffu, b[3 + d], o));
    }
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int d = 0; d < 6; ++d) red[threadIdx.x >> 5][d] = b[d];
  __syncthreads();
  if (threadIdx.x < 6) {
    double r = red[0][threadIdx.x];
    for (int q = 1; q < kWarps; ++q)
      r = threadIdx.x < 3 ? fmin(r, red[q][threadIdx.x]) : fmax(r, red[q][threadIdx.x]);
    out[threadIdx.x] = r;
  }
}

// boxes[b]: of points [256 b, 256 b + 256); with order, the points and weights of
// that order are written too
__global__ void __launch_bounds__(kThreads) gather_kernel(
    const double* __restrict__ raw, const double* __restrict__ raw_w, int64_t n,
    const uint32_t* __restrict__ order, double* __restrict__ pts, double* __restrict__ w,
    double* __restrict__ boxes) {
  const int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x;
  double v[3] = {};
  if (i < n) {
    const int64_t j = order ? order[i] : i;
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] = raw[3 * j + d];
    if (order) {
#pragma unroll
      for (int d = 0; d < 3; ++d) pts[3 * i + d] = v[d];
      w[i] = raw_w[j];
    }
  }
  block_box(v, i < n, boxes + 6 * (int64_t)blockIdx.x);
}

__global__ void keys_kernel(const double* __restrict__ raw, int64_t n, double x0, double y0, double z0,
                            uint64_t* __restrict__ key, uint32_t* __restrict__ idx) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  key[i] = spread((uint64_t)floor(raw[3 * i] - x0)) | spread((uint64_t)floor(raw[3 * i + 1] - y0)) << 1 |
           spread((uint64_t)floor(raw[3 * i + 2] - z0)) << 2;
  idx[i] = (uint32_t)i;
}

// hist[digit][block]: how many of a block's keys have the digit
__global__ void __launch_bounds__(kThreads) hist_kernel(const uint64_t* __restrict__ key, int64_t n,
                                                        int shift, int* __restrict__ hist) {
  __shared__ int h[kDigits];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t t0 = blockIdx.x * (int64_t)kTile;
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const int64_t i = t0 + j * kThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(key[i] >> shift) & (kDigits - 1)], 1);
  }
  __syncthreads();
  hist[threadIdx.x * (int64_t)gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// exclusive prefix sums of hist, in place, by one block
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) scan_kernel(int* __restrict__ hist, int64_t n) {
  __shared__ int warp_sum[kScanThreads / 32];
  const int64_t per = (n + kScanThreads - 1) / kScanThreads;
  const int64_t b = threadIdx.x * per < n ? threadIdx.x * per : n, e = b + per < n ? b + per : n;
  int sum = 0;
  for (int64_t i = b; i < e; ++i) sum += hist[i];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int v = warp_sum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    warp_sum[lane] = v;
  }
  __syncthreads();
  int run = inc - sum + (warp > 0 ? warp_sum[warp - 1] : 0);
  for (int64_t i = b; i < e; ++i) {
    const int c = hist[i];
    hist[i] = run;
    run += c;
  }
}

// to their places: the elements of a digit keep their order, block by block, warp
// by warp (a warp's run is contiguous) and, within a warp, 32 at a time by lane
__global__ void __launch_bounds__(kThreads) scatter_kernel(
    const uint64_t* __restrict__ key, const uint32_t* __restrict__ idx, int64_t n, int shift,
    const int* __restrict__ offs, uint64_t* __restrict__ key_out, uint32_t* __restrict__ idx_out) {
  __shared__ int at[kWarps][kDigits];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < kWarps; ++q) at[q][threadIdx.x] = 0;
  __syncthreads();
  const int64_t i0 = blockIdx.x * (int64_t)kTile + warp * 32 * kPerLane + lane;
  uint64_t k[kPerLane];
  int dig[kPerLane];   // kDigits: past the end
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const bool in = i0 + 32 * j < n;
    k[j] = in ? key[i0 + 32 * j] : 0;
    dig[j] = in ? (int)((k[j] >> shift) & (kDigits - 1)) : kDigits;
    if (in) atomicAdd(&at[warp][dig[j]], 1);
  }
  __syncthreads();
  int run = offs[threadIdx.x * (int64_t)gridDim.x + blockIdx.x];
#pragma unroll
  for (int q = 0; q < kWarps; ++q) {
    const int c = at[q][threadIdx.x];
    at[q][threadIdx.x] = run;
    run += c;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPerLane; ++j) {
    const unsigned same = __match_any_sync(0xffffffffu, dig[j]);
    const int rank = __popc(same & ((1u << lane) - 1));
    const int pos = dig[j] < kDigits ? at[warp][dig[j]] + rank : 0;
    __syncwarp();
    if (dig[j] < kDigits) {
      if (rank == 0) at[warp][dig[j]] = pos + __popc(same);
      key_out[pos] = k[j];
      idx_out[pos] = idx[i0 + 32 * j];
    }
    __syncwarp();
  }
}

}  // namespace

void sort_points(const double* pts_host, const double* w_host, int64_t n, DevBuf& pts, DevBuf& w,
                 std::vector<double>& boxes, cudaStream_t s) {
  if (n >= (int64_t)1 << 31) fail(DFJK_ERR_UNSUPPORTED, "%lld grid points", (long long)n);
  const int64_t nbox = (n + kXcBox - 1) / kXcBox, tiles = (n + kTile - 1) / kTile;
  static_assert(kXcBox == kThreads, "a box is a block's points");
  pts.alloc(3 * n * sizeof(double));
  w.alloc(n * sizeof(double));
  // one buffer for all scratch: each one taken from the cache may wait for the device
  DevBuf scratch;
  scratch.alloc((4 * n + 6 * nbox) * sizeof(double) + 2 * n * sizeof(uint64_t) +
                (2 * n + kDigits * tiles) * sizeof(uint32_t));
  double* raw = scratch.as<double>();
  double *raw_w = raw + 3 * n, *box = raw_w + n;
  uint64_t* key[2];
  key[0] = reinterpret_cast<uint64_t*>(box + 6 * nbox);
  key[1] = key[0] + n;
  uint32_t* idx[2];
  idx[0] = reinterpret_cast<uint32_t*>(key[1] + n);
  idx[1] = idx[0] + n;
  int* hist = reinterpret_cast<int*>(idx[1] + n);
  boxes.resize(6 * nbox);
  DFJK_CUDA(cudaMemcpyAsync(raw, pts_host, 3 * n * sizeof(double), cudaMemcpyHostToDevice, s));
  DFJK_CUDA(cudaMemcpyAsync(raw_w, w_host, n * sizeof(double), cudaMemcpyHostToDevice, s));
  auto gather = [&](const uint32_t* order) {
    gather_kernel<<<(unsigned)nbox, kThreads, 0, s>>>(raw, raw_w, n, order, pts.as<double>(),
                                                      w.as<double>(), box);
    DFJK_LAUNCHED();
    DFJK_CUDA(cudaMemcpyAsync(boxes.data(), box, 6 * nbox * sizeof(double), cudaMemcpyDeviceToHost, s));
    DFJK_CUDA(cudaStreamSynchronize(s));
  };
  gather(nullptr);
  double lo[3] = {INFINITY, INFINITY, INFINITY}, ext = 0.0;
  for (int64_t b = 0; b < nbox; ++b)
    for (int d = 0; d < 3; ++d) lo[d] = std::min(lo[d], boxes[6 * b + d]);
  for (int64_t b = 0; b < nbox; ++b)
    for (int d = 0; d < 3; ++d) ext = std::max(ext, boxes[6 * b + 3 + d] - lo[d]);
  // cells 0 .. floor(ext) a side: three bits of the key for each of theirs
  int bits = 0;
  while (bits < 21 && std::floor(ext) >= (double)((int64_t)1 << bits)) ++bits;
  keys_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(raw, n, lo[0], lo[1], lo[2], key[0], idx[0]);
  DFJK_LAUNCHED();
  int q = 0;
  for (int shift = 0; shift < 3 * bits; shift += 8, q ^= 1) {
    hist_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(key[q], n, shift, hist);
    DFJK_LAUNCHED();
    scan_kernel<<<1, kScanThreads, 0, s>>>(hist, kDigits * tiles);
    DFJK_LAUNCHED();
    scatter_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(key[q], idx[q], n, shift, hist, key[q ^ 1],
                                                        idx[q ^ 1]);
    DFJK_LAUNCHED();
  }
  gather(idx[q]);
}

}  // namespace dfjk
