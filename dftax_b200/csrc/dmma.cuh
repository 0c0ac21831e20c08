// Float64 tensor-core and copy instructions of the float64 products (K in
// jk.cu, the XC quadrature in xc.cu).
#pragma once

#include <cuda_runtime.h>

namespace dfjk {

// c += a b on an 8 x 8 x 4 fragment: lane l holds a[row l / 4][k l % 4],
// b[k l % 4][column l / 4] and c[row l / 4][columns 2 (l % 4), + 1]
__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// 16 bytes to shared memory; src-size 0 fills them with zeros (gmem must still
// be a valid address)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(smem))),
               "l"(gmem), "r"(valid ? 16 : 0)
               : "memory");
}

// bytes (a multiple of 16, at a 16-byte boundary) towards L2
__device__ __forceinline__ void prefetch_l2(const void* gmem, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(gmem)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// all but the newest N groups of this thread have landed
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace dfjk
