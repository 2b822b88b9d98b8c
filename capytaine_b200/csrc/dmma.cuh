// Complex products on the double-precision tensor cores, shared by the float64 LU
// and the tall products.
#pragma once
#include "common.cuh"

namespace bem {
namespace {

// Double-precision tensor-core MMA, 16 x 8 x 8 (36.5 TF/s with eight warps per
// SM, 36.0 for 8 x 8 x 4; plain float64 multiply-adds reach 27).  Lane l holds,
// with g = l / 4 and t = l % 4: A (g, t), (g + 8, t), (g, t + 4), (g + 8, t + 4);
// B (t, g), (t + 4, g); C (g, 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1).
__device__ __forceinline__ void dmma(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, bool valid) {
  const int bytes = valid ? 16 : 0;  // 0: the 16 bytes are filled with zeros, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
               "l"(gsrc), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Complex product of a warp: 16 rows x 8 NT columns, depth K (a multiple of
// 8), from shared memory.  A(m, k) at A[k * lda + m], B(k, n) at B[n * ldb + k]
// (both interleaved complex: one 16-byte load gives a fragment's real and
// imaginary parts); no bank conflicts when lda = 2 mod 8 and ldb = 4 mod 8.
template <int NT>
__device__ __forceinline__ void warp_zmma(const double2* __restrict__ A, int lda, const double2* __restrict__ B,
                                          int ldb, int K, double (&re)[NT][4], double (&im)[NT][4], int lane) {
  const int g = lane >> 2, t = lane & 3;
  A += t * lda + g;
  B += g * ldb + t;
#pragma unroll 2
  for (int k = 0; k < K; k += 8) {
    const double2 a0 = A[0], a1 = A[8], a2 = A[4 * lda], a3 = A[4 * lda + 8];
    const double ar[4] = {a0.x, a1.x, a2.x, a3.x}, ai[4] = {a0.y, a1.y, a2.y, a3.y};
    const double na[4] = {-a0.y, -a1.y, -a2.y, -a3.y};
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const double2 b0 = B[8 * j * ldb], b1 = B[8 * j * ldb + 4];
      const double br[2] = {b0.x, b1.x}, bi[2] = {b0.y, b1.y};
      dmma(re[j], ar, br);
      dmma(im[j], ar, bi);
      dmma(re[j], na, bi);
      dmma(im[j], ai, br);
    }
    A += 8 * lda;
    B += 8;
  }
}

}  // namespace
}  // namespace bem
