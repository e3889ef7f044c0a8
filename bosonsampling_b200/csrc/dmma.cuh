// FP64 tensor-core building blocks of the complex GEMM-shaped kernels (zgemm.cu,
// contract.cu): fragments of m8n8k4 and the product of a warp's complex tile.
#pragma once

#include "common.cuh"

// D += A B, m8n8k4: a = A[lane>>2][lane&3], b = B[lane&3][lane>>2],
// d = (D[lane>>2][2(lane&3)], D[lane>>2][2(lane&3)+1])
BSMPO_DEV void dmma8x8x4(double2& d, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d.x), "+d"(d.y)
               : "d"(a), "d"(b));
}

// 16 bytes global -> shared, zeros where !ok (src is not read then)
BSMPO_DEV void cp_async16(void* dst, const void* src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
BSMPO_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
BSMPO_DEV void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// acc[i][j] (re, im) += op(A)(8 i.., k) B(k, 8 j..) for KS steps of 4 complex k.  a(i, k) /
// b(j, k) give this lane's fragments: op(A)[8 i + lane/4][k + lane%4], B[k + lane%4][8 j + lane/4];
// CONJ: op conjugates.  Four real products per complex one: the split into three would
// cancel.
template <int MI, int NJ, int KS, bool CONJ, typename FA, typename FB>
BSMPO_DEV void cmma_tile(double2 (&re)[MI][NJ], double2 (&im)[MI][NJ], FA a, FB b) {
#pragma unroll
  for (int ks = 0; ks < KS; ++ks) {
    double2 av[MI], bv[NJ];
#pragma unroll
    for (int i = 0; i < MI; ++i) av[i] = a(i, 4 * ks);
#pragma unroll
    for (int j = 0; j < NJ; ++j) bv[j] = b(j, 4 * ks);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const double ni = -av[i].y;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        dmma8x8x4(re[i][j], av[i].x, bv[j].x);
        dmma8x8x4(im[i][j], av[i].x, bv[j].y);
        dmma8x8x4(re[i][j], CONJ ? av[i].y : ni, bv[j].y);
        dmma8x8x4(im[i][j], CONJ ? ni : av[i].y, bv[j].x);
      }
    }
  }
}
