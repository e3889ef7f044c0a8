// Grouped complex128 GEMM for the contraction-shaped steps of the BS update
// (the Theta block products, the Gram matrices, V = T Y / sigma, W = V^H C).
//
// FP64 has no tcgen05 kind on sm_100a, so this runs on the FP64 tensor path (m8n8k4): 32 x 32
// output tile per CTA, 4 warps of 16 x 16, K in slabs of 8 complex through a ring of three
// shared-memory stages filled by cp.async (zeros past the edges).  op(A) and B keep their
// storage order in shared memory, padded so that a fragment load (four k by two rows a
// quarter warp) falls on distinct banks.  All groups of one launch share the grid; a CTA
// finds its group by binary search over tile_start.  A Hermitian group (C = A^H A) forms its
// upper tiles only and writes the others as their adjoints.
// What bounds it: the FP64 tensor rate for large groups, the slabs' latency for small ones.
// 128-bit shared-memory reads take 4 cycles of the SM a warp: the vector form (4 x 4 complex
// a thread) needed as many cycles for its operands as for its arithmetic, the fragments need
// a quarter.  Measured, all GEMMs of one chi = 1024 update alone: 0.55 ms against 1.05 (64 x 64
// tiles).  Why 32 x 32: a launch's sectors give 20 to 300 tiles of 64 x 64, less than a wave or
// a ragged one, and a CTA's slabs wait for loads and barriers that other CTAs of the SM
// fill.  64 and 32, ms: update at chi = 1024 3.05 and 2.83 (Gram route), 10.1 and 9.7 (fp64);
// chi = 256 0.638 and 0.582, 1.575 and 1.450; 24 modes chi = 256 33.2 and 29.9; two layers at N =
// 64, chi = 1024 (thousands of tiles) 45.2 and 43.5.
#include "dmma.cuh"
#include "kernels.h"

namespace {

constexpr int TM = 32, TN = 32, TK = 8, NT = 128, STAGES = 3;
constexpr int MI = 2, NJ = 2;  // 8 x 8 tiles of a warp
constexpr int LDK = TK + 4;    // op(A) = A, stored [m][k]: 4 mod 8
constexpr int LDM = TM + 2;    // A^H, stored [k][m], and B [k][n]: 2 mod 8
constexpr int A_ELEMS = TM * LDK > TK * LDM ? TM * LDK : TK * LDM, B_ELEMS = TK * (TN + 2);
constexpr size_t SMEM = (size_t)STAGES * (A_ELEMS + B_ELEMS) * sizeof(double2);

template <bool OPA>
__device__ __forceinline__ void tile_loop(const GemmGroup& g, const cplx* __restrict__ a, const cplx* __restrict__ b,
                                          int m0, int n0, double2* smem, double2 (&re)[MI][NJ], double2 (&im)[MI][NJ]) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = g.M, N = g.N, K = g.K;
  auto stage_a = [&](int s) { return smem + s * (A_ELEMS + B_ELEMS); };
  auto stage_b = [&](int s) { return smem + s * (A_ELEMS + B_ELEMS) + A_ELEMS; };
  auto fill = [&](int s, int k0) {
    double2 *as = stage_a(s), *bs = stage_b(s);
#pragma unroll
    for (int i = 0; i < TM * TK / NT; ++i) {
      const int e = tid + i * NT;
      if (OPA) {
        const int k = e / TM, m = e % TM;
        const bool ok = m0 + m < M && k0 + k < K;
        cp_async16(as + k * LDM + m, ok ? a + (int64_t)(k0 + k) * g.lda + m0 + m : a, ok);
      } else {
        const int m = e / TK, k = e % TK;
        const bool ok = m0 + m < M && k0 + k < K;
        cp_async16(as + m * LDK + k, ok ? a + (int64_t)(m0 + m) * g.lda + k0 + k : a, ok);
      }
    }
#pragma unroll
    for (int i = 0; i < TK * TN / NT; ++i) {
      const int e = tid + i * NT, k = e / TN, n = e % TN;
      const bool ok = n0 + n < N && k0 + k < K;
      cp_async16(bs + k * (TN + 2) + n, ok ? b + (int64_t)(k0 + k) * g.ldb + n0 + n : b, ok);
    }
  };
  const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16, li = lane >> 2, lk = lane & 3;
  const bool live = m0 + wm < M && n0 + wn < N;   // a warp's tile past the edge does nothing
  const int slabs = (K + TK - 1) / TK;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < slabs) fill(s, s * TK);
    cp_async_commit();
  }
  for (int t = 0; t < slabs; ++t) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (t + STAGES - 1 < slabs) fill((t + STAGES - 1) % STAGES, (t + STAGES - 1) * TK);
    cp_async_commit();
    if (!live) continue;
    const double2 *as = stage_a(t % STAGES), *bs = stage_b(t % STAGES);
    cmma_tile<MI, NJ, TK / 4, OPA>(
        re, im,
        [&](int i, int k) { return OPA ? as[(k + lk) * LDM + wm + 8 * i + li] : as[(wm + 8 * i + li) * LDK + k + lk]; },
        [&](int j, int k) { return bs[(k + lk) * (TN + 2) + wn + 8 * j + li]; });
  }
}

__global__ __launch_bounds__(NT, 4) void zgemm_grouped_kernel(const cplx* __restrict__ A, const cplx* __restrict__ B,
                                                              cplx* __restrict__ C, const double* __restrict__ scale,
                                                              const GemmGroup* __restrict__ groups, int n_groups,
                                                              const SectorDesc* __restrict__ sd) {
  extern __shared__ __align__(16) double2 smem[];
  __shared__ GemmGroup g;
  const int tid = threadIdx.x;
  if (tid == 0) {
    int lo = 0, hi = n_groups - 1;
    const int t = blockIdx.x;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (groups[mid].tile_start <= t) lo = mid; else hi = mid - 1;
    }
    g = groups[lo];
    if (g.sec >= 0) {
      const int kept = sd[g.sec].kept;
      if (g.kdim == 1) { g.M = kept; g.lda = kept; }
      else if (g.kdim == 3) { g.M = kept < 0 ? 0 : g.M; }
      else { g.N = kept; g.ldb = kept; g.ldc = kept; }
    }
  }
  __syncthreads();
  const int tile = blockIdx.x - g.tile_start;
  const int m0 = (tile / g.tiles_n) * TM, n0 = (tile % g.tiles_n) * TN;
  // tiles are laid out for the host's bound; a Hermitian group forms n0 >= m0
  if (m0 >= g.M || n0 >= g.N || (g.herm && n0 < m0)) return;
  double2 re[MI][NJ], im[MI][NJ];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) re[i][j] = im[i][j] = make_double2(0.0, 0.0);
  if (g.opA) tile_loop<true>(g, A + g.a_off, B + g.b_off, m0, n0, smem, re, im);
  else tile_loop<false>(g, A + g.a_off, B + g.b_off, m0, n0, smem, re, im);
  const int lane = tid & 31, warp = tid >> 5;
  const int row0 = m0 + (warp >> 1) * 16 + (lane >> 2), col0 = n0 + (warp & 1) * 16 + 2 * (lane & 3);
  const double* cs = g.cs_off >= 0 ? scale + g.cs_off : nullptr;
  cplx* c = C + g.c_off;
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int n = col0 + 8 * j + x;
      if (n >= g.N) continue;
      const double f = cs ? cs[n] : 1.0;
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int m = row0 + 8 * i;
        if (m >= g.M) continue;
        const cplx v = cmake(f * (x ? re[i][j].y : re[i][j].x), f * (x ? im[i][j].y : im[i][j].x));
        stc(c + (int64_t)m * g.ldc + n, v);
        if (g.herm && n0 > m0) stc(c + (int64_t)n * g.ldc + m, cconj(v));
      }
    }
}

}  // namespace

int zgemm_tile_m() { return TM; }
int zgemm_tile_n() { return TN; }

cudaError_t launch_zgemm_grouped(const void* a, const void* b, void* c, const double* scale,
                                 const GemmGroup* groups_dev, int n_groups, int total_tiles,
                                 const SectorDesc* sd_dev, cudaStream_t s) {
  if (total_tiles <= 0 || n_groups <= 0) return cudaSuccess;
  static const cudaError_t attr =
      cudaFuncSetAttribute(zgemm_grouped_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
  if (attr != cudaSuccess) return attr;
  zgemm_grouped_kernel<<<total_tiles, NT, SMEM, s>>>(
      reinterpret_cast<const cplx*>(a), reinterpret_cast<const cplx*>(b),
      reinterpret_cast<cplx*>(c), scale, groups_dev, n_groups, sd_dev);
  return cudaGetLastError();
}
