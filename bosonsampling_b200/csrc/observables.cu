// Trace and single-mode photon-number marginals of the MPO, in FP64.
//
// Generalises summary.Probability (src/summary.py:11-26): the trace keeps, on every
// bond, only entries whose ket and bra charges agree (and Lambda > 0), and contracts
// the Gamma chain.  Right environments R_b (b = n..0) and left environments L_b
// (b = 0..n) are masked matrix-vector products; the marginal of mode i is
//     P_i(k) = sum_{a, j : c0(a) - c0(j) = k} L_i[a] Gamma_i[a, j] R_{i+1}[j].
// All reductions run in a fixed order (no floating-point atomics), so results are
// bit-reproducible from run to run.
//
// A bond's kept entries are at most d charge blocks (c, c), each a contiguous range, about
// one entry in d; only rows and columns of kept entries are read (a fraction ~1/d^2 of
// Gamma), through a list of their positions per bond.  The two environment recursions do
// not depend on each other: step t of one launch does right bond n - 1 - t and left bond
// t + 1.  What bounds it: the n dependent launches (a step reads ~0.7 MB at chi = 1024), not
// the memory.  Measured at n = 64, chi = 1024, d = 5: 0.79 ms the call; reading every row
// and column in two launches a site took 3.66.
#include "common.cuh"
#include "kernels.h"

namespace {

__device__ __forceinline__ bool diag_ok(int2 c, double lam, int d) {
  return c.x < d && c.x == c.y && lam > 0.0;
}

// Per bond: the positions of the kept entries (ascending) and their number, one CTA per
// bond; R_n and L_0 (ones on the kept entries, in list order)
constexpr int DL_NT = 256;
__global__ __launch_bounds__(DL_NT) void diag_list_kernel(int n, int d, int chi, const int2* __restrict__ charge,
                                                          const double* __restrict__ lam, int* __restrict__ list,
                                                          int* __restrict__ count, cplx* __restrict__ envr,
                                                          cplx* __restrict__ envl) {
  __shared__ int sums[DL_NT / 32], base;
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int2* cb = charge + (int64_t)b * chi;
  const double* lb = lam + (int64_t)b * chi;
  int* out = list + (int64_t)b * chi;
  if (tid == 0) base = 0;
  __syncthreads();
  for (int i0 = 0; i0 < chi; i0 += DL_NT) {
    const int i = i0 + tid;
    const bool ok = i < chi && diag_ok(cb[i], lb[i], d);
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    if (lane == 0) sums[warp] = __popc(m);
    __syncthreads();
    int at = base;
    for (int w = 0; w < warp; ++w) at += sums[w];
    at += __popc(m & ((1u << lane) - 1));
    if (ok) {
      out[at] = i;
      if (b == n) envr[(int64_t)b * chi + at] = cmake(1.0, 0.0);
      if (b == 0) envl[at] = cmake(1.0, 0.0);
    }
    __syncthreads();
    if (tid == 0)
      for (int w = 0; w < DL_NT / 32; ++w) base += sums[w];
    __syncthreads();
  }
  if (tid == 0) count[b] = base;
}

// Step t: blockIdx.y 0: R_b from R_{b+1}, b = n - 1 - t, one warp per kept row;
// blockIdx.y 1: L_{t+1} from L_t, 8 kept columns per CTA.
// Environments are in list order.
constexpr int ES_NT = 256;
__global__ __launch_bounds__(ES_NT) void env_step_kernel(int n, int chi, int t, const cplx* __restrict__ gamma,
                                                         const int* __restrict__ list, const int* __restrict__ count,
                                                         cplx* __restrict__ envr, cplx* __restrict__ envl) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (blockIdx.y == 0) {
    const int b = n - 1 - t, rows = count[b], cols = count[b + 1];
    const int* lr = list + (int64_t)b * chi;
    const int* lc = lr + chi;
    const cplx* rn = envr + (int64_t)(b + 1) * chi;
    for (int a = blockIdx.x * (ES_NT / 32) + warp; a < rows; a += gridDim.x * (ES_NT / 32)) {
      const cplx* g = gamma + ((int64_t)b * chi + lr[a]) * chi;
      cplx acc = cmake(0.0, 0.0);
#pragma unroll 8
      for (int j = lane; j < cols; j += 32) cfma(acc, ldc(g + lc[j]), ldc(rn + j));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
      }
      if (lane == 0) envr[(int64_t)b * chi + a] = acc;
    }
    return;
  }
  // 8 columns to a CTA, a lane's rows 4 apart, the warps' 32
  __shared__ double2 part[ES_NT / 8][9];
  const int rows = count[t], cols = count[t + 1];
  const int* lr = list + (int64_t)t * chi;
  const int* lc = lr + chi;
  const cplx* l0 = envl + (int64_t)t * chi;
  const int x = tid & 7, y = tid >> 3;
  for (int j0 = blockIdx.x * 8; j0 < cols; j0 += gridDim.x * 8) {
    const int j = j0 + x;
    cplx acc = cmake(0.0, 0.0);
    if (j < cols) {
      const cplx* g = gamma + (int64_t)t * chi * chi + lc[j];
#pragma unroll 8
      for (int a = y; a < rows; a += ES_NT / 8) cfma(acc, ldc(l0 + a), ldc(g + (int64_t)lr[a] * chi));
    }
    part[y][x] = make_double2(acc.x, acc.y);
    __syncthreads();
    if (tid < 8 && j < cols) {
      cplx s = cmake(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < ES_NT / 8; ++q) s = cadd(s, cmake(part[q][tid].x, part[q][tid].y));
      envl[(int64_t)(t + 1) * chi + j] = s;
    }
    __syncthreads();
  }
}

// part[site][chunk][k] = sum over the chunk's kept rows; one CTA per (site, chunk)
constexpr int MNT = 256;
__global__ __launch_bounds__(MNT) void marginal_kernel(int n, int d, int chi,
                                                        const cplx* __restrict__ gamma,
                                                        const int2* __restrict__ charge,
                                                        const int* __restrict__ list,
                                                        const int* __restrict__ count,
                                                        const cplx* __restrict__ envl,
                                                        const cplx* __restrict__ envr,
                                                        int chunk_rows, cplx* __restrict__ part) {
  __shared__ double2 red[MNT / 32][BSMPO_MAX_D];
  const int site = blockIdx.y, chunk = blockIdx.x;
  const int nchunk = gridDim.x;
  const int rows = count[site], cols = count[site + 1];
  const int* lr = list + (int64_t)site * chi;
  const int* lc = lr + chi;
  const cplx* g = gamma + (int64_t)site * chi * chi;
  const int2* ca = charge + (int64_t)site * chi;
  const int2* cj = charge + (int64_t)(site + 1) * chi;
  const cplx* L = envl + (int64_t)site * chi;
  const cplx* R = envr + (int64_t)(site + 1) * chi;
  cplx acc[BSMPO_MAX_D];
#pragma unroll
  for (int k = 0; k < BSMPO_MAX_D; ++k) acc[k] = cmake(0.0, 0.0);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int r0 = chunk * chunk_rows, r1 = min(rows, r0 + chunk_rows);
  // a warp to a row
  for (int a = r0 + wid; a < r1; a += MNT / 32) {
    const int ra = lr[a], ka = ca[ra].x;
    const cplx la = ldc(L + a);
#pragma unroll 2
    for (int j = lane; j < cols; j += 32) {
      const int cjx = lc[j], k = ka - cj[cjx].x;
      if (k < 0 || k >= d) continue;
      const cplx v = cmul(cmul(la, ldc(g + (int64_t)ra * chi + cjx)), ldc(R + j));
#pragma unroll
      for (int kk = 0; kk < BSMPO_MAX_D; ++kk)
        if (kk == k) acc[kk] = cadd(acc[kk], v);
    }
  }
#pragma unroll
  for (int k = 0; k < BSMPO_MAX_D; ++k) {
    double x = acc[k].x, y = acc[k].y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if (lane == 0) red[wid][k] = make_double2(x, y);
  }
  __syncthreads();
  if (threadIdx.x < d) {
    cplx s = cmake(0.0, 0.0);
    for (int w = 0; w < MNT / 32; ++w)
      s = cadd(s, cmake(red[w][threadIdx.x].x, red[w][threadIdx.x].y));
    part[((int64_t)site * nchunk + chunk) * d + threadIdx.x] = s;
  }
}

// marginals from their chunks' parts, and the trace (the sum of R_0) in the last entry
__global__ __launch_bounds__(256) void observables_reduce_kernel(int n, int d, int nchunk, const cplx* __restrict__ part,
                                                                 const int* __restrict__ count,
                                                                 const cplx* __restrict__ envr, cplx* __restrict__ out) {
  if (blockIdx.x == 0) {
    __shared__ double2 red[256];
    cplx acc = cmake(0.0, 0.0);
    for (int i = threadIdx.x; i < count[0]; i += 256) acc = cadd(acc, ldc(envr + i));
    red[threadIdx.x] = make_double2(acc.x, acc.y);
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
      if (threadIdx.x < s) {
        red[threadIdx.x].x += red[threadIdx.x + s].x;
        red[threadIdx.x].y += red[threadIdx.x + s].y;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) out[n * d] = cmake(red[0].x, red[0].y);
    return;
  }
  const int e = (blockIdx.x - 1) * 256 + threadIdx.x;
  if (e >= n * d || nchunk == 0) return;
  const int site = e / d, k = e % d;
  cplx s = cmake(0.0, 0.0);
  for (int c = 0; c < nchunk; ++c) s = cadd(s, part[((int64_t)site * nchunk + c) * d + k]);
  out[e] = s;
}

}  // namespace

cudaError_t launch_diag_lists(int n, int d, int chi, const int* charge, const double* lam, int* list, int* count,
                              void* env_r, void* env_l, cudaStream_t s) {
  diag_list_kernel<<<n + 1, DL_NT, 0, s>>>(n, d, chi, reinterpret_cast<const int2*>(charge), lam, list, count,
                                           reinterpret_cast<cplx*>(env_r), reinterpret_cast<cplx*>(env_l));
  return cudaGetLastError();
}

cudaError_t launch_env_step(int n, int chi, int t, int max_rows, bool left, const void* gamma, const int* list,
                            const int* count, void* env_r, void* env_l, cudaStream_t s) {
  // max_rows: a bound on the kept entries of the bonds concerned (the kernel loops past it)
  const dim3 grid(ceil_div(max_rows > 0 ? max_rows : 1, ES_NT / 32), left ? 2 : 1);
  env_step_kernel<<<grid, ES_NT, 0, s>>>(n, chi, t, reinterpret_cast<const cplx*>(gamma), list, count,
                                         reinterpret_cast<cplx*>(env_r), reinterpret_cast<cplx*>(env_l));
  return cudaGetLastError();
}

cudaError_t launch_marginals(int n, int d, int chi, const void* gamma, const int* charge, const int* list,
                             const int* count, const void* env_l, const void* env_r, void* part, int chunk_rows,
                             int nchunk, void* out, cudaStream_t s) {
  if (nchunk > 0) {
    marginal_kernel<<<dim3(nchunk, n), MNT, 0, s>>>(n, d, chi, reinterpret_cast<const cplx*>(gamma),
                                                    reinterpret_cast<const int2*>(charge), list, count,
                                                    reinterpret_cast<const cplx*>(env_l),
                                                    reinterpret_cast<const cplx*>(env_r), chunk_rows,
                                                    reinterpret_cast<cplx*>(part));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  observables_reduce_kernel<<<1 + (nchunk > 0 ? ceil_div(n * d, 256) : 0), 256, 0, s>>>(
      n, d, nchunk, reinterpret_cast<const cplx*>(part), count, reinterpret_cast<const cplx*>(env_r),
      reinterpret_cast<cplx*>(out));
  return cudaGetLastError();
}
