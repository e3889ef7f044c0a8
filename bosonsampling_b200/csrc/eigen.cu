// Gram / Hermitian-eigen route of the per-sector SVD (the mixed-precision form).
//
// The reference takes a thin SVD of every sector (cuSOLVER gesvd,
// src/beam_splitter_parallel/Rank.py:122-125; LAPACK, src/MPO.py:258).  The truncation
// keeps only the largest chi singular triplets over all sectors (at chi = 1024 about a
// third of the candidates, cut near 3e-3 of the largest singular value), so this route
// forms the Gram matrix of each sector in FP64 and solves a Hermitian eigenproblem:
//   X = T (|L| >= |R|) or T^H (|L| < |R|), G = X^H X (k x k, k = min(|L|, |R|)),
//   1. Householder reduction of G to a real symmetric tridiagonal (d, e): G = Q T Q^H,
//      Q = H_0 ... H_{k-2}, H_j = I - tau_j v_j v_j^H (LAPACK's zhetd2 conventions,
//      lower storage), one thread-block cluster per sector, rows owned cyclically by
//      the cluster's CTAs and kept in their shared memory, the rank-2 update of step j - 1
//      fused with the matrix-vector product of step j, one cluster barrier per step;
//   2. every eigenvalue by multisection of Sturm counts (one warp per eigenvalue, 32
//      points per pass), sigma = sqrt(lambda), zero below the numerical floor;
//   3. after the global top-chi selection: eigenvectors of the kept eigenvalues by
//      inverse iteration on T - lambda I (partial pivoting; members of tight clusters
//      of eigenvalues are orthogonalised against each other), then y = Q z.
// V = y directly when X = T^H (G = T T^H), else V = T Y diag(1/sigma) (a GEMM).
// Eigenvalue errors are about eps ||G||: singular values above ~1e-6 of the largest
// are accurate to ~1e-10 relative, far below the truncation cut.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "dmma.cuh"
#include "kernels.h"
#include "pipeline.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr double EPS = 2.220446049250313e-16;
// Streamed tridiagonalisation (sectors too large for tridiag_resident_kernel): one cluster of
// TD_CL CTAs per sector
constexpr int TD_NT = 256, TD_NW = TD_NT / 32;
constexpr int TD_CL = 16;
// bulk-copy ring of each warp: about TD_RING_KB per CTA, 1, 2 or TD_MAXSLOT row slots (pairs
// of rows share one pass over the vectors)
constexpr int TD_RING_KB = 64;
constexpr int TD_MAXSLOT = 4;

// shared memory of the tridiagonalisation with `slots` ring slots per warp (kmax = the
// launch's largest k, cl = CTAs per sector): the row rings, v and w of two steps, the
// published and the copied row, p of the own rows (two steps), 64 scalars and the rings'
// mbarriers
__host__ __device__ inline size_t td_smem_for(int kmax, int cl, int slots, int nw) {
  const int own = kmax / cl + 1;
  return sizeof(cplx) * ((size_t)nw * slots * kmax + 6 * (size_t)kmax + 2 * (size_t)own) +
         64 * sizeof(double) + nw * TD_MAXSLOT * sizeof(uint64_t);
}

// ring slots per warp: a power of two, 2 to TD_MAXSLOT within about TD_RING_KB per
// CTA, fewer where a sector of size kmax would not fit in 227 KB
__host__ __device__ inline int td_slots(int kmax, int nw) {
  const long long fit = (long long)TD_RING_KB * 1024 / ((long long)nw * kmax * (long long)sizeof(cplx));
  int s = fit >= TD_MAXSLOT ? TD_MAXSLOT : 2;
  while (s > 1 && td_smem_for(kmax, TD_CL, s, nw) > 227 * 1024) s >>= 1;
  return s;
}

// dynamic shared memory of a tridiagonalisation launch with nw warps per CTA
__host__ __device__ inline size_t td_smem_bytes(int kmax, int cl, int nw) {
  return td_smem_for(kmax, cl, td_slots(kmax, nw), nw);
}

__device__ __forceinline__ cplx warp_sum(cplx v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// The warp's sum in every lane: as the right operand of an FP64 m8n8k4 product with ones,
// lane 4 n + c's value is entry (c, n), so the product holds the sums over c; of those,
// lane x holds two, and a second product adds the four pairs.  Two matrix instructions and
// an addition (60 cycles) where five shuffles and additions take 210.
__device__ __forceinline__ double warp_sum(double v) {
  double2 a = make_double2(0.0, 0.0), t = a;
  dmma8x8x4(a, 1.0, v);
  dmma8x8x4(t, 1.0, a.x + a.y);
  return t.x;
}

// a - (x conj(y) + u conj(z)), eight fused multiply-adds (the rank-2 update of one entry)
__device__ __forceinline__ cplx crank2(cplx a, cplx x, cplx y, cplx u, cplx z) {
  a.x = fma(-x.x, y.x, a.x);
  a.x = fma(-x.y, y.y, a.x);
  a.x = fma(-u.x, z.x, a.x);
  a.x = fma(-u.y, z.y, a.x);
  a.y = fma(-x.y, y.x, a.y);
  a.y = fma(x.x, y.y, a.y);
  a.y = fma(-u.y, z.x, a.y);
  a.y = fma(u.x, z.y, a.y);
  return a;
}

// a / b for complex b != 0
__device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
  const double den = b.x * b.x + b.y * b.y;
  return cmake((a.x * b.x + a.y * b.y) / den, (a.y * b.x - a.x * b.y) / den);
}

// ---------------------------------------------------------------------------------
// 1a. Tridiagonalisation with the matrix resident in shared memory: cluster c handles
//     sector list[c]; CTA `rank` of its cl CTAs holds the rows i = rank (mod cl), stored by
//     columns so that a lane works on a row of its own and a row's dot product needs no
//     exchange between lanes.  Step j (trailing size t = k - j - 1), all in shared memory:
//     1   alpha = -|tau|^2 v^H A v / 2 of step j - 1 from the partials (zhetd2's
//         -tau p^H v / 2, which is real because A is Hermitian); v = sc y and
//         w = p + alpha v of step j - 1 (in y's and p's place); row j minus the pending
//         rank-2 update gives d_j and, conjugated, y, the vector the reflector is formed
//         from; its norm.  Done redundantly in every CTA on bit-identical inputs and in the
//         same order, so every CTA holds the same y without exchanging it;
//     2   own rows i > j, up to four to a lane, the columns dealt out to the warps and spare
//         lanes in runs: A[i][l] -= v'_i conj(w'_l) + w'_i conj(v'_l)
//         (v', w' of step j - 1) and the dot products with y.  A warp of its own computes
//         the reflector beside them (zlarfg: beta real, tau_j, v_j = sc y but 1 at j + 1);
//         it enters in 3, so its square root and division are off the step's chain;
//     3   p_i = tau (A[i][j + 1] + sc sum_l A[i][l] y_l); p_i, A[i][j + 1] (row j + 1 of the
//         next step, by symmetry) and the rows' part of alpha go into every CTA of the
//         cluster.
//     Two barriers within a CTA and one of the cluster per step; p, the row and the partials
//     of alpha are double-buffered by step parity, so a CTA that runs ahead writes what nobody
//     reads before the next barrier.
//     What bounds it: shared-memory instructions -- a 128-bit access of a warp takes four
//     cycles of the SM even where all lanes read one address, so an entry's load and store
//     and three vector loads would take longer than its 12 fused multiply-adds; four rows to
//     a lane share the vector loads (44 cycles for 128 entries) -- and the latency of the
//     step's chain (three warp sums, three barriers).
//     Measured, one sector alone, us (k = 27, 50, 100, 209, 310, 430): 41, 84, 213, 594,
//     1,062, 1,565, where the streamed form with 1 to 4 CTAs of 128 threads took 120, 312, 756,
//     2,847, 7,205, 8,553.  31 sectors of k = 430 at once take 7.8 ms against 9.0 (seven
//     clusters of 16 fit the GPU).
constexpr int TD_RES_CLASSES = 7;
// largest k, CTAs per sector and threads per CTA of a class.  The bounds of the classes
// from 2 on are what 227 KB of shared memory per CTA hold; below, several sectors share an
// SM, with about four warps to every 32 rows.
constexpr int TD_RES_K[TD_RES_CLASSES] = {28, 56, 113, 158, 224, 310, 430};
constexpr int TD_RES_MAX = TD_RES_K[TD_RES_CLASSES - 1];
constexpr int TD_RES_CL[TD_RES_CLASSES] = {1, 1, 1, 2, 4, 8, 16};
constexpr int TD_RES_NT[TD_RES_CLASSES] = {128, 256, 256, 256, 256, 256, 256};

// v, p and the next row, two of each; the partials of the dot products and (two sets, real)
// of alpha; 64 scalars; the rows
__host__ __device__ constexpr int td_res_rows(int k, int cl) { return (k + cl - 1) / cl; }
// 32-row slots of a CTA's rows, a power of two
__host__ __device__ constexpr int td_res_slots(int k, int cl) {
  const int rows = td_res_rows(k, cl);
  return rows > 64 ? 4 : rows > 32 ? 2 : 1;
}
__host__ __device__ constexpr size_t td_res_smem(int k, int cl, int nt) {
  return sizeof(cplx) * (6 * (size_t)k + (size_t)nt * td_res_slots(k, cl) + (size_t)cl * td_res_slots(k, cl) +
                         (size_t)td_res_rows(k, cl) * k) +
         64 * sizeof(double);
}
constexpr bool td_res_fits() {
  for (int c = 0; c < TD_RES_CLASSES; ++c)
    if (td_res_smem(TD_RES_K[c], TD_RES_CL[c], TD_RES_NT[c]) > 227 * 1024 ||
        td_res_rows(TD_RES_K[c], TD_RES_CL[c]) > 128 || td_res_slots(TD_RES_K[c], TD_RES_CL[c]) > TD_RES_NT[c] / 32)
      return false;
  return true;
}
static_assert(td_res_fits(), "a class exceeds a CTA's shared memory, or its warps do not cover its rows");

// Phase 2 of one group of lanes: rows r, r + RL, .. (RPL of them, the first n stored), columns
// l .. end - 1.  UPD: with the rank-2 update (not in step 0).
template <int RPL, bool UPD>
__device__ __forceinline__ void td_res_columns(cplx* ap, const int (&ro)[4], int ld, int n, const cplx* vprev,
                                               const cplx* wprev, const cplx* ycur, const int (&ri)[4], int l, int end,
                                               cplx (&acc)[4]) {
  constexpr int UN = RPL > 2 ? 2 : 4;  // columns in flight
  cplx vi[RPL], wi[RPL];
  if (UPD) {
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      vi[q] = ldc(vprev + ri[q]);
      wi[q] = ldc(wprev + ri[q]);
    }
  }
  auto columns = [&](auto un) {
    constexpr int U = decltype(un)::value;
    cplx y[U], vp[U], wp[U], a[U][RPL];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int q = 0; q < RPL; ++q) a[u][q] = ldc(ap + u * ld + ro[q]);
      if (UPD) {
        wp[u] = ldc(wprev + l + u);
        vp[u] = ldc(vprev + l + u);
      }
      y[u] = ldc(ycur + l + u);
    }
    if (UPD) {
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < RPL; ++q) a[u][q] = crank2(a[u][q], vi[q], wp[u], wi[q], vp[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < RPL; ++q)
          if (q < n) stc(ap + u * ld + ro[q], a[u][q]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < RPL; ++q) cfma(acc[q], a[u][q], y[u]);
    l += U;
    ap += U * ld;
  };
#pragma unroll 1
  while (l + UN <= end) columns(std::integral_constant<int, UN>());
#pragma unroll 1
  while (l < end) columns(std::integral_constant<int, 1>());
}

// NT worker threads and one warp more, which forms the reflectors
template <int NT>
__global__ void __launch_bounds__(NT + 32)
    tridiag_resident_kernel(const SectorDesc* __restrict__ sd, const int* __restrict__ list,
                            cplx* __restrict__ gbuf, double* __restrict__ dbuf,
                            double* __restrict__ ebuf, cplx* __restrict__ taubuf) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int cl = (int)cluster.num_blocks(), cls = __ffs(cl) - 1;   // a power of two
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SectorDesc& S = sd[list[blockIdx.x >> cls]];
  // what is left of the sector where the streamed kernel has reduced its first `off` rows
  const int ldg = S.k, off = max(S.k - TD_RES_MAX, 0);
  const int k = S.k - off;             // the same for every CTA of the cluster
  const int slots = td_res_slots(k, cl), nc = cl * slots;   // partials of alpha, at most 32
  const int sls = slots >> 1;          // log2 of 1, 2, 4
  const int ld = td_res_rows(k, cl);
  cplx* vb = reinterpret_cast<cplx*>(smem_raw);   // y, then v, of step j: vb + (j & 1) k
  cplx* pb = vb + 2 * k;               // p, then w, of step j: pb + (j & 1) k
  cplx* xb = pb + 2 * k;               // row j + 1 as step j left it: xb + (j & 1) k
  cplx* part = xb + 2 * k;             // partials of the dot products: part + warp 32 slots
  double* cb = reinterpret_cast<double*>(part + NT * slots);   // partials of alpha of step j: cb + (j & 1) nc
  double* scal = cb + 2 * nc;          // [0, NW) norm, [46, 48) diagonal, [48, 50) first of y, [50, 54) tau, sc
  cplx* As = reinterpret_cast<cplx*>(scal + 64);   // row i = rank + r cl: As[l ld + r] = A[i][l]
  cplx* A = gbuf + S.g_off + (int64_t)off * ldg + off;
  double* dd = dbuf + S.s_off + off;
  double* ee = ebuf + S.s_off + off;
  cplx* tt = taubuf + S.s_off + off;
  if (k <= 1) {
    if (k == 1 && rank == 0 && tid == 0) dd[0] = A[0].x;
    return;                            // uniform over the cluster
  }
  const int own = (k - rank + cl - 1) >> cls;
  if (off > 0) {
    // the streamed kernel's last rank-2 update is pending: v in the row above, w in column
    // 0 of the whole matrix
    for (int l = tid; l < k; l += NT + 32) {
      stc(vb + l, ldc(A - ldg + l));
      stc(pb + l, ldc(A + (int64_t)l * ldg - off));
    }
    __syncthreads();
  }
  auto entry = [&](int i, int l) {
    const cplx a = ldc(A + (int64_t)i * ldg + l);
    return off > 0 ? crank2(a, ldc(vb + i), ldc(pb + l), ldc(pb + i), ldc(vb + l)) : a;
  };
  // A[i][l] = conj(A[l][i]): a warp reads along a row of the matrix
  for (int l = warp; l < k; l += NW + 1)
    for (int r = lane; r < own; r += 32) stc(As + l * ld + r, cconj(entry(l, rank + (r << cls))));
  // row 0 to every CTA (step -1 of the row buffers)
  for (int l = tid; l < k; l += NT + 32) stc(xb + k + l, entry(0, l));
  cluster.sync();                      // row 0 of the global matrix is overwritten from here on
  // alpha of step j from the partials
  auto alpha_of = [&](int j) { return warp_sum(lane < nc ? cb[(j & 1) * nc + lane] : 0.0); };
  for (int j = 0; j < k - 1; ++j) {
    const int par = j & 1;
    cplx* ycur = vb + par * k;
    cplx* vprev = vb + (par ^ 1) * k;  // y of step j - 1 until phase 1 has scaled it
    cplx* wprev = pb + (par ^ 1) * k;  // p of step j - 1 likewise
    // ---- 1 (v'_j = 1; entry j of v' and w' is not read again, so it is not written)
    const int na = min(NW, (k - j + 31) >> 5);   // warps with an entry
    if (warp < na) {
      const cplx* x = xb + (par ^ 1) * k;
      double al = 0.0;
      cplx w1 = cmake(0.0, 0.0), sc = w1;
      if (j > 0) {
        al = alpha_of(j - 1);
        w1 = ldc(wprev + j);
        w1.x += al;
        sc = cmake(scal[52], scal[53]);
      }
      const bool keeper = j > 0 && rank == ((j - 1) & (cl - 1));   // stores v_{j-1} for the back-transformation
      double part2 = 0.0;
      for (int l = j + tid; l < k; l += NT) {
        cplx a = ldc(x + l);
        if (j > 0) {
          cplx v = cmul(sc, ldc(vprev + l)), w = ldc(wprev + l);
          w = cmake(fma(al, v.x, w.x), fma(al, v.y, w.y));
          if (l > j) {
            stc(vprev + l, v);
            stc(wprev + l, w);
          } else {
            v = cmake(1.0, 0.0);
            w = w1;
          }
          if (keeper) stc(A + (int64_t)(j - 1) * ldg + l, v);
          // row j: a - (conj(w_l) + w_j conj(v_l))
          a = csub(a, cadd(cconj(w), cmulc(w1, v)));
        }
        // d_j, then the first of y: its part of the dot products is added in phase 3
        const bool head = l <= j + 1;
        if (head) {
          scal[46 + 2 * (l - j)] = a.x;
          scal[47 + 2 * (l - j)] = -a.y;
          a = cmake(0.0, 0.0);
        }
        stc(ycur + l, cconj(a));
        part2 += cabs2(a);
      }
      part2 = warp_sum(part2);
      if (lane == 0) scal[warp] = part2;
    }
    __syncthreads();
    // ---- 2: own rows r = r0 .. own - 1 (i = rank + r cl > j); 8, 16 or 32 lanes across them
    const int r0 = j >= rank ? ((j - rank) >> cls) + 1 : 0;
    const int rows = own - r0;
    if (warp == NW) {
      // the reflector
      double xn2 = scal[0];
      for (int q = 1; q < na; ++q) xn2 += scal[q];
      const cplx alpha = cmake(scal[48], scal[49]);
      double beta = alpha.x;
      cplx tau = cmake(0.0, 0.0), sc = tau;
      if (xn2 != 0.0 || alpha.y != 0.0) {
        beta = -copysign(sqrt(fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, xn2))), alpha.x);
        tau = cmake((beta - alpha.x) / beta, -alpha.y / beta);
        sc = cdiv(cmake(1.0, 0.0), cmake(alpha.x - beta, alpha.y));
      }
      if (lane == 0) {
        scal[50] = tau.x; scal[51] = tau.y;
        scal[52] = sc.x; scal[53] = sc.y;
        if (rank == (j & (cl - 1))) { dd[j] = scal[46]; ee[j] = beta; tt[j] = tau; }
      }
    } else if (rows > 0) {
      const int rls = rows > 64 ? 5 : rows > 32 ? 4 : 3;   // log2 of the lanes across rows
      const int idx = lane & ((1 << rls) - 1);
      // rows past the end repeat the last one; they are not stored
      int ro[4], ri[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ro[q] = min(r0 + idx + (q << rls), own - 1);
        ri[q] = rank + (ro[q] << cls);
      }
      const int n = (rows - idx + (1 << rls) - 1) >> rls;   // rows of this lane
      // the columns j + 1 .. k - 1 in equal runs, one to each group of lanes
      constexpr int NWS = NW == 4 ? 2 : 3;
      const int gs = NWS + 5 - rls;        // log2 of the groups
      const int run = (k - j - 2 + (1 << gs)) >> gs;
      const int l = j + 1 + ((warp << (5 - rls)) + (lane >> rls)) * run, end = min(l + run, k);
      cplx acc[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = cmake(0.0, 0.0);
      cplx* ap = As + l * ld;
      const int rpl = (rows + (1 << rls) - 1) >> rls;       // 1 .. 4, warp-uniform
      if (j == 0) td_res_columns<4, false>(ap, ro, ld, n, vprev, wprev, ycur, ri, l, end, acc);
      else if (rpl > 3) td_res_columns<4, true>(ap, ro, ld, n, vprev, wprev, ycur, ri, l, end, acc);
      else if (rpl > 2) td_res_columns<3, true>(ap, ro, ld, n, vprev, wprev, ycur, ri, l, end, acc);
      else if (rpl > 1) td_res_columns<2, true>(ap, ro, ld, n, vprev, wprev, ycur, ri, l, end, acc);
      else td_res_columns<1, true>(ap, ro, ld, n, vprev, wprev, ycur, ri, l, end, acc);
      __syncwarp();
      // sums over the groups within the warp, each exchange halving the rows a lane keeps:
      // with 8 lanes across the rows lane x ends with row x, with 16 with rows
      // (x mod 16) + 32 (x / 16) and 16 more
      const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
      cplx* pp = part + (warp * slots << 5);
      if (rls == 5) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < n) stc(pp + idx + 32 * q, acc[q]);
      } else {
        const cplx s0 = h16 ? acc[0] : acc[2], s1 = h16 ? acc[1] : acc[3];
        cplx k0 = h16 ? acc[2] : acc[0], k1 = h16 ? acc[3] : acc[1];
        k0.x += __shfl_xor_sync(0xffffffffu, s0.x, 16);
        k0.y += __shfl_xor_sync(0xffffffffu, s0.y, 16);
        k1.x += __shfl_xor_sync(0xffffffffu, s1.x, 16);
        k1.y += __shfl_xor_sync(0xffffffffu, s1.y, 16);
        if (rls == 4) {
          const int x = idx + (h16 ? 32 : 0);
          if (x < rows) stc(pp + x, k0);
          if (x + 16 < rows) stc(pp + x + 16, k1);
        } else {
          const cplx s = h8 ? k0 : k1;
          cplx p = h8 ? k1 : k0;
          p.x += __shfl_xor_sync(0xffffffffu, s.x, 8);
          p.y += __shfl_xor_sync(0xffffffffu, s.y, 8);
          if (lane < rows) stc(pp + lane, p);
        }
      }
    }
    __syncthreads();
    // ---- 3: a warp to a slot of 32 rows and every (NW >> sls)-th receiving CTA
    if (warp < NW && (warp >> sls) < cl) {
      const int slot = warp & (slots - 1), idx = (slot << 5) + lane;
      cplx p = cmake(0.0, 0.0), xi = p;
      double ai = 0.0;
      const int i = rank + ((r0 + idx) << cls);
      if (idx < rows) {
        const cplx tau = cmake(scal[50], scal[51]), sc = cmake(scal[52], scal[53]);
        cplx acc = ldc(part + idx);
#pragma unroll
        for (int c = 1; c < NW; ++c) acc = cadd(acc, ldc(part + (c * slots << 5) + idx));
        const cplx aj = ldc(As + (j + 1) * ld + r0 + idx);
        xi = cconj(aj);
        const cplx av = cadd(aj, cmul(sc, acc));   // (A v)_i
        p = cmul(tau, av);
        const cplx v = i == j + 1 ? cmake(1.0, 0.0) : cmul(sc, ldc(ycur + i));
        ai = -0.5 * cabs2(tau) * fma(v.x, av.x, v.y * av.y);
      }
      cplx* pd = pb + par * k + i;
      cplx* xd = xb + par * k + i;
      double* ad = cb + par * nc + rank * slots + slot;
      if (cl == 1) {
        if (idx < rows) { stc(pd, p); stc(xd, xi); }
        ai = warp_sum(ai);
        if (lane == 0) *ad = ai;
      } else {
        for (int q = warp >> sls; q < cl; q += NW >> sls)
          if (idx < rows) {
            stc(cluster.map_shared_rank(pd, q), p);
            stc(cluster.map_shared_rank(xd, q), xi);
          }
        ai = warp_sum(ai);
        for (int q = warp >> sls; q < cl; q += NW >> sls)
          if (lane == 0) *cluster.map_shared_rank(ad, q) = ai;
      }
    }
    if (cl > 1) cluster.sync(); else __syncthreads();
  }
  // last diagonal entry: row k - 1 minus the update of step k - 2 (v = 1 there)
  if (rank == 0 && warp == 0) {
    const int j = k - 1, par = (k - 2) & 1;
    const double w = pb[par * k + j].x + alpha_of(k - 2);
    if (lane == 0) {
      dd[j] = xb[par * k + j].x - 2.0 * w;
      stc(A + (int64_t)(k - 2) * ldg + j, cmake(1.0, 0.0));
    }
  }
}

// ---------------------------------------------------------------------------------
// 1b. The first k - TD_RES_MAX steps of the larger sectors, rows streamed from L2; the
//    resident kernel takes over there (a step costs about 10 us here at k = 445, 30 at 1,024,
//    and 3.6 in the resident kernel).  Cluster c handles sector list[c]; its TD_CL CTAs own
//    the rows i = rank (mod TD_CL).  Every CTA holds the reflector vectors
//    and a copy of the row being reduced, so one cluster barrier per step suffices.
//    Step j (trailing size t = k - j - 1):
//    R   every CTA (warp 0): row j as the previous pass left it, minus the pending
//        rank-2 update of step j - 1, gives d_j and the reflector (zlarfg: beta real,
//        tau_j, v_j), computed redundantly and bit-identically in every CTA (the same
//        inputs, the same warp reduction);
//    P   every CTA, its rows i > j: A[i][l] -= v'_i conj(w'_l) + w'_i conj(v'_l) (v', w'
//        of step j - 1), write back, p_i = tau sum_l A[i][l] v_l, partial
//        c = sum conj(p_i) v_i; the owner of row j + 1 also publishes that row;
//    --  cluster barrier
//    G   every CTA: c = sum of the partials (fixed order), w_j = p - tau c / 2 v from the
//        owners' p, and a copy of the published row j + 1 (the next step's R); the owner
//        of row j stores v_j there for the back-transformation, d_j, e_j = beta, tau_j.
//    p and the partials are double-buffered by step parity; the published row is written
//    again only cl steps later: every next write follows the next barrier, which no CTA
//    passes before every CTA has finished its G.
//    Rows stream through shared memory.  Warp w of a CTA handles its own rows number
//    r = w (mod 8) in every step (row i = rank + r cl), through a private ring of row
//    slots: its lane 0 issues a bulk copy (cp.async.bulk, completion counted on the
//    slot's mbarrier) of the row's trailing segment as soon as the slot is free and the
//    warp has written that row back in the previous step, so the copies run ahead of
//    the pass -- across the barrier, G and the next R into the next step's first rows
//    -- instead of one L2 round trip per load.  A row is read and written by one warp
//    only; its write-back is ordered before the next bulk read of it by a proxy fence
//    of the writing lanes and the warp's synchronisation.
__global__ void __launch_bounds__(TD_NT, 2)
    tridiag_kernel(const SectorDesc* __restrict__ sd, const int* __restrict__ list, int kmax,
                   cplx* __restrict__ gbuf, double* __restrict__ dbuf, double* __restrict__ ebuf,
                   cplx* __restrict__ taubuf, int* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  constexpr int cls = 4;               // log2 of TD_CL
  static_assert(TD_CL == 1 << cls, "rows are dealt out by shifts");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int own_cap = kmax / TD_CL + 1;
  const int nslot = td_slots(kmax, TD_NW);         // 1, 2 or 4
  const int nss = __ffs(nslot) - 1;
  cplx* ring = reinterpret_cast<cplx*>(smem_raw);  // slot s of warp w: ring + (w nslot + s) kmax
  cplx* vb = ring + (size_t)TD_NW * nslot * kmax;  // v of two consecutive steps: vb + (j & 1) kmax
  cplx* wb = vb + 2 * kmax;                        // w likewise
  cplx* pub = wb + 2 * kmax;                       // row j + 1 as published by its owner
  cplx* nrow = pub + kmax;                         // this CTA's copy of the row being reduced
  cplx* pown = nrow + kmax;                        // p of the own rows: pown + (j & 1) own_cap
  // [0..3] partial c of the two parities, [4..5] tau of this step, [8..] warp partials
  double* scal = reinterpret_cast<double*>(pown + 2 * own_cap);
  uint64_t* bars = reinterpret_cast<uint64_t*>(scal + 64) + warp * TD_MAXSLOT;   // this warp's
  cplx* wring = ring + (size_t)warp * nslot * kmax;
  const SectorDesc& S = sd[list[blockIdx.x / TD_CL]];
  const int k = S.k;                   // the same for every CTA of the cluster
  const int steps = k - TD_RES_MAX;    // >= 1; the rest is the resident kernel's
  cplx* A = gbuf + S.g_off;
  double* dd = dbuf + S.s_off;
  double* ee = ebuf + S.s_off;
  cplx* tt = taubuf + S.s_off;
  if (lane < TD_MAXSLOT) {
    mbar_init(bars + lane, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  // ---- this warp's row sequence: (step s, own row r) with rows i = rank + r cl > s,
  // r = warp (mod 8), in step order, then row order; copies are issued in the same order
  // as the pass consumes them, element q into slot q mod nslot
  auto first_row = [&](int s) {
    const int r0 = s >= rank ? ((s - rank) >> cls) + 1 : 0;
    return r0 + ((warp - r0) & (TD_NW - 1));
  };
  int is = 0, ir = first_row(0);       // next element to copy
  int issued = 0, done = 0;            // elements copied / consumed
  int ls = -1, lr = 0;                 // the last consumed element
  auto issue = [&]() {
    // a free slot, and the row's write-back of the previous step done (consumption is in
    // sequence order, so the last consumed element tells)
    while (is < steps && rank + (ir << cls) < k && issued < done + nslot &&
           (is == 0 || ls > is - 1 || (ls == is - 1 && lr >= ir))) {
      if (lane == 0) {
        const int slot = issued & (nslot - 1);
        const uint32_t bytes = (uint32_t)(k - is - 1) * (uint32_t)sizeof(cplx);
        mbar_expect_tx(bars + slot, bytes);
        bulk_load(wring + (size_t)slot * kmax, A + (int64_t)(rank + (ir << cls)) * k + is + 1, bytes,
                  bars + slot);
      }
      ++issued;
      ir += TD_NW;
      if (rank + (ir << cls) >= k) ir = first_row(++is);
    }
  };
  issue();

  double beta = 0.0;                   // this step's e_j (warp 0)
  for (int j = 0; j < steps; ++j) {
    const int par = j & 1;
    const bool owner = rank == (j & (TD_CL - 1));
    cplx* vcur = vb + par * kmax;
    const cplx* vprev = vb + (par ^ 1) * kmax;
    const cplx* wprev = wb + (par ^ 1) * kmax;
    // ---- R: the reflector of row j (warp 0 of every CTA; warp shuffles only)
    if (warp == 0) {
      const cplx* row = A + (int64_t)j * k;
      double part = 0.0;
      const cplx vj = j > 0 ? vprev[j] : cmake(0.0, 0.0), wj = j > 0 ? wprev[j] : cmake(0.0, 0.0);
      for (int l = j + lane; l < k; l += 32) {
        // row j as the previous pass left it (copied from its owner), the Gram at j = 0
        cplx a = j > 0 ? nrow[l] : ldc(row + l);
        if (j > 0) a = crank2(a, vj, ldc(wprev + l), wj, ldc(vprev + l));
        if (l == j) {
          if (owner) dd[j] = a.x;
        } else {
          const cplx x = cconj(a);
          vcur[l] = x;                  // x for now, scaled below
          if (l > j + 1) part += cabs2(x);
        }
      }
      const double xn2 = warp_sum(part);   // the same value in every lane
      __syncwarp();
      const cplx alpha = vcur[j + 1];
      cplx tau, sc;
      if (xn2 == 0.0 && alpha.y == 0.0) {
        tau = cmake(0.0, 0.0);
        beta = alpha.x;
        sc = cmake(0.0, 0.0);
      } else {
        beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn2), alpha.x);
        tau = cmake((beta - alpha.x) / beta, -alpha.y / beta);
        sc = cdiv(cmake(1.0, 0.0), cmake(alpha.x - beta, alpha.y));
      }
      __syncwarp();                     // alpha read by every lane before vcur[j + 1] changes
      for (int l = j + 1 + lane; l < k; l += 32)
        vcur[l] = l == j + 1 ? cmake(1.0, 0.0) : cmul(sc, vcur[l]);
      if (lane == 0) {
        scal[4] = tau.x;
        scal[5] = tau.y;
      }
    }
    __syncthreads();
    const cplx tau = cmake(scal[4], scal[5]);
    // ---- P: fused update + matrix-vector product on this warp's rows
    {
      double cpx = 0.0, cpy = 0.0;
      cplx* pw = pown + par * own_cap;
      // rows two at a time where the ring holds two slots: one pass over the vectors for
      // both rows
      for (int r = first_row(j); rank + (r << cls) < k;) {
        const int r2 = r + TD_NW;
        const int i = rank + (r << cls), i2 = rank + (r2 << cls);
        const bool two = nslot >= 2 && i2 < k;   // warp-uniform
        const int slot = done & (nslot - 1), slot2 = (done + 1) & (nslot - 1);
        // on expiry the error word is set and the pass goes on with what the slot holds
        mbar_wait_fast(bars + slot, (uint32_t)(done >> nss) & 1u, err);
        if (two) mbar_wait_fast(bars + slot2, (uint32_t)((done + 1) >> nss) & 1u, err);
        const cplx* srow = wring + (size_t)slot * kmax - (j + 1);     // srow[l], l > j
        const cplx* srow2 = wring + (size_t)slot2 * kmax - (j + 1);
        cplx* grow = A + (int64_t)i * k;
        cplx* grow2 = A + (int64_t)(two ? i2 : i) * k;
        const bool next = i == j + 1;  // the next reflector row (never the second): publish it
        const cplx vi = j > 0 ? vprev[i] : cmake(0.0, 0.0), wi = j > 0 ? wprev[i] : cmake(0.0, 0.0);
        const cplx vi2 = (j > 0 && two) ? vprev[i2] : cmake(0.0, 0.0);
        const cplx wi2 = (j > 0 && two) ? wprev[i2] : cmake(0.0, 0.0);
        cplx acc = cmake(0.0, 0.0), acc2 = cmake(0.0, 0.0);
        if (two && j > 0 && !next) {
          // the common case without per-entry tests
#pragma unroll 2
          for (int l = j + 1 + lane; l < k; l += 32) {
            const cplx vc = ldc(vcur + l), vp = ldc(vprev + l), wp = ldc(wprev + l);
            const cplx a = crank2(ldc(srow + l), vi, wp, wi, vp);
            const cplx a2 = crank2(ldc(srow2 + l), vi2, wp, wi2, vp);
            stc(grow + l, a);
            stc(grow2 + l, a2);
            cfma(acc, a, vc);
            cfma(acc2, a2, vc);
          }
        } else {
#pragma unroll 2
          for (int l = j + 1 + lane; l < k; l += 32) {
            cplx a = ldc(srow + l);
            cplx a2 = two ? ldc(srow2 + l) : cmake(0.0, 0.0);
            const cplx vc = ldc(vcur + l);
            if (j > 0) {
              const cplx vp = ldc(vprev + l), wp = ldc(wprev + l);
              a = crank2(a, vi, wp, wi, vp);
              stc(grow + l, a);
              if (two) {
                a2 = crank2(a2, vi2, wp, wi2, vp);
                stc(grow2 + l, a2);
              }
            }
            if (next) pub[l] = a;
            cfma(acc, a, vc);
            cfma(acc2, a2, vc);
          }
        }
        // the write-back before the next bulk read of these rows (async proxy)
        if (j > 0) asm volatile("fence.proxy.async.global;" ::: "memory");
        if (two) {
          // both rows in one butterfly: after the first exchange lanes 0-15 carry row i and
          // lanes 16-31 row i2; lane 0 ends with row i's sum and fetches row i2's from lane 16
          const bool hi = (lane & 16) != 0;
          const cplx send = hi ? acc : acc2;
          cplx keep = hi ? acc2 : acc;
          keep.x += __shfl_xor_sync(0xffffffffu, send.x, 16);
          keep.y += __shfl_xor_sync(0xffffffffu, send.y, 16);
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) {
            keep.x += __shfl_xor_sync(0xffffffffu, keep.x, o);
            keep.y += __shfl_xor_sync(0xffffffffu, keep.y, o);
          }
          acc = keep;
          acc2 = cmake(__shfl_sync(0xffffffffu, keep.x, 16), __shfl_sync(0xffffffffu, keep.y, 16));
        } else {
          acc = warp_sum(acc);
        }
        if (lane == 0) {
          // p_i, and conj(p_i) v_i summed by lane 0 of each warp in row order
          const cplx p = cmul(tau, acc);
          pw[r] = p;
          const cplx cv = ccmul(p, vcur[i]);
          cpx += cv.x;
          cpy += cv.y;
          if (two) {
            const cplx p2 = cmul(tau, acc2);
            pw[r2] = p2;
            const cplx cv2 = ccmul(p2, vcur[i2]);
            cpx += cv2.x;
            cpy += cv2.y;
          }
        }
        __syncwarp();                  // every lane done with the slots and the rows
        done += two ? 2 : 1;
        ls = j;
        lr = two ? r2 : r;
        issue();
        r = two ? r2 + TD_NW : r2;
      }
      if (lane == 0) {
        scal[8 + 2 * warp] = cpx;
        scal[9 + 2 * warp] = cpy;
      }
      __syncthreads();
      if (tid == 0) {
        double sx = 0.0, sy = 0.0;
        for (int w = 0; w < TD_NW; ++w) { sx += scal[8 + 2 * w]; sy += scal[9 + 2 * w]; }
        scal[2 * par] = sx;
        scal[2 * par + 1] = sy;
      }
    }
    cluster.sync();
    // ---- G: w_j from every owner's p, the next row from its owner
    {
      double cx = 0.0, cy = 0.0;
      for (int q = 0; q < TD_CL; ++q) {   // fixed order: the same sum in every CTA
        const double* qs = cluster.map_shared_rank(scal, q);
        cx += qs[2 * par];
        cy += qs[2 * par + 1];
      }
      const cplx a2 = cscale(cmul(tau, cmake(cx, cy)), -0.5);
      cplx* wcur = wb + par * kmax;
      const cplx* rpub = cluster.map_shared_rank(pub, (j + 1) & (TD_CL - 1));
      for (int l = j + 1 + tid; l < k; l += TD_NT) {
        const cplx* rp = cluster.map_shared_rank(pown, l & (TD_CL - 1));
        wcur[l] = cadd(rp[par * own_cap + (l >> cls)], cmul(a2, vcur[l]));
        nrow[l] = rpub[l];
      }
      if (owner) {
        // v_j kept in row j for the back-transformation (row j has been read by every
        // CTA before the barrier, and no copy of it is issued after step j - 1)
        cplx* row = A + (int64_t)j * k;
        for (int l = j + 1 + tid; l < k; l += TD_NT) stc(row + l, vcur[l]);
        if (tid == 0) {
          ee[j] = beta;                 // thread 0 is lane 0 of warp 0, which formed it
          tt[j] = tau;
        }
      }
      __syncthreads();
    }
  }
  // w of the last step, whose update of the rows i >= steps is pending, into column 0
  for (int r = tid; rank + (r << cls) < k; r += TD_NT) {
    const int i = rank + (r << cls);
    if (i >= steps) stc(A + (int64_t)i * k, wb[((steps - 1) & 1) * kmax + i]);
  }
  cluster.sync();   // no CTA leaves while another may still read its shared memory
}

// ---------------------------------------------------------------------------------
// 2. Eigenvalues: warp i of sector s finds the i-th largest eigenvalue of (d, e) by
//    multisection: 32 Sturm counts per pass (one per lane), the interval shrinks 33x.
//    The counts use the three-term recurrence of the leading minors, p_i = (d_i - x) p_{i-1}
//    - e_{i-1}^2 p_{i-2} (Givens 1954; Barth, Martin, Wilkinson 1967), on the matrix scaled
//    to a norm of at most one: two dependent operations a step, where the ratio form has a
//    division in its chain.  The pair is rescaled by a power of two every BI_RS steps, in
//    which it can grow by 3^BI_RS and, with e^2 held above BI_E2, shrink by at most
//    BI_E2^(BI_RS / 2) or eps^BI_RS.  A minor of exactly zero changes the count by one over
//    its two steps whatever its sign bit.
//    Measured, all sectors of a chi = 1024 update alone: 144 us against 469 with divisions.
constexpr int BI_NT = 256;
constexpr int BI_RS = 8;
constexpr double BI_E2 = 1e-60;

// number of eigenvalues below x of the scaled matrix, de[i] = (d_i, e_{i-1}^2)
__device__ __forceinline__ int sturm_count(const double2* de, int k, double x) {
  double pp = 1.0, p = de[0].x - x;
  int c = (unsigned)__double2hiint(p) >> 31;
  auto step = [&](double2 v) {
    const double n = fma(v.x - x, p, -v.y * pp);
    c += (unsigned)(__double2hiint(n) ^ __double2hiint(p)) >> 31;
    pp = p;
    p = n;
  };
  auto rescale = [&]() {
    // the larger of the two to [1, 2)
    const int h = max(__double2hiint(p) & 0x7ff00000, __double2hiint(pp) & 0x7ff00000);
    const double f = __hiloint2double(0x7fe00000 - h, 0);
    p *= f;
    pp *= f;
  };
  int i = 1;
  for (; i + BI_RS <= k; i += BI_RS) {
    double2 v[BI_RS];
#pragma unroll
    for (int q = 0; q < BI_RS; ++q) v[q] = de[i + q];
#pragma unroll
    for (int q = 0; q < BI_RS; ++q) step(v[q]);
    rescale();
  }
  for (; i < k; ++i) step(de[i]);
  return c;
}

// a launch's sectors: all of them, or a list
__device__ __forceinline__ int sector_of(const int* list, int i) { return list ? list[i] : i; }

__global__ __launch_bounds__(BI_NT) void bisect_kernel(const SectorDesc* __restrict__ sd,
                                                       const int* __restrict__ list,
                                                       const double* __restrict__ dbuf,
                                                       const double* __restrict__ ebuf,
                                                       double* __restrict__ lam) {
  extern __shared__ double2 de[];
  const SectorDesc& S = sd[sector_of(list, blockIdx.y)];
  const int k = S.k;
  const int first = blockIdx.x * (BI_NT / 32);
  if (first >= k) return;             // uniform over the CTA
  __shared__ double red[2][BI_NT / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* dg = dbuf + S.s_off;
  const double* eg = ebuf + S.s_off;
  double lo = 1e300, hi = -1e300;
  for (int i = tid; i < k; i += BI_NT) {
    const double di = dg[i];
    const double ea = i > 0 ? fabs(eg[i - 1]) : 0.0, eb = i < k - 1 ? fabs(eg[i]) : 0.0;
    de[i] = make_double2(di, ea);
    lo = fmin(lo, di - ea - eb);
    hi = fmax(hi, di + ea + eb);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) { red[0][warp] = lo; red[1][warp] = hi; }
  __syncthreads();
  lo = red[0][0];
  hi = red[1][0];
  for (int w = 1; w < BI_NT / 32; ++w) { lo = fmin(lo, red[0][w]); hi = fmax(hi, red[1][w]); }
  const double span = fmax(fabs(lo), fabs(hi));
  if (span == 0.0) {                   // a zero matrix (uniform over the CTA)
    if (tid < BI_NT / 32 && first + tid < k) lam[S.s_off + first + tid] = 0.0;
    return;
  }
  // a power of two above the bound of the spectrum
  int ex;
  frexp(span, &ex);
  for (int i = tid; i < k; i += BI_NT) {
    const double e = scalbn(de[i].y, -ex);
    de[i] = make_double2(scalbn(de[i].x, -ex), fmax(e * e, BI_E2));
  }
  __syncthreads();
  const int i = first + warp;
  if (i >= k) return;
  const int target = k - 1 - i;        // eigenvalues below lambda_(i) (ascending index)
  // widen by a few ulps of the bound so the extreme eigenvalues stay inside
  const double sspan = scalbn(span, -ex);
  double a = scalbn(lo, -ex) - 4.0 * EPS * sspan - 1e-300, b = scalbn(hi, -ex) + 4.0 * EPS * sspan + 1e-300;
  const double tol_abs = 4.0 * EPS * fmax(fabs(a), fabs(b));
  for (int it = 0; it < 16; ++it) {
    const double x = a + (double)(lane + 1) * ((b - a) / 33.0);
    const int c = sturm_count(de, k, x);
    const unsigned below = __ballot_sync(0xffffffffu, c <= target);
    const int L = __popc(below);       // counts rise with x: lanes 0..L-1 lie below
    const double xl = __shfl_sync(0xffffffffu, x, L > 0 ? L - 1 : 0);
    const double xh = __shfl_sync(0xffffffffu, x, L < 32 ? L : 31);
    const double na = L > 0 ? xl : a, nb = L < 32 ? xh : b;
    a = na;
    b = nb;
    // absolute accuracy of a few eps ||T|| (the tridiagonalisation's own error) is all
    // the selection and sigma = sqrt(lambda) need
    if (b - a <= tol_abs) break;   // warp-uniform
  }
  if (lane == 0) lam[S.s_off + i] = scalbn(0.5 * (a + b), ex);
}

// Monotone order (bisection rounds independently), numerical floor, sigma and 1/sigma.
constexpr int FI_NT = 1024;
__global__ __launch_bounds__(FI_NT) void eig_finish_kernel(const SectorDesc* __restrict__ sd,
                                                           const double* __restrict__ lam,
                                                           double* __restrict__ sig,
                                                           double* __restrict__ invsig) {
  __shared__ double buf[2][FI_NT];
  const SectorDesc& S = sd[blockIdx.x];
  const int k = S.k;
  const int tid = threadIdx.x;
  // k <= FI_NT * 2 handled in two halves of the scan
  const double lmax = k > 0 ? lam[S.s_off] : 0.0;
  const double floor_l = 32.0 * EPS * (double)k * fabs(lmax);
  double carry = 1e300;
  for (int base = 0; base < k; base += FI_NT) {
    const int i = base + tid;
    double v = i < k ? lam[S.s_off + i] : 1e300;
    int cur = 0;
    buf[0][tid] = v;
    __syncthreads();
    for (int off = 1; off < FI_NT; off <<= 1) {   // inclusive prefix minimum
      const double x = buf[cur][tid];
      const double y = tid >= off ? buf[cur][tid - off] : 1e300;
      buf[cur ^ 1][tid] = fmin(x, y);
      cur ^= 1;
      __syncthreads();
    }
    v = fmin(buf[cur][tid], carry);
    if (i < k) {
      const double s = v > floor_l ? sqrt(v) : 0.0;
      sig[S.s_off + i] = s;
      invsig[S.s_off + i] = s > 0.0 ? 1.0 / s : 0.0;
    }
    carry = fmin(carry, buf[cur][FI_NT - 1]);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------
// 3a. Eigenvectors of the tridiagonal by inverse iteration, one thread per kept
//     eigenvalue, one CTA per sector.  T - lambda I = P L U with partial pivoting (U has
//     two superdiagonals), stored column-interleaved in the scratch (entry l of vector t
//     at l * kept + t, so a warp's accesses coalesce).  Start vector: a fixed
//     pseudo-random one; three solves, normalised.  Eigenvalues closer than `gaptol`
//     form a group; after the second and the third solve the whole CTA orthogonalises each
//     group's vectors in order (classical Gram-Schmidt, twice).
//     What bounds it: each thread's recurrences (k dependent steps, seven passes).  The
//     passes move IV_B steps of a column between registers and scratch at a time, one
//     batch ahead, and the factorisation keeps the pivots' reciprocals, so a step costs its
//     two or three dependent operations and not a division and an L2 round trip.
//     Measured: 3.1 ms of kernel time in two layers at N = 64, chi = 1024 (62 updates)
//     against 33.5 with one thread per group and a division and scratch access per step.
constexpr int IV_NT = 128;
constexpr int IV_B = 8;        // steps of a batch
constexpr int IV_GT = 32;      // group members one pass of the orthogonalisation takes
constexpr double IV_GAP_ALL = 1e-10;   // orthogonalise_kernel's groups, of the norm

__device__ __forceinline__ double start_entry(int l, int t) {
  unsigned h = (unsigned)l * 2654435761u ^ ((unsigned)t * 40503u + 0x9e3779b9u);
  h ^= h >> 15;
  h *= 2246822519u;
  h ^= h >> 13;
  return ((double)(h & 0xffffu) + 0.5) / 32768.0 - 1.0;
}

// Whether the eigenvalues show a sector to be better left as it is than preconditioned (whole
// warp): where fewer than chi values of its update lie above PRE_MIN of its largest and some
// of its own lie between that and the eigenvalues' floor, those would be kept and the update
// done again; where all values are equal within 5%, X's columns are nearly orthogonal.  Only a
// matter of time: what is kept too small after all is found by the selection.  Update of four
// 420 x 420 sectors, values over ten decades, chi = 1,260: 17.3 ms without the preconditioner,
// 50.0 with it and the second run, 18.9 left as they are; all values equal: 1.6, 11.2 and 2.9.
__device__ __forceinline__ bool better_plain(const SectorDesc* __restrict__ sds, int sec,
                                             const UpdateTables* __restrict__ tabs, int n_updates,
                                             const double* __restrict__ lam, double cutoff, int chi) {
  const int lane = threadIdx.x & 31;
  // its update: the last one that starts at or before it (a group has at most 32)
  const unsigned m = __ballot_sync(0xffffffffu, lane < n_updates && tabs[lane].sec0 <= sec);
  const UpdateTables* tab = tabs + (31 - __clz(m));
  const SectorDesc* sd = sds + tab->sec0;
  const int ns = tab->n_sectors, s = sec - tab->sec0, k = sd[s].k;
  auto pre = [&](int t) { return sd[t].t_off != sd[t].a_off; };
  auto above = [&](int t, double v) {   // eigenvalues of sector t above v
    const double* x = lam + sd[t].s_off;
    int lo = 0, hi = sd[t].k;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (x[mid] > v) lo = mid + 1; else hi = mid;
    }
    return lo;
  };
  const double l0 = lam[sd[s].s_off], ln = lam[sd[s].s_off + k - 1], x = PRE_MIN * PRE_MIN * l0;
  int n = 0;
  double top = 0.0;
  for (int t = lane; t < ns; t += 32) {
    n += pre(t) ? above(t, x) : sd[t].k;   // the others' values are not known yet
    top = fmax(top, pre(t) ? lam[sd[t].s_off] : 0.0);
  }
  n = __reduce_add_sync(0xffffffffu, n);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
  if (ln > 0.9 * l0) return true;
  if (n >= chi || cutoff * cutoff * top >= x) return false;
  const int own = lane < 2 ? above(s, lane == 0 ? 32.0 * EPS * k * l0 : x) : 0;
  return __shfl_sync(0xffffffffu, own, 0) > __shfl_sync(0xffffffffu, own, 1);
}

// tabs (preconditioner: every eigenvector, and the sectors better left as they are flagged
// with kept = -1) or null (the kept ones).
__global__ __launch_bounds__(IV_NT) void invit_kernel(SectorDesc* __restrict__ sd, const int* __restrict__ list,
                                                      const UpdateTables* __restrict__ tabs, int n_updates,
                                                      double cutoff, int chi,
                                                      const double* __restrict__ dbuf,
                                                      const double* __restrict__ ebuf,
                                                      const double* __restrict__ lam,
                                                      double* __restrict__ scratch,
                                                      unsigned char* __restrict__ swp,
                                                      double* __restrict__ zbuf) {
  extern __shared__ double ism[];
  __shared__ double dots[IV_NT / 32][IV_GT], coef[IV_GT], nrm2[IV_NT / 32];
  __shared__ int left;
  const bool all = tabs != nullptr;
  const int sec = sector_of(list, blockIdx.x);
  const SectorDesc& S = sd[sec];
  const int k = S.k, kept = all ? k : S.kept;
  if (kept == 0) return;
  if (all) {
    if (threadIdx.x < 32) {
      const bool yes = better_plain(sd, sec, tabs, n_updates, lam, cutoff, chi);
      if (threadIdx.x == 0) {
        left = yes;
        if (yes) sd[sec].kept = -1;
      }
    }
    __syncthreads();
    if (left) return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* d = ism;
  double* e = ism + k;
  for (int i = tid; i < k; i += IV_NT) {
    d[i] = dbuf[S.s_off + i];
    e[i] = i < k - 1 ? ebuf[S.s_off + i] : 0.0;
  }
  const double* lv = lam + S.s_off;
  const double norm = fmax(fabs(lv[0]), fabs(lv[k - 1]));
  const double gaptol = 1e-9 * norm;
  const double tiny = EPS * norm + 1e-300;
  // scratch of this sector: 1 / pivot, the superdiagonals, the multipliers (k x kept
  // each), and the row exchanges, IV_B of them to a byte
  double* RP = scratch + 4 * S.y_off;
  double* U1 = RP + (int64_t)k * kept;
  double* U2 = U1 + (int64_t)k * kept;
  double* MU = U2 + (int64_t)k * kept;
  unsigned char* SW = swp + S.y_off;
  double* Z = zbuf + S.y_off;
  __syncthreads();
  bool grouped = false;
  // with `all`, orthogonalise_kernel does the groups
  for (int m = tid; m < kept && !all; m += IV_NT) grouped |= m > 0 && lv[m - 1] - lv[m] <= gaptol;
  grouped = __syncthreads_or(grouped);
  for (int m = tid; m < kept; m += IV_NT) {
    // factor T - lambda I
    const double lambda = lv[m];
    double p = d[0] - lambda, q = k > 1 ? e[0] : 0.0;
    for (int i0 = 0; i0 < k; i0 += IV_B) {
      unsigned sw = 0;
#pragma unroll
      for (int b = 0; b < IV_B; ++b) {
        const int i = i0 + b;
        if (i >= k) break;
        const int64_t o = (int64_t)i * kept + m;
        const double ei = i < k - 1 ? e[i] : 0.0, en = i + 1 < k - 1 ? e[i + 1] : 0.0;
        const double an = i < k - 1 ? d[i + 1] - lambda : 0.0;
        const bool x = fabs(ei) > fabs(p);
        if (!x && p == 0.0) p = tiny;
        const double r = 1.0 / (x ? ei : p), mu = (x ? p : ei) * r;
        RP[o] = r;
        U1[o] = x ? an : q;
        U2[o] = x ? en : 0.0;
        MU[o] = mu;
        sw |= x ? 1u << b : 0u;
        p = x ? q - mu * an : an - mu * q;
        q = x ? -mu * en : en;
      }
      SW[(int64_t)(i0 / IV_B) * kept + m] = (unsigned char)sw;
    }
  }
  for (int it = 0; it < 3; ++it) {
    for (int m = tid; m < kept; m += IV_NT) {
      // right-hand side: the start vector, or L^{-1} P z; the solution's scale is applied
      // where it is read next (a solve's scale is dropped before the next one's matters)
      if (it == 0) {
        for (int i = 0; i < k; ++i) Z[(int64_t)i * kept + m] = start_entry(i, m);
      } else {
        double zc = Z[m];
        double zn[IV_B], mu[IV_B];
        unsigned sw = 0;
        auto load = [&](int i0) {
#pragma unroll
          for (int b = 0; b < IV_B; ++b) {
            const int i = i0 + b;
            zn[b] = i + 1 < k ? Z[(int64_t)(i + 1) * kept + m] : 0.0;
            mu[b] = i < k ? MU[(int64_t)i * kept + m] : 0.0;
          }
          sw = i0 < k ? SW[(int64_t)(i0 / IV_B) * kept + m] : 0;
        };
        load(0);
        for (int i0 = 0; i0 < k - 1; i0 += IV_B) {
          double cz[IV_B], cm[IV_B];
          const unsigned cs = sw;
#pragma unroll
          for (int b = 0; b < IV_B; ++b) { cz[b] = zn[b]; cm[b] = mu[b]; }
          load(i0 + IV_B);
#pragma unroll
          for (int b = 0; b < IV_B; ++b) {
            if (i0 + b >= k - 1) break;
            const bool x = (cs >> b) & 1u;
            const double bi = x ? cz[b] : zc, bn = x ? zc : cz[b];
            Z[(int64_t)(i0 + b) * kept + m] = bi;
            zc = fma(-cm[b], bi, bn);
          }
        }
        Z[(int64_t)(k - 1) * kept + m] = zc;
      }
      // back substitution U z = b, batches from the last row up
      double z1 = 0.0, z2 = 0.0, nrm = 0.0;
      double zb[IV_B], rp[IV_B], u1[IV_B], u2[IV_B];
      auto load = [&](int i1) {   // rows i1, i1 - 1, ...
#pragma unroll
        for (int b = 0; b < IV_B; ++b) {
          const int i = i1 - b;
          const int64_t o = (int64_t)i * kept + m;
          zb[b] = i >= 0 ? Z[o] : 0.0;
          rp[b] = i >= 0 ? RP[o] : 0.0;
          u1[b] = i >= 0 ? U1[o] : 0.0;
          u2[b] = i >= 0 ? U2[o] : 0.0;
        }
      };
      load(k - 1);
      for (int i1 = k - 1; i1 >= 0; i1 -= IV_B) {
        double cb[IV_B], cr[IV_B], c1[IV_B], c2[IV_B];
#pragma unroll
        for (int b = 0; b < IV_B; ++b) { cb[b] = zb[b]; cr[b] = rp[b]; c1[b] = u1[b]; c2[b] = u2[b]; }
        load(i1 - IV_B);
#pragma unroll
        for (int b = 0; b < IV_B; ++b) {
          if (i1 - b < 0) break;
          const double z = fma(-c1[b], z1, fma(-c2[b], z2, cb[b])) * cr[b];
          Z[(int64_t)(i1 - b) * kept + m] = z;
          z2 = z1;
          z1 = z;
          nrm = fma(z, z, nrm);
        }
      }
      const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
      for (int i0 = 0; i0 < k; i0 += IV_B) {
        double zs[IV_B];
#pragma unroll
        for (int b = 0; b < IV_B; ++b) zs[b] = i0 + b < k ? Z[(int64_t)(i0 + b) * kept + m] : 0.0;
#pragma unroll
        for (int b = 0; b < IV_B; ++b)
          if (i0 + b < k) Z[(int64_t)(i0 + b) * kept + m] = zs[b] * inv;
      }
    }
    if (!grouped || it == 0) continue;   // uniform over the CTA
    __syncthreads();
    int first = 0;
    for (int m = 1; m < kept; ++m) {
      if (lv[m - 1] - lv[m] > gaptol) { first = m; continue; }
      // z_m against the group's earlier vectors first .. m - 1, twice
      for (int pass = 0; pass < 2; ++pass) {
        for (int g0 = first; g0 < m; g0 += IV_GT) {
          const int g = g0 + lane, ng = min(IV_GT, m - g0);
          double dot = 0.0;
          if (g < m)
            for (int i = warp; i < k; i += IV_NT / 32)
              dot = fma(Z[(int64_t)i * kept + g], Z[(int64_t)i * kept + m], dot);
          dots[warp][lane] = dot;
          __syncthreads();
          if (tid < IV_GT) {
            double s = 0.0;
            for (int w = 0; w < IV_NT / 32; ++w) s += dots[w][tid];
            coef[tid] = s;
          }
          __syncthreads();
          // a thread per entry of z_m
          for (int i = tid; i < k; i += IV_NT) {
            double z = Z[(int64_t)i * kept + m];
            for (int c = 0; c < ng; ++c) z = fma(-coef[c], Z[(int64_t)i * kept + g0 + c], z);
            Z[(int64_t)i * kept + m] = z;
          }
          __syncthreads();
        }
      }
      double s = 0.0;
      for (int i = tid; i < k; i += IV_NT) {
        const double z = Z[(int64_t)i * kept + m];
        s = fma(z, z, s);
      }
      s = warp_sum(s);
      if (lane == 0) nrm2[warp] = s;
      __syncthreads();
      s = 0.0;
      for (int w = 0; w < IV_NT / 32; ++w) s += nrm2[w];
      const double inv = s > 0.0 ? 1.0 / sqrt(s) : 0.0;
      for (int i = tid; i < k; i += IV_NT) Z[(int64_t)i * kept + m] *= inv;
      __syncthreads();
    }
  }
}

// 3b. y = Q z = H_0 (H_1 (... H_{k-2} z)), one warp per kept vector, lane holding the entries
//     l = lane (mod 32) in registers; the reflectors' vectors come through shared memory, BT_R
//     rows at a time and one block ahead (cp.async, zeros outside the reflector, so the
//     products need no tests).  Writes V = y ([k][kept], X = T^H) or Y for the GEMM.
//     What bounds it: a reflector's chain (loads, dot product, warp sum, update) and its
//     instructions; the chunks of 32 entries are unrolled for the number still reached (in
//     steps of two), so they carry no tests.  Measured, all sectors of a chi = 1024 update
//     alone: 193 us, 527 with the vectors read from L2 by every warp, a test per chunk
//     and sums by shuffles.
constexpr int BT_NT = 128, BT_NW = BT_NT / 32;
constexpr int BT_R = 4;        // reflectors of a block

// Reflectors r = BT_R - 1 .. 0 of a block on a lane's entries y[i], chunk nc - 1 - i, of
// which the first N can be reached; v: this lane's entry of the first reflector's last chunk.
template <int N, int NPL>
__device__ __forceinline__ void bt_block(cplx (&y)[NPL], const double2* v0, int ks, const cplx* taus) {
  constexpr bool HOLD = N <= 16;       // v in registers between the two products
#pragma unroll 1
  for (int r = BT_R - 1; r >= 0; --r) {
    const double2* v = v0 + r * ks;
    const cplx tj = ldc(taus + r);
    double2 x[HOLD ? N : 1];
    cplx dot[2] = {cmake(0.0, 0.0), cmake(0.0, 0.0)};
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const double2 e = v[-32 * i];
      if (HOLD) x[HOLD ? i : 0] = e;
      ccfma(dot[i & 1], cmake(e.x, e.y), y[i]);
    }
    const cplx f = cmul(tj, cmake(warp_sum(dot[0].x + dot[1].x), warp_sum(dot[0].y + dot[1].y)));
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const double2 e = HOLD ? x[HOLD ? i : 0] : v[-32 * i];
      y[i].x = fma(-f.x, e.x, fma(f.y, e.y, y[i].x));
      y[i].y = fma(-f.x, e.y, fma(-f.y, e.x, y[i].y));
    }
  }
}

template <int N, int NPL>
__device__ __forceinline__ void bt_blocks(int n, cplx (&y)[NPL], const double2* v0, int ks, const cplx* taus) {
  if constexpr (N > 2) {
    if (n <= N - 2) return bt_blocks<N - 2, NPL>(n, y, v0, ks, taus);
  }
  bt_block<N, NPL>(y, v0, ks, taus);
}

template <int NPL>
__global__ __launch_bounds__(BT_NT) void backtransform_kernel(const SectorDesc* __restrict__ sd,
                                                              const cplx* __restrict__ gbuf,
                                                              const cplx* __restrict__ taubuf,
                                                              const double* __restrict__ zbuf,
                                                              cplx* __restrict__ vbuf, cplx* __restrict__ ybuf) {
  extern __shared__ __align__(16) double2 vs[];   // [2][BT_R][ks], then tau [ks]
  const SectorDesc& S = sd[blockIdx.y];
  const int k = S.k, kept = S.kept;
  if ((int)blockIdx.x * BT_NW >= kept) return;    // uniform over the CTA
  const int tid = threadIdx.x, lane = tid & 31, t = blockIdx.x * BT_NW + (tid >> 5);
  const bool live = t < kept;
  const int nc = ((k + 63) >> 6) << 1, ks = nc << 5;   // chunks, an even number
  const cplx* A = gbuf + S.g_off;
  const cplx* tau = taubuf + S.s_off;
  const double* Z = zbuf + S.y_off;
  cplx y[NPL];
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int l = lane + 32 * (nc - 1 - i);
    y[i] = cmake(live && l >= 0 && l < k ? Z[(int64_t)l * kept + t] : 0.0, 0.0);
  }
  cplx* taus = reinterpret_cast<cplx*>(vs + 2 * BT_R * ks);
  for (int j = tid; j < ks; j += BT_NT) stc(taus + j, j < k - 1 ? ldc(tau + j) : cmake(0.0, 0.0));
  const int nb = (k - 1 + BT_R - 1) / BT_R;
  // block b: v_j of j = b BT_R .. (at columns j+1 .. k-1 of row j, v[j+1] = 1), from the first
  // pair of chunks that it reaches
  auto fill = [&](int b) {
    const int l0 = (b * BT_R + 1) & ~63;
    for (int r = 0; r < BT_R; ++r) {
      const int j = b * BT_R + r;
      double2* dst = vs + ((b & 1) * BT_R + r) * ks;
      const cplx* src = A + (int64_t)j * k;
      for (int l = l0 + tid; l < ks; l += BT_NT) {
        const bool ok = l > j && l < k && j < k - 1;
        cp_async16(dst + l, ok ? src + l : A, ok);
      }
    }
  };
  if (nb > 0) fill(nb - 1);
  cp_async_commit();
  for (int b = nb - 1; b >= 0; --b) {
    if (b > 0) fill(b - 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    bt_blocks<NPL, NPL>(nc - 2 * ((b * BT_R + 1) >> 6), y, vs + (b & 1) * BT_R * ks + 32 * (nc - 1) + lane, ks,
                        taus + b * BT_R);
    __syncthreads();
  }
  if (!live) return;
  cplx* out = S.left ? vbuf + S.v_off : ybuf + S.y_off;
#pragma unroll
  for (int i = 0; i < NPL; ++i) {
    const int l = lane + 32 * (nc - 1 - i);
    if (l >= 0 && l < k) stc(out + (int64_t)l * kept + t, y[i]);
  }
}

// 3c. The same for every eigenvector of the preconditioned sectors (section 4), the
//     reflectors in blocks of WY_B: H_j0 .. H_{j0+15} = I - V T V^H (V the block's vectors as
//     columns, T upper triangular).  wy_t_kernel forms T of every block; wy_apply_kernel
//     applies the blocks, last first, to WY_C vectors held in shared memory: W = V^H Z with
//     the rows split over the warps, W2 = T W, Z -= V W2, the two products on the FP64 tensor
//     path with the fragments of V read straight from the Householder vectors.
//     Why not for 3b: its vectors leave the Gram route's marginals three times further off (T
//     adds its own rounding); here the Newton-Schulz steps take that out again.  Measured,
//     one layer at N = 64, chi = 1024, every eigenvector: 3.0 ms against 11.5 with 3b's
//     kernel.
constexpr int WY_B = 16;      // reflectors of a block
constexpr int WY_C = 8;       // vectors of a CTA
constexpr int WY_NT = 256, WY_NW = WY_NT / 32;
static_assert(WY_NT == WY_B * WY_B, "a thread to an entry of T");
constexpr int WY_LDZ = WY_C + 2;   // 2 mod 8: a fragment's four rows on distinct banks

// T of block b of sector s
__device__ __forceinline__ int64_t wy_t_off(const SectorDesc& S, int s, int b) {
  return WY_B * S.s_off + (int64_t)WY_B * WY_B * (s + b);
}

// v_j[l], zero outside the reflector
__device__ __forceinline__ cplx wy_v(const cplx* A, int k, int j, int l) {
  return j < k - 1 && l > j && l < k ? ldc(A + (int64_t)j * k + l) : cmake(0.0, 0.0);
}

constexpr int WT_NT = 128;
__global__ __launch_bounds__(WT_NT) void wy_t_kernel(const SectorDesc* __restrict__ sd, const int* __restrict__ list,
                                                     const cplx* __restrict__ gbuf,
                                                     const cplx* __restrict__ taubuf, cplx* __restrict__ tbuf) {
  __shared__ double2 G[WT_NT / 32][WY_B][WY_B + 1];
  __shared__ cplx T[WY_B][WY_B + 1];
  const int sec = list[blockIdx.y];
  const SectorDesc& S = sd[sec];
  const int k = S.k, j0 = blockIdx.x * WY_B;
  if (j0 >= k - 1 || S.kept < 0) return;
  const cplx* A = gbuf + S.g_off;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, li = lane >> 2, lk = lane & 3;
  // G = V^H V, rows j0 + 1 .. k - 1 in quarters
  double2 re[2][2], im[2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) re[i][j] = im[i][j] = make_double2(0.0, 0.0);
  for (int l = j0 + 1 + 4 * warp; l < k; l += 4 * (WT_NT / 32)) {
    auto frag = [&](int i, int) {
      const cplx v = wy_v(A, k, j0 + 8 * i + li, l + lk);
      return make_double2(v.x, v.y);
    };
    cmma_tile<2, 2, 1, true>(re, im, frag, frag);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      G[warp][8 * i + li][8 * j + 2 * lk] = make_double2(re[i][j].x, im[i][j].x);
      G[warp][8 * i + li][8 * j + 2 * lk + 1] = make_double2(re[i][j].y, im[i][j].y);
    }
  __syncthreads();
  if (warp == 0) {
    // column i of T: tau_i on the diagonal, -tau_i T(:, < i) (V^H v_i) above
    const cplx* tau = taubuf + S.s_off;
    for (int i = 0; i < WY_B; ++i) {
      const cplx ti = j0 + i < k - 1 ? tau[j0 + i] : cmake(0.0, 0.0);
      if (lane < WY_B) {
        cplx acc = cmake(0.0, 0.0);
        for (int c = lane; c < i; ++c) {
          cplx g = cmake(0.0, 0.0);
          for (int w = 0; w < WT_NT / 32; ++w) g = cadd(g, cmake(G[w][c][i].x, G[w][c][i].y));
          cfma(acc, T[lane][c], g);
        }
        acc = cmul(ti, acc);
        T[lane][i] = lane < i ? cmake(-acc.x, -acc.y) : lane == i ? ti : cmake(0.0, 0.0);
      }
      __syncwarp();
    }
  }
  __syncthreads();
  cplx* out = tbuf + wy_t_off(S, sec, blockIdx.x);
  for (int e = tid; e < WY_B * WY_B; e += WT_NT) stc(out + e, T[e / WY_B][e % WY_B]);
}

__global__ __launch_bounds__(WY_NT) void wy_apply_kernel(const SectorDesc* __restrict__ sd,
                                                         const int* __restrict__ list,
                                                         const cplx* __restrict__ gbuf,
                                                         const cplx* __restrict__ tbuf,
                                                         const double* __restrict__ zbuf,
                                                         cplx* __restrict__ ybuf) {
  extern __shared__ __align__(16) double2 Z[];   // [k][WY_LDZ]
  __shared__ double2 Wp[WY_NW][WY_B][WY_C + 1], W[WY_B][WY_LDZ];
  const int sec = list[blockIdx.y];
  const SectorDesc& S = sd[sec];
  const int k = S.k, c0 = blockIdx.x * WY_C;
  if (c0 >= k || S.kept < 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, li = lane >> 2, lk = lane & 3;
  const cplx* A = gbuf + S.g_off;
  const double* z = zbuf + S.y_off;
  for (int e = tid; e < k * WY_C; e += WY_NT) {
    const int l = e / WY_C, c = e % WY_C;
    Z[l * WY_LDZ + c] = make_double2(c0 + c < k ? z[(int64_t)l * k + c0 + c] : 0.0, 0.0);
  }
  const int nb = (k - 1 + WY_B - 1) / WY_B;
  for (int b = nb - 1; b >= 0; --b) {
    const int j0 = b * WY_B;
    const cplx* T = tbuf + wy_t_off(S, sec, b);
    const cplx te = ldc(T + tid);   // this thread's entry of T
    __syncthreads();
    // W = V^H Z, four rows a step, the steps over the warps
    {
      double2 re[2][1], im[2][1];
#pragma unroll
      for (int i = 0; i < 2; ++i) re[i][0] = im[i][0] = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int l = j0 + 1 + 4 * warp; l < k; l += 4 * WY_NW)
        cmma_tile<2, 1, 1, true>(
            re, im,
            [&](int i, int) {
              const cplx v = wy_v(A, k, j0 + 8 * i + li, l + lk);
              return make_double2(v.x, v.y);
            },
            [&](int, int) { return l + lk < k ? Z[(l + lk) * WY_LDZ + li] : make_double2(0.0, 0.0); });
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        Wp[warp][8 * i + li][2 * lk] = make_double2(re[i][0].x, im[i][0].x);
        Wp[warp][8 * i + li][2 * lk + 1] = make_double2(re[i][0].y, im[i][0].y);
      }
    }
    __syncthreads();
    // the warps' parts summed, then W2 = T W
    if (tid < WY_B * WY_C) {
      const int j = tid / WY_C, c = tid % WY_C;
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int w = 0; w < WY_NW; ++w) { s.x += Wp[w][j][c].x; s.y += Wp[w][j][c].y; }
      W[j][c] = s;
    }
    // T into the parts' place once they are read
    __syncthreads();
    cplx* Ts = reinterpret_cast<cplx*>(&Wp[0][0][0]);
    stc(Ts + tid, te);
    __syncthreads();
    cplx w2 = cmake(0.0, 0.0);
    if (tid < WY_B * WY_C) {
      const int j = tid / WY_C, c = tid % WY_C;
      for (int q = j; q < WY_B; ++q) cfma(w2, ldc(Ts + j * WY_B + q), cmake(W[q][c].x, W[q][c].y));
    }
    __syncthreads();
    if (tid < WY_B * WY_C) W[tid / WY_C][tid % WY_C] = make_double2(w2.x, w2.y);
    __syncthreads();
    // Z -= V W2, eight rows a tile
    for (int l0 = j0 + 1 + 8 * warp; l0 < k; l0 += 8 * WY_NW) {
      double2 re[1][1], im[1][1];
      re[0][0] = im[0][0] = make_double2(0.0, 0.0);
      cmma_tile<1, 1, WY_B / 4, false>(
          re, im,
          [&](int, int q) {
            const cplx v = wy_v(A, k, j0 + q + lk, l0 + li);
            return make_double2(v.x, v.y);
          },
          [&](int, int q) { return W[q + lk][li]; });
      if (l0 + li < k) {
        double2* p = Z + (l0 + li) * WY_LDZ + 2 * lk;
        p[0].x -= re[0][0].x;
        p[0].y -= im[0][0].x;
        p[1].x -= re[0][0].y;
        p[1].y -= im[0][0].y;
      }
    }
  }
  __syncthreads();
  cplx* out = ybuf + S.y_off;
  for (int e = tid; e < k * WY_C; e += WY_NT) {
    const int l = e / WY_C, c = e % WY_C;
    if (c0 + c < k) {
      const double2 v = Z[l * WY_LDZ + c];
      stc(out + (int64_t)l * k + c0 + c, cmake(v.x, v.y));
    }
  }
}

// ---------------------------------------------------------------------------------
// 4. The preconditioner of the blocked Jacobi SVD (plain path): a unitary Y close to the
//    eigenvectors of X^H X, so that the columns of X Y are nearly orthogonal and sorted, and
//    two or three sweeps replace 8 to 18.  Y comes from every eigenvector of the
//    tridiagonal (invit_kernel with `all`), orthogonalised within groups of close
//    eigenvalues here and, after the back-transformation, as a whole by three Newton-Schulz
//    steps Y <- Y (3 I - Y^H Y) / 2, which square the departure from unitarity and leave it
//    at rounding level.  The SVD itself stays the one-sided Jacobi iteration on X Y with its
//    own test, so Y decides how fast it converges, not what it converges to.  Measured: one
//    layer at N = 64, chi = 1024 on the plain path 223 ms without and 56 with it, an N = 24,
//    chi = 256 circuit 118 and 57 (30 with the later one-CTA form of its small sectors); the
//    marginals of N = 13 to 20 circuits are 9.9e-15 from a 64-bit CPU computation at most,
//    1.5e-13 without.  A sector whose Y was not unitary to NS_TOL before the last step
//    (flagged in sd[].kept, which the selection sets later) starts from X itself; an update
//    that keeps values far below a sector's largest is done again without Y (PRE_MIN).
constexpr int OR_NT = 512, OR_NW = OR_NT / 32;
constexpr int OR_P = 8;        // vectors of a panel
constexpr double NS_TOL = 1e-11;   // (k NS_TOL)^2 is below eps; about 1e-15 in use

// Panels of OR_P vectors of a group, in order: each against the group's earlier vectors (32 at
// a time, two products on the FP64 tensor path) and within itself (Gram-Schmidt), the whole
// twice.  What bounds it: the reads of the group's vectors by one CTA, twice a chunk; the
// sectors below chi's cut share one group of up to a few hundred values.  With scalar
// products, a thread to a row in the second one (uncoalesced), the largest launch of a layer
// at N = 64, chi = 1024 took 6.5 ms, now 2.6; one such update 10.9 and 10.1.
__global__ __launch_bounds__(OR_NT) void orthogonalise_kernel(const SectorDesc* __restrict__ sd,
                                                              const int* __restrict__ list,
                                                              const double* __restrict__ lam,
                                                              double* __restrict__ zbuf) {
  extern __shared__ __align__(16) double zp[];   // the panel, [k][OR_P]
  __shared__ double dots[OR_NW][32][OR_P], coef[32][OR_P], part[OR_NW][OR_P], tots[OR_P];
  const SectorDesc& S = sd[list[blockIdx.x]];
  if (S.kept < 0) return;
  const int k = S.k, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, li = lane >> 2, lk = lane & 3;
  const double* lv = lam + S.s_off;
  double* Z = zbuf + S.y_off;      // [k][k]
  const double gaptol = IV_GAP_ALL * fmax(fabs(lv[0]), fabs(lv[k - 1]));
  int first = 0;
  while (first < k) {
    int end = first + 1;
    while (end < k && lv[end - 1] - lv[end] <= gaptol) ++end;
    for (int m0 = first; end > first + 1 && m0 < end; m0 += OR_P) {
      const int np = min(OR_P, end - m0);
      for (int e = tid; e < k * OR_P; e += OR_NT) {
        const int i = e / OR_P, p = e % OR_P;
        zp[e] = p < np ? Z[(int64_t)i * k + m0 + p] : 0.0;
      }
      __syncthreads();
      for (int pass = 0; pass < 2; ++pass) {
        for (int g0 = first; g0 < m0; g0 += 32) {
          // Z^T zp by the warps' rows, four at a time
          double2 acc[4];
#pragma unroll
          for (int m = 0; m < 4; ++m) acc[m] = make_double2(0.0, 0.0);
#pragma unroll 4
          for (int r0 = 4 * warp; r0 < k; r0 += 4 * OR_NW) {
            const int i = r0 + lk;
            const double b = i < k ? zp[i * OR_P + li] : 0.0;
            double a[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              const int g = g0 + 8 * m + li;
              a[m] = i < k && g < m0 ? Z[(int64_t)i * k + g] : 0.0;
            }
            __syncwarp();
#pragma unroll
            for (int m = 0; m < 4; ++m) dmma8x8x4(acc[m], a[m], b);
          }
#pragma unroll
          for (int m = 0; m < 4; ++m) *reinterpret_cast<double2*>(&dots[warp][8 * m + li][2 * lk]) = acc[m];
          __syncthreads();
          if (tid < 32 * OR_P) {
            const int c = tid / OR_P, p = tid % OR_P;
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < OR_NW; ++w) s += dots[w][c][p];
            coef[c][p] = s;
          }
          __syncthreads();
          // zp - Z (Z^T zp), eight rows at a time
          double cf[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) cf[q] = coef[4 * q + lk][li];
#pragma unroll 2
          for (int r0 = 8 * warp; r0 < k; r0 += 8 * OR_NW) {
            const int i = r0 + li;
            double a[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const int g = g0 + 4 * q + lk;
              a[q] = i < k && g < m0 ? -Z[(int64_t)i * k + g] : 0.0;
            }
            double2 v = i < k ? *reinterpret_cast<const double2*>(&zp[i * OR_P + 2 * lk]) : make_double2(0.0, 0.0);
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 8; ++q) dmma8x8x4(v, a[q], cf[q]);
            if (i < k) *reinterpret_cast<double2*>(&zp[i * OR_P + 2 * lk]) = v;
          }
          __syncthreads();
        }
        // within the panel: vector p normalised, then taken out of the later ones
        for (int p = 0; p < np; ++p) {
          double acc[OR_P];
#pragma unroll
          for (int q = 0; q < OR_P; ++q) acc[q] = 0.0;
          for (int i = tid; i < k; i += OR_NT) {
            const double z = zp[i * OR_P + p];
#pragma unroll
            for (int q = 0; q < OR_P; ++q) acc[q] = fma(z, zp[i * OR_P + q], acc[q]);
          }
#pragma unroll
          for (int q = 0; q < OR_P; ++q) {
            const double s = warp_sum(acc[q]);
            if (lane == 0) part[warp][q] = s;
          }
          __syncthreads();
          if (tid < OR_P) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < OR_NW; ++w) s += part[w][tid];
            tots[tid] = s;
          }
          __syncthreads();
          double tot[OR_P];
#pragma unroll
          for (int q = 0; q < OR_P; ++q) tot[q] = tots[q];
          double n2 = 0.0;
#pragma unroll
          for (int q = 0; q < OR_P; ++q) n2 = q == p ? tot[q] : n2;
          const double inv = n2 > 0.0 ? 1.0 / n2 : 0.0, rinv = sqrt(inv);
          for (int i = tid; i < k; i += OR_NT) {
            const double z = zp[i * OR_P + p];
#pragma unroll
            for (int q = 0; q < OR_P; ++q)
              if (q > p) zp[i * OR_P + q] = fma(-tot[q] * inv, z, zp[i * OR_P + q]);
            zp[i * OR_P + p] = z * rinv;
          }
          __syncthreads();
        }
      }
      for (int e = tid; e < k * OR_P; e += OR_NT) {
        const int i = e / OR_P, p = e % OR_P;
        if (p < np) Z[(int64_t)i * k + m0 + p] = zp[e];
      }
      __syncthreads();
    }
    first = end;
  }
}

// S = Y^H Y -> 3/2 I - S / 2 in place; with check, flags a sector where S is not within NS_TOL
// of I
__global__ __launch_bounds__(256) void newton_schulz_kernel(SectorDesc* __restrict__ sd, const int* __restrict__ list,
                                                            cplx* __restrict__ gbuf, bool check) {
  SectorDesc& S = sd[list[blockIdx.y]];
  if (!check && S.kept < 0) return;
  const int k = S.k;
  cplx* G = gbuf + S.g_off;
  bool bad = false;
  for (int e = blockIdx.x * 256 + threadIdx.x; e < k * k; e += gridDim.x * 256) {
    const double diag = e / k == e % k ? 1.0 : 0.0;
    const cplx s = ldc(G + e);
    bad |= !(fabs(s.x - diag) <= NS_TOL && fabs(s.y) <= NS_TOL);
    stc(G + e, cmake(1.5 * diag - 0.5 * s.x, -0.5 * s.y));
  }
  if (check && bad) S.kept = -1;   // every writer writes the same
}

// Y below X^H Y in the matrices [T^H; I] Y of the `left` sectors; a flagged sector's matrix
// is [X; I] or X itself
__global__ __launch_bounds__(256) void precondition_finish_kernel(const SectorDesc* __restrict__ sd,
                                                                  const int* __restrict__ list,
                                                                  const cplx* __restrict__ y, cplx* __restrict__ abuf) {
  const SectorDesc& S = sd[list[blockIdx.y]];
  const bool bad = S.kept < 0;
  const int k = S.k, top = S.rows_g * k, total = S.rows_tot * k;
  for (int e = (bad ? 0 : top) + blockIdx.x * 256 + threadIdx.x; e < total; e += gridDim.x * 256) {
    const int r = e - top;
    const cplx v = r < 0 ? ldc(abuf + S.t_off + e)
                   : bad ? cmake(r / k == r % k ? 1.0 : 0.0, 0.0)
                         : ldc(y + S.y_off + r);
    stc(abuf + S.a_off + e, v);
  }
}

}  // namespace

int eigen_max_k() {
  // every k up to the bound fits the tridiagonalisation's shared memory with one CTA per
  // sector (the row ring shrinks in steps as k grows, so the size is not monotone in k)
  static const int kmax = [] {
    int best = 0;
    for (int k = 1; k <= 32 * 32; ++k) {   // the back-transformation keeps 32 entries per lane
      if (td_smem_bytes(k, TD_CL, TD_NW) > 227 * 1024) break;
      best = k;
    }
    return best;
  }();
  return kmax;
}

// Size class of a sector: the resident kernel's classes, then the streamed kernel's.
int tridiag_class(int k) {
  for (int c = 0; c < TD_RES_CLASSES; ++c)
    if (k <= TD_RES_K[c]) return c;
  return TD_RES_CLASSES;
}

namespace {

template <typename F, typename... Args>
cudaError_t launch_cluster(F* kernel, int grid, int cl, int nt, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cl;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace

cudaError_t launch_tridiag(const SectorDesc* sd_dev, const int* list_dev, const int* class_count,
                           const int* class_kmax, void* gbuf, double* dbuf, double* ebuf,
                           void* taubuf, int* err, const cudaStream_t* streams) {
  static_assert(TD_CLASSES == TD_RES_CLASSES + 1, "one class more than the resident kernel's");
  // once per process: the largest dynamic shared memory any launch may ask for, and
  // clusters of 16 CTAs
  static const cudaError_t attr = [] {
    size_t most = 0;
    for (int k = 1; k <= eigen_max_k(); ++k) most = std::max(most, td_smem_bytes(k, TD_CL, TD_NW));
    const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(tridiag_kernel, dyn, (int)most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(tridiag_resident_kernel<128>, dyn, 227 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(tridiag_resident_kernel<256>, dyn, 227 * 1024);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(tridiag_resident_kernel<256>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(tridiag_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
  }();
  if (attr != cudaSuccess) return attr;
  cplx* G = reinterpret_cast<cplx*>(gbuf);
  cplx* tau = reinterpret_cast<cplx*>(taubuf);
  int first = 0;
  for (int c = 0; c < TD_CLASSES; ++c) {
    const int count = class_count[c];
    if (count == 0) continue;
    const int* list = list_dev + first;
    cudaStream_t s = streams[c];
    cudaError_t e;
    if (c == TD_RES_CLASSES) {
      e = launch_cluster(tridiag_kernel, count * TD_CL, TD_CL, TD_NT, td_smem_bytes(class_kmax[c], TD_CL, TD_NW), s,
                         sd_dev, list, class_kmax[c], G, dbuf, ebuf, tau, err);
      if (e != cudaSuccess) return e;
    }
    {
      const int rc = std::min(c, TD_RES_CLASSES - 1);
      const int cl = TD_RES_CL[rc], nt = TD_RES_NT[rc];
      const auto kernel = nt == 128 ? tridiag_resident_kernel<128> : tridiag_resident_kernel<256>;
      e = launch_cluster(kernel, count * cl, cl, nt + 32, td_res_smem(std::min(class_kmax[c], TD_RES_MAX), cl, nt), s,
                         sd_dev, list, G, dbuf, ebuf, tau);
    }
    if (e != cudaSuccess) return e;
    first += count;
  }
  return cudaSuccess;
}

namespace {

cudaError_t run_bisect(const SectorDesc* sd, const int* list, int n, int kmax, const double* dbuf, const double* ebuf,
                       double* lam, cudaStream_t s) {
  static const cudaError_t attr = cudaFuncSetAttribute(
      bisect_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, eigen_max_k() * (int)sizeof(double2));
  if (attr != cudaSuccess) return attr;
  bisect_kernel<<<dim3(ceil_div(kmax, BI_NT / 32), n), BI_NT, (size_t)kmax * sizeof(double2), s>>>(sd, list, dbuf, ebuf,
                                                                                               lam);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_bisect(const SectorDesc* sd_dev, int n_sectors, int kmax, const double* dbuf,
                          const double* ebuf, double* lam, double* sig, double* invsig,
                          cudaStream_t s) {
  if (n_sectors <= 0 || kmax <= 0) return cudaSuccess;
  const cudaError_t e = run_bisect(sd_dev, nullptr, n_sectors, kmax, dbuf, ebuf, lam, s);
  if (e != cudaSuccess) return e;
  eig_finish_kernel<<<n_sectors, FI_NT, 0, s>>>(sd_dev, lam, sig, invsig);
  return cudaGetLastError();
}

namespace {

cudaError_t run_invit(SectorDesc* sd, const int* list, int n, int kmax, const UpdateTables* tabs, int n_updates,
                      double cutoff, int chi, const double* dbuf, const double* ebuf, const double* lam, double* scratch, unsigned char* swp, double* zbuf,
                      cudaStream_t s) {
  static const cudaError_t attr = cudaFuncSetAttribute(
      invit_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * eigen_max_k() * (int)sizeof(double));
  if (attr != cudaSuccess) return attr;
  invit_kernel<<<n, IV_NT, (size_t)2 * kmax * sizeof(double), s>>>(sd, list, tabs, n_updates, cutoff, chi, dbuf, ebuf, lam,
                                                               scratch, swp, zbuf);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_eigvec(SectorDesc* sd_dev, int n_sectors, int kmax, const double* dbuf, const double* ebuf,
                          const double* lam, double* scratch, unsigned char* swp, double* zbuf, const void* gbuf,
                          const void* taubuf, void* vbuf, void* ybuf, cudaStream_t s) {
  if (n_sectors <= 0 || kmax <= 0) return cudaSuccess;
  static const cudaError_t attr = [] {
    const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const int most = (2 * BT_R + 1) * (eigen_max_k() + 63) * (int)sizeof(double2);
    cudaError_t e = cudaFuncSetAttribute(backtransform_kernel<4>, dyn, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(backtransform_kernel<8>, dyn, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(backtransform_kernel<16>, dyn, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(backtransform_kernel<32>, dyn, most);
    return e;
  }();
  if (attr != cudaSuccess) return attr;
  const cudaError_t e = run_invit(sd_dev, nullptr, n_sectors, kmax, nullptr, 0, 0.0, 0, dbuf, ebuf, lam, scratch, swp,
                                  zbuf, s);
  if (e != cudaSuccess) return e;
  const cplx* G = reinterpret_cast<const cplx*>(gbuf);
  const cplx* tau = reinterpret_cast<const cplx*>(taubuf);
  cplx* V = reinterpret_cast<cplx*>(vbuf);
  cplx* Y = reinterpret_cast<cplx*>(ybuf);
  const dim3 grid(ceil_div(kmax, BT_NW), n_sectors);
  const int npl = 2 * ceil_div(kmax, 64);
  const size_t smem = (size_t)(2 * BT_R + 1) * 32 * npl * sizeof(double2);
  if (npl <= 4) backtransform_kernel<4><<<grid, BT_NT, smem, s>>>(sd_dev, G, tau, zbuf, V, Y);
  else if (npl <= 8) backtransform_kernel<8><<<grid, BT_NT, smem, s>>>(sd_dev, G, tau, zbuf, V, Y);
  else if (npl <= 16) backtransform_kernel<16><<<grid, BT_NT, smem, s>>>(sd_dev, G, tau, zbuf, V, Y);
  else if (npl <= 32) backtransform_kernel<32><<<grid, BT_NT, smem, s>>>(sd_dev, G, tau, zbuf, V, Y);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

size_t precondition_t_elems(int64_t s_elems, int n_sectors) {
  return (size_t)(WY_B * s_elems + (int64_t)WY_B * WY_B * n_sectors);
}

cudaError_t launch_precondition_basis(const UpdateTables* tab_dev, SectorDesc* sd_dev, int n_updates,
                                      const int* list_dev, int count, int kmax, double cutoff, int chi,
                                      const double* dbuf, const double* ebuf, double* lam, double* scratch,
                                      unsigned char* swp, double* zbuf, const void* gbuf, const void* taubuf, void* tbuf,
                                      void* ybuf, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  static const cudaError_t attr = [] {
    const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(wy_apply_kernel, dyn, eigen_max_k() * WY_LDZ * (int)sizeof(double2));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(orthogonalise_kernel, dyn, OR_P * eigen_max_k() * (int)sizeof(double));
    return e;
  }();
  if (attr != cudaSuccess) return attr;
  cudaError_t e = run_bisect(sd_dev, list_dev, count, kmax, dbuf, ebuf, lam, s);
  if (e != cudaSuccess) return e;
  e = run_invit(sd_dev, list_dev, count, kmax, tab_dev, n_updates, cutoff, chi, dbuf, ebuf, lam, scratch, swp, zbuf, s);
  if (e != cudaSuccess) return e;
  orthogonalise_kernel<<<count, OR_NT, (size_t)OR_P * kmax * sizeof(double), s>>>(sd_dev, list_dev, lam, zbuf);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const cplx* G = reinterpret_cast<const cplx*>(gbuf);
  cplx* T = reinterpret_cast<cplx*>(tbuf);
  if (kmax > 1) {
    wy_t_kernel<<<dim3(ceil_div(kmax - 1, WY_B), count), WT_NT, 0, s>>>(sd_dev, list_dev, G,
                                                                        reinterpret_cast<const cplx*>(taubuf), T);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  wy_apply_kernel<<<dim3(ceil_div(kmax, WY_C), count), WY_NT, (size_t)kmax * WY_LDZ * sizeof(double2), s>>>(
      sd_dev, list_dev, G, T, zbuf, reinterpret_cast<cplx*>(ybuf));
  return cudaGetLastError();
}

cudaError_t launch_newton_schulz(SectorDesc* sd_dev, const int* list_dev, int count, int kmax, void* gbuf, bool check,
                                 cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  newton_schulz_kernel<<<dim3(std::min(ceil_div(kmax * kmax, 1024), 64), count), 256, 0, s>>>(
      sd_dev, list_dev, reinterpret_cast<cplx*>(gbuf), check);
  return cudaGetLastError();
}

cudaError_t launch_precondition_finish(const SectorDesc* sd_dev, const int* list_dev, int count, int max_elems,
                                       const void* ybuf, void* abuf, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  precondition_finish_kernel<<<dim3(std::min(ceil_div(std::max(max_elems, 1), 1024), 64), count), 256, 0, s>>>(
      sd_dev, list_dev, reinterpret_cast<const cplx*>(ybuf), reinterpret_cast<cplx*>(abuf));
  return cudaGetLastError();
}
