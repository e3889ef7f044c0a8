// Blocked one-sided (Hestenes) Jacobi SVD of every sector, in FP64.
//
// Replaces the reference's per-sector cuSOLVER gesvd (src/beam_splitter_parallel/
// Rank.py:123) / LAPACK svd (src/MPO.py:258).  The Jacobi matrix of a sector is
// T = C diag(Lambda_R) when |L| >= |R| (its orthogonalised columns are sigma * V),
// or [T^H; I] when |L| < |R| (the identity rows accumulate V).  Columns are cut in
// blocks of 16; a round pairs the blocks by the circle method (all sectors of the
// update in one launch pair), and each block pair's rows are cut in parts of at most
// 128 rows:
//   1. (gram kernel) every part holding Gram rows forms its partial 32 x 32 Gram; the
//      last part to finish sums the partials in part order, tests the pair and, if a
//      column pair is not orthogonal to `tol` (relative), runs one cyclic two-sided
//      Jacobi sweep on the Gram (complex rotations, 16 disjoint pairs per step),
//      accumulating the 32 x 32 unitary Q;
//   2. (apply kernel) every part of a rotated pair applies Q to its rows.
// A sector is converged after a sweep without rotations; later rounds of it exit
// at once.  One-sided Jacobi keeps high relative accuracy for small singular values.
// Numerical rank: a column whose norm is <= 16 eps sqrt(rows) ||T||_F is rounding
// noise (the null space of a rank-deficient block); it takes part in no rotation and
// its singular value is reported as 0, as is a column below tol times its partner
// in a pair test.  Without this, noise columns never test orthogonal.
#include "dmma.cuh"
#include "kernels.h"

namespace {

constexpr int JB = 16;        // columns per block
constexpr int JC = 2 * JB;    // columns per block pair
constexpr int JNT = 256;
constexpr int RMAX = 128;     // rows of one part (Gram tile in shared memory)

// Where a CTA of a round works: its sector, block pair and row part.
struct JacTask {
  JacobiWork W;
  int pair, part, sweep, rr, slot;
};

// Gram launch: CTAs [gram_start, gram_start + npairs cs_g) of a work entry, pair-major;
// apply launch: [apply_start, apply_start + npairs cs).
__device__ __forceinline__ JacTask jac_task(const JacobiWork* __restrict__ work, int n_work, int t,
                                            bool apply) {
  const int b = blockIdx.x;
  int lo = 0, hi = n_work - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const int st = apply ? work[mid].apply_start : work[mid].gram_start;
    if (st <= b) lo = mid; else hi = mid - 1;
  }
  JacTask T;
  T.W = work[lo];
  const int per = apply ? T.W.cs : T.W.cs_g;
  const int local = b - (apply ? T.W.apply_start : T.W.gram_start);
  T.pair = local / per;
  T.part = local % per;
  T.sweep = t / T.W.rounds;
  T.rr = t % T.W.rounds;
  T.slot = T.W.slot_start + T.pair;
  return T;
}

// circle method over n (even) positions: the item at position pos in step s; position 0
// is fixed, the others turn by one place per step, pairs are (P, n - 1 - P)
__device__ __forceinline__ int circle_at(int pos, int s, int n) {
  return pos == 0 ? 0 : 1 + (pos - 1 + s) % (n - 1);
}

// the pair's c-th column (c < 16: first block, else second; -1: padding)
__device__ __forceinline__ int jac_col(const JacTask& T, int c, int k) {
  const int nbp = T.W.nblk + (T.W.nblk & 1);
  const int b = c < JB ? circle_at(T.pair, T.rr, nbp) : circle_at(nbp - 1 - T.pair, T.rr, nbp);
  const int col = b * JB + (c % JB);
  return (b < T.W.nblk && col < k) ? col : -1;
}

struct GramSmem {
  union {
    double2 tile[RMAX][JC + 1];   // this part's Gram rows of the pair's 32 columns
    double2 G[JC][JC + 1];        // then the pair Gram (upper triangle, i <= j, is used)
  } u;
  double rc[JC / 2];              // rotations of the current inner step
  double2 rs[JC / 2];
  int cols[JC];
  int rotate, last;
  double z2;
};

// pair-Gram element (i, j) from the stored upper triangle
__device__ __forceinline__ cplx gget(const GramSmem& S, int i, int j) {
  if (i <= j) {
    const double2 v = S.u.G[i][j];
    return cmake(v.x, v.y);
  }
  const double2 v = S.u.G[j][i];
  return cmake(v.x, -v.y);
}

__device__ __forceinline__ void gput(GramSmem& S, int i, int j, cplx v) {
  if (i < j) S.u.G[i][j] = make_double2(v.x, v.y);
  else S.u.G[j][i] = make_double2(v.x, -v.y);
}

// the ordered column pair (p < q) of pair P in inner step s
__device__ __forceinline__ void inner_pq(int P, int s, int& p, int& q) {
  p = circle_at(P, s, JC);
  q = circle_at(JC - 1 - P, s, JC);
  if (p > q) { const int x = p; p = q; q = x; }
}

// Round kernel 1: the pair Gram and, in the pair's last CTA to finish, the test and one
// cyclic Jacobi sweep on it.
//   a. every part (up to RMAX Gram rows) loads its rows of the pair's 32 columns and
//      forms a partial Gram on the FP64 tensor path; with several parts the partials go
//      to global memory and the last part to arrive (an arrival counter per pair) sums
//      them in part order, so the Gram does not depend on arrival order;
//   b. no rotation if every column pair is orthogonal to `tol` (relative); else
//   c. a cyclic two-sided sweep (circle order, 16 disjoint rotations per step) on the
//      Gram, accumulating the 32 x 32 unitary Q, which goes to global memory with a
//      flag for the apply kernel.
// The step's rotations are computed once (16 threads) and read by all; the Gram keeps
// only its upper triangle; Q lives in registers in circle-position order -- thread
// (pair L, rows g, g + 16) holds the entries of the two positions of pair L and passes
// them to the neighbouring pairs by warp shuffles when the circle turns, so Q never
// touches shared memory.  After the 31 steps the circle is back at its start and every
// thread holds columns L and 31 - L.
__global__ __launch_bounds__(JNT) void jacobi_gram_kernel(const SectorDesc* __restrict__ sd,
                                                          const JacobiWork* __restrict__ work,
                                                          int n_work, int t,
                                                          const cplx* __restrict__ abuf,
                                                          int* __restrict__ rot_count,
                                                          const double* __restrict__ nf2,
                                                          double tol, int max_sweeps,
                                                          cplx* __restrict__ pbuf,
                                                          int* __restrict__ pcnt,
                                                          cplx* __restrict__ qbuf,
                                                          int* __restrict__ qflag,
                                                          unsigned long long* __restrict__ executed) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GramSmem& S = *reinterpret_cast<GramSmem*>(smem_raw);
  const int tid = threadIdx.x;
  const JacTask T = jac_task(work, n_work, t, false);
  if (T.part == 0 && tid == 0) qflag[T.slot] = 0;
  // every exit before the arrival counter depends on (sector, t) only
  if (T.sweep >= max_sweeps) return;
  int* cnt = rot_count + 3 * T.W.sector;
  // the counter of sweep w+1 is cleared during sweep w (nobody else touches it then),
  // before the converged exit so that a converged sector keeps reading zeros
  if (T.rr == 0 && T.pair == 0 && T.part == 0 && tid == 0) cnt[(T.sweep + 1) % 3] = 0;
  if (T.sweep >= 1 && cnt[(T.sweep - 1) % 3] == 0) return;   // converged
  const SectorDesc& D = sd[T.W.sector];
  const int k = D.k, rows_g = D.rows_g;
  const int r0 = T.part * T.W.chunk;
  const int ng = min(rows_g, r0 + T.W.chunk) - r0;   // >= 1: parts cover the Gram rows
  if (tid < JC) S.cols[tid] = jac_col(T, tid, k);
  if (tid == 0) {
    // numerical-rank floor: columns with |a|^2 <= z2 are exact zeros for the SVD
    const double zf = 16.0 * 2.220446049250313e-16 * sqrt((double)rows_g);
    S.z2 = zf * zf * nf2[T.W.sector];
    S.rotate = 0;
  }
  __syncthreads();

  // ---- a. rows -> shared memory (all loads of a thread in flight), partial Gram
  {
    const cplx* A = abuf + D.a_off;
    const int lane = tid & 31, wrow = tid >> 5;
    const int col = S.cols[lane];
    constexpr int PER = RMAX * JC / JNT;
    double2 v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int r = wrow + i * (JNT / JC);
      v[i] = make_double2(0.0, 0.0);
      if (r < ng && col >= 0) v[i] = *reinterpret_cast<const double2*>(A + (int64_t)(r0 + r) * k + col);
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int r = wrow + i * (JNT / JC);
      if (r < ng) S.u.tile[r][lane] = v[i];
    }
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31, li = lane >> 2, lk = lane & 3;
  // G[i][j] = sum_r conj(X[r][i]) X[r][j] on 8 x 8 tiles, rows in chunks of 4;
  // (ar - i ai)(br + i bi) = (ar br + ai bi) + i (ar bi - ai br)
  // The Gram is Hermitian: only its 10 upper 8 x 8 tiles (I <= J) are formed, spread
  // over the warps so that no scheduler (warps w and w + 4) carries more than three.
  int I0, J0, I1 = 0, J1 = 0, nt = 1;
  switch (warp) {
    case 0: I0 = 0; J0 = 0; I1 = 0; J1 = 1; nt = 2; break;
    case 1: I0 = 0; J0 = 3; I1 = 1; J1 = 1; nt = 2; break;
    case 2: I0 = 1; J0 = 3; break;
    case 3: I0 = 2; J0 = 3; break;
    case 4: I0 = 0; J0 = 2; break;
    case 5: I0 = 1; J0 = 2; break;
    case 6: I0 = 2; J0 = 2; break;
    default: I0 = 3; J0 = 3; break;
  }
  double2 gre[2] = {make_double2(0, 0), make_double2(0, 0)};
  double2 gim[2] = {make_double2(0, 0), make_double2(0, 0)};
  for (int k0 = 0; k0 < ng; k0 += 4) {
    const int r = k0 + lk;
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      if (jj >= nt) break;   // warp-uniform
      const int I = jj == 0 ? I0 : I1, J = jj == 0 ? J0 : J1;
      const double2 a = r < ng ? S.u.tile[r][8 * I + li] : make_double2(0.0, 0.0);
      const double2 b = r < ng ? S.u.tile[r][8 * J + li] : make_double2(0.0, 0.0);
      dmma8x8x4(gre[jj], a.x, b.x);
      dmma8x8x4(gre[jj], a.y, b.y);
      dmma8x8x4(gim[jj], a.x, b.y);
      dmma8x8x4(gim[jj], -a.y, b.x);
    }
  }
  __syncthreads();   // the tile is dead; G takes its place
  if (tid == 0) atomicAdd(executed, (unsigned long long)ng);   // executed: ng rows of 10 Gram tiles
  const int cs_g = T.W.cs_g;
  if (cs_g == 1) {
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      if (jj >= nt) break;
      const int row = 8 * (jj == 0 ? I0 : I1) + li, c0 = 8 * (jj == 0 ? J0 : J1) + 2 * lk;
      S.u.G[row][c0] = make_double2(gre[jj].x, gim[jj].x);
      S.u.G[row][c0 + 1] = make_double2(gre[jj].y, gim[jj].y);
    }
  } else {
    cplx* pp = pbuf + (int64_t)blockIdx.x * JC * JC;
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      if (jj >= nt) break;
      const int row = 8 * (jj == 0 ? I0 : I1) + li, c0 = 8 * (jj == 0 ? J0 : J1) + 2 * lk;
      __stcg(reinterpret_cast<double2*>(pp + row * JC + c0), make_double2(gre[jj].x, gim[jj].x));
      __stcg(reinterpret_cast<double2*>(pp + row * JC + c0 + 1), make_double2(gre[jj].y, gim[jj].y));
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      const int old = atomicAdd(pcnt + T.slot, 1);
      __threadfence();
      S.last = (old == cs_g - 1);
    }
    __syncthreads();
    if (!S.last) return;
    // the last part: fixed-order sum of the upper triangles of the pair's partials
    const cplx* p0 = pbuf + (int64_t)(blockIdx.x - T.part) * JC * JC;
    for (int e = tid; e < JC * JC; e += JNT) {
      const int i = e / JC, j = e % JC;
      if (j < i) continue;
      double sx = 0.0, sy = 0.0;
#pragma unroll 4
      for (int q = 0; q < cs_g; ++q) {
        const double2 v = __ldcg(reinterpret_cast<const double2*>(p0 + (int64_t)q * JC * JC + e));
        sx += v.x;
        sy += v.y;
      }
      S.u.G[i][j] = make_double2(sx, sy);
    }
    if (tid == 0) pcnt[T.slot] = 0;   // ready for the next round
  }
  __syncthreads();

  // ---- b. convergence test (relative tolerance on |a_i^H a_j|)
  if (tol <= 0.0) tol = fmax(8.0 * 2.220446049250313e-16, 4.0 * 2.220446049250313e-16 * sqrt((double)rows_g));
  const double t2 = tol * tol, z2 = S.z2;
  for (int e = tid; e < JC * JC; e += JNT) {
    const int i = e / JC, j = e % JC;
    if (j <= i) continue;
    const double dii = S.u.G[i][i].x, djj = S.u.G[j][j].x;
    const double2 g = S.u.G[i][j];
    const double a2 = g.x * g.x + g.y * g.y;
    // a column at the numerical-rank floor, or below tol times its partner, is rounding
    // noise along the partner and is never rotated against it
    if (dii > z2 && djj > z2 && dii > t2 * djj && djj > t2 * dii && a2 > t2 * dii * djj) S.rotate = 1;
  }
  __syncthreads();
  if (!S.rotate) return;
  if (tid == 0) atomicAdd(cnt + T.sweep % 3, 1);

  // ---- c. one cyclic Jacobi sweep on the Gram
  // block roles: thread < 136 updates the 2 x 2 block (P1, P2), P1 <= P2, of the pair
  // positions; lanes 0-15 of the last warp compute the step's rotations
  int P1 = -1, P2 = -1;
  if (tid < (JC / 2) * (JC / 2 + 1) / 2) {
    int rem = tid;
    P1 = 0;
    while (rem >= JC / 2 - P1) { rem -= JC / 2 - P1; ++P1; }
    P2 = P1 + rem;
  }
  const int rt = tid - (JNT - 32);
  const int L = tid & 15, grp = tid >> 4;
  // Q at step 0 is the identity: positions hold columns L (upper) and 31 - L (lower);
  // rows grp < 16 meet column L only on the diagonal, rows grp + 16 meet 31 - L
  cplx qu0 = cmake(grp == L ? 1.0 : 0.0, 0.0), qu1 = cmake(0.0, 0.0);
  cplx ql0 = cmake(0.0, 0.0), ql1 = cmake(grp + 16 == JC - 1 - L ? 1.0 : 0.0, 0.0);
  for (int step = 0; step < JC - 1; ++step) {
    // ---- phase A: rotations (zero-division form) and block operands
    if (rt >= 0 && rt < JC / 2) {
      int p, q;
      inner_pq(rt, step, p, q);
      const double a = S.u.G[p][p].x, d = S.u.G[q][q].x;
      const double2 g = S.u.G[p][q];
      const double g2 = g.x * g.x + g.y * g.y;
      double c = 1.0;
      double2 se = make_double2(0.0, 0.0);
      // cos 2t = |d - a| / r, r = sqrt((d - a)^2 + 4 |g|^2), c = sqrt((1 + cos 2t) / 2),
      // s e^{i alpha} = sign(d - a) g / (r c).  The off-diagonal threshold is tol / 4: a
      // pair the pair test flags must be rotated here even if this Gram's rounding
      // puts it slightly lower.
      if (g2 > 0.0 && a > z2 && d > z2 && a > t2 * d && d > t2 * a && g2 > 0.0625 * t2 * a * d) {
        const double dd = d - a;
        const double ir = rsqrt(fma(dd, dd, 4.0 * g2));
        const double c2 = fma(0.5 * fabs(dd), ir, 0.5);
        const double ic = rsqrt(c2);
        c = c2 * ic;
        const double f = copysign(ir * ic, dd);
        se = make_double2(f * g.x, f * g.y);
      }
      S.rc[rt] = c;
      S.rs[rt] = se;
    }
    int p1 = 0, q1 = 0, p2 = 0, q2 = 0;
    cplx B00 = cmake(0.0, 0.0), B01 = B00, B10 = B00, B11 = B00;
    if (P1 >= 0) {
      inner_pq(P1, step, p1, q1);
      inner_pq(P2, step, p2, q2);
      B00 = gget(S, p1, p2);
      B01 = gget(S, p1, q2);
      B10 = gget(S, q1, p2);
      B11 = gget(S, q1, q2);
    }
    const int cu = circle_at(L, step, JC), cl = circle_at(JC - 1 - L, step, JC);
    __syncthreads();
    // ---- phase B: block updates G' = J^H G J, and Q' = Q J
    if (P1 >= 0) {
      const double c1 = S.rc[P1], c2v = S.rc[P2];
      const cplx s1 = cmake(S.rs[P1].x, S.rs[P1].y), s2 = cmake(S.rs[P2].x, S.rs[P2].y);
      const bool r1 = !(c1 == 1.0 && s1.x == 0.0 && s1.y == 0.0);
      const bool r2 = !(c2v == 1.0 && s2.x == 0.0 && s2.y == 0.0);
      if (r1 || r2) {
        // B J2: columns (p2, q2)
        const cplx x00 = csub(cscale(B00, c2v), cmulc(B01, s2)), x01 = cadd(cmul(B00, s2), cscale(B01, c2v));
        const cplx x10 = csub(cscale(B10, c2v), cmulc(B11, s2)), x11 = cadd(cmul(B10, s2), cscale(B11, c2v));
        // J1^H (B J2): rows (p1, q1)
        const cplx y00 = csub(cscale(x00, c1), cmul(s1, x10)), y01 = csub(cscale(x01, c1), cmul(s1, x11));
        const cplx y10 = cadd(cmulc(x00, s1), cscale(x10, c1)), y11 = cadd(cmulc(x01, s1), cscale(x11, c1));
        if (P1 == P2) {
          S.u.G[p1][p1] = make_double2(y00.x, 0.0);
          S.u.G[p1][q1] = make_double2(0.0, 0.0);
          S.u.G[q1][q1] = make_double2(y11.x, 0.0);
        } else {
          gput(S, p1, p2, y00);
          gput(S, p1, q2, y01);
          gput(S, q1, p2, y10);
          gput(S, q1, q2, y11);
        }
      }
    }
    {
      const double c = S.rc[L];
      const cplx se = cmake(S.rs[L].x, S.rs[L].y);
      if (!(c == 1.0 && se.x == 0.0 && se.y == 0.0)) {
        // columns (p, q) = (cu, cl) or (cl, cu): v = Q[:, p], w = Q[:, q]
        const bool up = cu < cl;
        const cplx v0 = up ? qu0 : ql0, w0 = up ? ql0 : qu0;
        const cplx v1 = up ? qu1 : ql1, w1 = up ? ql1 : qu1;
        const cplx n0 = csub(cscale(v0, c), cmulc(w0, se)), m0 = cadd(cmul(v0, se), cscale(w0, c));
        const cplx n1 = csub(cscale(v1, c), cmulc(w1, se)), m1 = cadd(cmul(v1, se), cscale(w1, c));
        qu0 = up ? n0 : m0;
        ql0 = up ? m0 : n0;
        qu1 = up ? n1 : m1;
        ql1 = up ? m1 : n1;
      }
      // turn the circle: position j takes the column of position j + 1 (31 -> 1), so
      // pair L's upper entry comes from pair L + 1's upper (pair 15: its own lower) and
      // its lower from pair L - 1's lower (pair 0: pair 1's upper); position 0 stays
      const cplx du0 = cmake(__shfl_down_sync(0xffffffffu, qu0.x, 1, 16), __shfl_down_sync(0xffffffffu, qu0.y, 1, 16));
      const cplx du1 = cmake(__shfl_down_sync(0xffffffffu, qu1.x, 1, 16), __shfl_down_sync(0xffffffffu, qu1.y, 1, 16));
      const cplx ul0 = cmake(__shfl_up_sync(0xffffffffu, ql0.x, 1, 16), __shfl_up_sync(0xffffffffu, ql0.y, 1, 16));
      const cplx ul1 = cmake(__shfl_up_sync(0xffffffffu, ql1.x, 1, 16), __shfl_up_sync(0xffffffffu, ql1.y, 1, 16));
      const cplx nu0 = L == 0 ? qu0 : (L == 15 ? ql0 : du0), nu1 = L == 0 ? qu1 : (L == 15 ? ql1 : du1);
      const cplx nl0 = L == 0 ? du0 : ul0, nl1 = L == 0 ? du1 : ul1;
      qu0 = nu0;
      qu1 = nu1;
      ql0 = nl0;
      ql1 = nl1;
    }
    __syncthreads();
  }
  // ---- Q (column order again) and the flag for the apply kernel
  cplx* qo = qbuf + (int64_t)T.slot * JC * JC;
  stc(qo + grp * JC + L, qu0);
  stc(qo + (grp + 16) * JC + L, qu1);
  stc(qo + grp * JC + (JC - 1 - L), ql0);
  stc(qo + (grp + 16) * JC + (JC - 1 - L), ql1);
  if (tid == 0) qflag[T.slot] = 1;
}

// Round kernel 2: every part of a rotated pair applies Q to its rows on the FP64 tensor
// path, straight from global memory into mma fragments: warp w owns rows
// [16 w, 16 w + 16), one 8-row tile at a time, x the four 8-column tiles.  The complex
// product takes three real products (Gauss):
// (tr + i ti)(qr + i qi) = (tr qr - ti qi) + i ((tr + ti)(qr + qi) - tr qr - ti qi).
__global__ __launch_bounds__(JNT) void jacobi_apply_kernel(const SectorDesc* __restrict__ sd,
                                                           const JacobiWork* __restrict__ work,
                                                           int n_work, int t, cplx* __restrict__ abuf,
                                                           int max_sweeps,
                                                           const cplx* __restrict__ qbuf,
                                                           const int* __restrict__ qflag,
                                                           unsigned long long* __restrict__ executed) {
  __shared__ double2 Qs[JC][JC + 1];
  __shared__ double Qsum[JC][JC + 1];   // Re Q + Im Q
  __shared__ int cols[JC];
  const int tid = threadIdx.x;
  const JacTask T = jac_task(work, n_work, t, true);
  if (T.sweep >= max_sweeps) return;
  if (!qflag[T.slot]) return;   // converged sector, or a pair without rotation
  const SectorDesc& D = sd[T.W.sector];
  const int k = D.k;
  const int r0 = T.part * T.W.chunk;
  const int nr = min(D.rows_tot, r0 + T.W.chunk) - r0;
  if (tid == 0) atomicAdd(executed + 1, (unsigned long long)nr);   // executed: nr rows rotated
  if (tid < JC) cols[tid] = jac_col(T, tid, k);
  const cplx* qi = qbuf + (int64_t)T.slot * JC * JC;
#pragma unroll
  for (int i = 0; i < JC * JC / JNT; ++i) {
    const int e = tid + i * JNT;
    const cplx v = ldc(qi + e);
    Qs[e / JC][e % JC] = make_double2(v.x, v.y);
    Qsum[e / JC][e % JC] = v.x + v.y;
  }
  __syncthreads();
  cplx* A = abuf + D.a_off;
  const int warp = tid >> 5, lane = tid & 31, li = lane >> 2, lk = lane & 3;
  if (16 * warp >= nr) return;
#pragma unroll 1
  for (int a = 0; a < 2; ++a) {
    const int row = 16 * warp + 8 * a + li;
    double2 tv[JC / 4];
#pragma unroll
    for (int kk = 0; kk < JC / 4; ++kk) {
      const int col = cols[4 * kk + lk];
      tv[kk] = make_double2(0.0, 0.0);
      if (row < nr && col >= 0) tv[kk] = *reinterpret_cast<const double2*>(A + (int64_t)(r0 + row) * k + col);
    }
    // t1 = Tr Qr, t2 = Ti Qi, t3 = (Tr + Ti)(Qr + Qi) on the four column tiles
    double2 t1[4], t2[4], t3[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      t1[c] = make_double2(0, 0);
      t2[c] = make_double2(0, 0);
      t3[c] = make_double2(0, 0);
    }
#pragma unroll
    for (int kk = 0; kk < JC / 4; ++kk) {
      const double ts = tv[kk].x + tv[kk].y;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const double2 q = Qs[4 * kk + lk][8 * c + li];
        const double qs = Qsum[4 * kk + lk][8 * c + li];
        dmma8x8x4(t1[c], tv[kk].x, q.x);
        dmma8x8x4(t2[c], tv[kk].y, q.y);
        dmma8x8x4(t3[c], ts, qs);
      }
    }
    if (row < nr) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int c0 = cols[8 * c + 2 * lk], c1 = cols[8 * c + 2 * lk + 1];
        if (c0 >= 0)
          stc(A + (int64_t)(r0 + row) * k + c0, cmake(t1[c].x - t2[c].x, t3[c].x - t1[c].x - t2[c].x));
        if (c1 >= 0)
          stc(A + (int64_t)(r0 + row) * k + c1, cmake(t1[c].y - t2[c].y, t3[c].y - t1[c].y - t2[c].y));
      }
    }
  }
}

constexpr int FNT = 512;

__global__ __launch_bounds__(FNT) void jacobi_finish_kernel(const SectorDesc* __restrict__ sd,
                                                            const int* __restrict__ list,
                                                            const cplx* __restrict__ abuf,
                                                            const double* __restrict__ nf2,
                                                            double* __restrict__ sig,
                                                            int* __restrict__ perm) {
  extern __shared__ unsigned char smem_raw[];
  const SectorDesc& S = sd[list[blockIdx.x]];
  const int k = S.k;
  if (k == 0) return;
  int np2 = 1;
  while (np2 < k) np2 <<= 1;
  double* sv = reinterpret_cast<double*>(smem_raw);
  int* si = reinterpret_cast<int*>(sv + np2);
  const cplx* A = abuf + S.a_off;
  const double zf = 16.0 * 2.220446049250313e-16 * sqrt((double)S.rows_g);
  const double z2 = zf * zf * nf2[list[blockIdx.x]];
  for (int j = threadIdx.x; j < np2; j += FNT) {
    double s2 = -1.0;
    if (j < k) {
      s2 = 0.0;
      for (int r = 0; r < S.rows_g; ++r) s2 += cabs2(ldc(A + (int64_t)r * k + j));
      if (s2 <= z2) s2 = 0.0;   // below the numerical-rank floor: an exact zero
    }
    sv[j] = s2 >= 0.0 ? sqrt(s2) : -1.0;
    si[j] = j;
  }
  __syncthreads();
  // bitonic sort: descending value, ascending index
  for (int size = 2; size <= np2; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < np2; i += FNT) {
        const int j = i ^ stride;
        if (j > i) {
          const bool up = (i & size) == 0;
          const double a = sv[i], b = sv[j];
          const int ia = si[i], ib = si[j];
          // "a before b" in the final order
          const bool a_first = (a > b) || (a == b && ia < ib);
          if (a_first != up) {
            sv[i] = b; sv[j] = a;
            si[i] = ib; si[j] = ia;
          }
        }
      }
      __syncthreads();
    }
  }
  for (int j = threadIdx.x; j < k; j += FNT) {
    sig[S.s_off + j] = sv[j];
    perm[S.s_off + j] = si[j];
  }
}

// ||T_s||_F^2 over the Gram rows, one CTA per sector, fixed-order reduction
constexpr int NNT = 256;
__global__ __launch_bounds__(NNT) void sector_norm_kernel(const SectorDesc* __restrict__ sd,
                                                          const int* __restrict__ list,
                                                          const cplx* __restrict__ abuf,
                                                          double* __restrict__ nf2) {
  __shared__ double red[NNT];
  const SectorDesc& S = sd[list[blockIdx.x]];
  const int64_t total = (int64_t)S.rows_g * S.k;
  const cplx* A = abuf + S.a_off;
  double acc = 0.0;
  for (int64_t e = threadIdx.x; e < total; e += NNT) acc += cabs2(ldc(A + e));
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = NNT / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) nf2[list[blockIdx.x]] = red[0];
}

// ---------------------------------------------------------------------------------
// Small sectors: the whole SVD of a sector in one CTA, preconditioned by QR with column
// pivoting (Drmac and Veselic, SIAM J. Matrix Anal. Appl. 29, 2008).  X is the Jacobi matrix's
// Gram part, rows x k, in shared memory by columns:
//   X P = Q R;  left sectors (X = T^H): T = P R^H Q^H, so T's left vectors are P times those
//   of L = R^H; the others (X = T): R^H P2 = Q2 R2, T's left vectors are Q P2 times those of
//   L = R2^H.
// One-sided Jacobi on the k columns of L gives L W = U Sigma; its normalised columns are the
// left vectors, so no rotation is accumulated.  A sweep is the circle method over single
// columns, eight lanes to a column pair with the columns in their registers: dot products,
// the rotation, its application, with the tests and the floor of the blocked form above.
// All sweeps, the norms and the sort run here: no rounds of launches, no convergence polls.
// What bounds it: a step's latency and its FP64 issue on one SM.  At k = 48 a step of a sweep
// takes 1,225 cycles (five to seven sweeps of k - 1 steps), a step of a QR 2,250 up to 64 rows
// and 4,100 up to 128.  Without the factorisations, a warp to a pair over all rows and the
// accumulated rotations (six to twelve sweeps where the sector is graded), before and after,
// us: k = 28, 128 rows 209 and 154 (X = T), 230 and 107 (X = T^H); k = 48, 128 rows 545 and
// 360, 674 and 287; graded sectors of a 24-mode circuit up to 1,090 and 340.  A 24-mode chi =
// 256 circuit 40.6 ms and 36.3, 32 modes on the Gram route 30.7 and 27.0, 24 modes chi = 64
// 13.8 and 10.0, chi = 128 31 and 20.5.
constexpr int JS_KMAX = 64;
// Up to JS_TINY columns the sweeps run on X itself, the rotations of a left sector accumulated:
// two factorisations of one to four columns add more rounding than they take away sweeps.
// Mean relative error of 1, 2, 3 and 4 square columns' values, 1e-16: 1.9, 1.7, 2.1 and 2.5 with
// the factorisations, 0.9, 1.2, 1.8 and 2.0 without; Lambda of a chi = 32 update under way 3.0e-15
// and 2.3e-15 off, at equal time (235 us).  Updates of four such sectors, us, with and without: 1,000
// x 3 215 and 192, 4 x 300 108 and 104, 3 x 1,000 132 and 147 (a warp to a pair is long there).
constexpr int JS_TINY = 4;
constexpr int JS_SMEM = 216 * 1024;
constexpr int JS_EX = 100;     // binary exponents of X's largest entry that need no scaling

// leading dimension of a column: odd in units of 16 B, so lanes across columns fall on
// different banks
__host__ __device__ inline int js_ld(int rows) { return rows | 1; }
__host__ __device__ inline int js_ldl(int k) { return (k + 15) / 16 * 16 + 1; }   // of L

// a summed over each LPC consecutive lanes (8, 16 or 32), in every one of them: a product
// with ones leaves lane i & 3 the four-lane sums of columns 2 i and 2 i + 1, lanes 8 i..8 i + 7
template <int LPC>
__device__ __forceinline__ double group_sum(double a) {
  double2 s = make_double2(0, 0);
  __syncwarp();
  dmma8x8x4(s, 1.0, a);
  const double e = s.x + s.y;
  const int first = (threadIdx.x & 31) / LPC * (LPC / 8);
  double t = __shfl_sync(0xffffffffu, e, first);
#pragma unroll
  for (int i = 1; i < LPC / 8; ++i) t += __shfl_sync(0xffffffffu, e, first + i);
  return t;
}

// X P = Q R of one matrix: the reflectors H_j = 1 - t_j v_j v_j^H, v_j the rows below j of
// column piv[j] under v1[j]; R's diagonal rd, its row i < j in row i of column piv[j].
struct JsQr {
  // squared norms of the columns' rows below the reduced ones; reduced: < 0, which a NaN is
  // not, so piv ends as a permutation whatever the numbers are
  double nn[2][JS_KMAX];
  double2 rd[JS_KMAX], v1[JS_KMAX];
  double t[JS_KMAX];
  int piv[JS_KMAX];
};

// Steps [j0, j1) of the factorisation, whose rows below j lie in chunks F..RPL - 1 of LPC rows
// (chunk F alone holds rows above them too): no test per chunk, so a column's loads are in
// flight together.  Returns false where nothing is left to reduce.
template <int LPC, int RPL, int F>
__device__ __forceinline__ bool js_qr_steps(double2* X, int ld, int rows, int k, JsQr& q, int n_warps, int j0, int j1) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int GPW = 32 / LPC, R = RPL > 0 ? RPL : 1;
  const int g = lane / LPC, l = lane % LPC;
  for (int j = j0; j < j1; ++j) {
    const double* nn = q.nn[j & 1];
    double* next = q.nn[(j + 1) & 1];
    // a largest column, by the leading 32 bits of its norm
    auto key = [&](int c) { return c >= k ? -2 : nn[c] < 0.0 ? -1 : __double2hiint(nn[c]) & 0x7fffffff; };
    const int h0 = key(lane), h1 = key(lane + 32);
    const int hm = __reduce_max_sync(0xffffffffu, max(h0, h1));
    const unsigned in0 = __ballot_sync(0xffffffffu, h0 == hm), in1 = __ballot_sync(0xffffffffu, h1 == hm);
    const int p = in0 ? __ffs(in0) - 1 : 31 + __ffs(in1);
    const double n2 = nn[p];
    if (n2 < 1e-270) {                 // nothing left (f2 >= 2^-200; uniform over the CTA): R's other rows are zero
      if (tid == 0) {
        int at = j;
        for (int c = 0; c < k; ++c)
          if (!(nn[c] < 0.0)) q.piv[at++] = c;
      }
      for (int i = j + tid; i < k; i += 32 * n_warps) {
        q.rd[i] = q.v1[i] = make_double2(0.0, 0.0);
        q.t[i] = 0.0;
      }
      return false;
    }
    const double2 *vp = X + p * ld, al = vp[j];
    double2 v[R];                      // the reflector below its head
    if (RPL > 0) {
#pragma unroll
      for (int i = F; i < R; ++i) {
        const int r = l + LPC * i;
        v[i] = (i > F || r > j) && r < rows ? vp[r] : make_double2(0.0, 0.0);
      }
    }
    const double a2 = fma(al.x, al.x, al.y * al.y), nx = n2 * rsqrt(n2);
    double t;
    double2 v1, beta;
    if (a2 > 1e-34 * n2) {
      const double ra = rsqrt(a2), f = nx * ra;
      t = __drcp_rn(fma(nx, a2 * ra, n2));
      beta = make_double2(-al.x * f, -al.y * f);
      v1 = make_double2(al.x - beta.x, al.y - beta.y);
    } else {
      // a head below the rounding of nx
      t = __drcp_rn(n2);
      beta = make_double2(-nx, 0.0);
      v1 = make_double2(nx, 0.0);
    }
    if (tid == 0) {
      q.piv[j] = p;
      q.rd[j] = beta;
      q.v1[j] = v1;
      q.t[j] = t;
    }
    for (int base = warp * GPW; base < k; base += n_warps * GPW) {
      const int c = base + g;
      const bool act = c < k && c != p && !(nn[c] < 0.0);
      double2* x = X + (act ? c : p) * ld;
      double dx = 0.0, dy = 0.0, s = 0.0;
      auto dot = [&](double2 a, double2 b) {   // conj(a) b
        dx = fma(a.x, b.x, fma(a.y, b.y, dx));
        dy = fma(a.x, b.y, fma(-a.y, b.x, dy));
      };
      auto sub = [&](double2 a, double2 b) {   // b - w a, w in (dx, dy)
        return make_double2(fma(-dx, a.x, fma(dy, a.y, b.x)), fma(-dx, a.y, fma(-dy, a.x, b.y)));
      };
      const double2 xj = x[j];
      auto weight = [&] {
        dx = group_sum<LPC>(dx);
        dy = group_sum<LPC>(dy);
        dot(v1, xj);
        dx *= t;
        dy *= t;
      };
      if (RPL > 0) {
        double2 u[R];
#pragma unroll
        for (int i = F; i < R; ++i) {
          const int r = l + LPC * i;
          u[i] = (i > F || r > j) && r < rows ? x[r] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int i = F; i < R; ++i) dot(v[i], u[i]);
        weight();
#pragma unroll
        for (int i = F; i < R; ++i) {
          const int r = l + LPC * i;
          u[i] = sub(v[i], u[i]);
          s = fma(u[i].x, u[i].x, fma(u[i].y, u[i].y, s));
          if (act && (i > F || r > j) && r < rows) x[r] = u[i];
        }
      } else {
        for (int r = j + 1 + l; r < rows; r += LPC) dot(vp[r], x[r]);
        weight();
        for (int r = j + 1 + l; r < rows; r += LPC) {
          const double2 o = sub(vp[r], x[r]);
          if (act) x[r] = o;
          s = fma(o.x, o.x, fma(o.y, o.y, s));
        }
      }
      if (act && l == 0) x[j] = sub(v1, xj);
      s = group_sum<LPC>(s);
      if (l == 0 && c < k) next[c] = act ? s : -1.0;
    }
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"r"(32 * n_warps) : "memory");
  }
  return true;
}

template <int LPC, int RPL, int F>
__device__ __forceinline__ void js_qr_from(double2* X, int ld, int rows, int k, JsQr& q, int n_warps) {
  // rows below j start in chunk F for j + 1 in [LPC F, LPC (F + 1))
  if (!js_qr_steps<LPC, RPL, F>(X, ld, rows, k, q, n_warps, max(LPC * F - 1, 0), min(LPC * (F + 1) - 1, k))) return;
  if constexpr (LPC * (F + 1) - 1 < JS_KMAX && F + 1 < RPL) {
    if (LPC * (F + 1) - 1 < k) js_qr_from<LPC, RPL, F + 1>(X, ld, rows, k, q, n_warps);
  } else if constexpr (LPC * (F + 1) - 1 < JS_KMAX) {
    // rows = k = LPC RPL: the last column has no rows below its head
    js_qr_steps<LPC, RPL, RPL - 1>(X, ld, rows, k, q, n_warps, LPC * (F + 1) - 1, k);
  }
}

// The factorisation; q.nn[0] holds the squared column norms.  LPC lanes take a column, its
// rows in their registers (up to LPC RPL rows; RPL 0: read twice): its dot product with
// the reflector, its update, and the norm of what is left of it, summed anew.  No more warps
// than the columns need take part: each computes the reflector's scalars.
template <int LPC, int RPL>
__device__ void js_qr(double2* X, int ld, int rows, int k, JsQr& q, int n_warps) {
  n_warps = min(n_warps, (k + 32 / LPC - 1) / (32 / LPC));
  if ((int)(threadIdx.x >> 5) < n_warps) {
    if constexpr (RPL > 0) js_qr_from<LPC, RPL, 0>(X, ld, rows, k, q, n_warps);
    else js_qr_steps<LPC, 0, 0>(X, ld, rows, k, q, n_warps, 0, k);
  }
  __syncthreads();
}

// y = H_j1 .. H_j0 y (j1 the lower) of a column's rows in registers; chunks F.. hold rows j..
template <int LPC, int RPL, int F>
__device__ __forceinline__ void js_q_steps(const double2* X, int ld, int rows, const JsQr& q, double2 (&y)[RPL], int j0, int j1) {
  const int l = threadIdx.x % LPC;
  constexpr bool KEEP = RPL <= 8;      // the reflector in registers too
  for (int j = j0; j >= j1; --j) {
    const double2* x = X + q.piv[j] * ld;
    const double2 v1 = q.v1[j];
    const double t = q.t[j];
    auto at = [&](int i) {
      const int r = l + LPC * i;
      const double2 w = (i > F || r > j) && r < rows ? x[r] : make_double2(0.0, 0.0);
      return i == F && r == j ? v1 : w;
    };
    double2 v[KEEP ? RPL : 1];
    double dx = 0.0, dy = 0.0;
    if (KEEP) {
#pragma unroll
      for (int i = F; i < RPL; ++i) v[KEEP ? i : 0] = at(i);
    }
#pragma unroll
    for (int i = F; i < RPL; ++i) {
      const double2 w = KEEP ? v[KEEP ? i : 0] : at(i);
      dx = fma(w.x, y[i].x, fma(w.y, y[i].y, dx));
      dy = fma(w.x, y[i].y, fma(-w.y, y[i].x, dy));
    }
    dx = t * group_sum<LPC>(dx);
    dy = t * group_sum<LPC>(dy);
#pragma unroll
    for (int i = F; i < RPL; ++i) {
      const double2 w = KEEP ? v[KEEP ? i : 0] : at(i);
      y[i] = make_double2(fma(-dx, w.x, fma(dy, w.y, y[i].x)), fma(-dx, w.y, fma(-dy, w.x, y[i].y)));
    }
  }
}

template <int LPC, int RPL, int F>
__device__ __forceinline__ void js_q_from(const double2* X, int ld, int rows, int k, const JsQr& q, double2 (&y)[RPL]) {
  js_q_steps<LPC, RPL, F>(X, ld, rows, q, y, min(LPC * (F + 1), k) - 1, LPC * F);
  if constexpr (F > 0) js_q_from<LPC, RPL, F - 1>(X, ld, rows, k, q, y);
}

// A's columns = Q [P2 Y; 0], LPC lanes to a column (y0(c, i): entry i of P2 Y's column c), a
// column's rows in their registers
template <int LPC, int RPL, typename F>
__device__ void js_q_apply(const double2* X, int ld, int rows, int k, const JsQr& q, cplx* A, int n_warps, F y0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int GPW = 32 / LPC;
  const int g = lane / LPC, l = lane % LPC;
  for (int base = warp * GPW; base < k; base += n_warps * GPW) {
    const int c = base + g;
    double2 y[RPL];
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int r = l + LPC * i;
      y[i] = r < k && c < k ? y0(c, r) : make_double2(0.0, 0.0);
    }
    js_q_from<LPC, RPL, (JS_KMAX - 1) / LPC>(X, ld, rows, k, q, y);
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int r = l + LPC * i;
      if (r < rows && c < k) stc(A + (int64_t)r * k + c, cmake(y[i].x, y[i].y));
    }
  }
}

// All sweeps over the k columns of L (k rows, zeros up to 8 RL), by the first n_warps warps: four column pairs
// to a warp, eight lanes and RL rows a lane to a pair.  Returns the sweeps done (max_sweeps
// + 1: not converged) and adds this lane's rotations to `turned`.
template <int RL>
__device__ int js_sweeps(double2* L, int ld, int k, double z2, double t2, int max_sweeps, int n_warps, int* rot,
                         unsigned long long& turned) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 3, l = lane & 7;
  const int n = k + (k & 1), P = 4 * warp + g;
  auto barrier = [&] { asm volatile("bar.sync 1, %0;" ::"r"(32 * n_warps) : "memory"); };
  for (int sweep = 0;; ++sweep) {
    if (sweep == max_sweeps) return max_sweeps + 1;
    int mine = 0;
    for (int step = 0; step < n - 1; ++step) {
      // circle_at without its division
      int p = P + step, q = n - 1 - P + step;
      if (p > n - 1) p -= n - 1;
      if (q > n - 1) q -= n - 1;
      if (P == 0) p = 0;
      if (p > q) { const int x = p; p = q; q = x; }
      const bool ok = P < n / 2 && q < k;   // q == k: the padding column
      double2 *x = L + (ok ? p * ld : 0) + l, *y = L + (ok ? q * ld : 0) + l;
      double2 u[RL], v[RL];
      double a = 0.0, b = 0.0, gx = 0.0, gy = 0.0;
#pragma unroll
      for (int i = 0; i < RL; ++i) {
        u[i] = x[8 * i];
        v[i] = y[8 * i];
      }
#pragma unroll
      for (int i = 0; i < RL; ++i) {
        a = fma(u[i].x, u[i].x, fma(u[i].y, u[i].y, a));
        b = fma(v[i].x, v[i].x, fma(v[i].y, v[i].y, b));
        gx = fma(u[i].x, v[i].x, fma(u[i].y, v[i].y, gx));
        gy = fma(u[i].x, v[i].y, fma(-u[i].y, v[i].x, gy));
      }
      // sums over the eight lanes: a product with ones leaves lane j & 3 the four-lane sums
      // of columns 2 j and 2 j + 1, which are the lanes of pair j
      double2 s0 = make_double2(0, 0), s1 = s0, s2 = s0, s3 = s0;
      __syncwarp();
      dmma8x8x4(s0, 1.0, a);
      dmma8x8x4(s1, 1.0, b);
      dmma8x8x4(s2, 1.0, gx);
      dmma8x8x4(s3, 1.0, gy);
      a = __shfl_sync(0xffffffffu, s0.x + s0.y, g);
      b = __shfl_sync(0xffffffffu, s1.x + s1.y, g);
      gx = __shfl_sync(0xffffffffu, s2.x + s2.y, g);
      gy = __shfl_sync(0xffffffffu, s3.x + s3.y, g);
      const double g2 = fma(gx, gx, gy * gy);
      const bool turn = ok && a > z2 && b > z2 && a > t2 * b && b > t2 * a && g2 > t2 * a * b;
      if (turn) {
        // the rotation of the blocked form: c, s e^{i alpha} of the small angle
        const double dd = b - a, ir = rsqrt(fma(dd, dd, 4.0 * g2)), c2 = fma(0.5 * fabs(dd), ir, 0.5), ic = rsqrt(c2);
        const double c = c2 * ic, f = copysign(ir * ic, dd), sx = f * gx, sy = f * gy;
        ++mine;
#pragma unroll
        for (int i = 0; i < RL; ++i) {
          // u' = c u - conj(s) v, v' = s u + c v
          x[8 * i] = make_double2(fma(c, u[i].x, fma(-sx, v[i].x, -(sy * v[i].y))),
                                  fma(c, u[i].y, fma(-sx, v[i].y, sy * v[i].x)));
          y[8 * i] = make_double2(fma(c, v[i].x, fma(sx, u[i].x, -(sy * u[i].y))),
                                  fma(c, v[i].y, fma(sx, u[i].y, sy * u[i].x)));
        }
      }
      __syncwarp();
      barrier();
    }
    turned += mine;
    if (l == 0 && mine) rot[sweep & 1] = 1;
    __syncwarp();
    barrier();
    const bool again = rot[sweep & 1] != 0;
    if (threadIdx.x == 0) rot[(sweep + 1) & 1] = 0;   // the next sweep's flag, which nobody sets before its barriers
    if (!again) return sweep + 1;
  }
}

// a summed over the warp, in every lane: the second product with ones adds the four pairs that
// the first leaves in a row (no shuffles)
__device__ __forceinline__ double lane_sum(double a) {
  double2 s = make_double2(0, 0), t = s;
  __syncwarp();
  dmma8x8x4(s, 1.0, a);
  dmma8x8x4(t, 1.0, s.x + s.y);
  return t.x;
}

// All sweeps over up to JS_TINY columns of X as they are, a warp to a pair: the rotations
// also go to the nv rows of V (below the identity they started from).  Returns as js_sweeps.
__device__ int js_sweeps_tiny(double2* X, int ldx, int rows, double2* V, int ldv, int nv, int k, double z2, double t2,
                              int max_sweeps, int* rot, unsigned long long& turned) {
  const int lane = threadIdx.x & 31, P = threadIdx.x >> 5, n = k + (k & 1);
  auto barrier = [&] { asm volatile("bar.sync 1, %0;" ::"r"(16 * n) : "memory"); };   // the n / 2 warps
  for (int sweep = 0;; ++sweep) {
    if (sweep == max_sweeps) return max_sweeps + 1;
    int mine = 0;
    for (int step = 0; step < n - 1; ++step) {
      int p = circle_at(P, step, n), q = circle_at(n - 1 - P, step, n);
      if (p > q) { const int x = p; p = q; q = x; }
      if (q < k) {                     // q == k: the padding column
        double2 *x = X + p * ldx, *y = X + q * ldx;
        double a = 0.0, b = 0.0, gx = 0.0, gy = 0.0;
#pragma unroll 4
        for (int r = lane; r < rows; r += 32) {
          const double2 u = x[r], v = y[r];
          a = fma(u.x, u.x, fma(u.y, u.y, a));
          b = fma(v.x, v.x, fma(v.y, v.y, b));
          gx = fma(u.x, v.x, fma(u.y, v.y, gx));
          gy = fma(u.x, v.y, fma(-u.y, v.x, gy));
        }
        a = lane_sum(a);
        b = lane_sum(b);
        gx = lane_sum(gx);
        gy = lane_sum(gy);
        const double g2 = fma(gx, gx, gy * gy);
        if (a > z2 && b > z2 && a > t2 * b && b > t2 * a && g2 > t2 * a * b) {
          const double dd = b - a, ir = rsqrt(fma(dd, dd, 4.0 * g2)), c2 = fma(0.5 * fabs(dd), ir, 0.5), ic = rsqrt(c2);
          const double c = c2 * ic, f = copysign(ir * ic, dd), sx = f * gx, sy = f * gy;
          ++mine;
          auto turn = [&](double2* x, double2* y, int n_rows) {
#pragma unroll 4
            for (int r = lane; r < n_rows; r += 32) {
              const double2 u = x[r], v = y[r];
              x[r] = make_double2(fma(c, u.x, fma(-sx, v.x, -(sy * v.y))), fma(c, u.y, fma(-sx, v.y, sy * v.x)));
              y[r] = make_double2(fma(c, v.x, fma(sx, u.x, -(sy * u.y))), fma(c, v.y, fma(sx, u.y, sy * u.x)));
            }
          };
          turn(x, y, rows);
          turn(V + p * ldv, V + q * ldv, nv);
        }
      }
      __syncwarp();
      barrier();
    }
    turned += mine;
    if (lane == 0 && mine) rot[sweep & 1] = 1;
    __syncwarp();
    barrier();
    const bool again = rot[sweep & 1] != 0;
    if (threadIdx.x == 0) rot[(sweep + 1) & 1] = 0;
    if (!again) return sweep + 1;
  }
}

// squared norms of a matrix's columns, a warp to a column
__device__ __forceinline__ void js_norms(const double2* X, int ld, int rows, int k, double* nn, int n_warps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int c = warp; c < k; c += n_warps) {
    double s = 0.0;
    for (int r = lane; r < rows; r += 32) {
      const double2 v = X[c * ld + r];
      s = fma(v.x, v.x, fma(v.y, v.y, s));
    }
    s = group_sum<32>(s);
    if (lane == 0) nn[c] = s;
  }
}

template <int NT>
__global__ __launch_bounds__(NT) void jacobi_small_kernel(const SectorDesc* __restrict__ sd,
                                                          const int* __restrict__ list, cplx* __restrict__ abuf,
                                                          int max_sweeps, double* __restrict__ sig,
                                                          int* __restrict__ perm, int* __restrict__ fail,
                                                          unsigned long long* __restrict__ executed) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ JsQr q1, q2;
  __shared__ double nrm[JS_KMAX];
  __shared__ int rot[2], inv2[JS_KMAX], top;
  const SectorDesc& S = sd[list[blockIdx.x]];
  const int k = S.k, rows = S.rows_g, ldx = js_ld(rows), ld = js_ldl(k);
  const bool left = S.left != 0;
  double2* X = reinterpret_cast<double2*>(smem_raw);   // column c: X + c ldx
  double2* Y = X + (size_t)k * ldx;                    // L, column c: Y + c ld
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cplx* A = abuf + S.a_off;
  if (tid < 2) rot[tid] = 0;
  if (tid == 0) top = 0;
  __syncthreads();
  int hi = 0;                                          // largest leading word of an entry's magnitude
  for (int e = tid; e < rows * k; e += NT) {
    const int r = e / k, c = e - r * k;
    const cplx v = ldc(A + e);
    X[c * ldx + r] = make_double2(v.x, v.y);
    hi = max(hi, max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff));
  }
  __syncwarp();
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) atomicMax(&top, hi);
  __syncthreads();
  // X 2^-ex where squares of its entries could leave the exponent's range (uniform over the
  // CTA), so the result does not depend on the scale; undone in the values and in X = T's columns
  int ex = (top >> 20) - 1023;
  if (top == 0 || top >= 0x7ff00000 || abs(ex) <= JS_EX) ex = 0;
  if (ex != 0) {
    for (int e = tid; e < rows * k; e += NT) {
      double2* x = X + (e % k) * ldx + e / k;
      *x = make_double2(scalbn(x->x, -ex), scalbn(x->y, -ex));
    }
    __syncthreads();
  }
  js_norms(X, ldx, rows, k, q1.nn[0], NW);
  __syncthreads();
  double f2 = 0.0;
  for (int c = 0; c < k; ++c) f2 += q1.nn[0][c];
  const double zf = 16.0 * 2.220446049250313e-16 * sqrt((double)rows), z2 = zf * zf * f2;
  // singular values from the squared norms in nrm (0 below the numerical-rank floor, -1 for a
  // NaN), in descending order (ties by column): perm is a permutation whatever nrm holds
  auto finish = [&] {
    if (tid < k) {
      const double s = nrm[tid];
      nrm[tid] = s <= z2 ? 0.0 : s >= 0.0 ? sqrt(s) : -1.0;
    }
    __syncthreads();
    if (tid < k) {
      const double s = nrm[tid];
      int at = 0;
      for (int c = 0; c < k; ++c) at += nrm[c] > s || (nrm[c] == s && c < tid);
      sig[S.s_off + at] = ex != 0 ? scalbn(s, ex) : s;
      perm[S.s_off + at] = tid;
    }
  };
  const bool finite = top < 0x7ff00000;
  if (k <= JS_TINY || !finite) {
    // X's columns as they are (see JS_TINY); where X has a NaN or an infinity none is rotated, as
    // in the blocked form, whose tests are all false then
    for (int e = tid; left && e < k * k; e += NT) Y[(e % k) * ld + e / k] = make_double2(e / k == e % k ? 1.0 : 0.0, 0.0);
    __syncthreads();
    if (finite && warp < k / 2 + (k & 1) && k > 1) {
      unsigned long long turned = 0;
      const double tol = fmax(8.0 * 2.220446049250313e-16, 4.0 * 2.220446049250313e-16 * sqrt((double)rows));
      const int nv = left ? k : 0, sweeps = js_sweeps_tiny(X, ldx, rows, Y, ld, nv, k, z2, tol * tol, max_sweeps, rot, turned);
      if (lane == 0 && turned) atomicAdd(executed, turned * 4ull * (unsigned)(rows + nv));
      if (tid == 0) {
        if (sweeps > max_sweeps) *fail = 1;
        atomicAdd(executed, (unsigned long long)min(sweeps, max_sweeps) * (unsigned)(k * (k - 1) / 2) * 2ull * (unsigned)rows);
        atomicMax(executed + 1, (unsigned long long)min(sweeps, max_sweeps));
      }
    }
    __syncthreads();
    js_norms(X, ldx, rows, k, nrm, NW);
    __syncthreads();
    finish();
    if (left) {
      for (int e = tid; e < k * k; e += NT) {
        const double2 v = Y[(e % k) * ld + e / k];
        stc(A + (int64_t)rows * k + e, cmake(v.x, v.y));
      }
    } else {
      for (int e = tid; e < rows * k; e += NT) {
        const double2 v = X[(e % k) * ldx + e / k];
        stc(A + e, ex != 0 ? cmake(scalbn(v.x, ex), scalbn(v.y, ex)) : cmake(v.x, v.y));
      }
    }
    return;
  }
  __syncthreads();                                     // q1.nn[0] is overwritten from the second step on
  const double tol = fmax(8.0 * 2.220446049250313e-16, 4.0 * 2.220446049250313e-16 * sqrt((double)k));
  const double t2 = tol * tol;
  if (rows <= 64) js_qr<8, 8>(X, ldx, rows, k, q1, NW);
  else if (rows <= 128) js_qr<16, 8>(X, ldx, rows, k, q1, NW);
  else if (rows <= 256) js_qr<32, 8>(X, ldx, rows, k, q1, NW);
  else js_qr<32, 0>(X, ldx, rows, k, q1, NW);
  // L = R^H
  for (int e = tid; e < ld * k; e += NT) {
    const int c = e / ld, r = e - c * ld;
    double2 v = make_double2(0.0, 0.0);
    if (r < k && r >= c) v = r > c ? X[q1.piv[r] * ldx + c] : q1.rd[c];
    Y[e] = make_double2(v.x, -v.y);
  }
  __syncthreads();
  if (!left) {
    js_norms(Y, ld, k, k, q2.nn[0], NW);
    __syncthreads();
    js_qr<8, 8>(Y, ld, k, k, q2, NW);
    // L = R2^H, in place through registers
    constexpr int PER = (JS_KMAX * JS_KMAX + 511) / 512;
    double2 keep[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = tid + i * NT;
      keep[i] = make_double2(0.0, 0.0);
      if (e < k * k) {
        const int c = e / k, r = e - c * k;
        if (r >= c) keep[i] = r > c ? Y[q2.piv[r] * ld + c] : q2.rd[c];
      }
    }
    if (tid < k) inv2[q2.piv[tid]] = tid;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = tid + i * NT;
      if (e < k * k) {
        const int c = e / k, r = e - c * k;
        Y[c * ld + r] = make_double2(keep[i].x, -keep[i].y);
      }
    }
    __syncthreads();
  }
  const int jw = (k + (k & 1)) / 8 + ((k + (k & 1)) % 8 != 0);   // four pairs a warp
  if (k > 1 && warp < jw) {
    unsigned long long turned = 0;
    int sweeps;
    if (k <= 16) sweeps = js_sweeps<2>(Y, ld, k, z2, t2, max_sweeps, jw, rot, turned);
    else if (k <= 32) sweeps = js_sweeps<4>(Y, ld, k, z2, t2, max_sweeps, jw, rot, turned);
    else if (k <= 48) sweeps = js_sweeps<6>(Y, ld, k, z2, t2, max_sweeps, jw, rot, turned);
    else sweeps = js_sweeps<8>(Y, ld, k, z2, t2, max_sweeps, jw, rot, turned);
    if ((lane & 7) == 0 && turned) atomicAdd(executed, turned * 4ull * k);
    if (tid == 0) {
      if (sweeps > max_sweeps) *fail = 1;
      sweeps = min(sweeps, max_sweeps);
      atomicAdd(executed, (unsigned long long)sweeps * (unsigned)(k * (k - 1) / 2) * 2ull * k + (unsigned long long)k * k * rows);
      atomicMax(executed + 1, (unsigned long long)sweeps);
    }
  }
  __syncthreads();
  js_norms(Y, ld, k, k, nrm, NW);
  __syncthreads();
  finish();
  if (left) {
    // the left vectors, where the blocked form accumulates its rotations
    for (int e = tid; e < k * k; e += NT) {
      const int r = e / k, c = e - r * k;
      const double2 v = Y[c * ld + r];
      const double is = nrm[c] > 0.0 ? 1.0 / nrm[c] : 0.0;
      stc(A + (int64_t)(rows + q1.piv[r]) * k + c, cmake(v.x * is, v.y * is));
    }
    return;
  }
  if (ex != 0) {
    for (int e = tid; e < ld * k; e += NT) Y[e] = make_double2(scalbn(Y[e].x, ex), scalbn(Y[e].y, ex));
    __syncthreads();
  }
  auto y0 = [&](int c, int r) { return Y[c * ld + inv2[r]]; };
  if (rows <= 64) js_q_apply<8, 8>(X, ldx, rows, k, q1, A, NW, y0);
  else if (rows <= 128) js_q_apply<16, 8>(X, ldx, rows, k, q1, A, NW, y0);
  else if (rows <= 256) js_q_apply<32, 8>(X, ldx, rows, k, q1, A, NW, y0);
  else if (rows <= 512) js_q_apply<32, 16>(X, ldx, rows, k, q1, A, NW, y0);
  else js_q_apply<32, 32>(X, ldx, rows, k, q1, A, NW, y0);
}

}  // namespace

int jacobi_block_cols() { return JB; }

// The whole SVD in one CTA: where X and L fit in shared memory and a column of X in a warp's
// registers (16 or, in the form for 16 columns, 32 a lane).  The blocked form pays two
// launches of 45 to 60 us a round, three rounds a sweep at k = 64: 64 x 128 945 us and more,
// here 480 to 620; k = 28, 400 rows 315 and 200 to 350.
int jacobi_small_elems(int rows_g, int k) { return (js_ld(rows_g) + js_ldl(k)) * k; }
bool jacobi_is_small(int rows_g, int k) {
  return k <= JS_KMAX && rows_g <= (k <= 16 ? 1024 : 512) && (size_t)jacobi_small_elems(rows_g, k) * sizeof(double2) <= JS_SMEM;
}

cudaError_t launch_jacobi_small(const SectorDesc* sd_dev, const int* list_dev, int count, int max_elems, int max_k,
                                void* abuf, int max_sweeps, double* sig, int* perm, int* fail,
                                unsigned long long* executed, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  static const cudaError_t attr = [] {
    cudaError_t e = cudaFuncSetAttribute(jacobi_small_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, JS_SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(jacobi_small_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, JS_SMEM);
    return e;
  }();
  if (attr != cudaSuccess) return attr;
  const size_t smem = (size_t)max_elems * sizeof(double2);
  cplx* A = reinterpret_cast<cplx*>(abuf);
  if (max_k <= 16)
    jacobi_small_kernel<256><<<count, 256, smem, s>>>(sd_dev, list_dev, A, max_sweeps, sig, perm, fail, executed);
  else
    jacobi_small_kernel<512><<<count, 512, smem, s>>>(sd_dev, list_dev, A, max_sweeps, sig, perm, fail, executed);
  return cudaGetLastError();
}

cudaError_t launch_sector_norms(const SectorDesc* sd_dev, const int* list_dev, int count, const void* abuf,
                                double* nf2, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  sector_norm_kernel<<<count, NNT, 0, s>>>(sd_dev, list_dev, reinterpret_cast<const cplx*>(abuf), nf2);
  return cudaGetLastError();
}

cudaError_t launch_jacobi_round(const SectorDesc* sd_dev, const JacobiWork* work_dev, int n_work,
                                int gram_ctas, int apply_ctas, int t, void* abuf, int* rot_count,
                                const double* nf2, double tol, int max_sweeps, void* pbuf,
                                int* pcnt, void* qbuf, int* qflag, unsigned long long* executed,
                                cudaStream_t s) {
  if (gram_ctas <= 0) return cudaSuccess;
  const int smem1 = (int)sizeof(GramSmem);
  // once per process (thread-safe initialisation; several host threads launch rounds)
  static const cudaError_t attr = cudaFuncSetAttribute(
      jacobi_gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GramSmem));
  if (attr != cudaSuccess) return attr;
  jacobi_gram_kernel<<<gram_ctas, JNT, smem1, s>>>(
      sd_dev, work_dev, n_work, t, reinterpret_cast<const cplx*>(abuf), rot_count, nf2, tol,
      max_sweeps, reinterpret_cast<cplx*>(pbuf), pcnt, reinterpret_cast<cplx*>(qbuf), qflag, executed);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  jacobi_apply_kernel<<<apply_ctas, JNT, 0, s>>>(sd_dev, work_dev, n_work, t,
                                                 reinterpret_cast<cplx*>(abuf), max_sweeps,
                                                 reinterpret_cast<const cplx*>(qbuf), qflag, executed);
  return cudaGetLastError();
}

int jacobi_rows_per_part() { return RMAX; }

cudaError_t launch_jacobi_finish(const SectorDesc* sd_dev, const int* list_dev, int count, int max_k,
                                 const void* abuf, const double* nf2, double* sig, int* perm,
                                 cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  int np2 = 1;
  while (np2 < max_k) np2 <<= 1;
  const size_t smem = (size_t)np2 * (sizeof(double) + sizeof(int));
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(jacobi_finish_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  jacobi_finish_kernel<<<count, FNT, smem, s>>>(sd_dev, list_dev, reinterpret_cast<const cplx*>(abuf), nf2, sig, perm);
  return cudaGetLastError();
}
