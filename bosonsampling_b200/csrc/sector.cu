// Charge-sector kernels of the BS update: gate mix, top-chi selection, vector
// extraction and the scatter into the new site tensors.
//
// Block structure (the reference's, src/MPO.py:182-254 and src/mpo_sort.py): bond
// entries are sorted by (ket, bra) charge, so every charge block is a contiguous
// range; sector cc = (cc0, cc1) uses left blocks a >= cc and right blocks b <= cc.
// The contraction is split into Theta_q = Glc[a, q] Gcr[q, b] (one GEMM per valid
// charge triple, zgemm.cu) and this mix,
//     C_cc[a, b] = sum_q U(a0-cc0, cc0-b0, a0-q0) conj U(a1-cc1, cc1-b1, a1-q1) Theta_q[a, b],
// which is the reference's block product (src/MPO.py:254) with the sum over centre
// charges reassociated: each triple product is formed once instead of once per sector.
#include "common.cuh"
#include "kernels.h"

#include <algorithm>

namespace {

constexpr int MIX_NT = 256;

template <int MD>
__global__ __launch_bounds__(MIX_NT) void mix_kernel(const UpdateTables* __restrict__ tabs,
                                                     const int* __restrict__ tidxs,
                                                     const ThetaDesc* __restrict__ td,
                                                     const SectorDesc* __restrict__ sd,
                                                     const MixPair* __restrict__ pairs, int n_pairs,
                                                     const cplx* __restrict__ u3s,
                                                     const cplx* __restrict__ theta,
                                                     const double* __restrict__ lam_all,
                                                     cplx* __restrict__ cbuf,
                                                     cplx* __restrict__ abuf) {
  __shared__ MixPair P;
  __shared__ cplx u0s[MD][MD], u1s[MD][MD];
  __shared__ int64_t qbase[MD][MD];
  __shared__ int qld[MD][MD];
  __shared__ int64_t cb[MD][MD], ab[MD][MD];
  __shared__ int cn[MD][MD], ck[MD][MD], cleft[MD][MD], crow[MD][MD], ccol[MD][MD], crt[MD][MD];
  const int tid = threadIdx.x;
  if (tid == 0) {
    int lo = 0, hi = n_pairs - 1;
    const int t = blockIdx.x;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (pairs[mid].tile_start <= t) lo = mid; else hi = mid - 1;
    }
    P = pairs[lo];
  }
  __syncthreads();
  const UpdateTables* tab = tabs + P.upd;
  const int d = tab->d;
  const int* tidx = tidxs + (int64_t)P.upd * d * d * d * d;
  const cplx* u3 = u3s + tab->gate_off;
  const double* lam_r = lam_all + (int64_t)(tab->mode + 2) * tab->chi;
  const int D0 = P.a0 - P.b0 + 1, D1 = P.a1 - P.b1 + 1;
  // per-box tables: index i0 <-> charge b0 + i0, i1 <-> b1 + i1
  if (tid < MD * MD) {
    const int i0 = tid / MD, i1 = tid % MD;
    // u0s[ic][iq] = U[a0-cc0][cc0-b0][a0-q0] with cc0 = b0+ic, q0 = b0+iq (same for 1)
    if (i0 < D0 && i1 < D0) {
      const int n0 = (D0 - 1) - i0, m0 = i0, l0 = (D0 - 1) - i1;
      u0s[i0][i1] = u3[(n0 * d + m0) * d + l0];
    } else {
      u0s[i0][i1] = cmake(0.0, 0.0);
    }
    if (i0 < D1 && i1 < D1) {
      const int n1 = (D1 - 1) - i0, m1 = i0, l1 = (D1 - 1) - i1;
      u1s[i0][i1] = u3[(n1 * d + m1) * d + l1];
    } else {
      u1s[i0][i1] = cmake(0.0, 0.0);
    }
    // Theta source of centre charge q = (b0 + i0, b1 + i1)
    qbase[i0][i1] = -1;
    qld[i0][i1] = 0;
    if (i0 < D0 && i1 < D1) {
      const int q0 = P.b0 + i0, q1 = P.b1 + i1;
      const int ti = tidx[((q0 * d + q1) * d + P.a0) * d + P.b0];
      if (ti >= 0) {
        const ThetaDesc T = td[ti];
        // rows of group start at left block (a0, q1); columns at right block (b0, 0)
        const int lr0 = P.row0 - tab->offL[P.a0 * d + q1];
        const int lc0 = P.col0 - tab->offR[P.b0 * d];
        qbase[i0][i1] = T.off + (int64_t)lr0 * T.ncol + lc0;
        qld[i0][i1] = T.ncol;
      }
    }
    // destination sector cc = (b0 + i0, b1 + i1)
    cb[i0][i1] = -1;
    if (i0 < D0 && i1 < D1) {
      const int cc0 = P.b0 + i0, cc1 = P.b1 + i1;
      const int s = tab->sidx[cc0 * d + cc1];
      if (s >= 0) {
        const SectorDesc& S = sd[s];
        cb[i0][i1] = S.c_off;
        ab[i0][i1] = S.t_off;
        cn[i0][i1] = S.n;
        ck[i0][i1] = S.k;
        cleft[i0][i1] = S.left;
        crt[i0][i1] = S.rows_tot;
        crow[i0][i1] = S.row_start[P.a0] + (P.row0 - tab->offL[P.a0 * d + cc1]);
        ccol[i0][i1] = S.col_start[P.b0] + (P.col0 - tab->offR[P.b0 * d]);
      }
    }
  }
  __syncthreads();
  const int le = (blockIdx.x - P.tile_start) * MIX_NT + tid;
  if (le >= P.nrow * P.ncol) return;
  const int lr = le / P.ncol, lc = le % P.ncol;
  const double lam = lam_r[P.col0 + lc];

  cplx th[MD][MD];
#pragma unroll
  for (int i0 = 0; i0 < MD; ++i0)
#pragma unroll
    for (int i1 = 0; i1 < MD; ++i1) {
      th[i0][i1] = cmake(0.0, 0.0);
      if (i0 < D0 && i1 < D1 && qbase[i0][i1] >= 0)
        th[i0][i1] = ldc(theta + qbase[i0][i1] + (int64_t)lr * qld[i0][i1] + lc);
    }
  // X[c0][q1] = sum_q0 u0[c0][q0] th[q0][q1]
  cplx X[MD][MD];
#pragma unroll
  for (int c0 = 0; c0 < MD; ++c0)
#pragma unroll
    for (int q1 = 0; q1 < MD; ++q1) {
      cplx acc = cmake(0.0, 0.0);
#pragma unroll
      for (int q0 = 0; q0 < MD; ++q0) cfma(acc, u0s[c0][q0], th[q0][q1]);
      X[c0][q1] = acc;
    }
#pragma unroll
  for (int c0 = 0; c0 < MD; ++c0) {
    if (c0 >= D0) continue;
#pragma unroll
    for (int c1 = 0; c1 < MD; ++c1) {
      if (c1 >= D1 || cb[c0][c1] < 0) continue;
      cplx acc = cmake(0.0, 0.0);
#pragma unroll
      for (int q1 = 0; q1 < MD; ++q1) ccfma(acc, u1s[c1][q1], X[c0][q1]);
      const int row = crow[c0][c1] + lr, col = ccol[c0][c1] + lc;
      stc(cbuf + cb[c0][c1] + (int64_t)row * cn[c0][c1] + col, acc);
      if (!cleft[c0][c1]) {
        stc(abuf + ab[c0][c1] + (int64_t)row * ck[c0][c1] + col, cscale(acc, lam));
      } else {
        stc(abuf + ab[c0][c1] + (int64_t)col * ck[c0][c1] + row, cscale(cconj(acc), lam));
      }
    }
  }
}

__global__ void identity_rows_kernel(const SectorDesc* __restrict__ sd, const int* __restrict__ list,
                                     cplx* __restrict__ abuf) {
  const SectorDesc& S = sd[list[blockIdx.y]];
  if (!S.left || S.t_off != S.a_off) return;   // a preconditioned sector gets Y there
  const int m = S.m;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m * m; e += gridDim.x * blockDim.x) {
    const int i = e / m, j = e % m;
    stc(abuf + S.a_off + (int64_t)(S.n + i) * S.k + j, cmake(i == j ? 1.0 : 0.0, 0.0));
  }
}

// ------------------------------------------------------------------ selection
__device__ __forceinline__ int count_gt(const double* key, int k, double v) {
  // keys sorted descending: number of entries > v
  int lo = 0, hi = k;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (key[mid] > v) lo = mid + 1; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ int count_ge(const double* key, int k, double v) {
  int lo = 0, hi = k;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (key[mid] >= v) lo = mid + 1; else hi = mid;
  }
  return lo;
}

constexpr int SEL_NT = 512;
constexpr int SEL_CAP = 5120;   // candidates whose keys are kept in shared memory

// One CTA per update.  The chi-th largest key is found by radix selection (8 bits of the
// keys' bit patterns a pass; keys are not negative, so the patterns order like the values),
// counted in shared-memory integers, so the result does not depend on any order.  Bound by
// the passes' barriers.  Measured (25 sectors, 2,595
// candidates): 18 us; a bisection over the patterns with a thread per sector took 118.
__global__ __launch_bounds__(SEL_NT) void select_kernel(const UpdateTables* __restrict__ tabs,
                                                        SectorDesc* __restrict__ sds, int n_sectors,
                                                        const double* __restrict__ sig,
                                                        double* __restrict__ keys, double cutoff,
                                                        int chi, double pre_min, int* __restrict__ kept_all,
                                                        double* __restrict__ trunc_all) {
  __shared__ double skey[SEL_CAP];
  __shared__ double tws[BSMPO_MAX_Q], smax_s;
  __shared__ int ks[BSMPO_MAX_Q], pair_s[BSMPO_MAX_Q], gt_s[BSMPO_MAX_Q], kept_s[BSMPO_MAX_Q], cut_s[BSMPO_MAX_Q];
  __shared__ int64_t offs[BSMPO_MAX_Q];
  __shared__ int hist[256], ncand, digit, above, redo;
  const UpdateTables* tab = tabs + blockIdx.x;
  const int sec0 = tab->sec0, ns = tab->n_sectors;
  SectorDesc* sd = sds + sec0;
  int* kept_out = kept_all + sec0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < ns) {
    ks[tid] = sd[tid].k;
    offs[tid] = sd[tid].s_off;
    pair_s[tid] = tab->pair_of[tid] - sec0;   // own index of the swapped sector, negative: none
  }
  if (tid == 0) ncand = redo = 0;
  __syncthreads();
  const int64_t off0 = offs[0];
  const int total = (int)(offs[ns - 1] + ks[ns - 1] - off0);
  double* const key = total <= SEL_CAP ? skey : keys + off0;   // sector s: key + offs[s] - off0
  if (warp == 0) {
    // largest singular value of the update
    double m = 0.0;
    for (int s = lane; s < ns; s += 32) m = fmax(m, ks[s] > 0 ? sig[offs[s]] : 0.0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) smax_s = m;
  }
  // keys: singular values made equal within ket/bra-swapped sector pairs
  for (int s = warp; s < ns; s += SEL_NT / 32) {
    const int p = pair_s[s], k = ks[s], kp = p >= 0 && p != s ? ks[p] : 0;
    for (int i = lane; i < k; i += 32) {
      double v = sig[offs[s] + i];
      if (i < kp) v = fmax(v, sig[offs[p] + i]);
      key[offs[s] - off0 + i] = v;
    }
  }
  __syncthreads();
  const double smax = smax_s, thr = fmax(cutoff * smax, 0.0);
  const bool own = tid < ns;
  const int k = own ? ks[tid] : 0;
  const double* kown = key + (own ? offs[tid] - off0 : 0);
  int kept = own ? count_gt(kown, k, thr) : 0;
  if (own) atomicAdd(&ncand, kept);
  __syncthreads();
  if (ncand > chi) {   // uniform
    // v* = chi-th largest candidate key
    unsigned long long prefix = 0;
    int want = chi;                      // its rank among the keys that share the prefix
    for (int shift = 56; shift >= 0; shift -= 8) {
      for (int b = tid; b < 256; b += SEL_NT) hist[b] = 0;
      __syncthreads();
      for (int i = tid; i < total; i += SEL_NT) {
        const double v = key[i];
        const unsigned long long u = (unsigned long long)__double_as_longlong(v);
        if (v > thr && (shift == 56 || (u >> (shift + 8)) == prefix)) atomicAdd(&hist[(u >> shift) & 255], 1);
      }
      __syncthreads();
      if (warp == 0) {
        // lane l sums the bins 255 - 8 l .. 248 - 8 l; the digit is where the count from
        // above reaches `want`
        int c = 0;
        for (int b = 0; b < 8; ++b) c += hist[255 - 8 * lane - b];
        int upto = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += y;
        }
        const int first = __ffs(__ballot_sync(0xffffffffu, upto >= want)) - 1;
        if (lane == first) {
          int before = upto - c, b = 255 - 8 * lane;
          while (before + hist[b] < want) before += hist[b--];
          digit = b;
          above = before;
        }
      }
      __syncthreads();
      prefix = (prefix << 8) | (unsigned)digit;
      want -= above;
    }
    const double vstar = __longlong_as_double((long long)prefix);
    if (own) {
      const int gt = count_gt(kown, k, vstar);
      gt_s[tid] = gt;
      kept_s[tid] = count_ge(kown, k, vstar) - gt;   // tied entries
    }
    __syncthreads();
    if (tid == 0) {
      // ties by sector order
      int need = chi;
      for (int i = 0; i < ns; ++i) need -= gt_s[i];
      for (int i = 0; i < ns; ++i) {
        const int take = min(kept_s[i], max(need, 0));
        kept_s[i] = take;
        need -= take;
      }
    }
    __syncthreads();
    if (own) kept = gt_s[tid] + kept_s[tid];
  }
  // a kept vector needs its own singular value > 0 (the key may come from the partner)
  if (own) {
    kept = min(kept, count_gt(sig + offs[tid], k, 0.0));
    cut_s[tid] = kept;
  }
  __syncthreads();
  // a cut inside a degenerate swapped pair keeps neither member
  if (own) {
    const int p = pair_s[tid];
    kept_s[tid] = p >= 0 && p != tid ? min(kept, cut_s[p]) : kept;
  }
  __syncthreads();
  // truncation weight: discarded sigma^2, a warp per sector, then in sector order
  for (int s = warp; s < ns; s += SEL_NT / 32) {
    double tw = 0.0;
    for (int i = kept_s[s] + lane; i < ks[s]; i += 32) {
      const double v = sig[offs[s] + i];
      tw += v * v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tw += __shfl_xor_sync(0xffffffffu, tw, o);
    if (lane == 0) tws[s] = tw;
  }
  __syncthreads();
  if (own) {
    int slot = 0;
    for (int i = 0; i < tid; ++i) slot += kept_s[i];
    // a preconditioned sector (not flagged to start from X) that keeps too small a value
    const double* v = sig + offs[tid];
    if (sd[tid].t_off != sd[tid].a_off && sd[tid].kept >= 0 && kept_s[tid] > 0 && v[kept_s[tid] - 1] < pre_min * v[0])
      redo = 1;
    sd[tid].kept = kept_s[tid];
    sd[tid].slot0 = slot;
    kept_out[tid] = kept_s[tid];
    if (tid == ns - 1) kept_all[n_sectors + blockIdx.x] = slot + kept_s[tid];
  }
  __syncthreads();
  if (tid == 0) {
    kept_all[n_sectors + gridDim.x + blockIdx.x] = redo;
    double tw = 0.0;
    for (int i = 0; i < ns; ++i) tw += tws[i];
    trunc_all[blockIdx.x] = tw;
  }
}

// conj-free V[l][t] (row-major [m][kept]) for the kept vectors of each sector
__global__ void extract_v_kernel(const SectorDesc* __restrict__ sd, const cplx* __restrict__ abuf,
                                 const double* __restrict__ sig, const int* __restrict__ perm,
                                 cplx* __restrict__ vbuf) {
  const SectorDesc& S = sd[blockIdx.y];
  const int kept = S.kept, m = S.m;
  const int total = kept * m;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    const int l = e / kept, t = e % kept;
    const int col = perm[S.s_off + t];
    cplx v;
    if (!S.left) {
      v = cscale(ldc(abuf + S.a_off + (int64_t)l * S.k + col), 1.0 / sig[S.s_off + t]);
    } else {
      v = ldc(abuf + S.a_off + (int64_t)(S.n + l) * S.k + col);
    }
    stc(vbuf + S.v_off + (int64_t)l * kept + t, v);
  }
}

constexpr int SC_NT = 256;

__global__ __launch_bounds__(SC_NT) void scatter_kernel(const UpdateTables* __restrict__ tabs,
                                                        const SectorDesc* __restrict__ sds,
                                                        const int* __restrict__ totals,
                                                        const int* __restrict__ err,
                                                        const cplx* __restrict__ vbuf,
                                                        const cplx* __restrict__ wbuf,
                                                        const double* __restrict__ sig,
                                                        cplx* __restrict__ gamma,
                                                        double* __restrict__ lam,
                                                        int2* __restrict__ charge) {
  // a failed group, or an update to be done again, leaves the state as it is
  if (err[0] != 0 || err[1] != 0 || totals[gridDim.y + blockIdx.y] != 0) return;
  const UpdateTables* tab = tabs + blockIdx.y;
  const SectorDesc* sd = sds + tab->sec0;
  const int ns = tab->n_sectors, total_kept = totals[blockIdx.y];
  const int64_t site = (int64_t)tab->chi * tab->chi;
  cplx* gamma_l = gamma + tab->mode * site;
  cplx* gamma_r = gamma_l + site;
  const int2* charge_l = charge + (int64_t)tab->mode * tab->chi;
  int2* charge_c = charge + (int64_t)(tab->mode + 1) * tab->chi;
  const int2* charge_r = charge + (int64_t)(tab->mode + 2) * tab->chi;
  double* lam_c = lam + (int64_t)(tab->mode + 1) * tab->chi;
  __shared__ int slot0[BSMPO_MAX_Q + 1];
  __shared__ SectorDesc S[BSMPO_MAX_Q];
  const int tid = threadIdx.x;
  const int d = tab->d, chi = tab->chi;
  for (int i = tid; i < ns; i += SC_NT) {
    S[i] = sd[i];
    slot0[i] = sd[i].slot0;
  }
  if (tid == 0) slot0[ns] = total_kept;
  __syncthreads();
  const int64_t chi2 = (int64_t)chi * chi;
  for (int64_t e = (int64_t)blockIdx.x * SC_NT + tid; e < 2 * chi2 + chi;
       e += (int64_t)gridDim.x * SC_NT) {
    int j, other;
    bool is_l = e < chi2, is_r = !is_l && e < 2 * chi2;
    if (is_l) { other = (int)(e / chi); j = (int)(e % chi); }
    else if (is_r) { j = (int)((e - chi2) / chi); other = (int)((e - chi2) % chi); }
    else { j = (int)(e - 2 * chi2); other = 0; }
    int s = -1, t = 0;
    if (j < total_kept) {
      int lo = 0, hi = ns - 1;
      while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (slot0[mid] <= j) lo = mid; else hi = mid - 1;
      }
      // skip sectors with zero kept vectors sharing the same slot0
      while (lo + 1 < ns && slot0[lo + 1] <= j) ++lo;
      s = lo;
      t = j - slot0[s];
    }
    if (is_l) {
      cplx v = cmake(0.0, 0.0);
      if (s >= 0) {
        const int2 c = charge_l[other];
        const SectorDesc& D = S[s];
        if (c.x < d && c.x >= D.cc0 && c.y >= D.cc1) {
          const int p = D.row_start[c.x] + (other - tab->offL[c.x * d + D.cc1]);
          v = ldc(vbuf + D.v_off + (int64_t)p * D.kept + t);
        }
      }
      stc(gamma_l + e, v);
    } else if (is_r) {
      cplx v = cmake(0.0, 0.0);
      if (s >= 0) {
        const int2 c = charge_r[other];
        const SectorDesc& D = S[s];
        if (c.x < d && c.x <= D.cc0 && c.y <= D.cc1) {
          const int p = D.col_start[c.x] + (other - tab->offR[c.x * d]);
          v = ldc(wbuf + D.w_off + (int64_t)t * D.n + p);
        }
      }
      stc(gamma_r + (e - chi2), v);
    } else {
      if (s >= 0) {
        lam_c[j] = sig[S[s].s_off + t];
        charge_c[j] = make_int2(S[s].cc0, S[s].cc1);
      } else {
        lam_c[j] = 0.0;
        charge_c[j] = make_int2(d, d);
      }
    }
  }
}

__global__ void phase_kernel(int d, int chi, double phi, const int2* __restrict__ cl,
                             const int2* __restrict__ cr, cplx* __restrict__ g) {
  const int64_t chi2 = (int64_t)chi * chi;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < chi2;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int a = (int)(e / chi), j = (int)(e % chi);
    const int2 x = cl[a], y = cr[j];
    if (x.x >= d || y.x >= d) continue;
    const int dn = (x.x - y.x) - (x.y - y.y);
    if (dn == 0) continue;
    double sn, cs;
    sincos(phi * (double)dn, &sn, &cs);
    stc(g + e, cmul(ldc(g + e), cmake(cs, sn)));
  }
}

}  // namespace

cudaError_t launch_mix_d(int d, const UpdateTables* tab_dev, const int* tidx_dev,
                         const ThetaDesc* td_dev, const SectorDesc* sd_dev,
                         const MixPair* pairs_dev, int n_pairs, int total_tiles, const void* u3,
                         const void* theta, const double* lam, void* cbuf, void* abuf,
                         cudaStream_t s) {
  if (total_tiles <= 0) return cudaSuccess;
  const cplx* U = reinterpret_cast<const cplx*>(u3);
  const cplx* T = reinterpret_cast<const cplx*>(theta);
  cplx* C = reinterpret_cast<cplx*>(cbuf);
  cplx* A = reinterpret_cast<cplx*>(abuf);
#define BSMPO_MIX(MD)                                                                        \
  mix_kernel<MD><<<total_tiles, MIX_NT, 0, s>>>(tab_dev, tidx_dev, td_dev, sd_dev, pairs_dev, \
                                                n_pairs, U, T, lam, C, A)
  switch (d) {
    case 1: case 2: BSMPO_MIX(2); break;
    case 3: BSMPO_MIX(3); break;
    case 4: BSMPO_MIX(4); break;
    case 5: BSMPO_MIX(5); break;
    case 6: BSMPO_MIX(6); break;
    default: BSMPO_MIX(8); break;
  }
#undef BSMPO_MIX
  return cudaGetLastError();
}

cudaError_t launch_identity_rows(const SectorDesc* sd_dev, const int* list_dev, int count, int max_elems,
                                 void* abuf, cudaStream_t s) {
  if (count <= 0 || max_elems <= 0) return cudaSuccess;
  dim3 grid(min(ceil_div(max_elems, 256), 1024), count);
  identity_rows_kernel<<<grid, 256, 0, s>>>(sd_dev, list_dev, reinterpret_cast<cplx*>(abuf));
  return cudaGetLastError();
}

cudaError_t launch_select(const UpdateTables* tab_dev, SectorDesc* sd_dev, int n_updates, int n_sectors,
                          const double* sig, double* keys, double cutoff, int chi, double pre_min, int* kept_out,
                          double* trunc_out, cudaStream_t s) {
  if (n_updates <= 0) return cudaSuccess;
  select_kernel<<<n_updates, SEL_NT, 0, s>>>(tab_dev, sd_dev, n_sectors, sig, keys, cutoff, chi, pre_min, kept_out,
                                             trunc_out);
  return cudaGetLastError();
}

cudaError_t launch_extract_v(const SectorDesc* sd_dev, int n_sectors, int max_elems,
                             const void* abuf, const double* sig, const int* perm, void* vbuf,
                             cudaStream_t s) {
  if (n_sectors <= 0 || max_elems <= 0) return cudaSuccess;
  dim3 grid(min(ceil_div(max_elems, 256), 1024), n_sectors);
  extract_v_kernel<<<grid, 256, 0, s>>>(sd_dev, reinterpret_cast<const cplx*>(abuf), sig, perm,
                                        reinterpret_cast<cplx*>(vbuf));
  return cudaGetLastError();
}

cudaError_t launch_scatter(const UpdateTables* tab_dev, const SectorDesc* sd_dev, int n_updates,
                           const int* totals, const int* err, int chi, const void* vbuf, const void* wbuf,
                           const double* sig, void* gamma, double* lam, int* charge, cudaStream_t s) {
  if (n_updates <= 0) return cudaSuccess;
  const int64_t total = 2 * (int64_t)chi * chi + chi;
  const int blocks = (int)std::min<int64_t>((total + SC_NT - 1) / SC_NT, 148 * 16);
  scatter_kernel<<<dim3(blocks, n_updates), SC_NT, 0, s>>>(
      tab_dev, sd_dev, totals, err, reinterpret_cast<const cplx*>(vbuf), reinterpret_cast<const cplx*>(wbuf), sig,
      reinterpret_cast<cplx*>(gamma), lam, reinterpret_cast<int2*>(charge));
  return cudaGetLastError();
}

cudaError_t launch_phase(int d, int chi, double phi, const int* charge_l, const int* charge_r,
                         void* gamma, cudaStream_t s) {
  const int64_t total = (int64_t)chi * chi;
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 8);
  phase_kernel<<<blocks, 256, 0, s>>>(d, chi, phi, reinterpret_cast<const int2*>(charge_l),
                                      reinterpret_cast<const int2*>(charge_r),
                                      reinterpret_cast<cplx*>(gamma));
  return cudaGetLastError();
}
