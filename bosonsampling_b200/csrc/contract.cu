// Standalone single-sector contraction: the drop-in for cuda_kernels.update_MPO
// (src/cuda_kernels.py:101-127) and its kernel (src/update_MPO_kernel.cu:193-733).
//
//   C[l][r] = sum_c Glc[l][c] Gcr[c][r] U(cl0-cc0, cc0-cr0, cl0-q0(c)) conj U(cl1-cc1, cc1-cr1, cl1-q1(c))
//
// with each charge taken per row / column / centre entry (so no x8 alignment
// padding or centre-charge change list is needed) and the term zero unless every U
// index lies in [0, d).  The whole-BS path (bsmpo_bs_update) does not use these kernels; it
// contracts charge blocks as GEMMs instead.
//
// The weight depends on the centre entry through its charge only.  So the centre entries are
// taken in runs of equal charge (any order of the entries is allowed; a window of them with more
// runs than there are charges is put in an order by charge first, stably): a run's plain
// products are accumulated on the FP64 tensor path (m8n8k4),
// and at its end each output adds its weight times the run's sum.  A run that no row and
// column of the tile can use is not read.  What bounds it: the FP64 tensor rate of the SM with
// the most tiles, so they are small (32 x 16, 4 warps): a sector of 443 x 389 is 350 CTAs.
// Measured there with 1,024 centre entries, d = 5: the kernel 74 us, the call with its wait 162
// us, 116 among others.  When the tiles were chosen, calls with their wait, 32 x 16 and 32 x
// 32 tiles (182 CTAs): 188 and 206 us; 700 x 1,024 x 300: 180 and 202; 1,500 x 1,024 x 1,400: 411
// and 411 (16 x 16 tiles with the weight applied per entry: the kernel alone 270 at the first).
// Entries in random order, calls with their wait, most of it the expansion of the change list on
// the host: 443 x 1,024 x 389 1,226 us, 2,222 with every entry a run of its own, 1,313 with the
// weight applied per entry.  The grouping's tables lie in the stages and the run list: 3 KB of
// shared memory more cost entries in order 2%.
#include "dmma.cuh"
#include "kernels.h"

namespace {

static_assert(BSMPO_MAX_D <= 1 << 10, "charges are far below the sentinel");
constexpr int CT = 32, CN = 16, CK = 8, CNT = 128, CSTAGES = 3;   // rows, columns, centre entries
constexpr int NJ = CN / 16;                // 8-column tiles of a warp
constexpr int CWIN = 1024;                 // centre entries whose runs are listed at once
constexpr int CLDA = CK + 4, CLDB = CN + 2;
constexpr int CSTAGE = CT * CLDA + CK * CLDB;

// (a, b) >= (x, y) in both components
__device__ __forceinline__ bool ge2(int2 a, int2 b) { return a.x >= b.x && a.y >= b.y; }

// The product of one tile over the centre entries, run by run: fold(q) is called with the
// run's first centre index once re / im hold its sum.  use is called by whole warps.
// code(i): entry i's charge as a number below CODES.
constexpr int CODES = BSMPO_MAX_Q + 1;
template <typename Same, typename Code, typename Use, typename Fold>
__device__ __forceinline__ void run_products(const cplx* __restrict__ glc, const cplx* __restrict__ gcr, int len_l,
                                             int len_c, int len_r, int most_runs, double2* smem, int* runs, double2 (&re)[2][NJ],
                                             double2 (&im)[2][NJ], Same same, Code code, Use use,
                                             Fold fold) {
  __shared__ int wsum[CNT / 32], n_runs;
  // to group a window: counts in the stages, and its entries by position behind its few runs
  int *at_code = reinterpret_cast<int*>(smem), (*in_warp)[CODES] = reinterpret_cast<int(*)[CODES]>(at_code + CODES);
  unsigned short* order = reinterpret_cast<unsigned short*>(runs + CWIN / 2);
  static_assert(CODES <= CWIN / 2 && (CNT / 32 + 1) * CODES * sizeof(int) <= CSTAGE * sizeof(double2), "no room");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.y * CT, n0 = blockIdx.x * CN;
  const int wm = (warp >> 1) * 16, wn = (warp & 1) * (CN / 2), li = lane >> 2, lk = lane & 3;
  for (int w0 = 0; w0 < len_c; w0 += CWIN) {
    const int w1 = min(w0 + CWIN, len_c);
    // starts of the window's runs, in order
    if (tid == 0) n_runs = 0;
    __syncthreads();
    for (int i0 = w0; i0 < w1; i0 += CNT) {
      const int i = i0 + tid;
      const bool start = i < w1 && (i == w0 || !same(i - 1, i));
      const unsigned m = __ballot_sync(0xffffffffu, start);
      if (lane == 0) wsum[warp] = __popc(m);
      __syncthreads();
      int at = n_runs + __popc(m & ((1u << lane) - 1));
      for (int w = 0; w < warp; ++w) at += wsum[w];
      if (start) runs[at] = i;
      __syncthreads();
      if (tid == 0)
        for (int w = 0; w < CNT / 32; ++w) n_runs += wsum[w];
      __syncthreads();
    }
    const bool grouped = n_runs > most_runs;   // uniform
    if (grouped) {
      for (int c = tid; c < CODES; c += CNT) at_code[c] = 0;
      for (int c = tid; c < CNT / 32 * CODES; c += CNT) in_warp[0][c] = 0;
      __syncthreads();
      for (int i = w0 + tid; i < w1; i += CNT) atomicAdd(&at_code[code(i)], 1);
      __syncthreads();
      if (tid == 0) {
        int at = 0, n = 0;
        for (int c = 0; c < CODES; ++c) {
          const int len = at_code[c];
          at_code[c] = at;
          if (len > 0) runs[n++] = w0 + at;
          at += len;
        }
        n_runs = n;
      }
      __syncthreads();
      for (int i0 = w0; i0 < w1; i0 += CNT) {
        // an entry's place: behind those of its code in the chunks, warps and lanes before it
        const int i = i0 + tid, c = i < w1 ? code(i) : CODES;
        const unsigned m = __match_any_sync(0xffffffffu, c), before = m & ((1u << lane) - 1);
        if (i < w1 && before == 0) in_warp[warp][c] = __popc(m);
        __syncthreads();
        if (i < w1) {
          int at = at_code[c] + __popc(before);
          for (int w = 0; w < warp; ++w) at += in_warp[w][c];
          order[at] = (unsigned short)(i - w0);
        }
        __syncthreads();
        for (int x = tid; x < CODES; x += CNT)
          for (int w = 0; w < CNT / 32; ++w) {
            at_code[x] += in_warp[w][x];
            in_warp[w][x] = 0;
          }
        __syncthreads();
      }
    }
    const int nr = n_runs;
    auto products = [&](auto entry) {   // entry at position i of the window
      // slabs of CK entries within a run, over the window's used runs; (run, k) walk in
      // step for the fills and the products
      auto end_of = [&](int r) { return r + 1 < nr ? runs[r + 1] : w1; };
      auto next_used = [&](int r) {
        while (r < nr && !use(entry(runs[r]))) ++r;
        return r;
      };
      int fr = next_used(0), fk = fr < nr ? runs[fr] : 0;   // next slab to fill
      auto fill = [&](int s) {
        if (fr >= nr) return;
        const int end = end_of(fr);
        double2 *as = smem + s * CSTAGE, *bs = as + CT * CLDA;
#pragma unroll
        for (int i = 0; i < CT * CK / CNT; ++i) {
          const int e = tid + i * CNT, m = e / CK, k = e % CK;
          const bool ok = m0 + m < len_l && fk + k < end;
          cp_async16(as + m * CLDA + k, ok ? glc + (int64_t)(m0 + m) * len_c + entry(fk + k) : glc, ok);
        }
#pragma unroll
        for (int i = 0; i < CN * CK / CNT; ++i) {
          const int e = tid + i * CNT, k = e / CN, n = e % CN;
          const bool ok = n0 + n < len_r && fk + k < end;
          cp_async16(bs + k * CLDB + n, ok ? gcr + (int64_t)entry(fk + k) * len_r + n0 + n : gcr, ok);
        }
        fk += CK;
        if (fk >= end) {
          fr = next_used(fr + 1);
          if (fr < nr) fk = runs[fr];
        }
      };
      int cr = fr, ck = fk;                                 // next slab to multiply
#pragma unroll
      for (int s = 0; s < CSTAGES - 1; ++s) {
        fill(s);
        cp_async_commit();
      }
      for (int t = 0; cr < nr; ++t) {
        cp_async_wait<CSTAGES - 2>();
        __syncthreads();
        fill((t + CSTAGES - 1) % CSTAGES);
        cp_async_commit();
        const double2 *as = smem + (t % CSTAGES) * CSTAGE, *bs = as + CT * CLDA;
        cmma_tile<2, NJ, CK / 4, false>(
            re, im, [&](int i, int k) { return as[(wm + 8 * i + li) * CLDA + k + lk]; },
            [&](int j, int k) { return bs[(k + lk) * CLDB + wn + 8 * j + li]; });
        ck += CK;
        if (ck >= end_of(cr)) {
          fold(entry(runs[cr]));
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) re[i][j] = im[i][j] = make_double2(0.0, 0.0);
          cr = next_used(cr + 1);
          if (cr < nr) ck = runs[cr];
        }
      }
    };
    if (grouped) products([&](int i) { return w0 + order[i - w0]; });
    else products([](int i) { return i; });
    __syncthreads();   // the stages and the run list are free for the next window
  }
}

// this lane's outputs of the tile: row of (i), column of (j, x)
struct TileLane {
  int row0, col0;
  __device__ TileLane() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    row0 = blockIdx.y * CT + (warp >> 1) * 16 + (lane >> 2);
    col0 = blockIdx.x * CN + (warp & 1) * (CN / 2) + 2 * (lane & 3);
  }
  __device__ int row(int i) const { return row0 + 8 * i; }
  __device__ int col(int j, int x) const { return col0 + 8 * j + x; }
};

__global__ __launch_bounds__(CNT) void contract_sector_kernel(int d, int cc0, int cc1, const cplx* __restrict__ u,
                                                              const cplx* __restrict__ glc, const cplx* __restrict__ gcr,
                                                              const int2* __restrict__ cl, const int2* __restrict__ cc,
                                                              const int2* __restrict__ cr, int len_l, int len_c, int len_r,
                                                              cplx* __restrict__ out) {
  __shared__ __align__(16) double2 smem[CSTAGES * CSTAGE];
  __shared__ cplx us[BSMPO_MAX_D * BSMPO_MAX_D * BSMPO_MAX_D];
  __shared__ int2 rows[CT], cols[CN];
  __shared__ int runs[CWIN];
  const int tid = threadIdx.x, d3 = d * d * d;
  for (int i = tid; i < d3; i += CNT) us[i] = u[i];
  // charges of the tile's rows and columns; (-1, -1) / (BIG, BIG): contributes nothing
  constexpr int BIG = 1 << 20;
  if (tid < CT) {
    const int l = blockIdx.y * CT + tid;
    const int2 a = l < len_l ? cl[l] : make_int2(d, d);
    rows[tid] = a.x < d && a.y < d && a.x >= cc0 && a.y >= cc1 ? a : make_int2(-1, -1);
  } else if (tid < CT + CN) {
    const int r = blockIdx.x * CN + tid - CT;
    const int2 b = r < len_r ? cr[r] : make_int2(d, d);
    cols[tid - CT] = b.x >= 0 && b.y >= 0 && b.x <= cc0 && b.y <= cc1 ? b : make_int2(BIG, BIG);
  }
  __syncthreads();
  const TileLane T;
  int2 a[2], b[NJ][2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    a[i] = rows[T.row(i) - blockIdx.y * CT];
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    b[j][0] = cols[T.col(j, 0) - blockIdx.x * CN];
    b[j][1] = cols[T.col(j, 1) - blockIdx.x * CN];
  }
  double2 re[2][NJ], im[2][NJ];
  cplx acc[2][NJ][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      re[i][j] = im[i][j] = make_double2(0.0, 0.0);
      acc[i][j][0] = acc[i][j][1] = cmake(0.0, 0.0);
    }
  run_products(
      glc, gcr, len_l, len_c, len_r, d * d + 1, smem, runs, re, im,
      [&](int i, int j) { return cc[i].x == cc[j].x && cc[i].y == cc[j].y; },
      [&](int i) { return cc[i].x < 0 || cc[i].y < 0 || cc[i].x >= d || cc[i].y >= d ? CODES - 1 : cc[i].x * d + cc[i].y; },
      [&](int i) {
        const int2 q = cc[i];
        if (q.x < 0 || q.y < 0 || q.x >= d || q.y >= d) return false;
        const int t = threadIdx.x & 31;   // a lane to a row and a column of the tile
        const bool r = __any_sync(0xffffffffu, ge2(rows[t], q)), c = __any_sync(0xffffffffu, ge2(q, cols[t % CN]));
        return r && c;
      },
      [&](int i0) {
        const int2 q = cc[i0];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (!ge2(a[i], q)) continue;
#pragma unroll
          for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int2 c = b[j][x];
              if (!ge2(q, c)) continue;
              const cplx u0 = us[((a[i].x - cc0) * d + (cc0 - c.x)) * d + (a[i].x - q.x)];
              const cplx u1 = us[((a[i].y - cc1) * d + (cc1 - c.y)) * d + (a[i].y - q.y)];
              cfma(acc[i][j][x], cmulc(u0, u1),
                   x ? cmake(re[i][j].y, im[i][j].y) : cmake(re[i][j].x, im[i][j].x));
            }
        }
      });
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (T.row(i) < len_l && T.col(j, x) < len_r) stc(out + (int64_t)T.row(i) * len_r + T.col(j, x), acc[i][j][x]);
}

// The pure-state (MPS) variant: the drop-in for cuda_kernels.update_MPS
// (src/cuda_kernels.py:72-90) and its kernel (src/update_kernel.cu:193-769), one charge
// per bond index:
//   T[l][r] = LL[l] LR[r] sum_c LC[c] Glc[l][c] Gcr[c][r] U(cl - tau, tau - cr, cl - q(c)),
// the term zero unless cl >= q(c) >= cr and every U index lies in [0, d).  The reference
// reloads LC in tiles of 256 centre indices and, on its last partial tile, from offset 0
// (src/update_kernel.cu:632-638) -- a quirk for k > 256; here LC[c] is read per index.
constexpr int MT = 16;
__global__ void contract_mps_kernel(int d, int tau, const cplx* __restrict__ u,
                                    const cplx* __restrict__ glc, const cplx* __restrict__ gcr,
                                    const double* __restrict__ ll, const double* __restrict__ lc,
                                    const double* __restrict__ lr, const int* __restrict__ cl,
                                    const int* __restrict__ cc, const int* __restrict__ cr, int len_l,
                                    int len_c, int len_r, cplx* __restrict__ out) {
  __shared__ cplx us[BSMPO_MAX_D * BSMPO_MAX_D * BSMPO_MAX_D];
  __shared__ cplx ga[MT][MT + 1], gb[MT][MT + 1];
  __shared__ int qc[MT];
  __shared__ double lcs[MT];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * MT + tx;
  const int d3 = d * d * d;
  for (int i = tid; i < d3; i += MT * MT) us[i] = u[i];
  const int l = blockIdx.y * MT + ty, r = blockIdx.x * MT + tx;
  const int a = l < len_l ? cl[l] : -1;
  const int b = r < len_r ? cr[r] : -1;
  const bool ok = a >= 0 && b >= 0 && a - tau >= 0 && a - tau < d && tau - b >= 0 && tau - b < d;
  cplx acc = cmake(0.0, 0.0);
  for (int c0 = 0; c0 < len_c; c0 += MT) {
    __syncthreads();
    {
      const int lrow = blockIdx.y * MT + ty, ccol = c0 + tx;
      ga[ty][tx] = (lrow < len_l && ccol < len_c) ? ldc(glc + (int64_t)lrow * len_c + ccol) : cmake(0.0, 0.0);
      const int crow = c0 + ty, rc = blockIdx.x * MT + tx;
      gb[ty][tx] = (crow < len_c && rc < len_r) ? ldc(gcr + (int64_t)crow * len_r + rc) : cmake(0.0, 0.0);
      if (ty == 0) {
        qc[tx] = (c0 + tx < len_c) ? cc[c0 + tx] : -1;
        lcs[tx] = (c0 + tx < len_c) ? lc[c0 + tx] : 0.0;
      }
    }
    __syncthreads();
    if (!ok) continue;
    for (int j = 0; j < MT; ++j) {
      const int q = qc[j];
      if (q < 0 || !(a >= q && q >= b) || a - q >= d) continue;
      const cplx w = cscale(us[((a - tau) * d + (tau - b)) * d + (a - q)], lcs[j]);
      cfma(acc, w, cmul(ga[ty][j], gb[j][tx]));
    }
  }
  if (l < len_l && r < len_r) out[(int64_t)l * len_r + r] = ok ? cscale(acc, ll[l] * lr[r]) : cmake(0.0, 0.0);
}

}  // namespace

cudaError_t launch_contract_mps(int d, int tau, const void* u, const void* glc, const void* gcr,
                                const double* ll, const double* lc, const double* lr, const int* cl,
                                const int* cc, const int* cr, int len_l, int len_c, int len_r, void* t,
                                cudaStream_t s) {
  if (len_l <= 0 || len_r <= 0) return cudaSuccess;
  dim3 grid(ceil_div(len_r, MT), ceil_div(len_l, MT));
  dim3 block(MT, MT);
  contract_mps_kernel<<<grid, block, 0, s>>>(d, tau, reinterpret_cast<const cplx*>(u),
                                             reinterpret_cast<const cplx*>(glc), reinterpret_cast<const cplx*>(gcr),
                                             ll, lc, lr, cl, cc, cr, len_l, len_c, len_r, reinterpret_cast<cplx*>(t));
  return cudaGetLastError();
}

cudaError_t launch_contract_sector(int d, int cc0, int cc1, const void* u, const void* glc,
                                   const void* gcr, const int* cl, const int* cc, const int* cr,
                                   int len_l, int len_c, int len_r, void* c, cudaStream_t s) {
  if (len_l <= 0 || len_r <= 0) return cudaSuccess;
  dim3 grid(ceil_div(len_r, CN), ceil_div(len_l, CT));
  contract_sector_kernel<<<grid, CNT, 0, s>>>(
      d, cc0, cc1, reinterpret_cast<const cplx*>(u), reinterpret_cast<const cplx*>(glc),
      reinterpret_cast<const cplx*>(gcr), reinterpret_cast<const int2*>(cl),
      reinterpret_cast<const int2*>(cc), reinterpret_cast<const int2*>(cr), len_l, len_c, len_r,
      reinterpret_cast<cplx*>(c));
  return cudaGetLastError();
}
