// Internal launch interface of libbsmpo's kernels (host side, C++).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/bsmpo.h"

// Message returned by bsmpo_last_error(NULL) (capi.cu).
void set_global_error(const char* msg);

// Largest local cutoff d supported (charge tables are d x d).
#define BSMPO_MAX_D 8
#define BSMPO_MAX_Q (BSMPO_MAX_D * BSMPO_MAX_D)

// ---------------------------------------------------------------- fock.cu
cudaError_t launch_fock_tensor(int d, int n_gates, const double* m4_dev, void* u_dev,
                               cudaStream_t s);
// One gate with M passed by value; writes interleaved complex (u_im == nullptr) or
// split real / imaginary double arrays.
struct M8 { double v[8]; };
// dL/dtheta, dL/dphi of every gate T(theta, phi) from the gradient of its tensor: m4 and
// dm4 (device) hold per gate M (8 doubles) and dM/dtheta, dM/dphi (16 doubles); grad gets
// 2 doubles per gate.
cudaError_t launch_fock_angle_grad(int d, int n_gates, const double* m4_dev, const double* dm4_dev,
                                   const void* ubar_dev, double* grad_dev, cudaStream_t s);
cudaError_t launch_fock_tensor_single(int d, M8 m, void* u_re_or_cplx, double* u_im,
                                      cudaStream_t s);

// ---------------------------------------------------------------- zgemm.cu
// One group of a grouped complex128 GEMM:  C = cs[n] sum_k op(A)(m,k) B(k,n), row-major
// A[m][k] (opA 0) or its conjugate transpose, A stored [k][m] (opA 1); B[k][n].  Offsets are
// in complex elements (the scale's in doubles) from the launch's base pointers; a negative
// scale offset means "none".  sd is read only for groups with sec >= 0.
struct GemmGroup {
  int M, N, K;
  int lda, ldb, ldc;
  int opA;
  int herm;          // 1: C is Hermitian (M = N), its lower tiles are written as adjoints
  int tiles_n;       // ceil(N / tile N)
  int tile_start;    // first flat tile index of this group
  int sec;           // >= 0: a dimension is sector sec's kept count, read on the device
  int kdim;          // (1: M and lda; 2: N, ldb and ldc); the host's value is its bound.
                     // 3: nothing is done where the kept count is negative
  int64_t a_off, b_off, c_off;
  int64_t cs_off;
};

cudaError_t launch_zgemm_grouped(const void* a, const void* b, void* c, const double* scale,
                                 const GemmGroup* groups_dev, int n_groups, int total_tiles,
                                 const struct SectorDesc* sd_dev, cudaStream_t s);
int zgemm_tile_m();
int zgemm_tile_n();

// ---------------------------------------------------------------- plan descriptors
// Theta group (q, a0, b0): Theta_q[rows of left group a0 with a1 >= q1]
//                                 [cols of right group b0 with b1 <= q1]
//                         = Glc[rows][centre block q] @ Gcr[centre block q][cols]
struct ThetaDesc {
  int q0, q1, a0, b0;
  int row0, nrow, col0, ncol, k0, nk;
  int64_t off;            // storage [nrow][ncol] in the Theta workspace
};

struct SectorDesc {
  int cc0, cc1;
  int m, n;            // |L_s|, |R_s|
  int k;               // columns of the Jacobi matrix: n when !left, m when left
  int left;            // 1: Jacobi on [T^H; I_m] (m < n), 0: on T (m >= n)
  int rows_g;          // rows entering the pair Gram (m or n)
  int rows_tot;        // stored rows of the Jacobi matrix (m or n + m)
  int kept;            // filled after selection
  int slot0;           // first slot of this sector on the new bond
  int64_t c_off;       // C[m][n] row-major (complex)
  int64_t a_off;       // Jacobi matrix, row-major [rows_tot][k] (complex)
  int64_t t_off;       // its first rows_g rows as the mix writes them (a_off, or where a
                       // preconditioned sector's T or T^H stays)
  int64_t s_off;       // singular values / keys / permutation (k entries)
  int64_t w_off;       // W = V^H C, [kept][n] row-major (complex)
  int64_t v_off;       // V, [m][kept] row-major (complex)
  // Gram route and preconditioned sectors only:
  int64_t g_off;       // Gram / Householder vectors, [k][k] (complex)
  int64_t y_off;       // k x k slots: eigenvectors [k][kept], scratch
  int row_start[BSMPO_MAX_D];   // row of L_s where left group a0 (a1 >= cc1 part) starts
  int col_start[BSMPO_MAX_D];   // column of R_s where right group b0 (b1 <= cc1 part) starts
};

// One (left block a, right block b), a >= b, of the gate mix, cut in tiles of 256 elements.
struct MixPair {
  int a0, a1, b0, b1;
  int row0, nrow;      // left-bond rows of block a
  int col0, ncol;      // right-bond columns of block b
  int tile_start;      // first flat CTA index of this pair
  int upd;             // its update in the group
};

// Tables of one update of a group, shared by several kernels (device copy).  Sector indices
// are the group's; the update's own sectors are sec0 .. sec0 + n_sectors - 1.
struct UpdateTables {
  int d, chi, mode;
  int n_sectors, sec0, pad_;
  int64_t gate_off;                               // its gate tensor, from the launch's base
  int offL[BSMPO_MAX_Q + 1], offC[BSMPO_MAX_Q + 1], offR[BSMPO_MAX_Q + 1];
  int sidx[BSMPO_MAX_Q];                          // sector index of centre charge, or -1
  int pair_of[BSMPO_MAX_Q];                       // per own sector: the (cc1, cc0) sector, or -1
};

// ---------------------------------------------------------------- sector.cu
// Theta -> C (every sector, row-major) and the Jacobi matrix (T or [T^H; I]).
cudaError_t launch_mix_d(int d, const UpdateTables* tab_dev, const int* tidx_dev,
                         const ThetaDesc* td_dev, const SectorDesc* sd_dev,
                         const MixPair* pairs_dev, int n_pairs, int total_tiles, const void* u3,
                         const void* theta, const double* lam, void* cbuf, void* abuf,
                         cudaStream_t s);
// Identity rows of [T^H; I_m] for the `left` sectors of a list (the blocked ones), but for the
// preconditioned ones.
cudaError_t launch_identity_rows(const SectorDesc* sd_dev, const int* list_dev, int count, int max_elems,
                                 void* abuf, cudaStream_t s);
// An update done with preconditioned matrices is done again from the plain ones where it
// keeps singular values below PRE_MIN of their sector's largest.  The preconditioner mixes the
// columns of values below ~1e-7 of the largest, a null space among them, and a column reduced
// to the numerical-rank floor z takes part in no more rotations, so it can leave (z / sigma)^2
// of a value sigma out.  At z of 4e-14 (100 rows) that is rounding at 1e-5; at 1e-8 the kept
// values of a rank-deficient 120 x 100 sector were 6.8e-11 off, without it 5.3e-14 (relative;
// values above 1e-5: 1e-15 and 1e-14).
constexpr double PRE_MIN = 1e-5;
// Deterministic top-chi with ket/bra pair symmetrisation, one CTA per update; writes kept
// counts into sd_dev[s].kept and kept_out[s], slot starts, every update's total into
// kept_out[n_sectors + u], whether it must be done again without the preconditioner into
// kept_out[n_sectors + n_updates + u] (it keeps a value below pre_min of its sector's largest), and its truncation weight into trunc_out[u].
cudaError_t launch_select(const UpdateTables* tab_dev, SectorDesc* sd_dev, int n_updates,
                          int n_sectors, const double* sig, double* keys, double cutoff, int chi,
                          double pre_min, int* kept_out, double* trunc_out, cudaStream_t s);
// conj(V) rows for the kept vectors of every sector.
cudaError_t launch_extract_v(const SectorDesc* sd_dev, int n_sectors, int max_elems,
                             const void* abuf, const double* sig, const int* perm, void* vbuf,
                             cudaStream_t s);
// New Gamma_L (= Gamma[mode]), Gamma_R (= Gamma[mode+1]), Lambda and charges of bond mode+1
// of every update not to be done again; gamma, lam, charge: the whole state's; totals: kept
// vectors per update, then the words of those to be done again; err: two words on the
// device, nothing is written unless both are zero.
cudaError_t launch_scatter(const UpdateTables* tab_dev, const SectorDesc* sd_dev, int n_updates,
                           const int* totals, const int* err, int chi, const void* vbuf, const void* wbuf,
                           const double* sig, void* gamma, double* lam, int* charge,
                           cudaStream_t s);
// exp(i phi (n_ket - n_bra)) on every element of one site tensor.
cudaError_t launch_phase(int d, int chi, double phi, const int* charge_l, const int* charge_r,
                         void* gamma, cudaStream_t s);

// ---------------------------------------------------------------- jacobi.cu
// One round of the blocked one-sided Jacobi SVD for every active sector.
struct JacobiWork {
  int sector;       // index into the SectorDesc array
  int nblk;         // column blocks
  int npairs;       // block pairs per round
  int rounds;       // rounds per sweep
  int cs;           // row parts per block pair (rows_tot in parts of `chunk` rows)
  int cs_g;         // parts holding Gram rows (the first rows_g rows)
  int chunk;        // rows per part (multiple of 16, at most jacobi_rows_per_part())
  int gram_start;   // first CTA of this sector in the gram launch (npairs * cs_g CTAs)
  int apply_start;  // first CTA in the apply launch (npairs * cs CTAs)
  int slot_start;   // first block-pair slot (Q, flag and arrival counter)
  int pad_[2];
};
// rows of one part of a block pair
int jacobi_rows_per_part();
int jacobi_block_cols();
// One round of every listed sector: the gram kernel (partial Grams -> pbuf, 32 x 32
// complex per gram CTA; the last part of a pair reduces, tests and solves, writing Q
// and the flag of its slot), then the apply kernel.  pcnt (one int per slot) must be
// zero before the first round; the kernels leave it zero.  executed[0] / executed[1]
// count the rows that formed a partial pair Gram / were rotated (the executed work).
cudaError_t launch_jacobi_round(const SectorDesc* sd_dev, const JacobiWork* work_dev, int n_work,
                                int gram_ctas, int apply_ctas, int t, void* abuf, int* rot_count,
                                const double* nf2, double tol, int max_sweeps, void* pbuf,
                                int* pcnt, void* qbuf, int* qflag, unsigned long long* executed,
                                cudaStream_t s);
// Small sectors: the whole SVD (QR, all sweeps, column norms, sort) in one CTA per listed
// sector.  jacobi_is_small: whether a Jacobi matrix of rows_g Gram rows and k columns goes
// there; max_elems: the largest jacobi_small_elems of the list.  A left sector's vectors are
// left in the rows below the Gram rows, the others' scaled columns in the Gram rows.  fail
// is set to 1 where max_sweeps do not converge; executed[0] += complex MACs done,
// executed[1] = the most sweeps.
bool jacobi_is_small(int rows_g, int k);
int jacobi_small_elems(int rows_g, int k);
cudaError_t launch_jacobi_small(const SectorDesc* sd_dev, const int* list_dev, int count, int max_elems, int max_k,
                                void* abuf, int max_sweeps, double* sig, int* perm, int* fail,
                                unsigned long long* executed, cudaStream_t s);
// ||T_s||_F^2 of the listed sectors' Jacobi matrices (Gram rows), fixed-order reduction.
cudaError_t launch_sector_norms(const SectorDesc* sd_dev, const int* list_dev, int count, const void* abuf,
                                double* nf2, cudaStream_t s);
// Column norms (0 below the numerical-rank floor), descending sort (ties by column
// index) of the listed sectors: sig[s_off..], perm[s_off..].
cudaError_t launch_jacobi_finish(const SectorDesc* sd_dev, const int* list_dev, int count, int max_k,
                                 const void* abuf, const double* nf2, double* sig, int* perm,
                                 cudaStream_t s);

// ---------------------------------------------------------------- eigen.cu
// Gram / Hermitian-eigen route of the sector SVD (see eigen.cu).  gbuf holds every
// sector's Gram G = X^H X (k x k at g_off), overwritten by the Householder vectors.
int eigen_max_k();
// Sectors go in one launch per size class (tridiag_class): list_dev holds the sector
// indices grouped by class, class_count / class_kmax (host, TD_CLASSES entries) the number
// of sectors and their largest k per class.  Class c goes on streams[c] (the caller forks
// and joins them).  err: a device word set to 1 when a bulk-copy wait expired (zeroed by
// the caller).
constexpr int TD_CLASSES = 8;
int tridiag_class(int k);
cudaError_t launch_tridiag(const SectorDesc* sd_dev, const int* list_dev, const int* class_count,
                           const int* class_kmax, void* gbuf, double* dbuf, double* ebuf,
                           void* taubuf, int* err, const cudaStream_t* streams);
// eigenvalues (lam, descending), singular values sig = sqrt(lam) (0 below the floor), 1/sig
cudaError_t launch_bisect(const SectorDesc* sd_dev, int n_sectors, int kmax, const double* dbuf,
                          const double* ebuf, double* lam, double* sig, double* invsig,
                          cudaStream_t s);
// eigenvectors of the kept eigenvalues (sd[s].kept): V ([k][kept] at v_off) of the
// sectors with X = T^H, Y ([k][kept] at y_off) of the others.
cudaError_t launch_eigvec(SectorDesc* sd_dev, int n_sectors, int kmax, const double* dbuf, const double* ebuf,
                          const double* lam, double* scratch, unsigned char* swp, double* zbuf, const void* gbuf,
                          const void* taubuf, void* vbuf, void* ybuf, cudaStream_t s);
// The preconditioner of the blocked Jacobi SVD (see eigen.cu) of the listed sectors, from
// their tridiagonals: the eigenvalues (lam, descending) and the sectors better left as they
// are, flagged with kept = -1; every eigenvector, nearly unitary, to ybuf ([k][k] at y_off);
// 3/2 I - S / 2 in place of S = Y^H Y (check: a sector whose S is too far from I is flagged);
// and Y into the matrices [T^H; I] Y, or the unpreconditioned matrix of a flagged sector
// (max_elems: the largest rows_tot k).  tbuf: precondition_t_elems complex entries.
size_t precondition_t_elems(int64_t s_elems, int n_sectors);
cudaError_t launch_precondition_basis(const UpdateTables* tab_dev, SectorDesc* sd_dev, int n_updates,
                                      const int* list_dev, int count, int kmax, double cutoff, int chi,
                                      const double* dbuf, const double* ebuf, double* lam, double* scratch,
                                      unsigned char* swp, double* zbuf, const void* gbuf, const void* taubuf, void* tbuf,
                                      void* ybuf, cudaStream_t s);
cudaError_t launch_newton_schulz(SectorDesc* sd_dev, const int* list_dev, int count, int kmax, void* gbuf, bool check,
                                 cudaStream_t s);
cudaError_t launch_precondition_finish(const SectorDesc* sd_dev, const int* list_dev, int count, int max_elems,
                                       const void* ybuf, void* abuf, cudaStream_t s);

// ---------------------------------------------------------------- tcgemm.cu
// One group of the tensor-core (tcgen05, 3 x TF32) grouped complex GEMM:
//   C[c_off + m ldc + n] = sum_k op(A)[m][k] B[k][n] (x scale[cs_off + n])
// A and B are read through TMA tensor maps (index mapA / mapB into the launch's map
// array, FP64 views of complex matrices): op(A) = A ([m][k] at row a_r0 + m, column
// a_c0 + k; opA 0) or A^H (A stored [k][m] at row a_r0 + k, column a_c0 + m; opA 1);
// B [k][n] at row b_r0 + k, column b_c0 + n.  Offsets in complex elements.
struct TcGroup {
  int M, N, K;
  int opA;
  int tiles_n, tile_start;
  int mapA, mapB;
  int a_r0, a_c0, b_r0, b_c0;
  int ldc, pad_;
  int64_t c_off, cs_off;
};
int tc_tile_m();
int tc_tile_n();
size_t tc_map_bytes();
// Encodes a tensor map (tc_map_bytes() bytes at map_out) of the complex matrix at base
// (rows x cols, leading dimension ld, complex elements) with the box of operand `kind`:
// 0 = A [m][k], 1 = A stored [k][m], 2 = B [k][n].
cudaError_t tc_encode_map(void* map_out, const void* base, int rows, int cols, int ld, int kind);
// err: device int, set to nonzero if a pipeline wait of the kernel expired.
cudaError_t launch_tc_zgemm(const TcGroup* groups_dev, int n_groups, int total_tiles, const void* maps_dev,
                            void* c, const double* scale, int* err, cudaStream_t s);

// ---------------------------------------------------------------- contract.cu
// Standalone sector contraction with per-element charges (the update_MPO drop-in).
cudaError_t launch_contract_sector(int d, int cc0, int cc1, const void* u, const void* glc,
                                   const void* gcr, const int* cl, const int* cc, const int* cr,
                                   int len_l, int len_c, int len_r, void* c, cudaStream_t s);

// ---------------------------------------------------------------- state.cu
// Product-state Gamma from the bond charges (sorted, sentinel d) and the per-site
// density matrices rho[site][o_ket][o_bra] (complex, n d^2 entries).
cudaError_t launch_product_fill(int n, int d, int chi, const int* charge, const void* rho,
                                void* gamma, cudaStream_t s);

// Pure-state (MPS) variant of the contraction, one int32 charge per index.
cudaError_t launch_contract_mps(int d, int tau, const void* u, const void* glc, const void* gcr,
                                const double* ll, const double* lc, const double* lr, const int* cl,
                                const int* cc, const int* cr, int len_l, int len_c, int len_r, void* t,
                                cudaStream_t s);

// ---------------------------------------------------------------- observables.cu
// Per bond the positions of the entries with ket == bra charge and Lambda > 0 (list
// [n+1][chi], count [n+1]); env_r / env_l [n+1][chi] hold environments in list order, of
// which R_n and L_0 are set here.
cudaError_t launch_diag_lists(int n, int d, int chi, const int* charge, const double* lam, int* list, int* count,
                              void* env_r, void* env_l, cudaStream_t s);
// Step t = 0 .. n - 1: R_{n-1-t} and, with left, L_{t+1}.
cudaError_t launch_env_step(int n, int chi, int t, int max_rows, bool left, const void* gamma, const int* list,
                            const int* count, void* env_r, void* env_l, cudaStream_t s);
// Marginals (nchunk chunks of chunk_rows kept rows; nchunk 0: none) into out[n][d] through
// part[site][chunk][d], and the trace into out[n d].
cudaError_t launch_marginals(int n, int d, int chi, const void* gamma, const int* charge, const int* list,
                             const int* count, const void* env_l, const void* env_r, void* part, int chunk_rows,
                             int nchunk, void* out, cudaStream_t s);
