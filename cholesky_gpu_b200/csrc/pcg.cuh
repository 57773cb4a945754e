// Launchers of the PCG kernels (pcg.cu).
#pragma once
#include "common.cuh"

namespace mpchol {

int pcg_padded_nrhs(int nrhs);   // 1, 2, 4 or 8
int pcg_vgrid();                 // CTAs of the reduction kernels (partials per vector)

// ---- operator and preconditioner (solve.cu) ----
cudaError_t solve_init_attributes();
int solve_super_rows();
size_t solve_wsup_elems(int n);
int solve_setup_launches(int n);
// y += A x (the lower triangle of A, FP32 or FP64); y is zero on entry for a
// product.  An FP32 A is streamed through the staged kernel, which then also
// fills `fro` (shares of ||A||_F^2 for up to nfro CTAs, the rest zero).
cudaError_t launch_zero_vec(double* y, long long count, cudaStream_t stream);
template <typename TA>
cudaError_t launch_symv_skip(const TA* A, int lda, int n, const double* x, double* y, int nrhs,
                             const int* skip, cudaStream_t stream, double* fro = nullptr,
                             int nfro = 0);
// 128-block inverses into winv, then the super-block inverses into wsup.
cudaError_t launch_solve_setup(const float* L, int ldl, int n, float* wsup, cudaStream_t stream);
// out = L^-1 w (forward) or L^-T w (backward) through the super-block inverses
// wsup, one persistent cooperative launch: w is consumed, out (n x nrhs) and
// the trsv_counter_ints(n) counters are zero on entry.  launch_trsv_prep: w <-
// in, and for the forward-then-backward pair its targets mid and out and both
// sets of counters zero.  slots: trsv_slot_bytes() of device memory that no two
// solves use at once, zero when allocated and afterwards written by these
// launches only.
size_t trsv_counter_ints(int n);
size_t trsv_slot_bytes();
cudaError_t launch_trsv_prep(const double* in, double* w, double* mid, double* out, int n, int nrhs,
                             int* counters, cudaStream_t stream);
cudaError_t launch_trsv_persistent(bool backward, const float* L, int ldl, int n,
                                   const float* wsup, double* w, double* out, int nrhs, int* counters,
                                   void* slots, const int* skip, DevStatus* st, cudaStream_t stream);
// What the kernels of one solve work on: n x nr vectors (column-major, ld n;
// nr = 1, 2, 4 or 8), partial sums of pcg_vgrid() blocks, and the scalars
// that never leave the device.
struct PcgVectors {
  int n, nr;
  double *x, *r, *z, *p, *Ap, *b, *tmp, *work;
  double *part_pAp, *part_rr, *part_rz, *part_xx, *part_bb, *part_fro;
  double* rho;       // two sets of 8, used in turn by iteration
  double* bnorm2;    // 8
  double* misc;      // true ||r||^2 at 0, ||x||^2 at 8, ||A||_F^2 at 16, r^T z at 24
  int* done;         // [0] converged or failed, [1] iterations of the solve
  int* ctl;          // [0] iterations of the current loop, [1] its budget
  int* ctr;          // the two triangular solves' counters
  int nctr;
  DevStatus* status;
};
// In the order of a solve.  begin: b from B, the start state, and (x0) the
// inputs of the application that gives x.  residual: r = b - A x from Ap, and
// the inputs of z = M^-1 r; residual_reduce: its norms and *done.  start: p = z,
// rho, the loop's budget.  An iteration: Ap = A p, dot_pAp, update_xr (leaves
// the inputs of z = M^-1 r), the application, dot_rz (clears Ap), update_p
// (loop: sets the WHILE node's condition).
cudaError_t launch_pcg_begin(const PcgVectors& v, const double* B, int nrhs, bool x0, cudaStream_t stream);
cudaError_t launch_residual(const PcgVectors& v, cudaStream_t stream);
cudaError_t launch_residual_reduce(const PcgVectors& v, bool first, bool fro, double tol2,
                                   const DevStatus* factor_st, cudaStream_t stream);
cudaError_t launch_pcg_start(const PcgVectors& v, int budget, cudaStream_t stream);
cudaError_t launch_dot_pAp(const PcgVectors& v, cudaStream_t stream);
cudaError_t launch_update_xr(const PcgVectors& v, cudaStream_t stream);
cudaError_t launch_dot_rz(const PcgVectors& v, cudaStream_t stream);
cudaError_t launch_update_p(const PcgVectors& v, double tol2, const cudaGraphConditionalHandle* loop,
                            cudaStream_t stream);

// A whole solve in one cooperative launch (pcg_small.cu), for systems it fits:
// nr padded right-hand sides, operator elements of elem bytes.  bar: a zeroed
// word; v's status zero on entry.  Writes X (n x nrhs), the scalars of v, done
// (converged, iterations).
bool pcg_small_ok(int n, int nr, int elem, int nsm);
cudaError_t pcg_small_set_attributes();   // by solve_init_attributes
template <typename TA>
cudaError_t launch_pcg_small(const TA* A, int lda, const double* B, int nrhs, double* X, const float* W,
                             const PcgVectors& v, double tol2, int max_it, int max_restarts, bool x0,
                             const DevStatus* factor_st, unsigned* bar, cudaStream_t stream);

// misc device utilities (util.cu)
cudaError_t launch_extract_diag(const float* A, int lda, int n, float* d, float* dtilde,
                                cudaStream_t stream);
// Columns [c0, c1) of the lower block columns (rows from the column's block
// diagonal down, block b; b = 1: the lower triangle) of src (FP32, or FP64
// rounded to FP32) into dst, in one launch.
template <typename TS>
cudaError_t launch_copy_lower(const TS* src, int lds, float* dst, int ldd, int n, int b, int c0,
                              int c1, cudaStream_t stream);
// Equilibration: ex[i] = exponent of row i from A's diagonal; then the lower
// triangle of columns [c0, c1) is scaled to D A D
// (unscale_rows = false) or the factor's rows scaled back by 2^ex[i] (true).
cudaError_t launch_equil_exps(const float* A, int lda, int n, int8_t* ex, cudaStream_t stream);
cudaError_t launch_equil_scale(float* A, int lda, int n, const int8_t* ex, int c0, int c1,
                               bool unscale_rows, cudaStream_t stream);
// G = -(Lam X^T + X Lam^T) / 2, lower triangle (n x nrhs column-major inputs).
cudaError_t launch_sym_outer(const double* lam, const double* x, int n, int nrhs, double* G,
                             int ldg, cudaStream_t stream);
template <typename TA>
cudaError_t launch_frob_lower(const TA* A, int lda, int n, double* partials, cudaStream_t stream);
cudaError_t launch_pad_columns(const double* src, int n, int ncols, double* dst, int ncols_pad,
                               cudaStream_t stream);

// RBF kernel matrix (FP64 arithmetic) and its gradient contraction.
int rbf_grad_max_features();
int rbf_grad_work_elems(int n);
cudaError_t launch_rbf_build(const float* X, int n, int d, int ldx, double lengthscale,
                             double nugget, double* K64, float* K32, int ldk, int lower_only,
                             cudaStream_t stream);
cudaError_t launch_rbf_grad(const float* X, int n, int d, int ldx, double lengthscale,
                            const double* a, const double* b, double* P, double* s, double* work,
                            cudaStream_t stream);

// ---- batched solve side (solve.cu, pcg.cu): every launch serves all systems
struct BatchSys;
cudaError_t launch_vec_slot_batched(const BatchSys* sys, int nsys, int src, int dst, int nr,
                                    int use_skip, cudaStream_t stream);
cudaError_t launch_symv_batched(const BatchSys* sys, int nsys, int ntiles, int xslot, int yslot,
                                int nr, int use_skip, cudaStream_t stream);
cudaError_t launch_solve_setup_batched(const BatchSys* sys, int nsys, int max_n,
                                       cudaStream_t stream);
cudaError_t launch_trsv_batched(bool backward, const BatchSys* sys, int nsys, int max_n,
                                int in_slot, int out_slot, int work_slot, int nr, int use_skip,
                                cudaStream_t stream);

cudaError_t launch_dot_batched(const BatchSys* sys, int nsys, int aslot, int bslot, int group,
                               int nr, int use_skip, cudaStream_t stream);
cudaError_t launch_update_xr_batched(const BatchSys* sys, int nsys, int cur, int nr,
                                     cudaStream_t stream);
cudaError_t launch_update_p_batched(const BatchSys* sys, int nsys, int cur, int nrhs, int nr,
                                    double tol2, cudaStream_t stream);
cudaError_t launch_reduce_batched(const BatchSys* sys, int nsys, int group, int off, int nr,
                                  int use_skip, cudaStream_t stream);
cudaError_t launch_residual_batched(const BatchSys* sys, int nsys, int nr, cudaStream_t stream);
cudaError_t launch_check_true_batched(const BatchSys* sys, int nsys, int nrhs, double tol2,
                                      cudaStream_t stream);
cudaError_t launch_count_open(const BatchSys* sys, int nsys, int* out, cudaStream_t stream);
cudaError_t launch_load_rhs_batched(const BatchSys* sys, int nsys, const double* const* B, int nrhs,
                                    int nr, cudaStream_t stream);
cudaError_t launch_store_x_batched(const BatchSys* sys, int nsys, double* const* X, int nrhs,
                                   int nr, cudaStream_t stream);
cudaError_t launch_frob_batched(const BatchSys* sys, int nsys, cudaStream_t stream);

}  // namespace mpchol
