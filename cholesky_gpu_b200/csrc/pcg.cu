// PCG FP64 recurrences with device-resident scalars.
//
// Replaces the reference's Ddot/Daxpy/Dscal/Dcopy/Dnrm2 calls in host pointer
// mode (two host syncs per iteration, src/mixed_cholesky.cu:171-216) with
// reduction and update kernels whose alpha, beta and rho never leave the
// device -- the intent of the reference's unused computeAlphaKernel /
// x_r_update / update_search_dir (src/kernels_macros.cuh:547-550,599-632).
// Reductions use a fixed grid and a fixed summation order (deterministic).
// All vectors are n x nrhs, column-major, ld = n, nrhs <= 8.
#include "common.cuh"
#include "kernels.cuh"
#include "pcg.cuh"

namespace mpchol {
namespace {

constexpr int NTH = 256;     // 8 warps

// ---- FP64 vector kernels ----------------------------------------------------
constexpr int VG = 296;   // fixed grid for reductions (2 x 148 SMs): deterministic order

template <int NR>
__device__ __forceinline__ void block_reduce_store(double (&v)[NR], double* partials) {
  __shared__ double s_red[NTH / 32][NR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NR; ++k) v[k] = warp_sum(v[k]);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NR; ++k) s_red[warp][k] = v[k];
  __syncthreads();
  if (threadIdx.x < NR) {
    double s = 0.0;
    for (int w = 0; w < NTH / 32; ++w) s += s_red[w][threadIdx.x];
    partials[blockIdx.x * NR + threadIdx.x] = s;
  }
}

// Sum of the VG partials of each rhs, formed by the whole block with a fixed
// tree (two loads per thread, warp shuffles, then the eight warp sums in
// order), so every block -- and every launch -- gets the same bits.  Every
// thread of the block must call it; all receive the sums.
template <int NR>
__device__ __forceinline__ void sum_partials(const double* partials, double (&out)[NR]) {
  static_assert(VG <= 2 * NTH, "two partials per thread");
  __shared__ double s_w[NTH / 32][NR];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    double v = (t < VG) ? partials[t * NR + k] : 0.0;
    if (t + NTH < VG) v += partials[(t + NTH) * NR + k];
    v = warp_sum(v);
    if (lane == 0) s_w[warp][k] = v;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < NTH / 32; ++w) s += s_w[w][k];
    out[k] = s;
  }
  __syncthreads();
}

// ---- the kernels of one solve ------------------------------------------------
// What a solve launches beside its operator products and triangular solves.
// Each of these vector passes also prepares what the next kernels start from
// (zeroed accumulation targets, the triangular solves' input and counters), so
// that an iteration is seven launches; a boundary costs 1.5 us or more of an
// iteration that takes 40 at n = 1500.

// The inputs of one application z = M^-1 r: work = r, tmp and z zero, the two
// triangular solves' counters zero.
struct PrecPrep {
  double* work;
  double* tmp;
  double* z;
  int* ctr;
  int nctr;
};
__device__ __forceinline__ void clear_counters(const PrecPrep& pp) {
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < pp.nctr; i += NTH) pp.ctr[i] = 0;
}

// b (padded to NR columns), its partial ||b||^2, and the start of the solve:
// the first application's inputs (x0) or x = 0, Ap and z zero, the solve's
// status and done flags clear.
template <int NR>
__global__ void __launch_bounds__(NTH)
pcg_begin_kernel(const double* __restrict__ B, int nrhs, int n, double* __restrict__ bb, double* partials,
                 PrecPrep pp, double* __restrict__ Ap, double* __restrict__ z, bool x0, DevStatus* st,
                 int* done) {
  double v[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) v[k] = 0.0;
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += VG * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      const double t = k < nrhs ? B[o] : 0.0;
      bb[o] = t;
      v[k] = fma(t, t, v[k]);
      if (x0) {
        pp.work[o] = t;
        pp.tmp[o] = 0.0;
      }
      pp.z[o] = 0.0;   // x
      Ap[o] = 0.0;
      z[o] = 0.0;
    }
  clear_counters(pp);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *st = DevStatus{0, 0, 0, 0};
    done[0] = done[1] = 0;
  }
  block_reduce_store<NR>(v, partials);
}

// r = b - A x (Ap on entry, zero on exit), the partials of ||r||^2, ||x||^2 and
// r^T z (z: the last application's result), and the inputs of the next
// application to r.
template <int NR>
__global__ void __launch_bounds__(NTH)
residual_kernel(const double* __restrict__ b, double* __restrict__ Ap, double* __restrict__ r,
                const double* __restrict__ x, int n, double* rr_partials, double* xx_partials,
                double* rz_partials, PrecPrep pp) {
  double v[NR], w[NR], u[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) v[k] = w[k] = u[k] = 0.0;
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += VG * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      const double rv = b[o] - Ap[o], xv = x[o];
      Ap[o] = 0.0;
      r[o] = rv;
      v[k] = fma(rv, rv, v[k]);
      w[k] = fma(xv, xv, w[k]);
      u[k] = fma(rv, pp.z[o], u[k]);
      pp.work[o] = rv;
      pp.tmp[o] = 0.0;
      pp.z[o] = 0.0;
    }
  clear_counters(pp);
  block_reduce_store<NR>(v, rr_partials);
  __syncthreads();
  block_reduce_store<NR>(w, xx_partials);
  __syncthreads();
  block_reduce_store<NR>(u, rz_partials);
}

// Reduces the partials of a residual pass, one block each: ||r||^2 (and, in the
// first pass, ||b||^2), ||x||^2, r^T z, ||A||_F^2 (null: elsewhere).  done is
// set when every rhs meets the tolerance or the factor has failed, so that the
// iterations enqueued behind it return at once; it is cleared otherwise.
template <int NR>
__global__ void __launch_bounds__(NTH)
residual_reduce_kernel(const double* rr_partials, const double* bb_partials, const double* xx_partials,
                       const double* rz_partials, const double* fro_partials, double* misc, double* bnorm2,
                       double tol2, const DevStatus* factor_st, int* done) {
  double s[NR];
  if (blockIdx.x == 0) {
    double bn[NR];
    if (bb_partials != nullptr) {
      sum_partials<NR>(bb_partials, bn);
    } else {
#pragma unroll
      for (int k = 0; k < NR; ++k) bn[k] = bnorm2[k];
    }
    sum_partials<NR>(rr_partials, s);
    if (threadIdx.x == 0) {
      int all = 1;
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        misc[k] = s[k];
        bnorm2[k] = bn[k];
        if (!(s[k] <= tol2 * bn[k])) all = 0;
      }
      done[0] = (all || factor_st->code != 0) ? 1 : 0;
    }
  } else if (blockIdx.x == 3) {
    if (fro_partials == nullptr) return;
    double f[1];
    sum_partials<1>(fro_partials, f);
    if (threadIdx.x == 0) misc[16] = f[0];
  } else {
    sum_partials<NR>(blockIdx.x == 1 ? xx_partials : rz_partials, s);
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < NR; ++k) misc[(blockIdx.x == 1 ? 8 : 24) + k] = s[k];
  }
}

// p = z, partial r^T z: the first search direction.
template <int NR>
__global__ void __launch_bounds__(NTH)
pcg_start_kernel(const double* __restrict__ r, const double* __restrict__ z, double* __restrict__ p, int n,
                 double* partials, const int* skip) {
  if (*skip) return;
  double v[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) v[k] = 0.0;
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += VG * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      const double zv = z[o];
      p[o] = zv;
      v[k] = fma(r[o], zv, v[k]);
    }
  block_reduce_store<NR>(v, partials);
}

// rho_0 = r^T z from its partials; ctl: iterations begun by this loop, its budget.
template <int NR>
__global__ void __launch_bounds__(NTH)
pcg_loop_begin_kernel(const double* partials, double* rho, int* ctl, int budget) {
  double s[NR];
  sum_partials<NR>(partials, s);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NR; ++k) rho[k] = s[k];
    ctl[0] = 0;
    ctl[1] = budget;
  }
}

// partial a^T b.  count (null: none): the iteration count, incremented once (no
// block of this kernel reads it); zero (null: none): a vector cleared on the
// way, the product's target for the next iteration.
template <int NR>
__global__ void __launch_bounds__(NTH)
dot_kernel(const double* __restrict__ a, const double* __restrict__ b, int n, double* partials,
           const int* skip, int* count, double* __restrict__ zero) {
  if (skip != nullptr && *skip) return;
  if (count != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *count += 1;
  double v[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) v[k] = 0.0;
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += VG * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      v[k] = fma(a[o], b[o], v[k]);
      if (zero != nullptr) zero[o] = 0.0;
    }
  block_reduce_store<NR>(v, partials);
}

// alpha = rho / (p^T A p); x += alpha p; r -= alpha A p; partial ||r||^2; the
// inputs of the application to r.  A right-hand side whose pAp or rho is zero
// (already converged exactly) or not finite takes alpha = 0; a negative pAp
// records PCG_BREAKDOWN.  rho holds two sets of 8, used in turn: iteration c
// (ctl[0], from 1) reads set (c - 1) % 2 and writes the other.
template <int NR>
__global__ void __launch_bounds__(NTH)
update_xr_kernel(double* __restrict__ x, double* __restrict__ r, const double* __restrict__ p,
                 const double* __restrict__ Ap, int n, const double* pAp_partials,
                 const double* rho_sets, const int* ctl, double* rr_partials, const int* skip,
                 DevStatus* st, PrecPrep pp) {
  if (*skip) return;
  const double* rho = rho_sets + 8 * ((ctl[0] - 1) & 1);
  double pAp[NR], al[NR];
  sum_partials<NR>(pAp_partials, pAp);
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    const double a = rho[k] / pAp[k];
    al[k] = (pAp[k] != 0.0 && isfinite(a)) ? a : 0.0;
    if (!(pAp[k] >= 0.0) && threadIdx.x == 0 && blockIdx.x == 0) set_status(st, MPCHOL_PCG_BREAKDOWN, k);
  }
  double v[NR];
#pragma unroll
  for (int k = 0; k < NR; ++k) v[k] = 0.0;
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += VG * NTH) {
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      x[o] = fma(al[k], p[o], x[o]);
      const double rn = fma(-al[k], Ap[o], r[o]);
      r[o] = rn;
      v[k] = fma(rn, rn, v[k]);
      pp.work[o] = rn;
      pp.tmp[o] = 0.0;
      pp.z[o] = 0.0;
    }
  }
  clear_counters(pp);
  block_reduce_store<NR>(v, rr_partials);
}

// rho_new = r^T z (from partials); beta = rho_new / rho_old; p = z + beta p.
// From the ||r||^2 partials, sets *done when every rhs has ||r|| <= tol * ||b||
// (a block that starts after that skips its part of p, which nothing reads
// any more).  LOOP: also sets the condition of the device-side loop this
// iteration is the body of: continue while the recursive residual is above
// the tolerance, no error is recorded and the budget is not spent (the budget
// alone ends it, whatever the other flags hold).
template <int NR, bool LOOP>
__global__ void __launch_bounds__(NTH)
update_p_kernel(double* __restrict__ p, const double* __restrict__ z, int n, const double* rz_partials,
                double* rho_sets, const int* ctl, const double* rr_partials, const double* bnorm2,
                double tol2, int* done, const DevStatus* st, cudaGraphConditionalHandle handle) {
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  if (*reinterpret_cast<volatile int*>(done)) {
    if (LOOP && first) cudaGraphSetConditional(handle, 0u);
    return;
  }
  const int cur = (ctl[0] - 1) & 1;
  double rz[NR], be[NR];
  sum_partials<NR>(rz_partials, rz);
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    const double old = rho_sets[8 * cur + k];
    const double b = rz[k] / old;
    be[k] = (old != 0.0 && isfinite(b)) ? b : 0.0;
  }
  double rr[NR];
  sum_partials<NR>(rr_partials, rr);
  if (first) {
    int all = 1;
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      rho_sets[8 * (cur ^ 1) + k] = rz[k];
      if (!(rr[k] <= tol2 * bnorm2[k])) all = 0;
    }
    done[0] = all;
    done[1] += 1;
    if (LOOP) cudaGraphSetConditional(handle, (ctl[0] < ctl[1] && !all && st->code == 0) ? 1u : 0u);
  }
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += VG * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      p[o] = fma(be[k], p[o], z[o]);
    }
}

// ---- batched PCG (one launch for every system of a batch) ------------------
// grid (BATCH_VB, nsys): CTA (v, i) handles rows v*NTH + t, stride
// BATCH_VB*NTH, of system i.  Slots: 0 x, 1 r, 2 z, 3 p, 4 Ap, 5 b, 6 tmp,
// 7 work.  Partial groups: 0 pAp, 1 r^T r, 2 r^T z, 3 misc.  Scalars:
// rho[0] 0, rho[1] 8, alpha 16, ||b||^2 24, true ||r||^2 32, ||x||^2 40,
// ||A||_F^2 48 (eight parts of the sum), final r^T z 56.
namespace bslots { constexpr int X = 0, R = 1, Z = 2, P = 3, AP = 4, B = 5; }   // 6, 7: solve scratch

__device__ __forceinline__ double* bvec(const BatchSys& S, int slot, int nr) {
  return S.vec + (size_t)slot * S.n * nr;
}
__device__ __forceinline__ double* bpart(const BatchSys& S, int group) {
  return S.part + (size_t)group * BATCH_VB * 8;
}

template <int NR>
__device__ __forceinline__ void bsum(const double* part, double (&out)[NR]) {
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    double s = 0.0;
    for (int b = 0; b < BATCH_VB; ++b) s += part[b * NR + k];
    out[k] = s;
  }
}

template <int NR>
__device__ __forceinline__ void bstore(double (&v)[NR], double* part) {
  __shared__ double s_red[NTH / 32][NR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NR; ++k) v[k] = warp_sum(v[k]);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NR; ++k) s_red[warp][k] = v[k];
  __syncthreads();
  if (threadIdx.x < NR) {
    double s = 0.0;
    for (int w = 0; w < NTH / 32; ++w) s += s_red[w][threadIdx.x];
    part[blockIdx.x * NR + threadIdx.x] = s;
  }
}

template <int NR>
__global__ void __launch_bounds__(NTH)
dot_batched_kernel(const BatchSys* __restrict__ sys, int aslot, int bslot_, int group, int use_skip) {
  const BatchSys& S = sys[blockIdx.y];
  if (use_skip && S.done[0]) return;
  const int n = S.n;
  const double* a = bvec(S, aslot, NR);
  const double* b = bvec(S, bslot_, NR);
  double v[NR] = {};
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += BATCH_VB * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) v[k] = fma(a[(size_t)k * n + i], b[(size_t)k * n + i], v[k]);
  bstore<NR>(v, bpart(S, group));
}

template <int NR>
__global__ void __launch_bounds__(NTH)
update_xr_batched_kernel(const BatchSys* __restrict__ sys, int cur) {
  const BatchSys& S = sys[blockIdx.y];
  if (S.done[0]) return;
  const int n = S.n;
  double pAp[NR], al[NR];
  bsum<NR>(bpart(S, 0), pAp);
  const double* rho = S.scal + 8 * cur;
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    const double a = rho[k] / pAp[k];
    al[k] = (pAp[k] != 0.0 && isfinite(a)) ? a : 0.0;
    if (!(pAp[k] >= 0.0) && threadIdx.x == 0 && blockIdx.x == 0) set_status(S.st, MPCHOL_PCG_BREAKDOWN, k);
  }
  if (blockIdx.x == 0 && threadIdx.x < NR) S.scal[16 + threadIdx.x] = al[threadIdx.x];
  double* x = bvec(S, bslots::X, NR);
  double* r = bvec(S, bslots::R, NR);
  const double* p = bvec(S, bslots::P, NR);
  const double* Ap = bvec(S, bslots::AP, NR);
  double v[NR] = {};
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += BATCH_VB * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      x[o] = fma(al[k], p[o], x[o]);
      const double rn = fma(-al[k], Ap[o], r[o]);
      r[o] = rn;
      v[k] = fma(rn, rn, v[k]);
    }
  bstore<NR>(v, bpart(S, 1));
}

template <int NR>
__global__ void __launch_bounds__(NTH)
update_p_batched_kernel(const BatchSys* __restrict__ sys, int cur, int nrhs, double tol2) {
  const BatchSys& S = sys[blockIdx.y];
  if (S.done[0]) return;
  const int n = S.n;
  double rz[NR], be[NR], rr[NR];
  bsum<NR>(bpart(S, 2), rz);
  bsum<NR>(bpart(S, 1), rr);
  const double* rho_old = S.scal + 8 * cur;
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    const double b = rz[k] / rho_old[k];
    be[k] = (rho_old[k] != 0.0 && isfinite(b)) ? b : 0.0;
  }
  // CTA 0 writes rho into the other buffer (no CTA of this launch reads it)
  // and the done flag; a CTA that already sees done = 1 skips the p update,
  // which no later iteration of a converged system reads
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    int all = 1;
    for (int k = 0; k < NR; ++k) {
      S.scal[8 * (cur ^ 1) + k] = rz[k];
      if (k < nrhs && !(rr[k] <= tol2 * S.scal[24 + k])) all = 0;
    }
    S.done[1] += 1;
    S.done[0] = all;
  }
  double* p = bvec(S, bslots::P, NR);
  const double* z = bvec(S, bslots::Z, NR);
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += BATCH_VB * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      p[o] = fma(be[k], p[o], z[o]);
    }
}

// scal[off + k] = sum of the group's partials
template <int NR>
__global__ void reduce_batched_kernel(const BatchSys* __restrict__ sys, int group, int off,
                                      int use_skip) {
  const BatchSys& S = sys[blockIdx.y];
  if (use_skip && S.done[0]) return;
  if (threadIdx.x == 0) {
    double s[NR];
    bsum<NR>(bpart(S, group), s);
    for (int k = 0; k < NR; ++k) S.scal[off + k] = s[k];
  }
}

// r = b - Ap, partial ||r||^2 (group 1)
template <int NR>
__global__ void __launch_bounds__(NTH)
residual_batched_kernel(const BatchSys* __restrict__ sys) {
  const BatchSys& S = sys[blockIdx.y];
  const int n = S.n;
  const double* b = bvec(S, bslots::B, NR);
  const double* y = bvec(S, bslots::AP, NR);
  double* r = bvec(S, bslots::R, NR);
  double v[NR] = {};
  for (int i = blockIdx.x * NTH + threadIdx.x; i < n; i += BATCH_VB * NTH)
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const size_t o = (size_t)k * n + i;
      const double rv = b[o] - y[o];
      r[o] = rv;
      v[k] = fma(rv, rv, v[k]);
    }
  bstore<NR>(v, bpart(S, 1));
}

// done[0] = true residual of every rhs within tolerance (scal[32..] vs ||b||^2)
__global__ void check_true_batched_kernel(const BatchSys* __restrict__ sys, int nrhs, double tol2) {
  const BatchSys& S = sys[blockIdx.x];
  if (threadIdx.x != 0) return;
  int all = 1;
  for (int k = 0; k < nrhs; ++k)
    if (!(S.scal[32 + k] <= tol2 * S.scal[24 + k])) all = 0;
  S.done[0] = all;
}

__global__ void count_open_kernel(const BatchSys* __restrict__ sys, int nsys, int* out) {
  __shared__ int s_cnt;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  int c = 0;
  for (int i = threadIdx.x; i < nsys; i += blockDim.x) c += (sys[i].done[0] == 0);
  atomicAdd(&s_cnt, c);
  __syncthreads();
  if (threadIdx.x == 0) *out = s_cnt;
}

// b slot <- the caller's B_i (n x nrhs, ld n), zero-padded to nr columns
__global__ void load_rhs_batched_kernel(const BatchSys* __restrict__ sys,
                                        const double* const* __restrict__ B, int nrhs, int nr) {
  const BatchSys& S = sys[blockIdx.y];
  const double* src = B[blockIdx.y];
  double* dst = bvec(S, bslots::B, nr);
  const long long cnt = (long long)S.n * nr;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cnt;
       e += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(e / S.n);
    dst[e] = k < nrhs ? src[e] : 0.0;
  }
}

// the caller's X_i (n x nrhs, ld n) <- x slot
__global__ void store_x_batched_kernel(const BatchSys* __restrict__ sys, double* const* __restrict__ X,
                                       int nrhs, int nr) {
  const BatchSys& S = sys[blockIdx.y];
  double* dst = X[blockIdx.y];
  const double* src = bvec(S, bslots::X, nr);
  const long long cnt = (long long)S.n * nrhs;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cnt;
       e += (long long)gridDim.x * blockDim.x)
    dst[e] = src[e];
}

// partial ||A||_F^2 of the operator's lower triangle, CTA x of FROB_VB into
// entry x of group 3.  A warp per column, four loads in flight per lane (four
// CTAs per system with a column each at a time: 493 us for 128 systems of 64 to
// 2048, 91 with these).
constexpr int FROB_VB = 32;
static_assert(FROB_VB == BATCH_VB * 8, "the partials of group 3");
__global__ void __launch_bounds__(NTH)
frob_batched_kernel(const BatchSys* __restrict__ sys) {
  const BatchSys& S = sys[blockIdx.y];
  const int n = S.n, lane = threadIdx.x & 31;
  double diag = 0.0, s4[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = blockIdx.x * (NTH / 32) + threadIdx.x / 32; c < n; c += FROB_VB * (NTH / 32)) {
    const float* col = S.op + (size_t)c * S.op_ld;
    if (lane == 0) diag += (double)col[c] * (double)col[c];
    int r = c + 1 + lane;
    for (; r + 96 < n; r += 128) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = col[r + 32 * u];
#pragma unroll
      for (int u = 0; u < 4; ++u) s4[u] = fma((double)v[u], (double)v[u], s4[u]);
    }
    for (; r < n; r += 32) s4[0] = fma((double)col[r], (double)col[r], s4[0]);
  }
  double v[1] = {diag + 2.0 * ((s4[0] + s4[1]) + (s4[2] + s4[3]))};
  bstore<1>(v, bpart(S, 3));
}

}  // namespace

// ---- host launchers ---------------------------------------------------------
#define NR_DISPATCH(nrhs, CALL)            \
  switch (nrhs) {                          \
    case 1: { constexpr int NRC = 1; CALL; } break; \
    case 2: { constexpr int NRC = 2; CALL; } break; \
    case 4: { constexpr int NRC = 4; CALL; } break; \
    case 8: { constexpr int NRC = 8; CALL; } break; \
    default: return cudaErrorInvalidValue;          \
  }

int pcg_padded_nrhs(int nrhs) { return nrhs <= 1 ? 1 : nrhs <= 2 ? 2 : nrhs <= 4 ? 4 : 8; }
int pcg_vgrid() { return VG; }

namespace {
PrecPrep prep_of(const PcgVectors& v, double* target) {
  return PrecPrep{v.work, v.tmp, target, v.ctr, v.nctr};
}
}  // namespace

cudaError_t launch_pcg_begin(const PcgVectors& v, const double* B, int nrhs, bool x0, cudaStream_t stream) {
  NR_DISPATCH(v.nr, (pcg_begin_kernel<NRC><<<VG, NTH, 0, stream>>>(B, nrhs, v.n, v.b, v.part_bb, prep_of(v, v.x), v.Ap, v.z, x0, v.status, v.done)));
  return cudaGetLastError();
}
cudaError_t launch_residual(const PcgVectors& v, cudaStream_t stream) {
  NR_DISPATCH(v.nr, (residual_kernel<NRC><<<VG, NTH, 0, stream>>>(v.b, v.Ap, v.r, v.x, v.n, v.part_rr, v.part_xx, v.part_rz, prep_of(v, v.z))));
  return cudaGetLastError();
}
cudaError_t launch_residual_reduce(const PcgVectors& v, bool first, bool fro, double tol2,
                                   const DevStatus* factor_st, cudaStream_t stream) {
  NR_DISPATCH(v.nr, (residual_reduce_kernel<NRC><<<4, NTH, 0, stream>>>(v.part_rr, first ? v.part_bb : nullptr, v.part_xx, v.part_rz, fro ? v.part_fro : nullptr, v.misc, v.bnorm2, tol2, factor_st, v.done)));
  return cudaGetLastError();
}
cudaError_t launch_pcg_start(const PcgVectors& v, int budget, cudaStream_t stream) {
  NR_DISPATCH(v.nr, (pcg_start_kernel<NRC><<<VG, NTH, 0, stream>>>(v.r, v.z, v.p, v.n, v.part_rz, v.done)));
  NR_DISPATCH(v.nr, (pcg_loop_begin_kernel<NRC><<<1, NTH, 0, stream>>>(v.part_rz, v.rho, v.ctl, budget)));
  return cudaGetLastError();
}
cudaError_t launch_dot_pAp(const PcgVectors& v, cudaStream_t stream) {
  NR_DISPATCH(v.nr, (dot_kernel<NRC><<<VG, NTH, 0, stream>>>(v.p, v.Ap, v.n, v.part_pAp, v.done, v.ctl, nullptr)));
  return cudaGetLastError();
}
cudaError_t launch_update_xr(const PcgVectors& v, cudaStream_t stream) {
  NR_DISPATCH(v.nr, (update_xr_kernel<NRC><<<VG, NTH, 0, stream>>>(v.x, v.r, v.p, v.Ap, v.n, v.part_pAp, v.rho, v.ctl, v.part_rr, v.done, v.status, prep_of(v, v.z))));
  return cudaGetLastError();
}
cudaError_t launch_dot_rz(const PcgVectors& v, cudaStream_t stream) {
  NR_DISPATCH(v.nr, (dot_kernel<NRC><<<VG, NTH, 0, stream>>>(v.r, v.z, v.n, v.part_rz, v.done, nullptr, v.Ap)));
  return cudaGetLastError();
}
cudaError_t launch_update_p(const PcgVectors& v, double tol2, const cudaGraphConditionalHandle* loop,
                            cudaStream_t stream) {
  if (loop != nullptr) {
    NR_DISPATCH(v.nr, (update_p_kernel<NRC, true><<<VG, NTH, 0, stream>>>(v.p, v.z, v.n, v.part_rz, v.rho, v.ctl, v.part_rr, v.bnorm2, tol2, v.done, v.status, *loop)));
  } else {
    NR_DISPATCH(v.nr, (update_p_kernel<NRC, false><<<VG, NTH, 0, stream>>>(v.p, v.z, v.n, v.part_rz, v.rho, v.ctl, v.part_rr, v.bnorm2, tol2, v.done, v.status, cudaGraphConditionalHandle{})));
  }
  return cudaGetLastError();
}

cudaError_t launch_dot_batched(const BatchSys* sys, int nsys, int aslot, int bslot, int group,
                               int nr, int use_skip, cudaStream_t stream) {
  NR_DISPATCH(nr, (dot_batched_kernel<NRC><<<dim3(BATCH_VB, nsys), NTH, 0, stream>>>(sys, aslot, bslot, group, use_skip)));
  return cudaGetLastError();
}
cudaError_t launch_update_xr_batched(const BatchSys* sys, int nsys, int cur, int nr,
                                     cudaStream_t stream) {
  NR_DISPATCH(nr, (update_xr_batched_kernel<NRC><<<dim3(BATCH_VB, nsys), NTH, 0, stream>>>(sys, cur)));
  return cudaGetLastError();
}
cudaError_t launch_update_p_batched(const BatchSys* sys, int nsys, int cur, int nrhs, int nr,
                                    double tol2, cudaStream_t stream) {
  NR_DISPATCH(nr, (update_p_batched_kernel<NRC><<<dim3(BATCH_VB, nsys), NTH, 0, stream>>>(sys, cur, nrhs, tol2)));
  return cudaGetLastError();
}
cudaError_t launch_reduce_batched(const BatchSys* sys, int nsys, int group, int off, int nr,
                                  int use_skip, cudaStream_t stream) {
  NR_DISPATCH(nr, (reduce_batched_kernel<NRC><<<dim3(1, nsys), 32, 0, stream>>>(sys, group, off, use_skip)));
  return cudaGetLastError();
}
cudaError_t launch_residual_batched(const BatchSys* sys, int nsys, int nr, cudaStream_t stream) {
  NR_DISPATCH(nr, (residual_batched_kernel<NRC><<<dim3(BATCH_VB, nsys), NTH, 0, stream>>>(sys)));
  return cudaGetLastError();
}
cudaError_t launch_check_true_batched(const BatchSys* sys, int nsys, int nrhs, double tol2,
                                      cudaStream_t stream) {
  check_true_batched_kernel<<<nsys, 32, 0, stream>>>(sys, nrhs, tol2);
  return cudaGetLastError();
}
cudaError_t launch_count_open(const BatchSys* sys, int nsys, int* out, cudaStream_t stream) {
  count_open_kernel<<<1, NTH, 0, stream>>>(sys, nsys, out);
  return cudaGetLastError();
}
cudaError_t launch_load_rhs_batched(const BatchSys* sys, int nsys, const double* const* B, int nrhs,
                                    int nr, cudaStream_t stream) {
  load_rhs_batched_kernel<<<dim3(8, nsys), NTH, 0, stream>>>(sys, B, nrhs, nr);
  return cudaGetLastError();
}
cudaError_t launch_store_x_batched(const BatchSys* sys, int nsys, double* const* X, int nrhs,
                                   int nr, cudaStream_t stream) {
  store_x_batched_kernel<<<dim3(8, nsys), NTH, 0, stream>>>(sys, X, nrhs, nr);
  return cudaGetLastError();
}
cudaError_t launch_frob_batched(const BatchSys* sys, int nsys, cudaStream_t stream) {
  frob_batched_kernel<<<dim3(FROB_VB, nsys), NTH, 0, stream>>>(sys);
  return cudaGetLastError();
}


}  // namespace mpchol
