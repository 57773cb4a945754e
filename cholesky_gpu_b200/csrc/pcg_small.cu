// One whole solve of a small system (n <= 1024: one super-block) in one
// cooperative launch.
//
// Replaces, for such systems, the reference's host loop of Dgemv / Dpotrs / Ddot /
// Daxpy calls (src/mixed_cholesky.cu:171-216) and this library's own kernel
// per step of it: at n = 1024 an iteration is 2 MB of matrix reads that stay in
// L2 and takes as long as its seven launches and the loop node around them do
// (37 us).  Here CTA c owns rows 8 c .. 8 c + 7: their full rows of A, their
// rows of the super-block inverse W and their columns of it stay in shared
// memory for the whole solve, r and p are replicated in every CTA, and an
// iteration is three products from shared memory with a grid barrier after each:
//   Ap = A p            | p^T Ap -> alpha, r, ||r||^2
//   y  = W r            |
//   z  = W^T y          | r^T z  -> beta, p
// Each product's operand is spread over the threads (thread t holds elements t, t
// + 256, ..), which multiply their element with the eight rows and reduce over
// the block.  All sums run in a fixed order, the same in every CTA, so every CTA
// takes the same decisions.  Bound by the barriers' round trips through L2: about 12
// us an iteration.  Waits are bounded; a CTA that gives up records
// MPCHOL_ERR_TIMEOUT and leaves.
#include "common.cuh"
#include "kernels.cuh"
#include "pcg.cuh"

namespace mpchol {
namespace {

constexpr int NTH = 256, NW = NTH / 32;
constexpr int ROWS = 8;                      // rows of A and W, columns of W, per CTA
constexpr int LDW = 1024;                    // leading dimension of the super-block inverse
constexpr unsigned kMaxPolls = 1u << 22;

// Eight values per lane summed over the warp: lanes end with the sum of value
// (lane >> 2) (three halving exchanges, then the two low lane bits).
__device__ __forceinline__ double reduce8(double (&w)[8], int lane) {
#pragma unroll
  for (int h = 4, off = 16; h >= 1; h >>= 1, off >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double send = up ? w[i] : w[i + h], keep = up ? w[i + h] : w[i];
      w[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  double v = w[0];
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}

template <typename T>
__device__ __forceinline__ void load8(const T* strip, int n, int j, double (&s)[8]) {
  // two planes of four rows, four values of one j together
  if constexpr (sizeof(T) == 4) {
    const float4 a = *reinterpret_cast<const float4*>(strip + 4 * j);
    const float4 b = *reinterpret_cast<const float4*>(strip + 4 * n + 4 * j);
    s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
    s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double2 a = *reinterpret_cast<const double2*>(strip + 4 * n * h + 4 * j);
      const double2 b = *reinterpret_cast<const double2*>(strip + 4 * n * h + 4 * j + 2);
      s[4 * h] = a.x; s[4 * h + 1] = a.y; s[4 * h + 2] = b.x; s[4 * h + 3] = b.y;
    }
  }
}

template <int NR, typename TA>
__global__ void __launch_bounds__(NTH, 1)
pcg_small_kernel(const TA* __restrict__ A, int lda, const double* B, int nrhs, double* X,
                 const float* __restrict__ W, PcgVectors g, double tol2, int max_it,
                 int max_restarts, bool x0, const DevStatus* factor_st, unsigned* bar) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const int n = g.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x;
  TA* As = reinterpret_cast<TA*>(sm_raw);                     // [2][n][4]
  float* Wr = reinterpret_cast<float*>(As + (size_t)ROWS * n);
  float* Wc = Wr + (size_t)ROWS * n;
  double* rs = reinterpret_cast<double*>(Wc + (size_t)ROWS * n);   // [NR][n]
  double* ps = rs + (size_t)NR * n;                           // [NR][n]
  __shared__ double red[NW][ROWS * NR];
  __shared__ double s_sum[8];
  __shared__ int s_ok;
  if (factor_st->code != 0) return;                           // the host reports it
  const int row0 = ROWS * blockIdx.x, nrow = min(ROWS, n - row0);
  // ---- the CTA's strips ------------------------------------------------------
  auto at = [&](int j, int r) { return (size_t)(r >> 2) * 4 * n + 4 * j + (r & 3); };
#pragma unroll 4
  for (int e = tid; e < ROWS * n; e += NTH) {                 // j <= i: eight rows of a column
    const int r = e & 7, j = e >> 3, i = row0 + r;
    const bool in = r < nrow && j <= i;
    As[at(j, r)] = in ? A[(size_t)j * lda + i] : TA(0);
    Wr[at(j, r)] = in ? W[(size_t)j * LDW + i] : 0.0f;
  }
  __syncthreads();
  for (int r = 0; r < ROWS; ++r) {
    const int i = row0 + r;
#pragma unroll 2
    for (int j = tid; j < n; j += NTH) {                      // j > i: down column i
      if (r < nrow && j > i) As[at(j, r)] = A[(size_t)i * lda + j];
      Wc[at(j, r)] = (r < nrow && j >= i) ? W[(size_t)i * LDW + j] : 0.0f;
    }
  }
  __syncthreads();
  // ---- pieces ------------------------------------------------------------------
  unsigned round = 0;
  bool ok = true;
  auto grid_bar = [&]() {
    if (!ok) return;                                          // uniform over the CTA
    ++round;
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicAdd(bar, 1u);
      const unsigned want = round * (unsigned)G;
      unsigned it = 0;
      int good = 1;
      while (*reinterpret_cast<volatile unsigned*>(bar) < want)
        if (++it > kMaxPolls) {
          good = 0;
          set_status(g.status, MPCHOL_ERR_TIMEOUT, row0);
          break;
        }
      __threadfence();
      s_ok = good;
    }
    __syncthreads();
    ok = ok && s_ok != 0;
  };
  // thread t < 8 NR: row t % 8, rhs t / 8 of the CTA's slice
  const int sr = tid & 7, sk = tid >> 3;
  const bool slice = tid < ROWS * NR && sr < nrow;
  const size_t so = (size_t)sk * n + row0 + sr;
  // the slice of strip * (operand), in thread t < 8 NR
  auto product = [&](auto* strip, auto operand) -> double {
    double acc[NR][ROWS];
#pragma unroll
    for (int k = 0; k < NR; ++k)
#pragma unroll
      for (int r = 0; r < ROWS; ++r) acc[k][r] = 0.0;
#pragma unroll(NR <= 2 ? 4 : 1)
    for (int j = tid; j < n; j += NTH) {
      double s[ROWS];
      load8(strip, n, j, s);
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        const double m = operand((size_t)k * n + j);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[k][r] = fma(s[r], m, acc[k][r]);
      }
    }
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const double v = reduce8(acc[k], lane);
      if ((lane & 3) == 0) red[warp][k * ROWS + (lane >> 2)] = v;
    }
    __syncthreads();
    double v = 0.0;
    if (tid < ROWS * NR)
#pragma unroll
      for (int w = 0; w < NW; ++w) v += red[w][tid];
    return v;
  };
  // this CTA's partial of sum_i (slice value) per rhs
  auto put_partial = [&](double* part, double v) {
    v = slice ? v : 0.0;
    if (tid < ((ROWS * NR + 31) / 32) * 32) {
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      if (tid < ROWS * NR && sr == 0) part[(size_t)blockIdx.x * 8 + sk] = v;
    }
  };
  // the partials of all CTAs (after a barrier) -> out[k], in every thread
  auto sum_partials = [&](const double* part, double (&out)[NR]) {
    if (warp < NR) {
      double v = 0.0;
      for (int c = lane; c < G; c += 32) v += __ldcg(part + (size_t)c * 8 + warp);
      v = warp_sum(v);
      if (lane == 0) s_sum[warp] = v;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NR; ++k) out[k] = s_sum[k];
    __syncthreads();
  };
  // sums over the block's threads (replicated vectors: the same in every CTA)
  auto block_sum = [&](double (&v)[NR]) {
    __syncthreads();                                          // red's last readers are done
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      const double t = warp_sum(v[k]);
      if (lane == 0) red[warp][k] = t;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < NW; ++w) t += red[w][k];
      v[k] = t;
    }
    __syncthreads();
  };
  auto smem_at = [](const double* v) { return [v](size_t o) { return v[o]; }; };
  auto l2_at = [](const double* v) { return [v](size_t o) { return __ldcg(v + o); }; };
  // z = W^T (W r): the slice of z (one barrier inside)
  auto apply = [&]() -> double {
    const double y = product(Wr, smem_at(rs));
    if (slice) g.tmp[so] = y;
    grid_bar();
    return product(Wc, l2_at(g.tmp));
  };
  double xv = 0.0, zv = 0.0;                                  // the slice of x and of the latest z
  double rr[NR], xx[NR], bn[NR];
  // r = b - A x (two barriers), ||r||^2 and ||x||^2
  auto residual = [&]() {
    if (slice) g.x[so] = xv;
    grid_bar();
    const double ax = product(As, l2_at(g.x));
    if (slice) g.Ap[so] = ax;
#pragma unroll
    for (int k = 0; k < NR; ++k) xx[k] = rr[k] = 0.0;
    for (int j = tid; j < n; j += NTH)
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        const double t = __ldcg(g.x + (size_t)k * n + j);
        xx[k] = fma(t, t, xx[k]);
      }
    block_sum(xx);
    grid_bar();
    for (int j = tid; j < n; j += NTH)
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        const size_t o = (size_t)k * n + j;
        const double t = (k < nrhs ? B[o] : 0.0) - __ldcg(g.Ap + o);
        rs[o] = t;
        rr[k] = fma(t, t, rr[k]);
      }
    block_sum(rr);
  };
  // ---- the solve ---------------------------------------------------------------
  {
    double f[NR];
#pragma unroll
    for (int k = 0; k < NR; ++k) f[k] = bn[k] = 0.0;
    for (int j = tid; j < n; j += NTH) {
      double s[ROWS];
      load8(As, n, j, s);
#pragma unroll
      for (int r = 0; r < ROWS; ++r) f[0] = fma(s[r], s[r], f[0]);
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        const size_t o = (size_t)k * n + j;
        const double t = k < nrhs ? B[o] : 0.0;
        rs[o] = t;
        bn[k] = fma(t, t, bn[k]);
      }
    }
    block_sum(f);
    block_sum(bn);
    if (tid == 0) g.part_fro[blockIdx.x] = f[0];
  }
  if (x0) xv = apply();
  residual();
  int it = 0;
  bool broke = false, conv = false;
  for (int restart = 0; ok; ++restart) {
    conv = true;
#pragma unroll
    for (int k = 0; k < NR; ++k)
      if (k < nrhs && !(rr[k] <= tol2 * bn[k])) conv = false;
    if (conv || it >= max_it || restart > max_restarts) break;
    double rho[NR], al[NR], rz[NR];
    __syncthreads();
    zv = apply();
    if (slice) g.z[so] = zv;
    put_partial(g.part_rz, slice ? rs[so] * zv : 0.0);
    grid_bar();
    sum_partials(g.part_rz, rho);
    for (int j = tid; j < n; j += NTH)
#pragma unroll
      for (int k = 0; k < NR; ++k) ps[(size_t)k * n + j] = __ldcg(g.z + (size_t)k * n + j);
    for (bool more = true; more && ok;) {
      // the products below read ps and rs of the thread's own elements, the
      // slice values those of other threads: every block_sum and barrier in
      // between orders them
      const double ap = product(As, smem_at(ps));
      if (slice) g.Ap[so] = ap;
      const double pv = slice ? ps[so] : 0.0;
      put_partial(g.part_pAp, pv * ap);
      grid_bar();
      sum_partials(g.part_pAp, al);
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        const double pAp = al[k], a = rho[k] / pAp;
        al[k] = (pAp != 0.0 && isfinite(a)) ? a : 0.0;
        if (!(pAp >= 0.0)) {
          broke = true;
          if (tid == 0 && blockIdx.x == 0) set_status(g.status, MPCHOL_PCG_BREAKDOWN, k);
        }
        rr[k] = 0.0;
      }
#pragma unroll
      for (int k = 0; k < NR; ++k)
        if (sk == k) xv = fma(al[k], pv, xv);
      for (int j = tid; j < n; j += NTH)
#pragma unroll
        for (int k = 0; k < NR; ++k) {
          const size_t o = (size_t)k * n + j;
          const double t = fma(-al[k], __ldcg(g.Ap + o), rs[o]);
          rs[o] = t;
          rr[k] = fma(t, t, rr[k]);
        }
      block_sum(rr);
      zv = apply();
      if (slice) g.z[so] = zv;
      put_partial(g.part_rz, slice ? rs[so] * zv : 0.0);
      grid_bar();
      sum_partials(g.part_rz, rz);
      bool all = true;
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        const double b = rz[k] / rho[k];
        const double be = (rho[k] != 0.0 && isfinite(b)) ? b : 0.0;
        rho[k] = rz[k];
        for (int j = tid; j < n; j += NTH) {
          const size_t o = (size_t)k * n + j;
          ps[o] = fma(be, ps[o], __ldcg(g.z + o));
        }
        if (!(rr[k] <= tol2 * bn[k])) all = false;
      }
      __syncthreads();
      ++it;
      more = !all && !broke && it < max_it;
    }
    if (ok) residual();
  }
  if (!ok) return;
  // ---- results -------------------------------------------------------------------
  put_partial(g.part_rz, slice ? rs[so] * zv : 0.0);
  grid_bar();
  if (!ok) return;
  // X may be B itself: every CTA has read B for the last time before this barrier
  if (slice && sk < nrhs) X[so] = xv;
  if (blockIdx.x != 0) return;
  double rz[NR];
  sum_partials(g.part_rz, rz);
  if (warp == 0) {
    double f = 0.0;
    for (int c = lane; c < G; c += 32) f += __ldcg(g.part_fro + c);
    f = warp_sum(f);
    if (lane == 0) {
      g.misc[16] = f;
      g.done[0] = conv ? 1 : 0;
      g.done[1] = it;
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        g.misc[k] = rr[k];
        g.misc[8 + k] = xx[k];
        g.misc[24 + k] = rz[k];
        g.bnorm2[k] = bn[k];
      }
    }
  }
}

// Dynamic shared memory: the strips of A (elem bytes an element) and W, r and p.
size_t small_smem(int n, int nr, int elem) {
  return (size_t)ROWS * n * (elem + 2 * sizeof(float)) + (size_t)2 * nr * n * sizeof(double);
}
// What an SM leaves for it beside the static reduction buffers.
size_t small_smem_max(int nr) {
  return (size_t)227 * 1024 - (sizeof(double) * (NW * ROWS * nr + 8) + 64);
}

template <int NR, typename TA>
cudaError_t launch_small(const TA* A, int lda, const double* B, int nrhs, double* X, const float* W,
                         const PcgVectors& v, double tol2, int max_it, int max_restarts, bool x0,
                         const DevStatus* factor_st, unsigned* bar, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ceil_div(v.n, ROWS));
  cfg.blockDim = dim3(NTH);
  cfg.dynamicSmemBytes = small_smem(v.n, NR, sizeof(TA));
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, pcg_small_kernel<NR, TA>, A, lda, B, nrhs, X, W, v, tol2, max_it,
                            max_restarts, x0, factor_st, bar);
}

}  // namespace

// One super-block (its inverse is the whole preconditioner), one CTA per SM
// for every eight rows, and the strips and replicated vectors in an SM's shared
// memory.
bool pcg_small_ok(int n, int nr, int elem, int nsm) {
  if (n > LDW || ceil_div(n, ROWS) > nsm) return false;
  return small_smem(n, nr, elem) <= small_smem_max(nr);
}

// The most any n takes, once per device: the attribute is the kernel's, not the
// launch's, and a value set for one call would bound a concurrent one.
cudaError_t pcg_small_set_attributes() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto kernel, int nr) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small_smem_max(nr));
  };
  set(pcg_small_kernel<1, float>, 1);
  set(pcg_small_kernel<2, float>, 2);
  set(pcg_small_kernel<4, float>, 4);
  set(pcg_small_kernel<8, float>, 8);
  set(pcg_small_kernel<1, double>, 1);
  set(pcg_small_kernel<2, double>, 2);
  set(pcg_small_kernel<4, double>, 4);
  set(pcg_small_kernel<8, double>, 8);
  return e;
}

template <typename TA>
cudaError_t launch_pcg_small(const TA* A, int lda, const double* B, int nrhs, double* X, const float* W,
                             const PcgVectors& v, double tol2, int max_it, int max_restarts, bool x0,
                             const DevStatus* factor_st, unsigned* bar, cudaStream_t stream) {
  switch (v.nr) {
    case 1: return launch_small<1, TA>(A, lda, B, nrhs, X, W, v, tol2, max_it, max_restarts, x0, factor_st, bar, stream);
    case 2: return launch_small<2, TA>(A, lda, B, nrhs, X, W, v, tol2, max_it, max_restarts, x0, factor_st, bar, stream);
    case 4: return launch_small<4, TA>(A, lda, B, nrhs, X, W, v, tol2, max_it, max_restarts, x0, factor_st, bar, stream);
    case 8: return launch_small<8, TA>(A, lda, B, nrhs, X, W, v, tol2, max_it, max_restarts, x0, factor_st, bar, stream);
    default: return cudaErrorInvalidValue;
  }
}
template cudaError_t launch_pcg_small<float>(const float*, int, const double*, int, double*, const float*, const PcgVectors&, double, int, int, bool, const DevStatus*, unsigned*, cudaStream_t);
template cudaError_t launch_pcg_small<double>(const double*, int, const double*, int, double*, const float*, const PcgVectors&, double, int, int, bool, const DevStatus*, unsigned*, cudaStream_t);

}  // namespace mpchol
