// Gaussian RBF kernel matrices and their gradient contractions.
//
// The reference has only a stub for this (src/RBF.cu:1-45).  Forward:
//   K_ij = exp(-||x_i - x_j||^2 / (2 l^2)) + nugget * delta_ij
// from n points x_i (rows of X, FP32), formed in FP64 (differences, not the
// norm expansion, so close points lose no digits) and written as FP64 and/or
// FP32 column-major.  Backward: for a symmetric cotangent
// G_K = -(a b^T + b a^T) / 2 of the solve x = K^-1 y (a the adjoint solution,
// b = x), every gradient needs only
//   P = K_rbf [a, b, a*X, b*X]    (n x (2 + 2d), K_rbf without the nugget)
//   s = sum_ij a_i b_j K_ij r_ij^2
// which one kernel forms while recomputing the K tiles from X (K itself is
// never read back):
//   dL/dnugget = -a.b,   dL/dl = -s / l^3,   dL/dy = a,
//   dL/dX_i = (X_i (a_i (K b)_i + b_i (K a)_i) - a_i (K(b*X))_i - b_i (K(a*X))_i) / l^2.
#include <algorithm>

#include "common.cuh"
#include "pcg.cuh"

namespace mpchol {
namespace {

constexpr int NTH = 256;
constexpr int JT = 64;        // columns of a tile of K

// Squared distances of a thread's R x C block of (row, column) pairs over KC
// staged features: xi and xj are feature-major (ldi, ldj doubles per feature),
// the thread's rows come in pairs rows[u], rows[u] + 1 and its columns likewise, so every
// feature reads R/2 + C/2 16-byte vectors for 2 R C FP64 operations; the
// FP64 pipe, not shared memory, then sets the pace from R C = 32 up.
template <int R, int C>
__device__ __forceinline__ void dist_step(const double* xi, const double* xj, const int (&rows)[R / 2],
                                          const int (&cols)[C / 2], double (&acc)[R][C]) {
  double a[R], b[C];
#pragma unroll
  for (int u = 0; u < R / 2; ++u) {
    const double2 v = *reinterpret_cast<const double2*>(xi + rows[u]);
    a[2 * u] = v.x;
    a[2 * u + 1] = v.y;
  }
#pragma unroll
  for (int u = 0; u < C / 2; ++u) {
    const double2 v = *reinterpret_cast<const double2*>(xj + cols[u]);
    b[2 * u] = v.x;
    b[2 * u + 1] = v.y;
  }
#pragma unroll
  for (int u = 0; u < R; ++u)
#pragma unroll
    for (int v = 0; v < C; ++v) {
      const double df = a[u] - b[v];
      acc[u][v] = fma(df, df, acc[u][v]);
    }
}

// ---- K: one IT x 64 tile per CTA -------------------------------------------
// Bound by the FP64 pipe (a subtraction and an fma per pair and feature).
// The features advance in chunks of 16 staged as FP64 in two buffers, the
// next chunk travelling in registers, one barrier per chunk.  IT = 128 gives a
// thread 8 x 4 pairs (six 16-byte reads per 64 operations); IT = 64 (4 x 4)
// serves matrices whose 128-row tiles would not fill the GPU.  n = 8192, d =
// 784: 3.58 ms, 82 % of the FP64 pipe's 2.92 ms (4.80 with 4 x 4 blocks from
// 8-byte reads and two barriers per chunk).
constexpr int BK = 16;

template <int IT>
__global__ void __launch_bounds__(NTH, 2)
rbf_build_kernel(const float* __restrict__ X, int n, int d, int ldx, double inv2l2, double nugget,
                 double* __restrict__ K64, float* __restrict__ K32, int ldk, int lower_only) {
  constexpr int R = IT / 16, C = 4;
  constexpr int LI = IT + 2, LJ = JT + 2;              // doubles per staged feature
  const int i0 = blockIdx.y * IT, j0 = blockIdx.x * JT;
  if (lower_only && j0 > i0 + IT - 1) return;
  extern __shared__ __align__(16) double sm_build[];   // [2][BK][LI], [2][BK][LJ]
  double* xi = sm_build;
  double* xj = xi + 2 * BK * LI;
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  int rows[R / 2], cols[C / 2];
#pragma unroll
  for (int u = 0; u < R / 2; ++u) rows[u] = 32 * u + 2 * tx;
#pragma unroll
  for (int u = 0; u < C / 2; ++u) cols[u] = 32 * u + 2 * ty;
  // thread (k = tid % 16, r = tid / 16 + 16 u): consecutive threads,
  // consecutive features
  constexpr int NI = IT / 16, NJ = JT / 16;
  float vi[NI], vj[NJ];
  const int lk = tid % BK, lr = tid / BK;
  auto fetch = [&](int k0) {
    const bool ok = k0 + lk < d;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const int gi = i0 + lr + 16 * u;
      vi[u] = (ok && gi < n) ? X[(size_t)gi * ldx + k0 + lk] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < NJ; ++u) {
      const int gj = j0 + lr + 16 * u;
      vj[u] = (ok && gj < n) ? X[(size_t)gj * ldx + k0 + lk] : 0.0f;
    }
  };
  double acc[R][C] = {};
  fetch(0);
  for (int k0 = 0, buf = 0; k0 < d; k0 += BK, buf ^= 1) {
    double* bi = xi + buf * BK * LI;
    double* bj = xj + buf * BK * LJ;
#pragma unroll
    for (int u = 0; u < NI; ++u) bi[lk * LI + lr + 16 * u] = (double)vi[u];
#pragma unroll
    for (int u = 0; u < NJ; ++u) bj[lk * LJ + lr + 16 * u] = (double)vj[u];
    __syncthreads();   // the buffer's last readers passed the previous barrier
    if (k0 + BK < d) fetch(k0 + BK);
#pragma unroll 4
    for (int k = 0; k < BK; ++k) dist_step<R, C>(bi + k * LI, bj + k * LJ, rows, cols, acc);
  }
#pragma unroll
  for (int v = 0; v < C; ++v) {
    const int j = j0 + cols[v / 2] + v % 2;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int i = i0 + rows[u / 2] + u % 2;
      if (i < n && j < n && (!lower_only || i >= j)) {
        double kv = exp(-acc[u][v] * inv2l2);
        if (i == j) kv = 1.0 + nugget;
        if (K64) K64[(size_t)j * ldk + i] = kv;
        if (K32) K32[(size_t)j * ldk + i] = (float)kv;
      }
    }
  }
}
template <int IT>
constexpr size_t build_smem() { return (size_t)2 * BK * (IT + 2 + JT + 2) * sizeof(double); }

// ---- backward contraction ---------------------------------------------------
// One CTA owns RT rows and sweeps the column tiles, so P is written once (no
// atomics) and s is reduced in a fixed order.  Per 64-column tile the K values
// are formed from differences (SIMT, R x C pairs per thread) into shared
// memory, with the sums K a, K b and s on the way, and then multiply the
// tile's points on the FP64 tensor cores: warp (m-block mb, column group ng)
// keeps the 8-row blocks of K (a o X) and K (b o X) for its feature blocks in
// accumulator fragments, a and b being multiplied into the K fragments.  Both
// halves run at the FP64 pipe: 2 d + 2 (d + 1) operations per pair and an
// exponential.  RT = 64 needs the fewest shared-memory reads per pair; 32 and
// 16 keep the GPU busy for fewer points.  n = 8192, d = 64: 2.26 ms (10.8 with
// one thread per row and column of P from 8-byte shared reads, 32-row CTAs).
constexpr int MAXD = 128;     // largest feature count the kernel stages
constexpr int LJX = JT + 4;   // doubles per feature of the column tile (4 mod 16: DMMA
                              // fragments read 16 different 8-byte banks per half-warp)

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <int RT>
__global__ void __launch_bounds__(NTH, 1)
rbf_grad_kernel(const float* __restrict__ X, int n, int d, int ldx, double inv2l2,
                const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ P,
                double* __restrict__ s_part) {
  constexpr int R = RT == 64 ? 4 : 2, C = RT == 16 ? 2 : 4;
  constexpr int NTX = RT / R, NTY = NTH / NTX;         // NTY * C = 64 columns
  static_assert(NTY * C == JT, "the threads cover the tile");
  constexpr int LI = RT + 4;                           // also 4 mod 16
  constexpr int MB = RT / 8, NG = (NTH / 32) / MB;     // m-blocks, column groups of warps
  constexpr int NBW = MAXD / 8 / NG;                   // feature blocks per warp at most
  extern __shared__ __align__(16) double sm_grad[];
  const int dp = (d + 7) / 8 * 8;                      // features padded with zeros
  double* xi = sm_grad;                                // [d][LI]
  double* xj = xi + (size_t)d * LI;                    // [dp][LJX]
  double* kt = xj + (size_t)dp * LJX;                  // [JT][LI]: K(i, j) at j * LI + i
  double* aj = kt + JT * LI;                           // [JT]
  double* bj = aj + JT;                                // [JT]
  __shared__ double s_red[NTH / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = blockIdx.x * RT;
  const int tx = tid % NTX, ty = tid / NTX;
  int rows[R / 2], cols[C / 2];
#pragma unroll
  for (int u = 0; u < R / 2; ++u) rows[u] = 32 * u + 2 * tx;
#pragma unroll
  for (int u = 0; u < C / 2; ++u) cols[u] = 32 * u + 2 * ty;
  for (int r = warp; r < RT; r += NTH / 32)
    for (int k = lane; k < d; k += 32)
      xi[k * LI + r] = (i0 + r < n) ? (double)X[(size_t)(i0 + r) * ldx + k] : 0.0;
  for (int e = tid; e < (dp - d) * LJX; e += NTH) xj[(size_t)d * LJX + e] = 0.0;
  double ai[R], pa[R] = {}, pb[R] = {};
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int gi = i0 + rows[u / 2] + u % 2;
    ai[u] = gi < n ? a[gi] : 0.0;
  }
  double s_acc = 0.0;
  const int g = lane >> 2, t = lane & 3, mb = warp % MB, ng = warp / MB;
  const int nblk = dp / 8;
  double da[NBW][2], db[NBW][2];
#pragma unroll
  for (int q = 0; q < NBW; ++q) da[q][0] = da[q][1] = db[q][0] = db[q][1] = 0.0;
  // the next tile's points travel in registers: rows warp + 8 u, features
  // lane + 32 v
  float px[JT / 8][MAXD / 32];
  auto fetch = [&](int j0) {
#pragma unroll
    for (int u = 0; u < JT / 8; ++u)
#pragma unroll
      for (int v = 0; v < MAXD / 32; ++v) {
        const int gj = j0 + warp + 8 * u, k = lane + 32 * v;
        if (32 * v < d) px[u][v] = (gj < n && k < d) ? X[(size_t)gj * ldx + k] : 0.0f;
      }
  };
  fetch(0);
  for (int j0 = 0; j0 < n; j0 += JT) {
    __syncthreads();                                   // the previous tile's readers are done
#pragma unroll
    for (int u = 0; u < JT / 8; ++u)
#pragma unroll
      for (int v = 0; v < MAXD / 32; ++v)
        if (lane + 32 * v < d) xj[(lane + 32 * v) * LJX + warp + 8 * u] = (double)px[u][v];
    if (tid < JT) {
      aj[tid] = j0 + tid < n ? a[j0 + tid] : 0.0;
      bj[tid] = j0 + tid < n ? b[j0 + tid] : 0.0;
    }
    __syncthreads();
    double r2[R][C] = {};
#pragma unroll 4
    for (int k = 0; k < d; ++k) dist_step<R, C>(xi + k * LI, xj + k * LJX, rows, cols, r2);
    // s by tiles, then over the tiles: one chain of R C terms a tile loses more than
    // 32-row CTAs with half the terms did (relative error at n = 8192, d = 64,
    // geometric mean of 24 draws: 7.3e-16 with those, 1.3e-15 in one chain, 4.2e-16)
    double s_tile = 0.0;
#pragma unroll
    for (int v = 0; v < C; ++v) {
      const int jl = cols[v / 2] + v % 2;
      const double av = aj[jl], bv = bj[jl];
      double kv[R];
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const bool in = i0 + rows[u / 2] + u % 2 < n && j0 + jl < n;
        kv[u] = in ? exp(-r2[u][v] * inv2l2) : 0.0;
        s_tile += in ? ai[u] * bv * kv[u] * r2[u][v] : 0.0;
        pa[u] = fma(kv[u], av, pa[u]);
        pb[u] = fma(kv[u], bv, pb[u]);
      }
#pragma unroll
      for (int u = 0; u < R / 2; ++u)
        *reinterpret_cast<double2*>(kt + jl * LI + rows[u]) = make_double2(kv[2 * u], kv[2 * u + 1]);
    }
    s_acc += s_tile;
    __syncthreads();
    if (j0 + JT < n) fetch(j0 + JT);
#pragma unroll 2
    for (int jj = 0; jj < JT; jj += 4) {
      const double kv = kt[(jj + t) * LI + 8 * mb + g];
      const double fa = kv * aj[jj + t], fb = kv * bj[jj + t];
#pragma unroll
      for (int q = 0; q < NBW; ++q) {
        const int nb = ng + NG * q;
        if (nb < nblk) {
          const double x = xj[(8 * nb + g) * LJX + jj + t];
          dmma(da[q], fa, x);
          dmma(db[q], fb, x);
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < NBW; ++q)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int k = 8 * (ng + NG * q) + 2 * t + e, gi = i0 + 8 * mb + g;
      if (k < d && gi < n) {
        P[(size_t)(2 + k) * n + gi] = da[q][e];
        P[(size_t)(2 + d + k) * n + gi] = db[q][e];
      }
    }
  // K a and K b: the column threads' sums in order
  __syncthreads();
  double* red = sm_grad;                               // [2][NTY][RT]: within xi and kt
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int r = rows[u / 2] + u % 2;
    red[ty * RT + r] = pa[u];
    red[(NTY + ty) * RT + r] = pb[u];
  }
  s_acc = warp_sum(s_acc);
  if (lane == 0) s_red[warp] = s_acc;
  __syncthreads();
  for (int e = tid; e < 2 * RT; e += NTH) {
    const int c = e / RT, r = e % RT;
    double v = 0.0;
    for (int y = 0; y < NTY; ++y) v += red[(c * NTY + y) * RT + r];
    if (i0 + r < n) P[(size_t)c * n + i0 + r] = v;
  }
  if (tid == 0) {
    double v = 0.0;
    for (int w = 0; w < NTH / 32; ++w) v += s_red[w];
    // two 16-row CTAs share a slot (zeroed before): 0 + x + y has one value in
    // either order
    if (RT == 16) atomicAdd(s_part + blockIdx.x / 2, v);
    else s_part[blockIdx.x] = v;
  }
}

// s = sum of the per-CTA partials in index order (deterministic)
__global__ void sum_partials_kernel(const double* __restrict__ part, int count, double* out) {
  __shared__ double s_w[NTH / 32];
  double v = 0.0;
  for (int i = threadIdx.x; i < count; i += NTH) v += part[i];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < NTH / 32; ++w) t += s_w[w];
    *out = t;
  }
}

template <int RT>
size_t grad_smem(int d) {
  constexpr int R = RT == 64 ? 4 : 2, NTY = NTH / (RT / R);
  const size_t main = (size_t)d * (RT + 4) + (size_t)((d + 7) / 8 * 8) * LJX + JT * (RT + 4) + 2 * JT;
  return std::max(main, (size_t)2 * NTY * RT) * sizeof(double);
}

// Rows per CTA of the contraction: the largest tile that still gives two
// thirds of the SMs a CTA.
int grad_rows(int n) { return n >= 100 * 64 ? 64 : (n >= 100 * 32 ? 32 : 16); }

template <int RT>
cudaError_t launch_grad(const float* X, int n, int d, int ldx, double inv2l2, const double* a,
                        const double* b, double* P, double* work, cudaStream_t stream) {
  const size_t smem = grad_smem<RT>(d);
  cudaError_t e = cudaFuncSetAttribute(rbf_grad_kernel<RT>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)grad_smem<RT>(MAXD));
  if (e == cudaSuccess && RT == 16)
    e = cudaMemsetAsync(work, 0, sizeof(double) * ceil_div(n, 32), stream);
  if (e != cudaSuccess) return e;
  rbf_grad_kernel<RT><<<ceil_div(n, RT), NTH, smem, stream>>>(X, n, d, ldx, inv2l2, a, b, P, work);
  return cudaGetLastError();
}

template <int IT>
cudaError_t launch_build(const float* X, int n, int d, int ldx, double inv2l2, double nugget,
                         double* K64, float* K32, int ldk, int lower_only, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(rbf_build_kernel<IT>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)build_smem<IT>());
  if (e != cudaSuccess) return e;
  rbf_build_kernel<IT><<<dim3(ceil_div(n, JT), ceil_div(n, IT)), NTH, build_smem<IT>(), stream>>>(
      X, n, d, ldx, inv2l2, nugget, K64, K32, ldk, lower_only);
  return cudaGetLastError();
}

}  // namespace

int rbf_grad_max_features() { return MAXD; }
int rbf_grad_work_elems(int n) { return ceil_div(n, 32); }

cudaError_t launch_rbf_build(const float* X, int n, int d, int ldx, double lengthscale,
                             double nugget, double* K64, float* K32, int ldk, int lower_only,
                             cudaStream_t stream) {
  const double inv2l2 = 1.0 / (2.0 * lengthscale * lengthscale);
  // 128-row tiles once they make two CTAs per SM
  const long long t128 = (long long)ceil_div(n, 128) * ceil_div(n, JT) / (lower_only ? 2 : 1);
  return t128 >= 2 * 148
             ? launch_build<128>(X, n, d, ldx, inv2l2, nugget, K64, K32, ldk, lower_only, stream)
             : launch_build<64>(X, n, d, ldx, inv2l2, nugget, K64, K32, ldk, lower_only, stream);
}

cudaError_t launch_rbf_grad(const float* X, int n, int d, int ldx, double lengthscale,
                            const double* a, const double* b, double* P, double* s, double* work,
                            cudaStream_t stream) {
  const double inv2l2 = 1.0 / (2.0 * lengthscale * lengthscale);
  const int rt = grad_rows(n);
  cudaError_t e = rt == 64   ? launch_grad<64>(X, n, d, ldx, inv2l2, a, b, P, work, stream)
                  : rt == 32 ? launch_grad<32>(X, n, d, ldx, inv2l2, a, b, P, work, stream)
                             : launch_grad<16>(X, n, d, ldx, inv2l2, a, b, P, work, stream);
  if (e != cudaSuccess) return e;
  sum_partials_kernel<<<1, NTH, 0, stream>>>(work, ceil_div(n, std::max(rt, 32)), s);
  return cudaGetLastError();
}

}  // namespace mpchol
