// Diagonal-block Cholesky (POTRF) for the blocked factorization.
//
// Replaces the reference's per-step cusolverDnSpotrf of the b x b diagonal
// block (src/switching_chol.cuh:86-95) and its CPU micro_cholesky variant
// (src/micro_chol.hpp:14-44, src/sChol.cuh:66-79).  One CTA factors a block of
// up to 256 x 256 as a blocked right-looking Cholesky on dense 32 x 32 tiles in
// shared memory (column-major, lane i of a warp always owns row i, so every
// shared access is either contiguous across lanes or a broadcast):
//   * a warp owns a row of tiles: it solves them from left to right, each
//     close behind the factor of its diagonal tile, then factors its own;
//   * other warps update the tiles ahead of their turn;
//   * the inverses of the diagonal tiles are formed for the panel solve.
// Blocks flagged near-indefinite by the switching criterion are factored in
// FP64 by a second kernel on a global (L2-resident) scratch.
#include "common.cuh"
#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace mpchol {

namespace {

constexpr int TS = 32;          // tile size
constexpr int TSZ = TS * TS;    // elements per dense tile

__device__ __forceinline__ int tidx(int I, int J) { return I * (I + 1) / 2 + J; }

// 16-byte shared-memory vector load of 4 floats or 2 doubles.
__device__ __forceinline__ void load_vec16(const float* p, float (&v)[4]) {
  const float4 w = *reinterpret_cast<const float4*>(p);
  v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
}
__device__ __forceinline__ void load_vec16(const double* p, double (&v)[2]) {
  const double2 w = *reinterpret_cast<const double2*>(p);
  v[0] = w.x; v[1] = w.y;
}

template <typename T>
__device__ __forceinline__ T drsqrt(T x);
template <>
__device__ __forceinline__ float drsqrt<float>(float x) { return rsqrtf(x); }
template <>
__device__ __forceinline__ double drsqrt<double>(double x) { return rsqrt(x); }

// The pivot rule of column k, evaluated by every lane on its own candidate
// (no divergent branch on the chain; lane k's value is the pivot).
template <typename T>
struct Pivot {
  T piv, r;        // repaired pivot and 1/sqrt(piv)
  bool pert, bad;  // repaired by the floor; failed (non-positive without repair, or not finite)
};
template <typename T>
__device__ __forceinline__ Pivot<T> eval_pivot(T cand, bool real, T my_shift, T my_pmin,
                                               int diag_pert) {
  Pivot<T> p;
  T piv = real ? cand + my_shift : T(1);
  // a NaN or infinite pivot means the Schur complement has overflowed
  // (earlier pivots floored far below the rounding error of a low-precision
  // update): no repair makes that factor usable, so it fails as NOT_SPD
  const bool nonfin = real && !(piv - piv == T(0));
  p.pert = false;
  p.bad = nonfin;
  if (diag_pert) {
    // repair: max(|pivot|, floor), the reference's fixDiag rule
    // (src/kernels_macros.cuh:90-99)
    p.pert = real && !nonfin && !(piv > my_pmin);
    const T ap = piv < T(0) ? -piv : piv;
    piv = p.pert ? (ap > my_pmin ? ap : my_pmin) : piv;
  } else {
    p.bad = p.bad || (real && !(piv > T(0)));
  }
  p.piv = p.bad ? T(1) : piv;   // keep the arithmetic finite; the caller discards the result
  // one SFU reciprocal square root on the dependency chain:
  // r = 1/sqrt(piv), L(k,k) = piv * r
  p.r = drsqrt<T>(p.piv);
  return p;
}

// Factor the 32 x 32 tile t in place (lower triangle).  inv[k] receives
// 1 / L(k,k).  Returns false on a non-positive pivot when pivot flooring is
// off (first failing local row in *fail_row).
//
// Lane i holds row i of the tile in registers (a[j], j relative to the
// current block of CB columns): per column lane k's pivot is repaired, one
// shuffle broadcasts 1/sqrt(pivot), and the rank-1 update reads the column's
// multipliers from the 32-entry shared buffer col as 16-byte broadcasts.  The
// columns run as a loop over blocks of CB whose body is unrolled: after a
// block its finished columns are stored and the registers shift down by CB,
// so register indices stay compile-time constants while the kernel's code
// stays small (its instructions must stay cache-resident while the trailing
// update saturates L2 beside it).  The pivot of column k + 1 is lane k + 1's
// candidate a[k+1] - L(k+1,k)^2 (the same fma the rank-1 update applies to
// a[k+1]); it is evaluated, square-rooted and broadcast before column k's
// multipliers go through shared memory, so the pivot chain and the update's
// round trip overlap.  Registers past the tile's last column are updated
// with junk and never stored.
template <typename T, int CB>
__device__ bool factor_diag_tile(T* t, T* inv, int lane, int nreal, const T* shift, const T* pmin,
                                 int diag_pert, int* nperturbed, int* fail_row, T* col) {
  constexpr int V = 16 / sizeof(T);
  T a[TS];
#pragma unroll
  for (int j = 0; j < TS; ++j) a[j] = t[j * TS + lane];
  const T my_shift = (lane < nreal) ? shift[lane] : T(0);
  const T my_pmin = pmin[lane];
  bool failed = false, perturbed = false;
  T my_inv = T(1);
  Pivot<T> pv = eval_pivot<T>(a[0], 0 < nreal, my_shift, my_pmin, diag_pert);
  T rk = __shfl_sync(0xffffffffu, pv.r, 0);
#pragma unroll 1
  for (int c0 = 0; c0 < TS; c0 += CB) {
#pragma unroll
    for (int c = 0; c < CB; ++c) {
      const int k = c0 + c;
      const bool mine = lane == k;
      perturbed = perturbed || (mine && pv.pert);
      failed = failed || (mine && pv.bad);
      my_inv = mine ? pv.r : my_inv;
      const T lik = (lane > k) ? a[c] * rk : T(0);
      a[c] = mine ? pv.piv * pv.r : ((lane > k) ? lik : a[c]);
      if (k + 1 < TS) {
        pv = eval_pivot<T>(fma(-lik, lik, a[c + 1]), k + 1 < nreal, my_shift, my_pmin, diag_pert);
        rk = __shfl_sync(0xffffffffu, pv.r, k + 1);
      }
      // two multiplier buffers used in turn: the next column's write cannot
      // overtake a lane still reading this one, so one warp barrier suffices
      T* cb = col + (k & 1) * TS;
      cb[lane] = lik;
      __syncwarp();
#pragma unroll
      for (int q = (c + 1) / V; q < TS / V; ++q) {
        if (c0 + V * q < TS) {
          T l[V];
          load_vec16(cb + c0 + V * q, l);
#pragma unroll
          for (int e = 0; e < V; ++e) {
            const int j = V * q + e;
            if (j > c) a[j] = fma(-lik, l[e], a[j]);
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < CB; ++c)
      if (c0 + c <= lane) t[(c0 + c) * TS + lane] = a[c];
#pragma unroll
    for (int j = 0; j < TS - CB; ++j) a[j] = a[j + CB];
  }
  inv[lane] = my_inv;
  const unsigned fm = __ballot_sync(0xffffffffu, failed);
  const unsigned pm = __ballot_sync(0xffffffffu, perturbed);
  if (fm) *fail_row = __ffs(fm) - 1;
  if (lane == 0) *nperturbed += __popc(pm);
  __syncwarp();
  return fm == 0;
}

// X L^T = B for one tile (B in x, overwritten); lane i owns row i.
// Right-looking: once x(i, m) is final it is applied to the later columns,
// whose multipliers L(m+1.., m) are contiguous in the column-major tile l and
// arrive as 16-byte broadcasts.  Blocks of CB columns with register rotation,
// as in factor_diag_tile.
template <typename T, int CB>
__device__ void trsm_tile(T* x, const T* l, const T* inv, int lane) {
  constexpr int V = 16 / sizeof(T);
  T b[TS];
#pragma unroll
  for (int m = 0; m < TS; ++m) b[m] = x[m * TS + lane];
#pragma unroll 1
  for (int m0 = 0; m0 < TS; m0 += CB) {
#pragma unroll
    for (int c = 0; c < CB; ++c) {
      const int m = m0 + c;
      b[c] *= inv[m];
#pragma unroll
      for (int q = (c + 1) / V; q < TS / V; ++q) {
        if (m0 + V * q < TS) {
          T lv[V];
          load_vec16(l + m * TS + m0 + V * q, lv);
#pragma unroll
          for (int e = 0; e < V; ++e)
            if (V * q + e > c) b[V * q + e] = fma(-b[c], lv[e], b[V * q + e]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < CB; ++c) x[(m0 + c) * TS + lane] = b[c];
#pragma unroll
    for (int j = 0; j < TS - CB; ++j) b[j] = b[j + CB];
  }
}

// N contiguous elements of a shared tile (16-byte vectors, an 8-byte
// remainder; p aligned to the access size).
template <int N, typename T>
__device__ __forceinline__ void load_n(const T* p, T (&v)[N]) {
  constexpr int V = 16 / sizeof(T);
#pragma unroll
  for (int q = 0; q < N / V; ++q) {
    T w[V];
    load_vec16(p + V * q, w);
#pragma unroll
    for (int e = 0; e < V; ++e) v[V * q + e] = w[e];
  }
  if constexpr (N % V != 0) {
    static_assert(sizeof(T) == 4 && N % V == 2, "8-byte remainder of a float block");
    const float2 w = *reinterpret_cast<const float2*>(p + N - 2);
    v[N - 2] = w.x;
    v[N - 1] = w.y;
  }
}

// C(r0 .. r0+RR-1, c0 .. c0+CC-1) -= A B^T over the tiles' 32 k (32 x 32
// tiles, column-major).  The thread keeps its RR x CC block in registers and
// reads, per k, RR values of A's column and CC of B's as vectors, so a warp's
// shared-memory traffic per FMA is (RR + CC) / (RR CC) of a value (the
// return path of shared memory, not the FMA pipe, bounds these updates).
// Each output is the same fma chain in k order as a row-by-row update.
template <typename T, int RR, int CC>
__device__ __forceinline__ void syrk_block(T* c, const T* a, const T* b, int r0, int c0) {
  T acc[RR][CC];
#pragma unroll
  for (int j = 0; j < CC; ++j)
#pragma unroll
    for (int i = 0; i < RR; ++i) acc[i][j] = c[(c0 + j) * TS + r0 + i];
#pragma unroll 4
  for (int k = 0; k < TS; ++k) {
    T av[RR], bv[CC];
    load_n<RR>(a + k * TS + r0, av);
    load_n<CC>(b + k * TS + c0, bv);
#pragma unroll
    for (int i = 0; i < RR; ++i)
#pragma unroll
      for (int j = 0; j < CC; ++j) acc[i][j] = fma(-av[i], bv[j], acc[i][j]);
  }
#pragma unroll
  for (int j = 0; j < CC; ++j)
#pragma unroll
    for (int i = 0; i < RR; ++i) c[(c0 + j) * TS + r0 + i] = acc[i][j];
}

// A whole 32 x 32 tile C -= A B^T by one warp: lane (rg, cg) = (lane % 4,
// lane / 4) owns rows 8 rg .. and columns 4 cg .. (a quarter-warp reads four
// distinct 32-byte row groups and two column groups: no bank conflict).
template <typename T>
__device__ __forceinline__ void syrk_tile(T* c, const T* a, const T* b, int lane) {
  syrk_block<T, 8, 4>(c, a, b, 8 * (lane & 3), 4 * (lane >> 2));
}

// Inverse of the lower-triangular tile l into out (32 x 32 column-major,
// FP32).  Lane j solves L w = e_j for column j of L^-1, right-looking with the
// column held in registers; the column of L used at each step arrives as
// 16-byte broadcasts.  Blocks of CB steps with register rotation, as in
// factor_diag_tile; each block's finished entries go out as 16-byte vectors.
template <typename T, int CB>
__device__ void invert_tile(const T* l, const T* inv, float* out, int lane) {
  constexpr int V = 16 / sizeof(T);
  T w[TS];
#pragma unroll
  for (int i = 0; i < TS; ++i) w[i] = (i == lane) ? T(1) : T(0);
#pragma unroll 1
  for (int k0 = 0; k0 < TS; k0 += CB) {
#pragma unroll
    for (int c = 0; c < CB; ++c) {
      const int k = k0 + c;
      w[c] *= inv[k];
#pragma unroll
      for (int q = (c + 1) / V; q < TS / V; ++q) {
        if (k0 + V * q < TS) {
          T lv[V];
          load_vec16(l + k * TS + k0 + V * q, lv);
#pragma unroll
          for (int e = 0; e < V; ++e)
            if (V * q + e > c) w[V * q + e] = fma(-lv[e], w[c], w[V * q + e]);
        }
      }
    }
    // the finished entries k0 .. k0 + CB - 1 of column lane
    float4* o = reinterpret_cast<float4*>(out + lane * TS + k0);
#pragma unroll
    for (int q = 0; q < CB / 4; ++q)
      o[q] = make_float4((float)w[4 * q], (float)w[4 * q + 1], (float)w[4 * q + 2], (float)w[4 * q + 3]);
#pragma unroll
    for (int j = 0; j < TS - CB; ++j) w[j] = w[j + CB];
  }
}

// ---- FP64 blocks -------------------------------------------------------------
template <typename T, int CB>
__device__ void potrf_block(T* tiles, float* A, int lda, int s, int bs, const float* d, float* sh,
                            const PotrfParams& p, float* winv, DevStatus* st,
                            const StepState* prev, const float* rowsq) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int NT = (bs + TS - 1) / TS;
  __shared__ T s_shift[256];
  __shared__ T s_pmin[256];
  __shared__ T s_inv[256];
  __shared__ __align__(16) T s_col[2 * TS];
  __shared__ int s_fail, s_pert;
  if (tid == 0) { s_fail = -1; s_pert = 0; }
  const int prev_prec = (prev != nullptr && p.diag_pert && sh) ? prev->prec : FP32;
  for (int i = tid; i < NT * TS; i += blockDim.x) {
    T shv = T(0), pm = T(0);
    if (i < bs) {
      if (p.diag_pert && sh) {
        float shf = sh[s + i];
        if (prev_prec != FP32) {   // the previous step's shift for this row
          shf = __fmaf_rn(unit_roundoff(prev_prec), rowsq[s + i], shf);
          sh[s + i] = shf;
        }
        shv = T(p.pert) * T(shf);
      }
      pm = T(p.pivot_floor) * T(d[s + i]);
    }
    s_shift[i] = shv;
    s_pmin[i] = pm;
  }
  // FP64 path: batched loads from the FP32 matrix
  const int total = NT * NT * TSZ;
  for (int base = 0; base < total; base += 8 * blockDim.x) {
    float v[8];
    int dst[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = base + q * blockDim.x + tid;
      dst[q] = -1;
      v[q] = 0.0f;
      if (e < total) {
        const int T2 = e / TSZ, rc = e % TSZ;
        const int I = T2 % NT, J = T2 / NT, c = rc / TS, r = rc % TS;
        if (I >= J) {
          const int gr = I * TS + r, gc = J * TS + c;
          dst[q] = tidx(I, J) * TSZ + c * TS + r;
          if (gr < bs && gc < bs) v[q] = A[(size_t)(s + gc) * lda + (s + gr)];
          else v[q] = (gr == gc) ? 1.0f : 0.0f;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (dst[q] >= 0) tiles[dst[q]] = T(v[q]);
  }
  __syncthreads();
  // Step J: (A) the tiles below diagonal tile J are solved, one per warp;
  // (B) warps 0-3 apply column J to diagonal tile J+1 (8 columns each, one
  // warp per SM sub-partition) and warp 0 factors it at once, while warps
  // 1.. update the other trailing tiles, one tile per warp with 2-D register
  // blocks.  The factor of the next diagonal tile thus overlaps the trailing
  // update (look-ahead).
  auto factor_tile = [&](int J) {
    int nreal = bs - J * TS;
    nreal = nreal > TS ? TS : nreal;
    int fail = -1, npert = 0;
    const bool ok = factor_diag_tile<T, CB>(tiles + tidx(J, J) * TSZ, s_inv + J * TS, lane, nreal,
                                        s_shift + J * TS, s_pmin + J * TS, p.diag_pert, &npert,
                                        &fail, s_col);
    if (lane == 0) {
      if (!ok) s_fail = J * TS + fail;
      s_pert += npert;
    }
  };
  // J = -1 factors diagonal tile 0 alone; the factor has one call site, so
  // its code is in the kernel once.  Warp 0 carries the chain (the solve of
  // tile (J+1, J) and the factor of diagonal tile J+1) and has its SM
  // sub-partition to itself: the other warps of that sub-partition (warp %
  // 4 == 0) stay idle, and the helper warps (warp % 4 != 0) take the other
  // tile solves and the trailing updates.
  const int helper = (warp & 3) ? warp - (warp >> 2) - 1 : -1;
  const int nhelp = nwarps - nwarps / 4;
  for (int J = -1; J < NT - 1; ++J) {
    if (J >= 0) {
      if (s_fail >= 0) break;
      // warp 0 solves tile (J+1, J), the one the next diagonal tile waits
      // on; the helpers take the others
      if (warp == 0 && J + 1 < NT)
        trsm_tile<T, CB>(tiles + tidx(J + 1, J) * TSZ, tiles + tidx(J, J) * TSZ, s_inv + J * TS, lane);
      if (helper >= 0)
        for (int I = J + 2 + helper; I < NT; I += nhelp)
          trsm_tile<T, CB>(tiles + tidx(I, J) * TSZ, tiles + tidx(J, J) * TSZ, s_inv + J * TS, lane);
      __syncthreads();
    }
    if (warp < 4) {
      if (J >= 0) {
        // columns 8 warp .. +7 of diagonal tile J+1: lane (rg, cg) = (lane %
        // 8, lane / 8) owns rows 4 rg .. and columns 8 warp + 2 cg ..
        T* dt = tiles + tidx(J + 1, J + 1) * TSZ;
        const T* pj = tiles + tidx(J + 1, J) * TSZ;
        syrk_block<T, 4, 2>(dt, pj, pj, 4 * (lane & 7), 8 * warp + 2 * (lane >> 3));
        asm volatile("bar.sync 1, 128;" ::: "memory");   // warps 0-3
      }
      if (warp == 0) factor_tile(J + 1);
    }
    if (J >= 0 && helper >= 0) {
      // work items: the trailing tiles (I, K), J < K <= I, diagonal tile J+1
      // excluded, numbered down each tile column; one helper warp per tile
      int item = 0;
      for (int K = J + 1; K < NT; ++K) {
        const int i0 = (K == J + 1) ? K + 1 : K;
        for (int I = i0; I < NT; ++I, ++item) {
          if (item % nhelp != helper) continue;
          syrk_tile<T>(tiles + tidx(I, K) * TSZ, tiles + tidx(I, J) * TSZ,
                       tiles + tidx(K, J) * TSZ, lane);
        }
      }
    }
    __syncthreads();
  }
  if (s_fail >= 0) {
    if (tid == 0) set_status(st, MPCHOL_ERR_NOT_SPD, s + s_fail);
    return;
  }
  // write back, rounded to FP32
  for (int c = warp; c < bs; c += nwarps) {
    const int J = c / TS, cc = c % TS;
    for (int r = c + lane; r < bs; r += TS) {
      const int I = r / TS, rr = r % TS;
      A[(size_t)(s + c) * lda + (s + r)] = (float)tiles[tidx(I, J) * TSZ + cc * TS + rr];
    }
  }
  // inverses of the diagonal tiles, used by the panel solve
  for (int J = warp; J < NT; J += nwarps)
    invert_tile<T, CB>(tiles + tidx(J, J) * TSZ, s_inv + J * TS, winv + J * TS * TS, lane);
  if (tid == 0 && s_pert) atomicAdd(&st->perturbed, s_pert);
}

// ---- FP32 blocks -------------------------------------------------------------
// The chain of a block is its 256 pivots; the rest (28 tile solves and 84 tile
// products) has to stay off it.  Warp I (0 .. 7) owns tile row I, lane = row:
//   * for each tile column J < I it solves X(I, J), eight columns behind the
//     factor of diagonal tile J (follow_tile), having applied column J - 1 to
//     the tile itself;
//   * while it solves X(I, I - 1) it applies the finished columns to its
//     diagonal tile, kept in registers, so that its factor starts as soon as
//     the solve ends;
//   * it factors the diagonal tile (chain_tile), eight columns at a time: the
//     8 x 8 diagonal block goes to every lane through shared memory, each lane
//     factors it in registers (no shuffle on the pivot chain) and solves its
//     own row with it, and the update of the columns beyond the next eight
//     overlaps the next eight pivots;
//   * then it inverts the tile for the panel solve.
// The other warps apply columns 0 .. J - 2 to the tiles of column J >= 2 before
// their row's warp gets there, in the order of those deadlines.  The warps meet
// only on mbarriers (a column step of a factor, a solved tile, a tile brought
// up to date), all of one use and waited for in an order without cycles.
// Every element is one fma chain over the columns in order, whatever the
// schedule.  The loops stay rolled (register arrays shift by eight columns):
// instruction fetch, not arithmetic, bounded fully unrolled forms, whose code
// was refetched in every phase.  One SM's FP32 rate is the floor: 116 K warp
// fmas, about 41 K cycles at the 0.7 of peak that three-operand fmas reach.
// 256 x 256: 46 us a launch alone and 46 - 68 us (median 55, n = 8192) beside a
// trailing update, from its early start on; one
// pivot per shared-memory round trip with block barriers between tile solves
// and updates took 72 us, and 77 - 105 us beside the update.
constexpr int NPW = 8;          // panel warps: warp w holds tile row w
constexpr int SUB = 8;          // columns per step of the chain
constexpr int NSUB = TS / SUB;

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t d, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(d));
}
// two fused multiply-adds in one issue slot, each rounded as fmaf
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// a[0..7] -= x l[0..7], nx2 = (-x, -x), l 16-byte aligned
__device__ __forceinline__ void axpy8(float* a, uint64_t nx2, const float* l) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(l + 4 * q);
    unpack2(fma2(nx2, v.x, pack2(a[4 * q], a[4 * q + 1])), a[4 * q], a[4 * q + 1]);
    unpack2(fma2(nx2, v.y, pack2(a[4 * q + 2], a[4 * q + 3])), a[4 * q + 2], a[4 * q + 3]);
  }
}

// What the pivot rule needs of one tile column's rows, and what it found.
struct PivotRule {
  const float* shift;     // 32 entries each
  const float* pmin;
  const float* thr;       // a finite pivot above thr is taken as it is
  int nreal, diag_pert;
};
struct PivotLog {
  int fail = -1, npert = 0;
};

// Eight columns with the pivot rule in full (a pivot at or below its floor, not
// finite or denormal among them): D the 8 x 8 diagonal block by rows, x the
// lane's row, i its row in the block.  Uniform over the warp but for x.
__device__ __noinline__ void rare_block(const float* D, const PivotRule& pr, int c0, int i, float* x,
                                        float* my_inv, int lane, PivotLog* log) {
  float d[SUB * SUB];
  for (int e = 0; e < SUB * SUB; ++e) d[e] = D[e];
  for (int k = 0; k < SUB; ++k) {
    const Pivot<float> p = eval_pivot<float>(d[k * SUB + k], c0 + k < pr.nreal, pr.shift[c0 + k],
                                             pr.pmin[c0 + k], pr.diag_pert);
    log->npert += p.pert ? 1 : 0;
    if (p.bad && log->fail < 0) log->fail = c0 + k;
    if (lane == k) *my_inv = p.r;
    const float xk = i == k ? p.piv * p.r : x[k] * p.r;
    x[k] = xk;
    for (int e = k + 1; e < SUB; ++e) d[e * SUB + k] *= p.r;
    for (int e = k + 1; e < SUB; ++e)
      for (int c = k + 1; c <= e; ++c)
        d[e * SUB + c] = fmaf(-d[e * SUB + k], d[c * SUB + k], d[e * SUB + c]);
    for (int c = k + 1; c < SUB; ++c) x[c] = fmaf(-xk, d[c * SUB + k], x[c]);
  }
}

// The factor of a diagonal tile whose rows the lanes hold in a (column j of the
// lane's row in a[j]), into t (lower triangle); inv[k] = 1 / L(k,k); sub[s] is
// arrived at once columns 8 s .. 8 s + 7 are in shared memory.  D: an 8 x 8
// buffer.
__device__ __forceinline__ void chain_tile(float (&a)[TS], float* t, float* inv, float* D, int lane,
                                           const PivotRule& pr, uint64_t* sub, PivotLog& log) {
  float xp[SUB] = {};                              // the previous eight columns of the row
#pragma unroll 1
  for (int s = 0; s < NSUB; ++s) {
    const int c0 = SUB * s;
    const int i = lane - c0;                       // row of the diagonal block
    if (i >= 0 && i < SUB) {
      *reinterpret_cast<float4*>(D + i * SUB) = make_float4(a[0], a[1], a[2], a[3]);
      *reinterpret_cast<float4*>(D + i * SUB + 4) = make_float4(a[4], a[5], a[6], a[7]);
    }
    __syncwarp();
    float d[SUB][SUB];
#pragma unroll
    for (int r = 0; r < SUB; ++r)
#pragma unroll
      for (int q = 0; q <= r / 4; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(D + r * SUB + 4 * q);
        d[r][4 * q] = v.x; d[r][4 * q + 1] = v.y; d[r][4 * q + 2] = v.z; d[r][4 * q + 3] = v.w;
      }
    float sh[SUB], th[SUB];
    load_n<SUB>(pr.shift + c0, sh);
    load_n<SUB>(pr.thr + c0, th);
    // the columns after the next eight, by the previous eight
    if (s == 1 || s == 2) {
      const float* tp = t + (c0 - SUB) * TS + c0 + SUB;
#pragma unroll
      for (int m = 0; m < SUB; ++m) axpy8(a + SUB, pack2(-xp[m], -xp[m]), tp + m * TS);
      if (s == 1) {
#pragma unroll
        for (int m = 0; m < SUB; ++m) axpy8(a + 2 * SUB, pack2(-xp[m], -xp[m]), tp + m * TS + SUB);
      }
    }
    float x[SUB], my_inv = 1.0f;
    bool plain = true;
#pragma unroll
    for (int c = 0; c < SUB; ++c) x[c] = a[c];
#pragma unroll
    for (int k = 0; k < SUB; ++k) {
      const float piv = d[k][k] + sh[k];
      // rsqrtf's result (the bits agree for every positive normal argument, checked
      // over all of them; 2^-22.9 of the exact value at worst) at less than half its
      // latency.  A denormal pivot takes the full rule.
      float r;
      asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(piv));
      plain = plain && piv > th[k] && piv <= 3.402823466e38f;
      my_inv = lane == k ? r : my_inv;
      x[k] = i == k ? piv * r : x[k] * r;
#pragma unroll
      for (int e = k + 1; e < SUB; ++e) d[e][k] *= r;
#pragma unroll
      for (int e = k + 1; e < SUB; ++e)
#pragma unroll
        for (int c = k + 1; c <= e; ++c) d[e][c] = fmaf(-d[e][k], d[c][k], d[e][c]);
#pragma unroll
      for (int c = k + 1; c < SUB; ++c) x[c] = fmaf(-x[k], d[c][k], x[c]);
    }
    if (!plain) {
      float xr[SUB], ir = 1.0f;
#pragma unroll
      for (int c = 0; c < SUB; ++c) xr[c] = a[c];
      rare_block(D, pr, c0, i, xr, &ir, lane, &log);
#pragma unroll
      for (int c = 0; c < SUB; ++c) x[c] = xr[c];
      my_inv = ir;
    }
#pragma unroll
    for (int c = 0; c < SUB; ++c) {
      if (c <= i) t[(c0 + c) * TS + lane] = x[c];
      xp[c] = x[c];
    }
    if (lane < SUB) inv[c0 + lane] = my_inv;
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(&sub[s]);
    if (s + 1 < NSUB) {
#pragma unroll
      for (int m = 0; m < SUB; ++m)
        axpy8(a + SUB, pack2(-x[m], -x[m]), t + (c0 + m) * TS + c0 + SUB);
    }
#pragma unroll
    for (int j = 0; j < TS - SUB; ++j) a[j] = a[j + SUB];
  }
}

// A 32 x 32 tile spread over the warp as 8 x 4 blocks per lane, rows in pairs
// for packed fmas.  The blocks' numbers interleave the lane's bits so that four
// neighbouring lanes read two different vectors of each operand: such a
// 16-byte shared load takes 2.2 cycles of an SM, one with four different
// vectors 4.0.  The values are kept negated, so that the accumulation adds.
struct TileAcc {
  uint64_t v[4][4];                                // [column][row pair]
};
__device__ __forceinline__ int blk_row(int lane) { return 8 * ((lane & 1) | ((lane >> 1) & 2)); }
__device__ __forceinline__ int blk_col(int lane) { return 4 * (((lane >> 1) & 1) | ((lane >> 2) & 6)); }
constexpr uint64_t kSigns = 0x8000000080000000ull;
__device__ __forceinline__ void acc_load(TileAcc& c, const float* t, int lane) {
  t += blk_col(lane) * TS + blk_row(lane);
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(t + u * TS + 4 * q);
      c.v[u][2 * q] = w.x ^ kSigns;
      c.v[u][2 * q + 1] = w.y ^ kSigns;
    }
}
__device__ __forceinline__ void acc_store(const TileAcc& c, float* t, int lane) {
  t += blk_col(lane) * TS + blk_row(lane);
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      ulonglong2 w;
      w.x = c.v[u][2 * q] ^ kSigns;
      w.y = c.v[u][2 * q + 1] ^ kSigns;
      *reinterpret_cast<ulonglong2*>(t + u * TS + 4 * q) = w;
    }
}
// c -= A B^T over columns [k0, k1) (a multiple of 8) of the tiles a and b
__device__ __forceinline__ void acc_product(TileAcc& c, const float* a, const float* b, int lane, int k0,
                                            int k1) {
  a += blk_row(lane);
  b += blk_col(lane);
#pragma unroll 8
  for (int k = k0; k < k1; ++k) {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(a + k * TS);
    const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(a + k * TS + 4);
    const uint64_t av[4] = {a0.x, a0.y, a1.x, a1.y};
    float bv[4];
    load_n<4>(b + k * TS, bv);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint64_t bb = pack2(bv[u], bv[u]);
#pragma unroll
      for (int i = 0; i < 4; ++i) c.v[u][i] = fma2(av[i], bb, c.v[u][i]);
    }
  }
}

// X L^T = A for the tile whose rows the lanes hold in a, below diagonal tile l,
// eight columns behind its factor (sub as above), into x.  crit: dg, this
// row's diagonal tile, receives -X X^T on the way.
// Returns false if a bounded wait gave up.
__device__ __forceinline__ bool follow_tile(float (&a)[TS], float* x, const float* l, const float* inv,
                                            int lane, uint64_t* sub, bool crit, TileAcc& dg) {
  bool ok = true;
#pragma unroll 1
  for (int s = 0; s < NSUB; ++s) {
    const int c0 = SUB * s;
    ok = tc::mbar_wait(&sub[s], 0) && ok;
    const float* lb = l + c0 * TS + c0;            // L(c0 + c, c0 + m) at m * 32 + c
    float iv[SUB];
    load_n<SUB>(inv + c0, iv);
#pragma unroll
    for (int m = 0; m < SUB; ++m) {
      float lm[SUB];
      load_n<SUB>(lb + m * TS, lm);
      a[m] *= iv[m];
#pragma unroll
      for (int c = m + 1; c < SUB; ++c) a[c] = fmaf(-a[m], lm[c], a[c]);
    }
#pragma unroll
    for (int m = 0; m < SUB; ++m) x[(c0 + m) * TS + lane] = a[m];
#pragma unroll
    for (int g = 1; g < NSUB; ++g) {
      if (s + g < NSUB) {
#pragma unroll
        for (int m = 0; m < SUB; ++m) axpy8(a + SUB * g, pack2(-a[m], -a[m]), lb + m * TS + SUB * g);
      }
    }
    if (crit) {
      __syncwarp();
      acc_product(dg, x, x, lane, c0, c0 + SUB);
    }
#pragma unroll
    for (int j = 0; j < TS - SUB; ++j) a[j] = a[j + SUB];
  }
  return ok;
}

// Tile t of the lower ones (at most NPW rows of them), numbered by rows.
__device__ __forceinline__ void tile_of(int t, int& I, int& J) {
  I = 0;
#pragma unroll
  for (int r = 1; r < NPW; ++r) I += t >= r * (r + 1) / 2 ? 1 : 0;
  J = t - I * (I + 1) / 2;
}
// The block's lower tiles from global memory and back.  Whole tiles whose
// columns start on 16-byte boundaries move as 16-byte vectors, eight lanes to
// a column of 32 rows, nine loads in flight per thread (36 boxes by TMA take
// one thread's issue about 80 cycles each); anything else element by element,
// identity past the block.  The strictly upper part of a diagonal tile is
// left alone in global memory.
__device__ __forceinline__ void load_tiles(float* tiles, const float* A, int lda, int bs, int ntiles,
                                           bool vec, int tid) {
  if (vec) {
    const int r4 = 4 * (tid & 7), c = (tid & 255) >> 3;
    for (int t0 = tid >> 8; t0 < ntiles; t0 += 18) {
      float4 v[9];
#pragma unroll
      for (int u = 0; u < 9; ++u)
        if (t0 + 2 * u < ntiles) {
          int I, J;
          tile_of(t0 + 2 * u, I, J);
          v[u] = *reinterpret_cast<const float4*>(A + (size_t)(J * TS + c) * lda + I * TS + r4);
        }
#pragma unroll
      for (int u = 0; u < 9; ++u)
        if (t0 + 2 * u < ntiles) *reinterpret_cast<float4*>(tiles + (t0 + 2 * u) * TSZ + c * TS + r4) = v[u];
    }
  } else {
#pragma unroll 4
    for (int e = tid; e < ntiles * TSZ; e += 512) {
      int I, J;
      tile_of(e / TSZ, I, J);
      const int r = I * TS + e % TS, c = J * TS + e % TSZ / TS;
      tiles[e] = r < bs && c < bs ? A[(size_t)c * lda + r] : (r == c ? 1.0f : 0.0f);
    }
  }
}
// Tile t by the calling warp.
__device__ __forceinline__ void store_tile(const float* tiles, float* A, int lda, int bs, int t, bool vec,
                                           int lane) {
  int I, J;
  tile_of(t, I, J);
  tiles += t * TSZ;
  if (vec) {
    const int r4 = 4 * (lane & 7);
#pragma unroll 4
    for (int c = lane >> 3; c < TS; c += 4) {
      const float4 v = *reinterpret_cast<const float4*>(tiles + c * TS + r4);
      float* g = A + (size_t)(J * TS + c) * lda + I * TS + r4;
      if (I > J || r4 >= c) {
        *reinterpret_cast<float4*>(g) = v;
      } else if (r4 + 3 >= c) {                      // the vector the diagonal crosses
        if (r4 + 1 >= c) g[1] = v.y;
        if (r4 + 2 >= c) g[2] = v.z;
        g[3] = v.w;
      }
    }
  } else {
    const int r = I * TS + lane;
#pragma unroll 1
    for (int k = 0; k < TS; ++k) {
      const int c = J * TS + k;
      if (r < bs && c < bs && r >= c) A[(size_t)c * lda + r] = tiles[k * TS + lane];
    }
  }
}

__device__ __forceinline__ void
potrf_f32_block(float* tiles, float* A, int lda, int s, int bs, const float* d, float* sh,
                const PotrfParams& p, const int* fp64_flag, float* winv, DevStatus* st,
                const StepState* prev, const float* rowsq) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int NT = (bs + TS - 1) / TS;
  const int ntiles = NT * (NT + 1) / 2;
  __shared__ __align__(16) float s_shift[256];
  __shared__ __align__(16) float s_pmin[256];
  __shared__ __align__(16) float s_thr[256];
  __shared__ __align__(16) float s_inv[256];
  __shared__ __align__(16) float s_D[NPW][SUB * SUB];
  __shared__ int s_fail, s_pert, s_ok;
  // sub: column steps of the factors; done: solved tiles; fresh: tiles brought
  // up to date by the helpers
  __shared__ __align__(8) uint64_t sub[NPW * NSUB], done[NPW * (NPW + 1) / 2],
      fresh[NPW * (NPW + 1) / 2];
  float* const Ab = A + (size_t)s * lda + s;
  const bool vec = (reinterpret_cast<uintptr_t>(Ab) & 15) == 0 && lda % 4 == 0 && bs % TS == 0;
  if (tid >= 32 && tid < 32 + NPW * (NPW + 1) / 2) {
    if (tid - 32 < NPW * NSUB) tc::mbar_init(&sub[tid - 32], 1);
    tc::mbar_init(&done[tid - 32], 1);
    tc::mbar_init(&fresh[tid - 32], 1);
    tc::fence_mbar_init();
  }
  if (tid == 96) {
    s_fail = NPW * TS;       // none
    s_pert = 0;
    s_ok = st->code == 0 && (fp64_flag == nullptr || *fp64_flag == 0);
  }
  const int prev_prec = (prev != nullptr && p.diag_pert && sh) ? prev->prec : FP32;
  for (int i = tid; i < NT * TS; i += blockDim.x) {
    // rows past the block are identity: their pivots are 1
    float shv = 0.0f, pm = 0.0f, th = 1.175494351e-38f;
    if (i < bs) {
      if (p.diag_pert && sh) {
        float shf = sh[s + i];
        if (prev_prec != FP32)   // the previous step's shift for this row
          shf = __fmaf_rn(unit_roundoff(prev_prec), rowsq[s + i], shf);
        s_inv[i] = shf;          // stored once the block is known to be this kernel's
        shv = p.pert * shf;
      }
      pm = p.pivot_floor * d[s + i];
      // NaN bounds take every pivot to the full rule
      if (p.diag_pert && !(pm < th)) th = pm >= th ? pm : 3.402823466e38f;
    }
    s_shift[i] = shv;
    s_pmin[i] = pm;
    s_thr[i] = th;
  }
  load_tiles(tiles, Ab, lda, bs, ntiles, vec, tid);
  __syncthreads();
  if (!s_ok) return;
  if (p.diag_pert && sh && prev_prec != FP32)
    for (int i = tid; i < bs; i += blockDim.x) sh[s + i] = s_inv[i];
  __syncthreads();
  bool ok = true;
  if (warp < NT) {
    const int I = warp;
    float a[TS];
    TileAcc acc;
    float* const mine = tiles + tidx(I, I) * TSZ;
#pragma unroll 1
    for (int J = 0; J < I; ++J) {
      float* x = tiles + tidx(I, J) * TSZ;
      if (J >= 1) {
        if (J >= 2) ok = tc::mbar_wait(&fresh[tidx(I, J)], 0) && ok;
        ok = tc::mbar_wait(&done[tidx(J, J - 1)], 0) && ok;
        acc_load(acc, x, lane);
        acc_product(acc, tiles + tidx(I, J - 1) * TSZ, tiles + tidx(J, J - 1) * TSZ, lane, 0, TS);
        acc_store(acc, x, lane);
        __syncwarp();
      }
#pragma unroll
      for (int j = 0; j < TS; ++j) a[j] = x[j * TS + lane];
      const bool crit = J == I - 1;
      if (crit) {
        if (I >= 2) ok = tc::mbar_wait(&fresh[tidx(I, I)], 0) && ok;
        acc_load(acc, mine, lane);
      }
      ok = follow_tile(a, x, tiles + tidx(J, J) * TSZ, s_inv + J * TS, lane, sub + J * NSUB, crit, acc) && ok;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&done[tidx(I, J)]);
    }
    if (I > 0) acc_store(acc, mine, lane);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < TS; ++j) a[j] = mine[j * TS + lane];
    PivotLog log;
    const PivotRule pr{s_shift + I * TS, s_pmin + I * TS, s_thr + I * TS, min(TS, bs - I * TS), p.diag_pert};
    chain_tile(a, mine, s_inv + I * TS, s_D[I], lane, pr, sub + I * NSUB, log);
    if (lane == 0) {
      if (log.fail >= 0) atomicMin(&s_fail, I * TS + log.fail);
      if (log.npert) atomicAdd(&s_pert, log.npert);
    }
    // the inverse for the panel solve, where the SM has issue slots to spare: the
    // first two tiles' beside the last three columns, the last one's beside the
    // stores
    if (I < NT - 1) {
      if (I < 2) ok = tc::mbar_wait(&sub[max(I + 1, NT - 3) * NSUB], 0) && ok;
      invert_tile<float, SUB>(mine, s_inv + I * TS, winv + I * TS * TS, lane);
    }
  } else {
    // tile (I, K), K >= 2, by columns 0 .. K - 2, in column order over all
    // helpers: a task waits only for tiles that need tasks of earlier columns
    const int nhelp = nwarps - NT;
    int task = 0;
    for (int K = 2; K < NT; ++K)
      for (int I = K; I < NT; ++I, ++task) {
        if (task % nhelp != warp - NT) continue;
        TileAcc acc;
        acc_load(acc, tiles + tidx(I, K) * TSZ, lane);
#pragma unroll 1
        for (int j = 0; j < K - 1; ++j) {
          ok = tc::mbar_wait(&done[tidx(K, j)], 0) && ok;
          ok = tc::mbar_wait(&done[tidx(I, j)], 0) && ok;
          acc_product(acc, tiles + tidx(I, j) * TSZ, tiles + tidx(K, j) * TSZ, lane, 0, TS);
        }
        acc_store(acc, tiles + tidx(I, K) * TSZ, lane);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&fresh[tidx(I, K)]);
      }
  }
  if (__syncthreads_or(!ok)) {
    if (tid == 0) set_status(st, MPCHOL_ERR_TIMEOUT, s);
    return;
  }
  if (s_fail < NT * TS) {
    if (tid == 0) set_status(st, MPCHOL_ERR_NOT_SPD, s + s_fail);
    return;
  }
  if (warp == NT - 1) {
    invert_tile<float, SUB>(tiles + (ntiles - 1) * TSZ, s_inv + warp * TS, winv + warp * TS * TS, lane);
  } else {
    for (int t = warp < NT - 1 ? warp : warp - 1; t < ntiles; t += nwarps - 1)
      store_tile(tiles, Ab, lda, bs, t, vec, lane);
  }
  if (tid == 0 && s_pert) atomicAdd(&st->perturbed, s_pert);
}

// Separate kernels for the two precisions keep the FP64 register footprint out
// of the FP32 path.
__global__ void __launch_bounds__(512, 1)
potrf_f32_kernel(float* A, int lda, int s, int bs,
                 const float* d, float* sh, PotrfParams p, const int* fp64_flag, float* winv,
                 DevStatus* st, const StepState* prev, const float* rowsq) {
  tc::grid_dep_wait();      // the block's update and the step state are final
  tc::grid_dep_trigger();   // the next kernel may be scheduled (it waits too)
  extern __shared__ __align__(128) unsigned char smem_raw[];
  potrf_f32_block(reinterpret_cast<float*>(smem_raw), A, lda, s, bs, d, sh, p, fp64_flag, winv, st, prev,
                  rowsq);
}

// Batched: CTA i factors the current diagonal block of system i.
__global__ void __launch_bounds__(512, 1)
potrf_batched_kernel(BatchSys* __restrict__ sys, int s, int b, PotrfParams p) {
  const BatchSys& S = sys[blockIdx.x];
  const int bs = min(b, S.n - s);
  if (bs <= 0 || S.st->code != 0) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  potrf_f32_block(reinterpret_cast<float*>(smem_raw), S.A, S.ld, s, bs, S.d, S.sh, p, nullptr, S.winv,
                  S.st, nullptr, nullptr);
}

// FP64 blocks (flagged near-indefinite): tiles in a global scratch.
__global__ void __launch_bounds__(256, 1)
potrf_f64_kernel(float* A, int lda, int s, int bs, const float* d, float* sh,
                 PotrfParams p, const int* fp64_flag, double* scratch64, float* winv, DevStatus* st,
                 const StepState* prev, const float* rowsq) {
  if (st->code != 0) return;
  if (fp64_flag == nullptr || *fp64_flag == 0) return;
  potrf_block<double, 8>(scratch64, A, lda, s, bs, d, sh, p, winv, st, prev, rowsq);
}

}  // namespace

// the lower tiles of the block
size_t potrf_scratch64_elems(int bs) {
  const int NT = (bs + TS - 1) / TS;
  return (size_t)NT * (NT + 1) / 2 * TSZ;
}
size_t potrf_smem_bytes(int bs) { return potrf_scratch64_elems(bs) * sizeof(float); }

cudaError_t launch_potrf(float* A, int lda, int s, int bs,
                         const float* d, float* sh, const PotrfParams& p,
                         const int* fp64_flag, double* scratch64, float* winv, DevStatus* st,
                         bool may_fp64, cudaStream_t stream, const StepState* prev,
                         const float* rowsq) {
  const size_t smem = potrf_smem_bytes(256);
  cudaError_t e = cudaFuncSetAttribute(potrf_f32_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  PdlLaunch L(dim3(1), dim3(512), smem, stream);
  const int* flag = may_fp64 ? fp64_flag : nullptr;
  e = cudaLaunchKernelEx(&L.cfg, potrf_f32_kernel, A, lda, s, bs, d, sh, p, flag, winv, st,
                         prev, rowsq);
  if (e != cudaSuccess) return e;
  if (may_fp64)
    potrf_f64_kernel<<<1, 256, 0, stream>>>(A, lda, s, bs, d, sh, p, fp64_flag, scratch64, winv, st,
                                            prev, rowsq);
  return cudaGetLastError();
}

cudaError_t launch_potrf_batched(BatchSys* sys, int nact, int s, int b, const PotrfParams& p,
                                 cudaStream_t stream) {
  if (nact <= 0) return cudaSuccess;
  const size_t smem = potrf_smem_bytes(b);
  // the kernel's limit, not the launch's: the most any block needs
  cudaError_t e = cudaFuncSetAttribute(potrf_batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)potrf_smem_bytes(256));
  if (e != cudaSuccess) return e;
  potrf_batched_kernel<<<nact, 512, smem, stream>>>(sys, s, b, p);
  return cudaGetLastError();
}

}  // namespace mpchol
