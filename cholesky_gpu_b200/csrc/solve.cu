// PCG operator and preconditioner: y = A x and z = (L L^T)^-1 r.
//
// Replaces the reference's per-iteration cublasDgemv on FP64 A
// (src/mixed_cholesky.cu:185-191) and cusolverDnDpotrs on an FP64 copy of L
// (src/mixed_cholesky.cu:141,204-206).  Both read the FP32 lower triangle once
// per application, in 128 x 128 tiles, with FP64 vectors and accumulation.
//
// Triangular solves.  A row-by-row (or 128-block-by-block) substitution is a
// chain of n/128 dependent steps and runs at a few GB/s on one B200.  Instead,
// once per factor, the inverses W_S of the 1024-row diagonal super-blocks
// L_SS are formed by recursive doubling (FP64 128-block inverses, FP32 GEMM
// tiles above that).  A
// forward solve is then n/1024 steps of two fully parallel passes over tiles:
//     y_S  = W_S w_S                      (TRMV over the super-block's lower tiles)
//     w_T -= L_TS y_S   for T > S         (GEMV over the panel below)
// and the backward solve mirrors it with transposes; a single system's tiles
// run in one persistent launch, a batch's in a launch per pass.  The applied operator is
// (Lt Lt^T)^-1 with Lt = blockdiag(W_S^-1) + strictly-block-lower(L), which is
// symmetric positive definite whenever the W_S are nonsingular, so PCG stays
// well defined; it equals (L L^T)^-1 up to the FP32 rounding of the W_S.
// Partial sums of the products, of far panel tiles and of a batch's passes are
// combined with FP64 atomics; those on the persistent solve's chain go through
// tagged slots where there are one or two right-hand sides.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "pcg.cuh"

namespace mpchol {
cudaError_t solve_set_attributes();
namespace {

constexpr int RB = 128;     // tile size
constexpr int NTH = 256;    // 8 warps: warp w owns tile columns 16w..16w+15
constexpr int RS = 1024;    // super-block rows

template <typename TA>
__device__ __forceinline__ void load4(const TA* p, int nvalid, float out[4]);
template <>
__device__ __forceinline__ void load4<float>(const float* p, int nvalid, float out[4]) {
  if (nvalid >= 4 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p));
    out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
  } else {
#pragma unroll
    for (int r = 0; r < 4; ++r) out[r] = (r < nvalid) ? __ldg(p + r) : 0.0f;
  }
}

// Tile loaded into registers: lane covers rows 4*lane..4*lane+3, warp covers
// CH consecutive columns starting at col0.  Elements outside (rows_valid,
// cols_valid) are zero.  Every load of the batch is issued before any use.
// Tile values stay in the matrix's own type in registers (FP32 tiles take
// half the registers of a widened copy); they are widened at each use.
template <int CH>
__device__ __forceinline__ void load_cols(const float* T, int ld, int rloc, int rows_valid,
                                          int col0, int cols_valid, float (&v)[CH][4]) {
  const int nv = min(4, rows_valid - rloc);
#pragma unroll
  for (int cc = 0; cc < CH; ++cc) {
    const int c = col0 + cc;
    if (c < cols_valid && nv > 0) load4<float>(T + (size_t)c * ld + rloc, nv, v[cc]);
    else v[cc][0] = v[cc][1] = v[cc][2] = v[cc][3] = 0.0f;
  }
}

template <int CH>
__device__ __forceinline__ void load_cols(const double* T, int ld, int rloc, int rows_valid,
                                          int col0, int cols_valid, double (&v)[CH][4]) {
  const int nv = min(4, rows_valid - rloc);
#pragma unroll
  for (int cc = 0; cc < CH; ++cc) {
    const int c = col0 + cc;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      v[cc][r] = (c < cols_valid && r < nv) ? __ldg(T + (size_t)c * ld + rloc + r) : 0.0;
  }
}

// Sum each of the W per-lane values w[i] (W = 8 or 16) over the 32 lanes of
// the warp: a butterfly that halves the values a lane keeps at each step
// (W/2 + W/4 + ... shuffles), then plain xor steps for the remaining lane
// bits.  Lane l ends with the sum of column col_of_lane<W>(l); the lanes
// that differ only in the low 5 - log2(W) bits hold the same sum.
template <int W>
__device__ __forceinline__ int col_of_lane(int lane) {
  int c = 0;
#pragma unroll
  for (int off = 16, h = W / 2; h >= 1; off >>= 1, h >>= 1) c += ((lane & off) ? h : 0);
  return c;
}
template <int W>
__device__ __forceinline__ double butterfly(double (&w)[W], int lane) {
  int off = 16;
#pragma unroll
  for (int h = W / 2; h >= 1; h >>= 1, off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double send = upper ? w[i] : w[i + h];
      const double keep = upper ? w[i + h] : w[i];
      w[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  double v = w[0];
#pragma unroll
  for (; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// Accumulate a 128 x 128 tile times a vector segment.
//   NOTRANS: part[r][k] += T[r][c] * vin[k][c]   (per-thread rows, summed over the warp's columns)
//   TRANS  : colsum[k][c] = sum_r T[r][c] * vin[k][r], the CH columns of a chunk reduced
//            over the warp together by one butterfly per rhs
// (staged vectors and column sums are k-major: [k * RB + index])
// `mask`: 0 none, 1 keep r >= c (lower incl. diagonal), 2 keep r > c.
template <typename TA, int NR, int CH>
__device__ __forceinline__ void tile_pass(const TA* T, int ld, int rows_valid, int cols_valid,
                                          const double* vin_cols, const double* vin_rows,
                                          double (&acc)[4][NR], double* colsum_smem, int mask_nt,
                                          int mask_t, bool do_nt, bool do_t) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rloc = 4 * lane;
  constexpr int LOWBITS = (CH == 16) ? 1 : 3;   // lanes holding the same column sum
#pragma unroll
  for (int cb = 0; cb < 16; cb += CH) {
    TA v[CH][4];
    load_cols<CH>(T, ld, rloc, rows_valid, warp * 16 + cb, cols_valid, v);
    if (do_nt) {
#pragma unroll
      for (int cc = 0; cc < CH; ++cc) {
        const int c = warp * 16 + cb + cc;
#pragma unroll
        for (int k = 0; k < NR; ++k) {
          const double xc = vin_cols[k * RB + c];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const bool keep = mask_nt == 0 || (mask_nt == 1 ? (rloc + r >= c) : (rloc + r > c));
            if (keep) acc[r][k] = fma((double)v[cc][r], xc, acc[r][k]);
          }
        }
      }
    }
    if (do_t) {
      // one rhs at a time (bounded register pressure for NR > 2)
#pragma unroll 1
      for (int k = 0; k < NR; ++k) {
        // this lane's four rows of the rhs, read once (two 16-byte loads)
        const double2 x01 = *reinterpret_cast<const double2*>(vin_rows + k * RB + rloc);
        const double2 x23 = *reinterpret_cast<const double2*>(vin_rows + k * RB + rloc + 2);
        const double xr[4] = {x01.x, x01.y, x23.x, x23.y};
        double w[CH];
#pragma unroll
        for (int cc = 0; cc < CH; ++cc) {
          const int c = warp * 16 + cb + cc;
          double sacc = 0.0;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const bool keep = mask_t == 0 || (mask_t == 1 ? (rloc + r >= c) : (rloc + r > c));
            if (keep) sacc = fma((double)v[cc][r], xr[r], sacc);
          }
          w[cc] = sacc;
        }
        const double sum = butterfly<CH>(w, lane);
        if ((lane & LOWBITS) == 0)
          colsum_smem[k * RB + warp * 16 + cb + col_of_lane<CH>(lane)] = sum;
      }
    }
  }
}

// The per-warp row partials of tile_pass(NOTRANS) in shared memory (ends with a
// barrier) and the sum of element e = k * RB + r over the warps.
template <int NR>
__device__ __forceinline__ void stage_rows(double (&acc)[4][NR], double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int k = 0; k < NR; ++k) red[(warp * NR + k) * RB + 4 * lane + r] = acc[r][k];
  __syncthreads();
}
template <int NR>
__device__ __forceinline__ double row_sum(const double* red, int e) {
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < NTH / 32; ++w) s += red[w * NR * RB + e];
  return s;
}

// Reduce the per-warp row partials and add sign * sum into out[row0 + r]
// (rows < nvalid) with FP64 atomics.
template <int NR>
__device__ __forceinline__ void flush_rows(double (&acc)[4][NR], double* red, double* out, int n,
                                           int row0, int nvalid, double sign) {
  stage_rows<NR>(acc, red);
  for (int e = threadIdx.x; e < RB * NR; e += NTH) {
    const int k = e / RB, r = e % RB;
    if (r < nvalid) atomicAdd(&out[(size_t)k * n + row0 + r], sign * row_sum<NR>(red, e));
  }
}

// Vector segments are read from L2 (ld.global.cg): inside the persistent
// solve other CTAs produce them with atomics while this SM may hold older
// lines of the same arrays in L1.
template <int NR>
__device__ __forceinline__ void load_vec(const double* x, int n, int row0, int nvalid, double* s) {
  // k-major in shared memory (s[k * RB + r]): a lane's rows are contiguous
  for (int e = threadIdx.x; e < RB * NR; e += NTH) {
    const int k = e / RB, r = e % RB;
    s[e] = (r < nvalid) ? __ldcg(x + (size_t)k * n + row0 + r) : 0.0;
  }
}

__device__ __forceinline__ void tri_of(int t, int& i, int& j) {
  int a = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
  while (a * (a + 1) / 2 > t) --a;
  while ((a + 1) * (a + 2) / 2 <= t) ++a;
  i = a;
  j = t - a * (a + 1) / 2;
}

// ---- tiles staged in shared memory -------------------------------------------
// The streaming kernels (SYMV, the persistent triangular solve) copy each
// 128 x 128 FP32 tile into shared memory with cp.async, one stage per CTA and
// two or three CTAs per SM: the copies hold no registers, and one CTA's copy is
// in flight (64 KB) while the others compute on theirs.
constexpr int TILE_ELEMS = RB * RB;   // 64 KB of FP32
constexpr int SCH = 8;                // columns per widened chunk

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Copy the rows_valid x cols_valid tile at T (column-major, leading dimension
// ld; T and ld keep 16-byte alignment) into a dense 128 x 128 column-major
// tile; everything outside the valid part is zero-filled by the copies.
// A warp copies one 512-byte column per instruction.
__device__ __forceinline__ void stage_tile(float* dst, const float* T, int ld, int rows_valid,
                                           int cols_valid) {
#pragma unroll 4
  for (int e = threadIdx.x; e < TILE_ELEMS / 4; e += NTH) {
    const int c = e / (RB / 4), r = 4 * (e % (RB / 4));
    const bool ok = c < cols_valid && r < rows_valid;
    cp_async16(dst + c * RB + r, ok ? T + (size_t)c * ld + r : T, ok ? 4 * min(4, rows_valid - r) : 0);
  }
}

// x[k * n + row0 + r] -> s[k * RB + r], zero for r >= nvalid (8-byte copies:
// n may be odd)
template <int NR>
__device__ __forceinline__ void stage_vec(const double* x, int n, int row0, int nvalid, double* s) {
  for (int e = threadIdx.x; e < RB * NR; e += NTH) {
    const int k = e / RB, r = e % RB;
    const bool ok = r < nvalid;
    cp_async8(s + e, ok ? x + (size_t)k * n + row0 + r : x, ok ? 8 : 0);
  }
}

// tile_pass on a staged tile.  Each lane widens its 4 x SCH chunk to FP64
// once and uses it for every rhs of both products.  DIAG: a diagonal tile of
// a symmetric operator stored lower -- NOTRANS keeps r >= c, TRANS r > c.
// FRO: also adds the tile's share of ||A||_F^2 to *fsq (the lower triangle,
// off-diagonal entries twice).
template <int NR, bool DIAG, bool FRO = false>
__device__ __forceinline__ void tile_pass_staged(const float* Ts, const double* vin_cols,
                                                 const double* vin_rows, double (&acc)[4][NR],
                                                 double* colsum_smem, bool do_nt, bool do_t,
                                                 double* fsq = nullptr) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rloc = 4 * lane;
  constexpr int LOWBITS = 3;   // lanes holding the same column sum (SCH = 8)
#pragma unroll
  for (int cb = 0; cb < 16; cb += SCH) {
    double dv[SCH][4];
#pragma unroll
    for (int cc = 0; cc < SCH; ++cc) {
      const int c = warp * 16 + cb + cc;
      const float4 f = *reinterpret_cast<const float4*>(Ts + c * RB + rloc);
      dv[cc][0] = f.x; dv[cc][1] = f.y; dv[cc][2] = f.z; dv[cc][3] = f.w;
      if (DIAG) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (rloc + r < c) dv[cc][r] = 0.0;
      }
      if (FRO) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
          *fsq = fma((DIAG && rloc + r == c) ? dv[cc][r] : 2.0 * dv[cc][r], dv[cc][r], *fsq);
      }
    }
    if (do_nt) {
#pragma unroll
      for (int cc = 0; cc < SCH; cc += 2) {
        const int c = warp * 16 + cb + cc;
#pragma unroll
        for (int k = 0; k < NR; ++k) {
          const double2 xc = *reinterpret_cast<const double2*>(vin_cols + k * RB + c);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            acc[r][k] = fma(dv[cc][r], xc.x, acc[r][k]);
            acc[r][k] = fma(dv[cc + 1][r], xc.y, acc[r][k]);
          }
        }
      }
    }
    if (do_t) {
#pragma unroll 1
      for (int k = 0; k < NR; ++k) {
        const double2 x01 = *reinterpret_cast<const double2*>(vin_rows + k * RB + rloc);
        const double2 x23 = *reinterpret_cast<const double2*>(vin_rows + k * RB + rloc + 2);
        const double xr[4] = {x01.x, x01.y, x23.x, x23.y};
        double w[SCH];
#pragma unroll
        for (int cc = 0; cc < SCH; ++cc) {
          const int c = warp * 16 + cb + cc;
          double sacc = 0.0;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const double a = (DIAG && rloc + r == c) ? 0.0 : dv[cc][r];
            sacc = fma(a, xr[r], sacc);
          }
          w[cc] = sacc;
        }
        const double sum = butterfly<SCH>(w, lane);
        if ((lane & LOWBITS) == 0)
          colsum_smem[k * RB + warp * 16 + cb + col_of_lane<SCH>(lane)] = sum;
      }
    }
  }
}

// ---- eight right-hand sides on the FP64 tensor cores ---------------------
// With 8 rhs the tile passes are FP64-FMA bound (16 FMAs per tile element for
// the symmetric product), so they run as mma.sync m8n8k4 FP64 (DMMA): a warp
// owns 16 rows of the tile for the row sums and 16 columns for the column
// sums, and its accumulator fragments hold finished 8 x 8 (rows x rhs)
// blocks -- no butterflies and no cross-warp reduction.  Fragments follow the
// PTX ISA for m8n8k4.f64: a = A[lane / 4][lane % 4], b = B[lane % 4][lane / 4],
// d[i] = D[lane / 4][2 (lane % 4) + i].
//
// The tile is staged in a blocked layout in which both fragment patterns
// read 32 distinct banks: 4-row x 8-column blocks of 32 floats (column-major
// inside a block, so a 16-byte copy of 4 rows of one column lands contiguous),
// 16 blocks per 4-row group, and the groups 528 floats apart (16 banks of
// stagger between neighbouring groups).  Vector segments are staged k-major
// with a row of XS = 132 doubles per rhs.
constexpr int BL_RG = 16 * 32 + 16;          // floats per 4-row group
constexpr int BL_TILE = (RB / 4) * BL_RG;    // floats per blocked tile
constexpr int XS = RB + 4;                   // doubles per rhs in a staged segment

__device__ __forceinline__ int bl_off(int r, int c) {
  return (r >> 2) * BL_RG + (c >> 3) * 32 + (c & 7) * 4 + (r & 3);
}

__device__ __forceinline__ void dmma_m8n8k4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// stage_tile into the blocked layout
__device__ __forceinline__ void stage_tile_bl(float* dst, const float* T, int ld, int rows_valid,
                                              int cols_valid) {
#pragma unroll 4
  for (int e = threadIdx.x; e < TILE_ELEMS / 4; e += NTH) {
    const int c = e / (RB / 4), r = 4 * (e % (RB / 4));
    const bool ok = c < cols_valid && r < rows_valid;
    cp_async16(dst + bl_off(r, c), ok ? T + (size_t)c * ld + r : T,
               ok ? 4 * min(4, rows_valid - r) : 0);
  }
}

// x[k * n + row0 + r] -> s[k * XS + r] (zero past nvalid), 8 rhs
__device__ __forceinline__ void stage_vec_x8(const double* x, int n, int row0, int nvalid, double* s) {
  for (int e = threadIdx.x; e < RB * 8; e += NTH) {
    const int k = e / RB, r = e % RB;
    const bool ok = r < nvalid;
    cp_async8(s + k * XS + r, ok ? x + (size_t)k * n + row0 + r : x, ok ? 8 : 0);
  }
}
// the same through L2 loads (the persistent solve's segments are produced by
// other CTAs' atomics)
__device__ __forceinline__ void load_vec_x8(const double* x, int n, int row0, int nvalid, double* s) {
  for (int e = threadIdx.x; e < RB * 8; e += NTH) {
    const int k = e / RB, r = e % RB;
    s[k * XS + r] = (r < nvalid) ? __ldcg(x + (size_t)k * n + row0 + r) : 0.0;
  }
}

// One blocked tile T (rows i0.., columns j0..) times 8 rhs on the DMMA pipe:
//   do_nt: y_rows[row0 + r] += sign * sum_c T[r][c] x_c[c]   (rows < nrows)
//   do_t : y_cols[col0 + c] += sign * sum_r T[r][c] x_r[r]   (columns < ncols)
// by FP64 atomics.  DIAG (a diagonal tile of a symmetric operator stored
// lower): the row sums keep r >= c, the column sums r > c.  FRO: adds the
// tile's share of ||A||_F^2 (off-diagonal entries twice) to *fsq.
// KC k-steps of fragments are loaded (and widened) per chunk and UNR chunks
// are unrolled, so the next chunk's loads overlap this chunk's DMMAs; ONLY
// fixes the product at compile time (1: row sums, 2: column sums, 0: by
// do_nt / do_t).  Both products: KC = 8, UNR = 2 (the 128 registers of two
// CTAs per SM allow no more); one product: KC = 4 fully unrolled.
// NACC accumulators share the k-steps of an output in turn: each is a chain of
// 32 / NACC DMMAs.
template <bool DIAG, bool FRO, int KC = 8, int UNR = 2, int ONLY = 0, int NACC = 2>
__device__ __forceinline__ void tile_mma_x8(const float* Ts, const double* x_c, const double* x_r,
                                            double* y_rows, int row0, int nrows, double* y_cols,
                                            int col0, int ncols, int n, bool do_nt_rt, bool do_t_rt,
                                            double sign, double* fsq) {
  const bool do_nt = ONLY == 1 ? true : (ONLY == 2 ? false : do_nt_rt);
  const bool do_t = ONLY == 2 ? true : (ONLY == 1 ? false : do_t_rt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int B0 = 16 * warp;
  // accumulators: [m-block][k-step % NACC] -- eight independent DMMA chains
  // per warp when both products run with two
  double dn[2][NACC][2] = {};
  double dt[2][NACC][2] = {};
  static_assert(KC % NACC == 0, "a chunk's k-steps go round the accumulators whole times");
#pragma unroll(UNR)
  for (int kb = 0; kb < RB; kb += 4 * KC) {
    // every fragment of the chunk is loaded (and widened) before its DMMAs
    float an[2][KC], at[2][KC];
    double bn[KC], bt[KC];
#pragma unroll
    for (int j = 0; j < KC; ++j) {
      const int k0 = kb + 4 * j;
      if (do_nt) {
        bn[j] = x_c[g * XS + k0 + t];
#pragma unroll
        for (int mb = 0; mb < 2; ++mb) {
          const int r = B0 + 8 * mb + g, c = k0 + t;
          const float v = Ts[bl_off(r, c)];
          an[mb][j] = (DIAG && r < c) ? 0.0f : v;
        }
      }
      if (do_t) {
        bt[j] = x_r[g * XS + k0 + t];
#pragma unroll
        for (int mb = 0; mb < 2; ++mb) {
          const int c = B0 + 8 * mb + g, r = k0 + t;
          const float v = Ts[bl_off(r, c)];
          at[mb][j] = (DIAG && r <= c) ? 0.0f : v;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < KC; ++j) {
      if (do_nt) {
#pragma unroll
        for (int mb = 0; mb < 2; ++mb) {
          const double a = (double)an[mb][j];
          if (FRO) {
            const int r = B0 + 8 * mb + g, c = kb + 4 * j + t;
            *fsq = fma((DIAG && r == c) ? a : 2.0 * a, a, *fsq);
          }
          dmma_m8n8k4(dn[mb][j % NACC], a, bn[j]);
        }
      }
      if (do_t) {
#pragma unroll
        for (int mb = 0; mb < 2; ++mb) dmma_m8n8k4(dt[mb][j % NACC], (double)at[mb][j], bt[j]);
      }
    }
  }
#pragma unroll
  for (int mb = 0; mb < 2; ++mb) {
#pragma unroll
    for (int h = NACC / 2; h > 1; h >>= 1)             // the accumulators in pairs
#pragma unroll
      for (int q = 0; q < h; ++q)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          dn[mb][q][i] += dn[mb][q + h][i];
          dt[mb][q][i] += dt[mb][q + h][i];
        }
    const int idx = B0 + 8 * mb + g;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = 2 * t + i;
      if (do_nt && idx < nrows)
        atomicAdd(&y_rows[(size_t)k * n + row0 + idx], sign * (dn[mb][0][i] + dn[mb][1][i]));
      if (do_t && idx < ncols)
        atomicAdd(&y_cols[(size_t)k * n + col0 + idx], sign * (dt[mb][0][i] + dt[mb][1][i]));
    }
  }
}

// A tile whose columns need not start on 16-byte boundaries, by 4-byte
// copies into the plain (BL = false) or blocked (BL = true) layout.
template <bool BL>
__device__ __forceinline__ void stage_tile_4b(float* dst, const float* T, int ld, int rows_valid,
                                              int cols_valid) {
#pragma unroll 4
  for (int e = threadIdx.x; e < TILE_ELEMS; e += NTH) {
    const int c = e / RB, r = e % RB;
    const bool ok = c < cols_valid && r < rows_valid;
    cp_async4(dst + (BL ? bl_off(r, c) : c * RB + r), ok ? T + (size_t)c * ld + r : T, ok ? 4 : 0);
  }
}

// CTAs per SM of the staged SYMV, each with one stage (tile + x_J + x_I, and the
// column sums): a CTA's load overlaps the others' tile passes, and 16 or 24
// warps hide the FP64 and shared-memory latencies better than one CTA with its
// tiles staged two ahead.  One rhs, n = 8192: 36 us -> 30; two, 4100: 15.3 ->
// 13.8; four, 2999: 21.5 -> 18.3; eight, 16384: 331 -> 306.
template <int NR>
constexpr int symv_ctas() { return NR == 1 ? 3 : 2; }
template <int NR>
constexpr size_t symv_staged_smem() {
  if (NR == 8)   // blocked tiles and padded segments, no column-sum buffer
    return BL_TILE * sizeof(float) + 2 * (size_t)XS * 8 * sizeof(double);
  return TILE_ELEMS * sizeof(float) + 3 * (size_t)RB * NR * sizeof(double);
}

// ---- y += A x, FP32 symmetric A (lower triangle), persistent over the tiles.
// CTA b takes tiles b, b + grid, ...; each tile is staged together with its two
// vector segments.  The row partials are
// reduced in the stage's own tile buffer once the tile has been used.
// fro != nullptr: CTA b also writes its share of ||A||_F^2 (lower triangle,
// off-diagonal entries twice) to fro[b] and zeroes fro[gridDim.x ..nfro).
// al16: the columns of A start on 16-byte boundaries.  Eight right-hand sides
// (AL, fixed at compile time there): columns that do not start so used to be
// summed in short chains by FMAs, so their DMMA passes, one product at a time,
// spread the sums over eight accumulators (relative error of a product at n =
// 2999: 2.4e-16 with FMAs, 44 us; 3.3e-16 with two accumulators, 17.4; 2.5e-16
// with eight, 16.8).
template <int NR, bool AL = true>
__global__ void __launch_bounds__(NTH, symv_ctas<NR>())
symv_staged_kernel(const float* __restrict__ A, int lda, int n, const double* __restrict__ x,
                   double* __restrict__ y, const int* skip, double* fro, int nfro, int al16) {
  if (skip != nullptr && *skip) return;
  constexpr bool MMA = NR == 8;
  constexpr int TE = MMA ? BL_TILE : TILE_ELEMS;      // floats of the staged tile
  constexpr int VEC = MMA ? XS * 8 : RB * NR;         // doubles per staged segment
  extern __shared__ __align__(16) unsigned char sm_raw[];
  float* Ts = reinterpret_cast<float*>(sm_raw);
  double* xJ = reinterpret_cast<double*>(Ts + TE);
  double* xI = xJ + VEC;
  double* s_col = xI + VEC;
  const int T = ceil_div(n, RB);
  const int ntiles = T * (T + 1) / 2;
  auto issue = [&](int i0, int ni, int j0, int nj) {
    const float* T = A + (size_t)j0 * lda + i0;
    if (MMA) {
      if (AL) stage_tile_bl(Ts, T, lda, ni, nj);
      else stage_tile_4b<true>(Ts, T, lda, ni, nj);
      stage_vec_x8(x, n, j0, nj, xJ);
      stage_vec_x8(x, n, i0, ni, xI);
    } else {
      if (al16) stage_tile(Ts, T, lda, ni, nj);
      else stage_tile_4b<false>(Ts, T, lda, ni, nj);
      stage_vec<NR>(x, n, j0, nj, xJ);
      stage_vec<NR>(x, n, i0, ni, xI);
    }
  };
  double fsq = 0.0;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int I, J;
    tri_of(t, I, J);
    const int i0 = I * RB, j0 = J * RB;
    const int ni = min(RB, n - i0), nj = min(RB, n - j0);
    issue(i0, ni, j0, nj);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (MMA) {
      // row sums to y_I, column sums to y_J, straight from the fragments
      auto pass = [&](auto diag, auto f) {
        constexpr bool D = decltype(diag)::value, F = decltype(f)::value;
        if constexpr (AL) {
          tile_mma_x8<D, F>(Ts, xJ, xI, y, i0, ni, y, j0, nj, n, true, true, 1.0, &fsq);
        } else {
          tile_mma_x8<D, F, 8, 2, 1, 8>(Ts, xJ, xI, y, i0, ni, y, j0, nj, n, true, false, 1.0, &fsq);
          tile_mma_x8<D, false, 8, 2, 2, 8>(Ts, xJ, xI, y, i0, ni, y, j0, nj, n, false, true, 1.0, nullptr);
        }
      };
      if (fro != nullptr) {
        if (I == J) pass(std::true_type{}, std::true_type{});
        else pass(std::false_type{}, std::true_type{});
      } else {
        if (I == J) pass(std::true_type{}, std::false_type{});
        else pass(std::false_type{}, std::false_type{});
      }
      __syncthreads();   // the stage is free again
      continue;
    }
    double acc[4][NR] = {};
    if (fro != nullptr) {
      if (I == J) tile_pass_staged<NR, true, true>(Ts, xJ, xI, acc, s_col, true, true, &fsq);
      else tile_pass_staged<NR, false, true>(Ts, xJ, xI, acc, s_col, true, true, &fsq);
    } else {
      if (I == J) tile_pass_staged<NR, true>(Ts, xJ, xI, acc, s_col, true, true);
      else tile_pass_staged<NR, false>(Ts, xJ, xI, acc, s_col, true, true);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < VEC; e += NTH) {
      const int k = e / RB, c = e % RB;
      if (c < nj) atomicAdd(&y[(size_t)k * n + j0 + c], s_col[e]);
    }
    flush_rows<NR>(acc, reinterpret_cast<double*>(Ts), y, n, i0, ni, 1.0);
    __syncthreads();   // the stage and s_col are free again
  }
  if (fro != nullptr) {
    // block sum in a fixed order: warps, then the CTA's warps in turn
    double v = fsq;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    double* wsum = reinterpret_cast<double*>(Ts);   // the stage is free
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < NTH / 32; ++w) t += wsum[w];
      fro[blockIdx.x] = t;
    }
    for (int e = gridDim.x + blockIdx.x; e < nfro; e += gridDim.x)
      if (threadIdx.x == 0) fro[e] = 0.0;
  }
}

// ---- y += A x, symmetric A, lower triangle only (one CTA per lower tile) ----
template <typename TA, int NR>
__device__ __forceinline__ void
symv_body(const TA* __restrict__ A, int lda, int n, const double* __restrict__ x,
            double* __restrict__ y, const int* skip, uint3 bid) {
  if (skip != nullptr && *skip) return;
  __shared__ __align__(16) double s_xJ[RB * NR];
  __shared__ __align__(16) double s_xI[RB * NR];
  __shared__ double s_col[RB * NR];
  extern __shared__ double s_red[];
  int I, J;
  tri_of(bid.x, I, J);
  const int i0 = I * RB, j0 = J * RB;
  const int ni = min(RB, n - i0), nj = min(RB, n - j0);
  load_vec<NR>(x, n, j0, nj, s_xJ);
  load_vec<NR>(x, n, i0, ni, s_xI);
  __syncthreads();
  double acc[4][NR] = {};
  const bool diag = (I == J);
  tile_pass<TA, NR, 8>(A + (size_t)j0 * lda + i0, lda, ni, nj, s_xJ, s_xI, acc, s_col, diag ? 1 : 0, diag ? 2 : 0, true, true);
  __syncthreads();
  // column sums go to y_J
  for (int e = threadIdx.x; e < RB * NR; e += NTH) {
    const int k = e / RB, c = e % RB;
    if (c < nj) atomicAdd(&y[(size_t)k * n + j0 + c], s_col[e]);
  }
  flush_rows<NR>(acc, s_red, y, n, i0, ni, 1.0);
}

template <typename TA, int NR>
__global__ void __launch_bounds__(NTH)
symv_kernel(const TA* __restrict__ A, int lda, int n, const double* __restrict__ x,
            double* __restrict__ y, const int* skip) {
  symv_body<TA, NR>(A, lda, n, x, y, skip, blockIdx);
}

// ---- setup: super-block inverses by recursive doubling ---------------------
// For a lower-triangular [A 0; B C], inv = [A^-1 0; X C^-1] with
// X = -C^-1 (B A^-1).  The inverses W_S of the RS-row diagonal super-blocks
// are built bottom-up: the 128-row diagonal blocks in FP64 (32-row tiles on
// the FP64 tensor cores), then the 128 -> 1024 doublings as 32 x 32 FP32 GEMM
// tiles over all super-blocks at once.
// Storage: W_S is RS x RS column-major at wsup + S*RS*RS.  Its lower 128-tiles
// hold the inverse (diagonal tiles with a zero upper part); the strictly
// upper 128-tiles are scratch for the doubling products T = B A^-1 and are
// never read by the solves.

// FP64 32 x 32 tiles in shared memory: column-major, 36 doubles per column,
// so both DMMA fragment patterns (four consecutive rows of four columns 36
// apart) read 16 different 8-byte banks per half-warp.
constexpr int DT = 32;
constexpr int DLD = 36;
constexpr int DTSZ = DT * DLD;
constexpr int BT = RB / DT;                       // tiles per 128-block side
__host__ __device__ constexpr int dtri(int i, int j) { return i * (i + 1) / 2 + j; }
// the block's ten lower tiles, the column's solved tiles below its diagonal
// one, one product
constexpr int BI_TILES = BT * (BT + 1) / 2 + (BT - 1) + 1;
constexpr size_t kBlockInvSmem = (size_t)BI_TILES * DTSZ * sizeof(double);

// The 32 x 32 product A B added to the warp's two 8 x 8 blocks: rows 8 mb..,
// columns 8 nb.. and 8 (nb + 1)..
__device__ __forceinline__ void dtile_mma(const double* A, const double* B, int mb, int nb, int g,
                                          int t, double (&acc)[2][2]) {
#pragma unroll
  for (int k0 = 0; k0 < DT; k0 += 4) {
    const double a = A[(k0 + t) * DLD + 8 * mb + g];
#pragma unroll
    for (int u = 0; u < 2; ++u) dmma_m8n8k4(acc[u], a, B[(8 * (nb + u) + g) * DLD + k0 + t]);
  }
}

// Columns 32 q .. 32 q + 31 of the inverse of one 128-row diagonal block
// (bid.x = 4 block + q), 256 threads, FP64; the FP32 result goes to its
// diagonal tile of W_S.  Rows and columns past n are identity.  The columns
// of an inverse are independent, so four CTAs share a block and each runs
// only the tile rows from q down:
//   W_q = L_qq^-1,  W_i = -L_ii^-1 (L_iq W_q + .. + L_i,i-1 W_i-1)
// with the diagonal tiles inverted side by side, one warp each.  Latency
// bound (the 32 dependent steps of a tile inverse, then up to three pairs of
// products): 13 us for up to 37 blocks, 45 us for the 128 blocks of n = 16384
// (one CTA per block with 8-byte shared loads per FMA: 80 and 84 us).
__device__ __forceinline__ void
block_inverse_body(const float* __restrict__ L, int ldl, int n, float* __restrict__ wsup, uint3 bid) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  double* Lt = reinterpret_cast<double*>(sm_raw);           // tile (i, j) at dtri(i, j) * DTSZ
  double* Wt = Lt + BT * (BT + 1) / 2 * DTSZ;               // W_i, i > q, at (i - 1) * DTSZ
  double* Pt = Wt + (BT - 1) * DTSZ;                        // the product
  const int g0 = bid.x / BT, q = bid.x % BT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = g0 * RB;
  const int nb = min(RB, n - i0);
  // the lower tiles of tile columns q.., four loads in flight per thread
  for (int j = q; j < BT; ++j)
    for (int i = j; i < BT; ++i) {
      float v[DT * DT / NTH];
#pragma unroll
      for (int u = 0; u < DT * DT / NTH; ++u) {
        const int e = tid + u * NTH, c = DT * j + e / DT, r = DT * i + e % DT;
        v[u] = (r < nb && c < nb) ? (r >= c ? L[(size_t)(i0 + c) * ldl + i0 + r] : 0.0f)
                                  : (r == c ? 1.0f : 0.0f);
      }
#pragma unroll
      for (int u = 0; u < DT * DT / NTH; ++u) {
        const int e = tid + u * NTH;
        Lt[dtri(i, j) * DTSZ + (e / DT) * DLD + e % DT] = (double)v[u];
      }
    }
  __syncthreads();
  // diagonal tiles, in place: lane j of warp w solves L_tt w = e_j (t = q + w;
  // right-looking, the column held in registers)
  if (q + warp < BT) {
    double* T = Lt + dtri(q + warp, q + warp) * DTSZ;
    const double rinv = 1.0 / T[lane * DLD + lane];
    double w[DT];
#pragma unroll
    for (int i = 0; i < DT; ++i) w[i] = (i == lane) ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < DT; ++k) {
      w[k] *= __shfl_sync(0xffffffffu, rinv, k);
#pragma unroll
      for (int i = k + 1; i < DT; ++i) w[i] = fma(-T[k * DLD + i], w[k], w[i]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < DT; ++i) T[lane * DLD + i] = w[i];
  }
  __syncthreads();
  const int S = i0 / RS, tb = (i0 % RS) / RB;
  float* out = wsup + (size_t)S * RS * RS + (size_t)(tb * RB + DT * q) * RS + tb * RB;
  // rows above the tile column are zero, then its diagonal tile
  for (int e = tid; e < DT * DT * (q + 1); e += NTH) {
    const int c = e % DT, r = e / DT;              // r < 32 (q + 1)
    out[(size_t)c * RS + r] = r < DT * q ? 0.0f : (float)Lt[dtri(q, q) * DTSZ + c * DLD + r - DT * q];
  }
  const int g = lane >> 2, t = lane & 3, mb = warp >> 1, nb8 = 2 * (warp & 1);
  for (int i = q + 1; i < BT; ++i) {
    double acc[2][2] = {};
    dtile_mma(Lt + dtri(i, q) * DTSZ, Lt + dtri(q, q) * DTSZ, mb, nb8, g, t, acc);
    for (int j = q + 1; j < i; ++j)
      dtile_mma(Lt + dtri(i, j) * DTSZ, Wt + (j - 1) * DTSZ, mb, nb8, g, t, acc);
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int e = 0; e < 2; ++e) Pt[(8 * (nb8 + u) + 2 * t + e) * DLD + 8 * mb + g] = -acc[u][e];
    __syncthreads();
    double x[2][2] = {};
    dtile_mma(Lt + dtri(i, i) * DTSZ, Pt, mb, nb8, g, t, x);
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * (nb8 + u) + 2 * t + e, r = 8 * mb + g;
        Wt[(i - 1) * DTSZ + c * DLD + r] = x[u][e];
        out[(size_t)c * RS + DT * i + r] = (float)x[u][e];
      }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(NTH)
block_inverse_kernel(const float* __restrict__ L, int ldl, int n, float* __restrict__ wsup) {
  block_inverse_body(L, ldl, n, wsup, blockIdx);
}

// C(32 x 32) = A(32 x K) B(K x 32), all column-major, FP32 FMA, by 256 threads
// as four groups of 64: group q takes k = 16 q .. 16 q + 15 of every 64-deep
// chunk with 4 x 4 outputs per thread, and the groups' sums are added at the
// end in a fixed order.  The next chunk travels in registers; the lanes' bits
// interleave into tx and ty so that four neighbouring lanes read two different
// 16-byte vectors of each operand (2.2 cycles of shared memory a load; 4.0 with
// four).  A chunk costs its load latency before it costs its FMAs, so the small
// tile wins at every order: four CTAs per SM in place of two, and 256 tiles for
// a super-block's largest doubling.  All the levels (B200, n = 1024 / 3000 /
// 8192 / 16384): 103 / 121 / 176 / 306 us with 64 x 64 tiles and 8 x 8 outputs,
// 39 / 66 / 137 / 248 with these.
// Rows of A past a_rows are zero.  K is a multiple of 64.  Thread (tx, ty): rows
// 4 tx.., columns ty + 8 j.
constexpr int GT = 32;
constexpr int GKC = 64;
constexpr int GLDB = GKC + 4;                        // floats per staged column of B
constexpr int G_AS = GKC * GT, G_BS = GT * GLDB;
constexpr int G_SMEM = 2 * (G_AS + G_BS);            // two chunks; the reduction reuses them
static_assert(G_SMEM >= 2 * GT * GT, "two groups' sums fit");

__device__ __forceinline__ void gemm32_load(const float* A, int lda, int a_rows, const float* B, int ldb,
                                            int k0, float4 (&ra)[2], float4 (&rb)[2]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int e = threadIdx.x + NTH * u;
    const int r = 4 * (e % (GT / 4));
    const float* p = A + (size_t)(k0 + e / (GT / 4)) * lda + r;
    if (r + 3 < a_rows) {
      ra[u] = *reinterpret_cast<const float4*>(p);
    } else {
      ra[u].x = r < a_rows ? p[0] : 0.0f;
      ra[u].y = r + 1 < a_rows ? p[1] : 0.0f;
      ra[u].z = r + 2 < a_rows ? p[2] : 0.0f;
      ra[u].w = 0.0f;
    }
    rb[u] = *reinterpret_cast<const float4*>(B + (size_t)(e / (GKC / 4)) * ldb + k0 + 4 * (e % (GKC / 4)));
  }
}

__device__ __forceinline__ void gemm32_lane(int& tx, int& ty) {
  const int l = threadIdx.x % 32;
  tx = (l & 1) | ((l >> 1) & 6);
  ty = ((l >> 1) & 1) | ((l >> 3) & 2) | ((threadIdx.x >> 3) & 4);
}

__device__ __forceinline__ void gemm32(const float* A, int lda, int a_rows, const float* B, int ldb,
                                       int K, float (&acc)[4][4], float* sm) {
  const int tid = threadIdx.x, grp = tid / 64;
  int tx, ty;
  gemm32_lane(tx, ty);
  float4 ra[2], rb[2];
  gemm32_load(A, lda, a_rows, B, ldb, 0, ra, rb);
  for (int k0 = 0, buf = 0; k0 < K; k0 += GKC, buf ^= 1) {
    float* As = sm + buf * (G_AS + G_BS);          // [k][row]
    float* Bs = As + G_AS;                          // [column][k]
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int e = tid + NTH * u;
      *reinterpret_cast<float4*>(As + 4 * e) = ra[u];
      *reinterpret_cast<float4*>(Bs + (e / (GKC / 4)) * GLDB + 4 * (e % (GKC / 4))) = rb[u];
    }
    __syncthreads();   // this buffer's last reader passed the previous barrier
    if (k0 + GKC < K) gemm32_load(A, lda, a_rows, B, ldb, k0 + GKC, ra, rb);
#pragma unroll 1
    for (int kq = 0; kq < GKC / 4; kq += 4) {
      const int k = GKC / 4 * grp + kq;
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        b[j] = *reinterpret_cast<const float4*>(Bs + (ty + 8 * j) * GLDB + k);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 a = *reinterpret_cast<const float4*>(As + (k + e) * GT + 4 * tx);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float bv = e == 0 ? b[j].x : (e == 1 ? b[j].y : (e == 2 ? b[j].z : b[j].w));
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i][j] = fmaf(av[i], bv, acc[i][j]);
        }
      }
    }
  }
  // groups 2 and 3 onto 0 and 1, then 1 onto 0
#pragma unroll
  for (int half = 2; half >= 1; half >>= 1) {
    __syncthreads();
    if (grp >= half && grp < 2 * half) {
      float* d = sm + (grp - half) * GT * GT + (tid % 64);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) d[(j * 4 + i) * 64] = acc[i][j];
    }
    __syncthreads();
    if (grp < half) {
      const float* d = sm + grp * GT * GT + (tid % 64);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][j] += d[(j * 4 + i) * 64];
    }
  }
}

// One doubling level of half-size h (a multiple of RB) for pair bid.y of
// super-block bid.z; bid.x enumerates the (h/32)^2 output tiles.
//   PHASE 0:  T(ti,tj) = sum_{kt >= tj} L(h + ti, kt) A^-1(kt, tj)  -> upper-right scratch
//   PHASE 1:  X(ti,tj) = -sum_{kt <= ti} C^-1(ti, kt) T(kt, tj)     -> lower-left block
// (indices relative to the pair's origin a0 = 2 h * pair; the sums over k
// start and end at multiples of 64, where the inverses are zero on the wrong
// side of the diagonal).  64-row groups that start at or past n are skipped:
// the solves never read them.
template <int PHASE>
__device__ __forceinline__ void
superinv_gemm_body(const float* __restrict__ L, int ldl, int n, float* __restrict__ wsup, int h, uint3 bid) {
  __shared__ __align__(16) float sm[G_SMEM];
  const int tpr = h / GT;
  const int ti = bid.x / tpr, tj = bid.x % tpr;
  const int S = bid.z, s0 = S * RS, a0 = bid.y * 2 * h;
  const int r0 = ti * GT, c0 = tj * GT;
  if (s0 + a0 + h + (r0 & ~63) >= n) return;
  const int grow = s0 + a0 + h + r0;               // first global row of the output tile
  float* W = wsup + (size_t)S * RS * RS;
  float acc[4][4] = {};
  float* out;
  if (PHASE == 0) {
    const int k0 = c0 & ~63;
    gemm32(L + (size_t)(s0 + a0 + k0) * ldl + grow, ldl, min(GT, n - grow),
           W + (size_t)(a0 + c0) * RS + a0 + k0, RS, h - k0, acc, sm);
    out = W + (size_t)(a0 + h + c0) * RS + a0 + r0;
  } else {
    gemm32(W + (size_t)(a0 + h) * RS + a0 + h + r0, RS, GT,
           W + (size_t)(a0 + h + c0) * RS + a0, RS, (r0 & ~63) + 64, acc, sm);
    out = W + (size_t)(a0 + c0) * RS + a0 + h + r0;
  }
  if (threadIdx.x >= 64) return;                   // group 0 holds the sums
  const float sg = PHASE == 0 ? 1.0f : -1.0f;
  int tx, ty;
  gemm32_lane(tx, ty);
#pragma unroll
  for (int j = 0; j < 4; ++j)
    *reinterpret_cast<float4*>(out + (size_t)(ty + 8 * j) * RS + 4 * tx) =
        make_float4(sg * acc[0][j], sg * acc[1][j], sg * acc[2][j], sg * acc[3][j]);
}

template <int PHASE>
__global__ void __launch_bounds__(NTH, 4)
superinv_gemm_kernel(const float* __restrict__ L, int ldl, int n, float* __restrict__ wsup, int h) {
  superinv_gemm_body<PHASE>(L, ldl, n, wsup, h, blockIdx);
}

// ---- y_S += W_S w_S (TRANS: z_S += W_S^T w_S) over the super-block's lower tiles
template <int NR, bool TRANS>
__device__ __forceinline__ void
trmv_super_body(const float* __restrict__ W, int n, int s0, int rs, const double* __restrict__ in,
                  double* __restrict__ out, const int* skip, uint3 bid) {
  if (skip != nullptr && *skip) return;
  __shared__ __align__(16) double s_v[RB * NR];
  __shared__ double s_col[RB * NR];
  extern __shared__ double s_red[];
  int i, j;
  tri_of(bid.x, i, j);
  const int ri0 = s0 + i * RB, rj0 = s0 + j * RB;
  const int ni = min(RB, s0 + rs - ri0), nj = min(RB, s0 + rs - rj0);
  if (!TRANS) load_vec<NR>(in, n, rj0, nj, s_v);
  else load_vec<NR>(in, n, ri0, ni, s_v);
  __syncthreads();
  double acc[4][NR] = {};
  const float* T = W + (size_t)(j * RB) * RS + i * RB;
  tile_pass<float, NR, 16>(T, RS, ni, nj, s_v, s_v, acc, s_col, 0, 0, !TRANS, TRANS);
  __syncthreads();
  if (!TRANS) {
    flush_rows<NR>(acc, s_red, out, n, ri0, ni, 1.0);
  } else {
    for (int e = threadIdx.x; e < RB * NR; e += NTH) {
      const int k = e / RB, c = e % RB;
      if (c < nj) atomicAdd(&out[(size_t)k * n + rj0 + c], s_col[e]);
    }
  }
}


// ---- panel updates ---------------------------------------------------------
// forward: w[rows below the super-block] -= L(rows, super-block cols) y_S
// backward: w[cols left of the super-block] -= L(super-block rows, cols)^T z_S
template <int NR, bool TRANS>
__device__ __forceinline__ void
panel_body(const float* __restrict__ L, int ldl, int n, int s0, int rs,
             const double* __restrict__ v, double* __restrict__ w, const int* skip, uint3 bid) {
  if (skip != nullptr && *skip) return;
  __shared__ __align__(16) double s_v[RB * NR];
  __shared__ double s_col[RB * NR];
  extern __shared__ double s_red[];
  int r0, c0, nr_, nc_;
  if (!TRANS) {
    r0 = s0 + rs + bid.x * RB;  c0 = s0 + bid.y * RB;
    nr_ = min(RB, n - r0);           nc_ = min(RB, s0 + rs - c0);
    load_vec<NR>(v, n, c0, nc_, s_v);
  } else {
    r0 = s0 + bid.y * RB;       c0 = bid.x * RB;
    nr_ = min(RB, s0 + rs - r0);     nc_ = min(RB, s0 - c0);
    load_vec<NR>(v, n, r0, nr_, s_v);
  }
  __syncthreads();
  double acc[4][NR] = {};
  tile_pass<float, NR, 16>(L + (size_t)c0 * ldl + r0, ldl, nr_, nc_, s_v, s_v, acc, s_col, 0, 0,
                           !TRANS, TRANS);
  __syncthreads();
  if (!TRANS) {
    flush_rows<NR>(acc, s_red, w, n, r0, nr_, -1.0);
  } else {
    for (int e = threadIdx.x; e < RB * NR; e += NTH) {
      const int k = e / RB, c = e % RB;
      if (c < nc_) atomicAdd(&w[(size_t)k * n + c0 + c], -s_col[e]);
    }
  }
}


// ---- persistent triangular solve -------------------------------------------
// One launch per solve.  The tiles of a solve form a dependency DAG: the
// TRMV tiles of W_S (which need every panel contribution to their input
// segment) and the panel tiles below (forward) or left of (backward) S (which
// need their segment of y_S / z_S complete).  Units are handed out by an
// atomic counter in a topological order (trsv_job: grouped by the
// super-block they feed), so a unit only ever waits on units already taken
// by running CTAs; the launch is cooperative, so all CTAs are resident and
// every wait ends.
//
// The chain of a solve is TRMV tile -> panel tile from S into its neighbour
// S' ("near") -> TRMV tile of S', two links per super-block.  What a link costs
// beyond its tile is the hand-over.  With 1 or 2 right-hand sides each TRMV and
// near tile writes its 128 partial sums into a slot of its own, every number
// beside a tag that names the launch and the super-block, and the tiles that
// need the segment read the slots of its 1 to 8 contributors until the tags
// match, adding them in a fixed order: one L2 write and one read, no fence, no
// counter and no atomic in between.  The other panel tiles ("far") are off the
// chain: they add into the right-hand side with FP64 atomics and count per
// 128-row segment:
//   seg_in[g]   far contributions received by segment g (global 128-tile g)
//   seg_out[g]  segment g of the result is in `out` (the last TRMV tile that
//               contributes to it adds the slots and writes it)
// Slots are used in turn by odd and even super-blocks: a slot is written again
// only after tiles that wait, through the chain, for every reader of its last
// use.
// With 4 or 8 right-hand sides a segment's slots would hold as many bytes as the
// tile or twice that: there every tile adds with atomics, seg_in counts all
// panel tiles and seg_out the finished TRMV tiles of the segment (slots for 4:
// 0 to 5% slower).
// One right-hand side, forward / backward, against atomics and counters
// throughout, units in the order of need alone and bound to a CTA a unit early
// (B200): n = 6144 45 / 49 -> 39 / 45 us, 8192 63 / 69 -> 57 / 65, 16384 172 / 188
// -> 145 / 158; eight: 16384 291 / 291 -> 282 / 274.  With two super-blocks, where
// every unit runs at once, the decoding of the order shows: n = 2048, two
// right-hand sides, 13.7 / 16.7 -> 15.6 / 18.9 (the launches saved around a pair
// of solves make up for it: 86 -> 84 us for mpchol_apply_precond).
// Waits are bounded; a wait that runs out records MPCHOL_ERR_TIMEOUT and the
// unit proceeds (the result is then wrong, but no CTA waits forever).
constexpr long long kTrsvMaxPolls = 1ll << 24;

__device__ __forceinline__ void wait_count(const int* ctr, int need, DevStatus* st, int unit) {
  if (threadIdx.x == 0) {
    long long it = 0;
    while (*reinterpret_cast<const volatile int*>(ctr) < need) {
      if (++it > kTrsvMaxPolls) {
        if (st != nullptr) set_status(st, MPCHOL_ERR_TIMEOUT, unit);
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
  }
  __syncthreads();
}

__device__ __forceinline__ void signal_count(int* ctr) {
  __threadfence();                            // this thread's atomics visible device-wide
  __syncthreads();                            // ... for every thread of the unit
  if (threadIdx.x == 0) atomicAdd(ctr, 1);
}

// A slot's element: 16 bytes, written and read in one access.
struct __align__(16) TrsvSlot { double v; unsigned long long tag; };
constexpr int kSlotSegs = 64;                 // slots per parity and kind: 8 contributors of 8 segments
constexpr int kSlotNr = 2;                    // most right-hand sides that use them
constexpr long long kSlotMaxPolls = 1ll << 22;

__device__ __forceinline__ void slot_put(TrsvSlot* p, double v, unsigned long long tag) {
  asm volatile("{\n.reg .b128 t;\nmov.b128 t, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ void slot_get(const TrsvSlot* p, double& v, unsigned long long& tag) {
  long long lo;
  asm volatile("{\n.reg .b128 t;\nld.relaxed.gpu.global.b128 t, [%2];\nmov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(tag)
               : "l"(p)
               : "memory");
  v = __longlong_as_double(lo);
}

// s[e] = base(e) + the nin (1 to 8) contributions of a segment, in order, once
// their tags match; base(e): row0 + e of x (null: zero).  One right-hand side:
// two threads per element, which take the even and the odd contributions (the
// odd sums pass through tmp).  Ends with a barrier.
template <int NR>
__device__ __forceinline__ void gather_slots(const TrsvSlot* slots, int nin, unsigned long long tag,
                                             const double* x, int n, int row0, int nvalid, double* s,
                                             double* tmp, DevStatus* st, int unit) {
  constexpr int STR = NR == 1 ? 2 : 1, PER = 8 / STR;
  const int half = NR == 1 ? threadIdx.x / RB : 0;
  long long polls = 0;
#pragma unroll 1
  for (int e = NR == 1 ? threadIdx.x % RB : threadIdx.x; e < RB * NR; e += NTH) {
    const int r = e % RB;
    double sum = (half == 0 && x != nullptr && r < nvalid) ? __ldcg(x + (size_t)(e / RB) * n + row0 + r) : 0.0;
    double v[PER];
    bool all;
    do {
      unsigned long long t[PER];
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        t[q] = tag;
        v[q] = 0.0;
        const int p = q * STR + half;
        if (p < nin) slot_get(slots + (size_t)p * RB * NR + e, v[q], t[q]);
      }
      all = true;
#pragma unroll
      for (int q = 0; q < PER; ++q) all = all && t[q] == tag;
      if (!all && ++polls > kSlotMaxPolls) {
        if (st != nullptr) set_status(st, MPCHOL_ERR_TIMEOUT, unit);
        break;
      }
    } while (!all);
#pragma unroll
    for (int q = 0; q < PER; ++q) sum += v[q];
    if (half == 0) s[e] = sum;
    else tmp[e] = sum;
    if (NR == 1) break;
  }
  if (NR == 1) {
    __syncthreads();
    if (half == 0) s[threadIdx.x] += tmp[threadIdx.x];
  }
  __syncthreads();
}

// One unit of the solve: a tile, the vector segment it reads, where its
// result goes and the counters it waits on and signals.
struct TrsvJob {
  const float* T;       // tile origin (column-major)
  int ld, nrow, ncol;   // leading dimension, valid rows / columns
  int vin_row0, vin_n;  // input segment (of out for panels, of work for TRMV)
  int out_row0, out_n;  // output segment
  bool nt;              // NOTRANS (row sums) or TRANS (column sums)
  bool panel;           // L panel tile (reads out, writes work) or W_S tile
  const int* wait_ctr;
  int wait_need;
  int* sig_ctr;         // null: nothing waits on a counter of this unit
  // slots (0: the input is a vector / the result is added to one)
  int in_slot, nin;     // first slot and number of the input segment's contributions
  int in_blk;           // the super-block in their tags
  int out_slot, out_blk;
  int fin_slot, nfin;   // the unit that completes a segment: its contributions
};

// The order of the units.  Positions count super-blocks in solve order
// (forward: block p, backward: block NS-1-p); chain(p): the near tiles (p-1 ->
// p), then the TRMV tiles of p; far (a -> b), b >= a + 2: the other panel tiles.
//   chain(0);  for p = 0, 1, ..: chain(p+1), far tiles with 3 p + 2 <= 2 a + b < 3 p + 5
//   (by 2 a + b, then by a)
// Topological: 2 a + b < 3 p + 5 and b >= a + 2 give a <= p, so the sources of a
// stage's far tiles are solved by chains before it, and far tiles into p + 2
// (a <= p, so 2 a + b <= 3 p + 2) stand before chain(p+2).  The chain's tiles
// stand a stage ahead, so that they are staged when their input arrives, and
// 2 a + b brings a far tile up between its source and its need, which spreads
// the far work over the solve (in the order of need alone, grouped by b, half
// the CTAs waited on unsolved sources while tiles that were ready stood further
// back, and the chain waited for far tiles from the fourth super-block on).
// A CTA asks for numbers in increasing order, so the stage is found by moving
// on from that of its last unit.
struct TrsvCursor { int stage, first; };     // stage p (-1: chain(0)) and its first unit

template <bool TRANS, bool SLOTS>
__device__ __forceinline__ bool trsv_job(int u, TrsvCursor& cu, const float* L, int ldl, int n,
                                         const float* wsup, int* seg_in, int* seg_out, TrsvJob& jb) {
  const int ntiles = ceil_div(n, RB);
  const int NS = ceil_div(n, RS);
  constexpr int NSUB = RS / RB;              // segments of a full super-block
  jb.nin = jb.nfin = 0;
  jb.out_slot = -1;
  // first slot of segment q of super-block S: kind 0 its TRMV sums, kind 1 its
  // near panel contributions
  auto slot0 = [&](int S, int kind, int q) { return ((S & 1) * 2 + kind) * kSlotSegs + q * NSUB; };
  auto block = [&](int p) { return TRANS ? NS - 1 - p : p; };
  auto nsub = [&](int S) { return min(NSUB, ntiles - S * NSUB); };
  // panel tiles (source position a -> target position b)
  auto pair_units = [&](int a, int b) { return TRANS ? nsub(block(a)) * NSUB : NSUB * nsub(block(b)); };
  // far pairs with 2 a + b = k: a = lo .. lo + count - 1; the last super-block,
  // which may be partial, is in the first of them if in any
  auto far_lo = [&](int k) { return max(0, (k - NS + 2) / 2); };
  auto far_count = [&](int k) { return max(0, (k - 2) / 3 - far_lo(k) + 1); };
  auto far_units = [&](int k) {
    const int c = far_count(k);
    return c == 0 ? 0 : pair_units(far_lo(k), k - 2 * far_lo(k)) + (c - 1) * NSUB * NSUB;
  };
  auto trmv_units = [&](int p) {
    const int nb = nsub(block(p));
    return nb * (nb + 1) / 2;
  };
  int a = -1, b = 0;                         // positions; a < 0: a TRMV tile of b
  bool far = false;
  for (;; ++cu.stage) {
    const int p = cu.stage, near = p >= 0 ? pair_units(p, p + 1) : 0, trmv = trmv_units(p + 1);
    int v = u - cu.first, k = 3 * p + 2;
    if (v < near + trmv) {
      if (v < near) a = p;
      else v -= near;
      b = p + 1;
      u = v;
      break;
    }
    v -= near + trmv;
    int units = 0;
    if (p >= 0)
      for (; k < 3 * p + 5; ++k) {
        units = far_units(k);
        if (v < units) break;
        v -= units;
      }
    if (p >= 0 && k < 3 * p + 5) {
      far = true;
      a = far_lo(k);
      const int first = pair_units(a, k - 2 * a);
      if (v >= first) { a += 1 + (v - first) / (NSUB * NSUB); v = (v - first) % (NSUB * NSUB); }
      b = k - 2 * a;
      u = v;
      break;
    }
    if (p + 2 >= NS) return false;
    cu.first = u - v;
  }
  const int B = block(b), b0 = B * RS, nsubB = nsub(B), gB = b0 / RB;
  const int nsubN = b == 0 ? 0 : nsub(block(b - 1));   // segments of B's neighbour in the chain
  if (a >= 0) {
    const int T = block(a), t0 = T * RS, gT = t0 / RB, nsubT = nsub(T);
    jb.panel = true;
    jb.ld = ldl;
    // forward: w(rows r of B) -= L(r, T col c) y_T(c); backward: w(col segment c
    // of B) -= L(T row r, c)^T z_T(r)
    const int r = u / NSUB, c = u % NSUB;
    const int src = TRANS ? r : c, dst = TRANS ? c : r;
    const int r0 = (TRANS ? t0 : b0) + r * RB, c0 = (TRANS ? b0 : t0) + c * RB;
    jb.T = L + (size_t)c0 * ldl + r0;
    jb.nrow = min(RB, n - r0); jb.ncol = RB;
    jb.nt = !TRANS;
    jb.vin_row0 = TRANS ? r0 : c0; jb.vin_n = TRANS ? jb.nrow : RB;
    jb.out_row0 = TRANS ? c0 : r0; jb.out_n = TRANS ? RB : jb.nrow;
    if (!SLOTS || far) {
      jb.wait_ctr = seg_out + gT + src;
      jb.wait_need = SLOTS ? 1 : TRANS ? nsubT - src : src + 1;
      jb.sig_ctr = seg_in + gB + dst;
    } else {
      // polling the slots starts once the source's far contributions are in
      jb.wait_ctr = seg_in + gT + src;
      jb.wait_need = TRANS ? max(0, ntiles - gT - 2 * NSUB) : max(0, gT - NSUB);
      jb.sig_ctr = nullptr;
      jb.in_slot = slot0(T, 0, src) + (TRANS ? src : 0);
      jb.nin = TRANS ? nsubT - src : src + 1;
      jb.in_blk = T;
      jb.out_slot = slot0(B, 1, dst) + src;
      jb.out_blk = B;
    }
    return true;
  }
  int i, j;
  tri_of(u, i, j);
  const int ri0 = b0 + i * RB, rj0 = b0 + j * RB;
  jb.T = wsup + (size_t)B * RS * RS + (size_t)(j * RB) * RS + i * RB;
  jb.ld = RS;
  jb.nrow = min(RB, n - ri0);
  jb.ncol = min(RB, n - rj0);
  jb.panel = false;
  jb.nt = !TRANS;
  // forward: y_B(i) += W(i,j) w_B(j): w_B(j) has all gB panel contributions;
  // backward: z_B(j) += W(i,j)^T w_B(i): w_B(i) has the contributions of
  // every segment below B
  const int in = TRANS ? i : j, o = TRANS ? j : i;
  jb.vin_row0 = TRANS ? ri0 : rj0; jb.vin_n = TRANS ? jb.nrow : jb.ncol;
  jb.out_row0 = TRANS ? rj0 : ri0; jb.out_n = TRANS ? jb.ncol : jb.nrow;
  jb.wait_ctr = seg_in + gB + in;
  jb.wait_need = TRANS ? ntiles - gB - nsubB : gB;
  jb.sig_ctr = seg_out + gB + o;
  if (SLOTS) {
    jb.wait_need -= nsubN;                   // the near ones come through slots
    jb.in_slot = slot0(B, 1, in); jb.nin = nsubN; jb.in_blk = B;
    jb.out_slot = slot0(B, 0, o) + (TRANS ? i : j); jb.out_blk = B;
    // the last unit of segment o (in the order of the units) completes it
    const bool last = TRANS ? i == nsubB - 1 : i == j;
    if (last) { jb.fin_slot = slot0(B, 0, o) + (TRANS ? o : 0); jb.nfin = TRANS ? nsubB - o : i + 1; }
    else jb.sig_ctr = nullptr;
  }
  return true;
}

template <int NR>
constexpr size_t trsv_staged_smem() {
  if (NR == 8) return (size_t)BL_TILE * sizeof(float) + (size_t)XS * 8 * sizeof(double);
  return (size_t)TILE_ELEMS * sizeof(float) + 2 * (size_t)RB * NR * sizeof(double);
}
size_t trsv_smem_bytes(int nrhs) {
  switch (nrhs) {
    case 1: return trsv_staged_smem<1>();
    case 2: return trsv_staged_smem<2>();
    case 4: return trsv_staged_smem<4>();
    default: return trsv_staged_smem<8>();
  }
}

// Two (or three) CTAs per SM, each with one tile stage: a unit's tile copy is
// issued as soon as the unit is taken and overlaps the wait for its input
// segment; while one CTA waits on L2 round trips (dependency counter, vector
// segment, fence) the other computes.  A CTA finishes its unit before it starts
// the next, whose number it asks for only when the unit's input is there; every
// unit depends only on earlier ones, so the earliest unfinished unit always
// belongs to a CTA that is working on it, and every wait ends.
template <int NR>
constexpr int trsv_ctas() { return NR == 1 ? 3 : 2; }   // most per SM

template <int NR, bool TRANS>
__global__ void __launch_bounds__(NTH, trsv_ctas<NR>())
trsv_persistent_kernel(const float* __restrict__ L, int ldl, int n, const float* __restrict__ wsup,
                       double* __restrict__ work, double* __restrict__ out, int* ctr,
                       TrsvSlot* slots, const int* skip, DevStatus* st) {
  if (skip != nullptr && *skip) return;
  constexpr bool MMA = NR == 8;
  constexpr bool SLOTS = NR <= kSlotNr;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  float* Ts = reinterpret_cast<float*>(sm_raw);                           // one stage
  double* s_v = reinterpret_cast<double*>(Ts + (MMA ? BL_TILE : TILE_ELEMS));   // RB x NR
  double* s_col = s_v + RB * NR;                                          // RB x NR
  __shared__ int s_unit[2];
  __shared__ unsigned long long s_epoch;
  int* next = ctr;
  int* exits = ctr + 1;         // CTAs that are done
  int* seg_in = ctr + 2;
  int* seg_out = seg_in + ceil_div(n, RB);
  // The launch's number, which the tags carry: in the slots' header, one more
  // after each launch (the last CTA to leave raises it).
  unsigned long long* epoch = reinterpret_cast<unsigned long long*>(slots);
  if (threadIdx.x == 0) {
    if (SLOTS) s_epoch = *reinterpret_cast<volatile unsigned long long*>(epoch);
    s_unit[0] = atomicAdd(next, 1);
  }
  __syncthreads();
  int ucur = s_unit[0];
  TrsvSlot* slot = slots + 1;
  const unsigned long long tag0 = SLOTS ? (s_epoch << 20) + 1 : 0;
  TrsvCursor cursor{-1, 0};
  TrsvJob cur;
  for (int it = 1; trsv_job<TRANS, SLOTS>(ucur, cursor, L, ldl, n, wsup, seg_in, seg_out, cur); ++it) {
    if (MMA) stage_tile_bl(Ts, cur.T, cur.ld, cur.nrow, cur.ncol);
    else stage_tile(Ts, cur.T, cur.ld, cur.nrow, cur.ncol);
    cp_async_commit();
    wait_count(cur.wait_ctr, cur.wait_need, st, ucur);
    // the next number, asked for once this unit's input is there: its round trip
    // overlaps the tile pass, and no unit is bound to a CTA that still waits
    // (s_unit[it & 1] is read after this unit's barriers)
    auto take_next = [&]() {
      if (threadIdx.x == 32) s_unit[it & 1] = atomicAdd(next, 1);
    };
    double* dst = cur.panel ? work : out;
    const double sign = cur.panel ? -1.0 : 1.0;
    if constexpr (MMA) {
      load_vec_x8(cur.panel ? out : work, n, cur.vin_row0, cur.vin_n, s_v);
      take_next();
      cp_async_wait<0>();
      __syncthreads();
      if (cur.nt)
        tile_mma_x8<false, false, 4, RB / 16, 1>(Ts, s_v, s_v, dst, cur.out_row0, cur.out_n, dst,
                                                 cur.out_row0, cur.out_n, n, true, false, sign, nullptr);
      else
        tile_mma_x8<false, false, 4, RB / 16, 2>(Ts, s_v, s_v, dst, cur.out_row0, cur.out_n, dst,
                                                 cur.out_row0, cur.out_n, n, false, true, sign, nullptr);
      signal_count(cur.sig_ctr);   // its barrier also frees the stage and s_v
    } else {
      if (cur.nin == 0)
        load_vec<NR>(cur.panel ? out : work, n, cur.vin_row0, cur.vin_n, s_v);
      else
        gather_slots<NR>(slot + (size_t)cur.in_slot * RB * NR, cur.nin, tag0 + cur.in_blk,
                         cur.panel ? nullptr : work, n, cur.vin_row0, cur.vin_n, s_v, s_col, st, ucur);
      take_next();
      cp_async_wait<0>();
      __syncthreads();
      double acc[4][NR] = {};
      tile_pass_staged<NR, false>(Ts, s_v, s_v, acc, s_col, cur.nt, !cur.nt);
      __syncthreads();
      double* red = reinterpret_cast<double*>(Ts);
      if (cur.nt) stage_rows<NR>(acc, red);
      for (int e = threadIdx.x; e < RB * NR; e += NTH) {
        const int r = e % RB;
        const double v = sign * (cur.nt ? row_sum<NR>(red, e) : s_col[e]);
        if (cur.out_slot >= 0) slot_put(slot + (size_t)cur.out_slot * RB * NR + e, v, tag0 + cur.out_blk);
        else if (r < cur.out_n) atomicAdd(&dst[(size_t)(e / RB) * n + cur.out_row0 + r], v);
      }
      if (cur.nfin > 0) {
        // the segment's sums into the result (s_v is free; the odd sums pass
        // through the half of the stage that `red` leaves)
        gather_slots<NR>(slot + (size_t)cur.fin_slot * RB * NR, cur.nfin, tag0 + cur.out_blk, nullptr, n,
                         0, 0, s_v, red + TILE_ELEMS / 4, st, ucur);
        for (int e = threadIdx.x; e < RB * NR; e += NTH)
          if (e % RB < cur.out_n) __stcg(&out[(size_t)(e / RB) * n + cur.out_row0 + e % RB], s_v[e]);
      }
      // the barrier also frees the stage, s_v and s_col
      if (cur.sig_ctr != nullptr) signal_count(cur.sig_ctr);
      else __syncthreads();
    }
    ucur = s_unit[it & 1];
  }
  if (SLOTS && threadIdx.x == 0 && atomicAdd(exits, 1) == (int)gridDim.x - 1) *epoch = s_epoch + 1;
}

// ---- batched variants: one launch serves every system of a batch --------
// blockIdx.y (or .z) selects the system; CTAs past a system's own extent
// return at once.  Vectors live in the system's slots (n x NR column-major).
__device__ __forceinline__ double* bslot(const BatchSys& S, int slot, int nr) {
  return S.vec + (size_t)slot * S.n * nr;
}

// One unit of the batched operator product: tile (I, J) of one system's
// lower triangle.  A == nullptr: the system has converged, nothing to do.
struct SymvUnit {
  const float* A;
  int lda, n, I, J;
  const double* x;
  double* y;
  int al16;             // columns start on 16-byte boundaries
};

// Unit t -> its system (binary search of the per-system first units; the
// systems are numbered in order of their first unit) and its tile.
template <int NR>
__device__ __forceinline__ SymvUnit symv_unit(const BatchSys* __restrict__ sys, int nsys, int t,
                                              int xslot, int yslot, int use_skip) {
  int lo = 0, hi = nsys - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (sys[mid].sym_tile0 <= t) lo = mid;
    else hi = mid - 1;
  }
  const BatchSys& S = sys[lo];
  SymvUnit u;
  tri_of(t - S.sym_tile0, u.I, u.J);
  u.A = (use_skip && S.done[0]) ? nullptr : S.op;
  u.lda = S.op_ld;
  u.n = S.n;
  u.x = bslot(S, xslot, NR);
  u.y = bslot(S, yslot, NR);
  u.al16 = (reinterpret_cast<uintptr_t>(S.op) & 15) == 0 && S.op_ld % 4 == 0;
  return u;
}

// y = A x for every system of a batch, persistent over the concatenated
// 128-tiles of all systems' lower triangles, with the unit's system found per
// tile.  Two single-stage CTAs per SM: each copies its next tile and vector
// segments into shared memory while the other runs its tile pass (both A x
// and A^T x from the one copy).  For 1-4 rhs this replaces three stages in
// one 190-register CTA per SM and caps the FP64 tile pass at 128 registers:
// the 512-system batch step (4 rhs, 10 products) took 54.8 against 57.5 ms.
// y slots are zeroed beforehand.
template <int NR>
constexpr size_t symv_batched_smem() {
  if (NR == 8)
    return (size_t)BL_TILE * sizeof(float) + 2 * (size_t)XS * 8 * sizeof(double);
  return (size_t)TILE_ELEMS * sizeof(float) + 3 * (size_t)RB * NR * sizeof(double);
}
template <int NR>
__global__ void __launch_bounds__(NTH, 2)
symv_staged_batched_kernel(const BatchSys* __restrict__ sys, int nsys, int ntiles, int xslot,
                           int yslot, int use_skip) {
  constexpr bool MMA = NR == 8;
  constexpr int TE = MMA ? BL_TILE : TILE_ELEMS;
  constexpr int VEC = MMA ? XS * 8 : RB * NR;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  float* Ts = reinterpret_cast<float*>(sm_raw);
  double* xJ = reinterpret_cast<double*>(Ts + TE);
  double* xI = xJ + VEC;
  double* s_col = xI + VEC;
  __shared__ SymvUnit s_unit;   // read again after the copies: no registers held through the tile pass
  auto issue = [&](const SymvUnit& u) {
    const int i0 = u.I * RB, j0 = u.J * RB;
    const int ni = min(RB, u.n - i0), nj = min(RB, u.n - j0);
    const float* T = u.A + (size_t)j0 * u.lda + i0;
    if (MMA) {
      if (u.al16) stage_tile_bl(Ts, T, u.lda, ni, nj);
      else stage_tile_4b<true>(Ts, T, u.lda, ni, nj);
      stage_vec_x8(u.x, u.n, j0, nj, xJ);
      stage_vec_x8(u.x, u.n, i0, ni, xI);
    } else {
      if (u.al16) stage_tile(Ts, T, u.lda, ni, nj);
      else stage_tile_4b<false>(Ts, T, u.lda, ni, nj);
      stage_vec<NR>(u.x, u.n, j0, nj, xJ);
      stage_vec<NR>(u.x, u.n, i0, ni, xI);
    }
  };
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    {
      const SymvUnit u = symv_unit<NR>(sys, nsys, t, xslot, yslot, use_skip);
      if (u.A == nullptr) continue;                // uniform over the CTA
      if (threadIdx.x == 0) s_unit = u;
      issue(u);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const SymvUnit u = s_unit;
    const int i0 = u.I * RB, j0 = u.J * RB;
    const int ni = min(RB, u.n - i0), nj = min(RB, u.n - j0);
    if (MMA) {
      if (u.I == u.J)
        tile_mma_x8<true, false>(Ts, xJ, xI, u.y, i0, ni, u.y, j0, nj, u.n, true, true, 1.0, nullptr);
      else
        tile_mma_x8<false, false>(Ts, xJ, xI, u.y, i0, ni, u.y, j0, nj, u.n, true, true, 1.0, nullptr);
    } else {
      double acc[4][NR] = {};
      if (u.I == u.J) tile_pass_staged<NR, true>(Ts, xJ, xI, acc, s_col, true, true);
      else tile_pass_staged<NR, false>(Ts, xJ, xI, acc, s_col, true, true);
      __syncthreads();
      for (int e = threadIdx.x; e < VEC; e += NTH) {
        const int k = e / RB, c = e % RB;
        if (c < nj) atomicAdd(&u.y[(size_t)k * u.n + j0 + c], s_col[e]);
      }
      flush_rows<NR>(acc, reinterpret_cast<double*>(Ts), u.y, u.n, i0, ni, 1.0);
    }
    __syncthreads();   // the stage, the unit's record and s_col are free again
  }
}

// dst slot = 0 (src < 0) or a copy of the src slot
__global__ void vec_slot_batched_kernel(const BatchSys* __restrict__ sys, int src, int dst, int nr,
                                        int use_skip) {
  const BatchSys& S = sys[blockIdx.y];
  if (use_skip && S.done[0]) return;
  const long long cnt = (long long)S.n * nr;
  double* d = bslot(S, dst, nr);
  const double* a = src >= 0 ? bslot(S, src, nr) : nullptr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < cnt;
       i += (long long)gridDim.x * blockDim.x)
    d[i] = a ? a[i] : 0.0;
}

__global__ void __launch_bounds__(NTH)
block_inverse_batched_kernel(const BatchSys* __restrict__ sys) {
  const BatchSys& S = sys[blockIdx.y];
  if ((int)(blockIdx.x / BT) * RB >= S.n) return;
  block_inverse_body(S.A, S.ld, S.n, S.wsup, make_uint3(blockIdx.x, 0, 0));
}

template <int PHASE>
__global__ void __launch_bounds__(NTH, 4)
superinv_gemm_batched_kernel(const BatchSys* __restrict__ sys, int h, int max_super) {
  const BatchSys& S = sys[blockIdx.z / max_super];
  const int sup = blockIdx.z % max_super;
  if (sup * RS >= S.n) return;
  superinv_gemm_body<PHASE>(S.A, S.ld, S.n, S.wsup, h, make_uint3(blockIdx.x, blockIdx.y, sup));
}

template <int NR, bool TRANS>
__global__ void __launch_bounds__(NTH)
trmv_super_batched_kernel(const BatchSys* __restrict__ sys, int sup, int in_slot, int out_slot,
                          int use_skip) {
  const BatchSys& S = sys[blockIdx.y];
  const int s0 = sup * RS;
  if (s0 >= S.n) return;
  const int rs = min(RS, S.n - s0);
  const int nsub = ceil_div(rs, RB);
  if ((int)blockIdx.x >= nsub * (nsub + 1) / 2) return;
  trmv_super_body<NR, TRANS>(S.wsup + (size_t)sup * RS * RS, S.n, s0, rs, bslot(S, in_slot, NR),
                             bslot(S, out_slot, NR), use_skip ? S.done : nullptr,
                             make_uint3(blockIdx.x, 0, 0));
}

template <int NR, bool TRANS>
__global__ void __launch_bounds__(NTH)
panel_batched_kernel(const BatchSys* __restrict__ sys, int sup, int v_slot, int w_slot,
                     int use_skip) {
  const BatchSys& S = sys[blockIdx.z];
  const int s0 = sup * RS;
  if (s0 >= S.n) return;
  const int rs = min(RS, S.n - s0);
  const int nsub = ceil_div(rs, RB);
  const int span = TRANS ? s0 : S.n - s0 - rs;      // rows below (forward) / columns left (backward)
  if (span <= 0 || (int)blockIdx.x >= ceil_div(span, RB) || (int)blockIdx.y >= nsub) return;
  panel_body<NR, TRANS>(S.A, S.ld, S.n, s0, rs, bslot(S, v_slot, NR), bslot(S, w_slot, NR),
                        use_skip ? S.done : nullptr, make_uint3(blockIdx.x, blockIdx.y, 0));
}

// The inputs of a forward and a backward solve: w <- in, their targets zero and
// their dependency counters cleared.
__global__ void trsv_prep_kernel(const double* __restrict__ in, double* __restrict__ w,
                                 double* __restrict__ mid, double* __restrict__ out, long long count,
                                 int* counters, int ncounters) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  for (long long i = t0; i < count; i += stride) {
    w[i] = in[i];
    mid[i] = 0.0;
    out[i] = 0.0;
  }
  for (long long i = t0; i < ncounters; i += stride) counters[i] = 0;
}

__global__ void zero_vec_kernel(double* __restrict__ a, long long count) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
       i += (long long)gridDim.x * blockDim.x)
    a[i] = 0.0;
}

size_t red_bytes(int nr) { return (size_t)(NTH / 32) * RB * nr * sizeof(double); }

template <typename K>
cudaError_t set_dyn(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

#define NR_SWITCH(nrhs, CALL)                                 \
  switch (nrhs) {                                             \
    case 1: { constexpr int NRC = 1; CALL; } break;           \
    case 2: { constexpr int NRC = 2; CALL; } break;           \
    case 4: { constexpr int NRC = 4; CALL; } break;           \
    case 8: { constexpr int NRC = 8; CALL; } break;           \
    default: return cudaErrorInvalidValue;                    \
  }

int solve_super_rows() { return RS; }
size_t solve_wsup_elems(int n) {
  const int nbs = (n + RS - 1) / RS;
  return (size_t)nbs * RS * RS;
}

// What the launchers ask of a device: its SMs, and the resident CTAs per SM of
// the triangular solve (by direction; 1, 2, 4, 8 right-hand sides).
struct DeviceLimits {
  int sms = 0, trsv[2][4] = {};
};
// The kernels' attributes are set and the limits asked for once per device (both
// are per device), under a lock until all is complete: threads may make their
// first calls at the same time.
cudaError_t device_limits(const DeviceLimits** out) {
  static std::mutex mu;
  static DeviceLimits limits[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  DeviceLimits& d = limits[dev & 63];
  if (d.sms == 0) {
    DeviceLimits f;
    e = solve_set_attributes();
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&f.sms, cudaDevAttrMultiProcessorCount, dev);
    auto ask = [&](auto kernel, size_t smem, int& n) {
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, NTH, smem);
      n = std::max(1, n);
    };
    auto both = [&](auto fwd, auto bwd, size_t smem, int i) {
      ask(fwd, smem, f.trsv[0][i]);
      ask(bwd, smem, f.trsv[1][i]);
    };
    both(trsv_persistent_kernel<1, false>, trsv_persistent_kernel<1, true>, trsv_staged_smem<1>(), 0);
    both(trsv_persistent_kernel<2, false>, trsv_persistent_kernel<2, true>, trsv_staged_smem<2>(), 1);
    both(trsv_persistent_kernel<4, false>, trsv_persistent_kernel<4, true>, trsv_staged_smem<4>(), 2);
    both(trsv_persistent_kernel<8, false>, trsv_persistent_kernel<8, true>, trsv_staged_smem<8>(), 3);
    if (e != cudaSuccess) return e;
    d = f;
  }
  *out = &d;
  return cudaSuccess;
}

cudaError_t solve_init_attributes() {
  const DeviceLimits* lim = nullptr;
  return device_limits(&lim);
}

cudaError_t solve_set_attributes() {
  cudaError_t e;
  if ((e = set_dyn(block_inverse_kernel, kBlockInvSmem)) != cudaSuccess) return e;
#define SET_NR(NRC)                                                                         \
  if ((e = set_dyn(symv_kernel<double, NRC>, red_bytes(NRC))) != cudaSuccess) return e;
  SET_NR(1) SET_NR(2) SET_NR(4) SET_NR(8)
#undef SET_NR
#define SET_NRP(NRC)                                                                              \
  if ((e = set_dyn(trsv_persistent_kernel<NRC, false>, trsv_staged_smem<NRC>())) != cudaSuccess) return e; \
  if ((e = set_dyn(trsv_persistent_kernel<NRC, true>, trsv_staged_smem<NRC>())) != cudaSuccess) return e; \
  if ((e = set_dyn(symv_staged_kernel<NRC>, symv_staged_smem<NRC>())) != cudaSuccess) return e;
  SET_NRP(1) SET_NRP(2) SET_NRP(4) SET_NRP(8)
#undef SET_NRP
  if ((e = set_dyn(symv_staged_kernel<8, false>, symv_staged_smem<8>())) != cudaSuccess) return e;
  if ((e = set_dyn(block_inverse_batched_kernel, kBlockInvSmem)) != cudaSuccess) return e;
#define SET_NRB(NRC)                                                                              \
  if ((e = set_dyn(symv_staged_batched_kernel<NRC>, symv_batched_smem<NRC>())) != cudaSuccess) return e; \
  if ((e = set_dyn(trmv_super_batched_kernel<NRC, false>, red_bytes(NRC))) != cudaSuccess) return e; \
  if ((e = set_dyn(trmv_super_batched_kernel<NRC, true>, red_bytes(NRC))) != cudaSuccess) return e;  \
  if ((e = set_dyn(panel_batched_kernel<NRC, false>, red_bytes(NRC))) != cudaSuccess) return e;      \
  if ((e = set_dyn(panel_batched_kernel<NRC, true>, red_bytes(NRC))) != cudaSuccess) return e;
  SET_NRB(1) SET_NRB(2) SET_NRB(4) SET_NRB(8)
#undef SET_NRB
  return pcg_small_set_attributes();
}

cudaError_t launch_zero_vec(double* y, long long count, cudaStream_t stream) {
  zero_vec_kernel<<<148, 256, 0, stream>>>(y, count);
  return cudaGetLastError();
}

// FP32 operators stream through the staged persistent kernel (4-byte copies
// where columns do not start on 16-byte boundaries: n = 2999, 4 rhs, 28 us by
// register loads of one tile per CTA against 22 us); FP64 operators take one
// CTA per tile with register loads.
template <typename TA>
cudaError_t launch_symv_skip(const TA* A, int lda, int n, const double* x, double* y, int nrhs,
                             const int* skip, cudaStream_t stream, double* fro, int nfro) {
  const int T = ceil_div(n, RB);
  const int ntiles = T * (T + 1) / 2;
  if constexpr (sizeof(TA) == 4) {
    const DeviceLimits* lim = nullptr;
    const cudaError_t le = device_limits(&lim);
    if (le != cudaSuccess) return le;
    int grid = std::min(ntiles, (nrhs == 1 ? symv_ctas<1>() : symv_ctas<2>()) * lim->sms);
    if (fro != nullptr) grid = std::min(grid, nfro);   // one Frobenius partial per CTA
    const int al16 = (reinterpret_cast<uintptr_t>(A) & 15) == 0 && lda % 4 == 0;
    if (nrhs == 8 && !al16)
      symv_staged_kernel<8, false><<<grid, NTH, symv_staged_smem<8>(), stream>>>(A, lda, n, x, y, skip, fro, nfro, 0);
    else
      NR_SWITCH(nrhs, (symv_staged_kernel<NRC><<<grid, NTH, symv_staged_smem<NRC>(), stream>>>(A, lda, n, x, y, skip, fro, nfro, al16)));
  } else {
    NR_SWITCH(nrhs, (symv_kernel<TA, NRC><<<ntiles, NTH, red_bytes(NRC), stream>>>(A, lda, n, x, y, skip)));
  }
  return cudaGetLastError();
}
template cudaError_t launch_symv_skip<float>(const float*, int, int, const double*, double*, int, const int*, cudaStream_t, double*, int);
template cudaError_t launch_symv_skip<double>(const double*, int, int, const double*, double*, int, const int*, cudaStream_t, double*, int);

// Pairs of the doubling level h whose second half has rows below n, in a
// super-block of the first min(n, RS) rows; 0: the level is not launched.
int doubling_pairs(int n, int h) { return ceil_div(std::max(0, std::min(n, RS) - h), 2 * h); }

cudaError_t launch_solve_setup(const float* L, int ldl, int n, float* wsup, cudaStream_t stream) {
  block_inverse_kernel<<<BT * ceil_div(n, RB), NTH, kBlockInvSmem, stream>>>(L, ldl, n, wsup);
  const int nbs = ceil_div(n, RS);
  for (int h = RB; h < RS; h *= 2) {
    if (doubling_pairs(n, h) == 0) break;
    const dim3 grid((h / GT) * (h / GT), doubling_pairs(n, h), nbs);
    superinv_gemm_kernel<0><<<grid, NTH, 0, stream>>>(L, ldl, n, wsup, h);
    superinv_gemm_kernel<1><<<grid, NTH, 0, stream>>>(L, ldl, n, wsup, h);
  }
  return cudaGetLastError();
}

int solve_setup_launches(int n) {
  int k = 1;
  for (int h = RB; h < RS && doubling_pairs(n, h) > 0; h *= 2) k += 2;
  return k;
}

cudaError_t launch_vec_slot_batched(const BatchSys* sys, int nsys, int src, int dst, int nr,
                                    int use_skip, cudaStream_t stream) {
  vec_slot_batched_kernel<<<dim3(8, nsys), NTH, 0, stream>>>(sys, src, dst, nr, use_skip);
  return cudaGetLastError();
}

cudaError_t launch_symv_batched(const BatchSys* sys, int nsys, int ntiles, int xslot, int yslot,
                                int nr, int use_skip, cudaStream_t stream) {
  cudaError_t e = launch_vec_slot_batched(sys, nsys, -1, yslot, nr, use_skip, stream);
  if (e != cudaSuccess) return e;
  if (ntiles <= 0) return cudaSuccess;
  const DeviceLimits* lim = nullptr;
  if ((e = device_limits(&lim)) != cudaSuccess) return e;
  const int grid = std::min(ntiles, 2 * lim->sms);
  NR_SWITCH(nr, (symv_staged_batched_kernel<NRC><<<grid, NTH, symv_batched_smem<NRC>(), stream>>>(sys, nsys, ntiles, xslot, yslot, use_skip)));
  return cudaGetLastError();
}

cudaError_t launch_solve_setup_batched(const BatchSys* sys, int nsys, int max_n,
                                       cudaStream_t stream) {
  block_inverse_batched_kernel<<<dim3(BT * ceil_div(max_n, RB), nsys), NTH, kBlockInvSmem, stream>>>(sys);
  const int max_super = ceil_div(max_n, RS);
  for (int h = RB; h < RS; h *= 2) {
    if (doubling_pairs(max_n, h) == 0) break;
    const dim3 grid((h / GT) * (h / GT), doubling_pairs(max_n, h), nsys * max_super);
    superinv_gemm_batched_kernel<0><<<grid, NTH, 0, stream>>>(sys, h, max_super);
    superinv_gemm_batched_kernel<1><<<grid, NTH, 0, stream>>>(sys, h, max_super);
  }
  return cudaGetLastError();
}

cudaError_t launch_trsv_batched(bool backward, const BatchSys* sys, int nsys, int max_n,
                                int in_slot, int out_slot, int work_slot, int nr, int use_skip,
                                cudaStream_t stream) {
  cudaError_t e = launch_vec_slot_batched(sys, nsys, in_slot, work_slot, nr, use_skip, stream);
  if (e == cudaSuccess) e = launch_vec_slot_batched(sys, nsys, -1, out_slot, nr, use_skip, stream);
  if (e != cudaSuccess) return e;
  const int max_super = ceil_div(max_n, RS);
  const int nsub_max = ceil_div(min(max_n, RS), RB);
  const int span_tiles = ceil_div(max_n, RB);
  for (int t = 0; t < max_super; ++t) {
    const int sup = backward ? max_super - 1 - t : t;
    const dim3 gt(nsub_max * (nsub_max + 1) / 2, nsys);
    const dim3 gp(span_tiles, nsub_max, nsys);
    if (!backward) {
      NR_SWITCH(nr, (trmv_super_batched_kernel<NRC, false><<<gt, NTH, red_bytes(NRC), stream>>>(sys, sup, work_slot, out_slot, use_skip)));
      NR_SWITCH(nr, (panel_batched_kernel<NRC, false><<<gp, NTH, red_bytes(NRC), stream>>>(sys, sup, out_slot, work_slot, use_skip)));
    } else {
      NR_SWITCH(nr, (trmv_super_batched_kernel<NRC, true><<<gt, NTH, red_bytes(NRC), stream>>>(sys, sup, work_slot, out_slot, use_skip)));
      NR_SWITCH(nr, (panel_batched_kernel<NRC, true><<<gp, NTH, red_bytes(NRC), stream>>>(sys, sup, out_slot, work_slot, use_skip)));
    }
  }
  return cudaGetLastError();
}

size_t trsv_slot_bytes() {
  return sizeof(TrsvSlot) * (1 + (size_t)4 * kSlotSegs * RB * kSlotNr);
}

size_t trsv_counter_ints(int n) { return 2 + 2 * (size_t)ceil_div(n, RB); }

cudaError_t launch_trsv_prep(const double* in, double* w, double* mid, double* out, int n, int nrhs,
                             int* counters, cudaStream_t stream) {
  trsv_prep_kernel<<<148, 256, 0, stream>>>(in, w, mid, out, (long long)n * nrhs, counters,
                                            2 * (int)trsv_counter_ints(n));
  return cudaGetLastError();
}

// One cooperative launch over every resident CTA.
cudaError_t launch_trsv_persistent(bool backward, const float* L, int ldl, int n,
                                   const float* wsup, double* work, double* out, int nrhs, int* counters,
                                   void* slots, const int* skip, DevStatus* st, cudaStream_t stream) {
  const DeviceLimits* lim = nullptr;
  cudaError_t e = device_limits(&lim);
  if (e != cudaSuccess) return e;
  const int nri = nrhs == 1 ? 0 : nrhs == 2 ? 1 : nrhs == 4 ? 2 : 3;
  const int per_sm = lim->trsv[backward ? 1 : 0][nri];
  const size_t smem = trsv_smem_bytes(nrhs);
  auto launch = [&](auto kernel) -> cudaError_t {
    cudaLaunchConfig_t cfg = {};
    // The third CTA per SM (one right-hand side, or eight) pays once far tiles
    // bound the solve; before that it only slows the chain's tile passes.  Two and
    // three per SM, forward / backward in us.  One right-hand side: 24.0 / 27.5 and
    // 27.7 / 32.1 at n = 4096, 55 / 60 and 56 / 63 at 8192, 65 / 70 and 63 / 70 at
    // 9200, 78 / 88 and 76 / 82 at 10240, 168 / 185 and 145 / 158 at 16384.  Eight:
    // 22.8 / 23.4 and 24.7 / 26.8 at 2048, 46 / 46 and 51 / 51 at 4096, 100 / 98 and
    // 112 / 112 at 8192.  (With two or four only two fit.)
    cfg.gridDim = dim3((n > 9 * RS ? per_sm : std::min(per_sm, 2)) * lim->sms);
    cfg.blockDim = dim3(NTH);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, L, ldl, n, wsup, work, out, counters,
                              static_cast<TrsvSlot*>(slots), skip, st);
  };
  if (!backward) {
    NR_SWITCH(nrhs, (e = launch(trsv_persistent_kernel<NRC, false>)));
  } else {
    NR_SWITCH(nrhs, (e = launch(trsv_persistent_kernel<NRC, true>)));
  }
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}


}  // namespace mpchol
