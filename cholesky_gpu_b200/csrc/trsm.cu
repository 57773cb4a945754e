// Panel TRSM with the fused switching epilogue.
//
// Replaces the reference's cublasStrsm of the panel (src/switching_chol.cuh:98-110,
// correct form RIGHT/LOWER/TRANS at src/sChol.cuh:273-280), its update_diag
// kernel (src/kernels_macros.cuh:177-190) and the per-row part of can_switch
// (src/kernels_macros.cuh:191-211).
//
// X * L11^T = A21 for the m rows below the diagonal block.  Rows are
// independent, so one CTA of 16 warps owns a slab of 16, 32 or 64 rows (the
// smallest of which the panel has at most one per SM, else 64).  TMA stages the slab
// and all of L11: the strictly-lower 32 x 32 tiles L_{J,M} as 2-D boxes and
// the inverses of the diagonal tiles L_JJ, which the POTRF kernel wrote, as
// 1-D bulk copies, one mbarrier per tile row.  The solve is a pipeline over
// the 32-column tiles J of the slab, a warp pair per tile (each thread a
// register block of 4 or 8 rows x 4 columns, so a k step reads two or three
// 16-byte vectors for 16 or 32 FMAs; the shared-memory return path, not the
// FMA rate, bounds these small products):
//   X_J = (A_J - sum_{K<J} X_K L_{J,K}^T) L_JJ^-T,
// where the pair of tile J applies X_K as soon as the pair of tile K has
// published it (an mbarrier per tile, bounded waits), so the only chain is
// one tile update plus one diagonal multiply per tile column.  A finished pair
// sums its tile's rows and columns and writes its MX codes while the chain goes
// on.  The epilogue writes the slab back (TMA stores), folds each row's sum of
// squares into the Schur-diagonal tracker dtilde, reduces the switching
// statistics (max d/dtilde, min dtilde, the reference-literal choice) and the
// near-indefinite flag of the next diagonal block, and writes the slab's codes
// in the other candidate formats, straight from the slab.  The last CTA to take
// a ticket (a counter) resolves the step precision.
//
// Against one thread that issued every copy (about 80 cycles each), sums after
// the solve and codes staged in shared memory on their way out (n = 1024 / 8192
// solve, b = 256, B200): 580 -> 561 and 4459 -> 4260 us end to end.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "quant.cuh"
#include "tc_ptx.cuh"

namespace mpchol {
namespace {

constexpr int NTHR = 512;    // 16 warps: two per 32-column tile of a 256-wide block
constexpr int TSZ = 32 * 32; // dense 32 x 32 tile
constexpr int MAXNT = 8;     // tiles per block column (b <= 256)

__device__ __forceinline__ int tl(int I, int M) { return I * (I - 1) / 2 + M; }  // I > M

// The slab of TR rows in shared memory: parts of HR = min(TR, 32) rows, each
// column-major with its rows contiguous (the layout of an HR x bs TMA box), so
// lane l reading row l of one column of a 32- or 64-row slab touches 32
// different banks.
template <int TR>
struct Slab {
  static constexpr int HR = TR < 32 ? TR : 32;   // rows per part
  static constexpr int RPL = TR / HR;            // parts
  static constexpr int RT = HR / 8;              // rows of a part per thread of the solve
};
template <int TR>
__device__ __forceinline__ int xoff(int r, int c, int bs) {
  constexpr int HR = Slab<TR>::HR;
  return (r / HR) * bs * HR + c * HR + r % HR;
}
template <int N>
__device__ __forceinline__ void load_rows(const float* p, float (&v)[N]) {
  if constexpr (N == 4) {
    const float4 w = *reinterpret_cast<const float4*>(p);
    v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
  } else {
    static_assert(N == 2, "two or four rows per thread");
    const float2 w = *reinterpret_cast<const float2*>(p);
    v[0] = w.x; v[1] = w.y;
  }
}
template <int N>
__device__ __forceinline__ void store_rows(float* p, const float (&v)[N]) {
  if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

// Shared memory of both panel kernels (floats): the slab, L11's strictly-lower
// tiles and the inverses of its diagonal tiles.
size_t trsm_smem_floats(int tr, int bs) {
  const int NT = bs / 32;
  return (size_t)bs * tr + (size_t)(NT * (NT - 1) / 2 + NT) * TSZ;
}

__device__ __forceinline__ void pair_sync(int J) {   // the two warps of tile column J
  asm volatile("bar.sync %0, 64;" ::"r"(J + 1) : "memory");
}

// The slab solve.  The warp pair of tile column J (warps 2J, 2J + 1; w = 2J +
// h) computes the TR x 32 tile X_J: thread t of the pair (t = 32 h + lane)
// holds RT rows of each part (rows RT rg ..) x 4 columns (4 cg ..) in
// registers, so every k step of the tile products reads a vector of X per part
// and one of L.  The lane's bits interleave into rg and cg so that four
// neighbouring lanes read two different vectors of each (2.2 cycles of the
// SM's shared memory per 16-byte load; 4.0 when they read four).  Lt: L11's
// tiles L_{I,M} (I > M) at tl(I, M) * TSZ; Wt: the inverses W_JJ = L_JJ^-1,
// tile J at J * TSZ; both column-major (L(c, m) at m * 32 + c, W(c, m) zero
// for m > c).  lrow[J] (null: already staged) completes when tile row J has
// landed; ready[J] (64 arrivals) when X_J is final:
//   X_J = (A_J - sum_{K<J} X_K L_{J,K}^T) W_JJ^T.
// post(J, t) runs in the pair's threads once both warps' parts of X_J are
// written.  Each output is one fma chain in a fixed order: the update over K,
// then m; the diagonal multiply over m.  Returns false if a bounded wait gave
// up.
template <int TR, typename Post>
__device__ bool slab_solve(float* Xs, int bs, const float* Lt, const float* Wt, uint64_t* lrow,
                           uint64_t* ready, int tid, Post post) {
  constexpr int HR = Slab<TR>::HR, RPL = Slab<TR>::RPL, RT = Slab<TR>::RT;
  const int NT = bs / 32;
  const int warp = tid >> 5, lane = tid & 31;
  const int J = warp >> 1, h = warp & 1;
  if (J >= NT) return true;
  const int XH = bs * HR;                              // floats per part
  const int rg = (lane & 1) | ((lane >> 1) & 6), cg = ((lane >> 1) & 1) | ((lane >> 3) & 2) | (h << 2);
  const int r0 = RT * rg;                              // rows r0.. of each part
  const int cl = 4 * cg;                               // columns cl.. of the tile
  bool ok = lrow == nullptr || tc::mbar_wait(&lrow[J], 0);
  float acc[RPL][4][RT];                               // [part][column][row]
#pragma unroll
  for (int q = 0; q < RPL; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) load_rows<RT>(Xs + q * XH + (32 * J + cl + j) * HR + r0, acc[q][j]);
#pragma unroll 1
  for (int K = 0; K < J; ++K) {
    ok = tc::mbar_wait(&ready[K], 0) && ok;
    const float* L = Lt + (size_t)tl(J, K) * TSZ + cl;
    const float* xk = Xs + 32 * K * HR + r0;
#pragma unroll 8
    for (int m = 0; m < 32; ++m) {
      const float4 lv = *reinterpret_cast<const float4*>(L + m * 32);
      const float l[4] = {lv.x, lv.y, lv.z, lv.w};
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        float x[RT];
        load_rows<RT>(xk + q * XH + m * HR, x);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < RT; ++i) acc[q][j][i] = fmaf(-x[i], l[j], acc[q][j][i]);
      }
    }
  }
  // the updated tile into the slab, then X_J = Y W_JJ^T
  float* xj = Xs + 32 * J * HR + r0;
#pragma unroll
  for (int q = 0; q < RPL; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) store_rows<RT>(xj + q * XH + (cl + j) * HR, acc[q][j]);
  pair_sync(J);
  const float* W = Wt + (size_t)J * TSZ + cl;
#pragma unroll
  for (int q = 0; q < RPL; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < RT; ++i) acc[q][j][i] = 0.0f;
  const int mend = 16 * h + 16;                        // W(c, m) = 0 for m > c (the warp's columns)
#pragma unroll 8
  for (int m = 0; m < mend; ++m) {
    const float4 wv = *reinterpret_cast<const float4*>(W + m * 32);
    const float w[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      float y[RT];
      load_rows<RT>(xj + q * XH + m * HR, y);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < RT; ++i) acc[q][j][i] = fmaf(y[i], w[j], acc[q][j][i]);
    }
  }
  pair_sync(J);                                        // every read of Y is done
#pragma unroll
  for (int q = 0; q < RPL; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) store_rows<RT>(xj + q * XH + (cl + j) * HR, acc[q][j]);
  tc::mbar_arrive(&ready[J]);                          // release: X_J to the later tiles
  pair_sync(J);
  post(J, 32 * h + lane);
  return ok;
}

// Per-row sums of squares of the solved slab (batched kernel): thread (r, part)
// = (tid % TR, tid / TR) covers row r's 32 columns `part` (a chain of FMAs in
// column order), leaving the partials in s_sq[part][r]; the row's sum is then
// the partials added in part order (row_sq).  The streaming kernel's pairs sum
// in the same order, so both give the same bits.
template <int TR>
__device__ __forceinline__ void slab_row_partials(const float* Xs, int bs, float (*s_sq)[TR], int tid) {
  const int NT = bs / 32;
  const int r = tid % TR, part = tid / TR;
  float sq = 0.0f;
  if (part < NT) {
#pragma unroll 8
    for (int c = part * 32; c < part * 32 + 32; ++c) {
      const float v = Xs[xoff<TR>(r, c, bs)];
      sq = __fmaf_rn(v, v, sq);
    }
  }
  s_sq[part][r] = sq;
}
template <int TR>
__device__ __forceinline__ float row_sq(float (*s_sq)[TR], int NT, int r) {
  float sq = s_sq[0][r];
  for (int q = 1; q < NT; ++q) sq += s_sq[q][r];
  return sq;
}

// Two elements as 8-bit codes of format FMT (already scaled): E4M3 / E5M2
// by the hardware conversion; the FP6/FP4 MX elements rounded onto their
// grid first (the rounded value is exact in E4M3).
template <int FMT>
__device__ __forceinline__ uint32_t code8_x2(float a, float b) {
  if constexpr (FMT == E5M2) return f32x2_to_e5m2x2(a, b);
  else if constexpr (FMT == E4M3 || FMT == MXFP8) return f32x2_to_e4m3x2(a, b);
  else {
    const MxElem me = mx_elem(FMT);
    return f32x2_to_e4m3x2(mx_round_elem(a, me), mx_round_elem(b, me));
  }
}

// N scaled values as N bytes at dst (N = 8, 16 or 32; dst aligned to the
// smaller of N and 16).
template <int FMT, int N>
__device__ __forceinline__ void put_codes8(const float (&v)[N], float inv, uint8_t* dst) {
  uint32_t w[N / 4];
#pragma unroll
  for (int c = 0; c < N; c += 4)
    w[c / 4] = code8_x2<FMT>(v[c] * inv, v[c + 1] * inv) | (code8_x2<FMT>(v[c + 2] * inv, v[c + 3] * inv) << 16);
  if constexpr (N == 8) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
  else
#pragma unroll
    for (int q = 0; q < N / 16; ++q)
      reinterpret_cast<uint4*>(dst)[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
}

// One row's 32-column block (values v, largest magnitude amax) in an MX format:
// its own E8M0 scale, then its codes.
template <int FMT>
__device__ __forceinline__ void put_mx_block(const float (&v)[32], float amax, const QuantAll& qa, int gi,
                                             int block) {
  const int eb = mx_scale_exp(amax, FMT);
  qa.mxexp[(size_t)gi * qa.ldmx + block] = (uint8_t)(eb + 127);
  put_codes8<FMT>(v, pow2f(-eb), qa.q8[q8_slot(FMT)] + (size_t)gi * qa.ldq + 32 * block);
}

// The codes of a solved slab that take the row's power-of-two scale (FP16 and
// FP16X2, E4M3, E5M2), straight from the slab to global memory: thread (r,
// part) = (tid % TR, tid / TR) converts TR / 2 columns of row r, 16 bytes or
// more of codes in one piece.
template <int TR>
__device__ __forceinline__ void quantize_rows_of_slab(const float* Xs, int bs, int nrows, int gi0, int m,
                                                      float (*s_rmax)[TR], const QuantAll& qa, int tid) {
  constexpr int CW = TR / 2;
  const int r = tid % TR, c0 = tid / TR * CW;
  if (r >= nrows || c0 >= bs) return;
  const bool f16 = (qa.cand >> FP16) & 1u, f16x2 = (qa.cand >> FP16X2) & 1u;
  const bool e4 = (qa.cand >> E4M3) & 1u, e5 = (qa.cand >> E5M2) & 1u;
  if (!(f16 || f16x2 || e4 || e5)) return;
  const int gi = gi0 + r;
  float rmax = 0.0f, v[CW];
  for (int q = 0; q < bs / 32; ++q) rmax = fmaxf(rmax, s_rmax[q][r]);
#pragma unroll
  for (int u = 0; u < CW; ++u) v[u] = Xs[xoff<TR>(r, c0 + u, bs)];
  if (f16 || f16x2) {
    const int e = row_scale_exp(rmax, FP16);
    const float inv = pow2f(-e);
    if (c0 == 0) qa.rexp[2][gi] = (int8_t)e;
    uint4* dh = reinterpret_cast<uint4*>(qa.q16 + (size_t)gi * qa.ldq + c0);
    uint4* dl = reinterpret_cast<uint4*>(qa.q16 + (size_t)(m + gi) * qa.ldq + c0);
#pragma unroll
    for (int q = 0; q < CW / 8; ++q) {
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float x0 = v[8 * q + 2 * u] * inv, x1 = v[8 * q + 2 * u + 1] * inv;
        const __half2 h = __floats2half2_rn(x0, x1);
        hi[u] = *reinterpret_cast<const uint32_t*>(&h);
        const float2 hf = __half22float2(h);   // x - hi is exact in FP32
        lo[u] = f32x2_to_f16x2(x0 - hf.x, x1 - hf.y);
      }
      dh[q] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      if (f16x2) dl[q] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
  if (e4) {
    const int e = row_scale_exp(rmax, E4M3);
    if (c0 == 0) qa.rexp[rexp_slot(E4M3)][gi] = (int8_t)e;
    put_codes8<E4M3>(v, pow2f(-e), qa.q8[q8_slot(E4M3)] + (size_t)gi * qa.ldq + c0);
  }
  if (e5) {
    const int e = row_scale_exp(rmax, E5M2);
    if (c0 == 0) qa.rexp[rexp_slot(E5M2)][gi] = (int8_t)e;
    put_codes8<E5M2>(v, pow2f(-e), qa.q8[q8_slot(E5M2)] + (size_t)gi * qa.ldq + c0);
  }
}

// Panel solve with the quantization of the panel fused in; one slab of TR
// rows per CTA (the launch may exceed the resident CTAs: no CTA
// waits on another).  Each CTA stages its slab and L11 by TMA, solves the
// slab, writes it back, folds its rows into the diagonal tracker and the
// switching statistics, and writes the slab's codes in every candidate
// format (the step's precision is not known yet; the trailing update reads
// the panel of the one the step picks).  The CTA that finishes last (a
// ticket counter) resolves the step precision.
template <int TR>
__global__ void __launch_bounds__(NTHR, 1)
trsm_panel_kernel(const __grid_constant__ CUtensorMap tmapX, const __grid_constant__ CUtensorMap tmap32,
                  float* __restrict__ A, int lda, int n, int s, int bs, const float* __restrict__ winv,
                  const float* __restrict__ d, float* __restrict__ dtilde, float* __restrict__ rowsq,
                  StepState* step, StepState* next, int next_bs, DecisionParams dp, DevStatus* st,
                  QuantAll qa, const StepState* prev, double* __restrict__ colacc) {
  constexpr int HR = Slab<TR>::HR, RPL = Slab<TR>::RPL;
  constexpr int SW = TR > 32 ? 2 : 1;                    // warps that hold the slab's rows
  extern __shared__ __align__(128) float sm[];
  const int NT = bs / 32;
  float* Xs = sm;                                        // the slab (xoff layout)
  float* Lt = Xs + (size_t)bs * TR;                      // L_{I,M}, I > M
  float* Wt = Lt + (size_t)(NT * (NT - 1) / 2) * TSZ;    // L_JJ^-1
  __shared__ double red_coh[NTHR / 32];
  __shared__ float s_rmax[MAXNT][TR];                    // by tile column and row
  __shared__ float s_sq[MAXNT][TR];
  __shared__ __align__(8) uint64_t barx, lrow[MAXNT], ready[MAXNT];
  __shared__ int s_ok, s_last;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m = n - s - bs;
  const int slab = blockIdx.x;
  const int row0 = s + bs + slab * TR;                   // first global row of the slab
  const int nrows = min(TR, n - row0);
  const int gi0 = slab * TR;                             // first trailing row of the slab
  if (tid == 0) {
    tc::mbar_init(&barx, 1);
    for (int J = 0; J < NT; ++J) {
      tc::mbar_init(&lrow[J], 1);
      tc::mbar_init(&ready[J], 64);
    }
    tc::fence_mbar_init();
    s_last = 0;
  }
  __syncthreads();
  tc::grid_dep_wait();   // the POTRF (and the trailing update) before it are complete
  // the copies, spread over the warps (a copy takes its thread about 80 cycles
  // to issue): the slab, and each pair its own tile row of L11
  if (lane == 0) {
    if (warp == 1) {
      tc::mbar_expect_tx(&barx, (uint32_t)(TR * bs * sizeof(float)));
      for (int q = 0; q < RPL; ++q) tc::tma_load_2d(Xs + q * bs * HR, &tmapX, &barx, row0 + HR * q, s);
    }
    if ((warp & 1) == 0 && warp / 2 < NT) {
      const int J = warp / 2;
      tc::mbar_expect_tx(&lrow[J], (uint32_t)((J + 1) * TSZ * sizeof(float)));
      tc::bulk_load_1d(Wt + (size_t)J * TSZ, winv + (size_t)J * TSZ, (uint32_t)(TSZ * sizeof(float)), &lrow[J]);
      for (int M = 0; M < J; ++M)
        tc::tma_load_2d(Lt + (size_t)tl(J, M) * TSZ, &tmap32, &lrow[J], s + 32 * J, s + 32 * M);
    }
  }
  // the previous step's rounding shift for the slab's rows, before this
  // step's sums of squares replace the previous ones in rowsq
  if (prev != nullptr && qa.sh != nullptr && tid < nrows) {
    const int pp = prev->prec;
    if (pp != FP32) {
      float* shp = qa.sh + slab * TR + tid;
      *shp = __fmaf_rn(unit_roundoff(pp), rowsq[row0 + tid], *shp);
    }
  }
  if (tid == NTHR - 1) s_ok = st->code == 0;
  // every copy has landed before the CTA may leave (bounded, twice)
  const bool landed = tc::mbar_wait(&barx, 0) || tc::mbar_wait(&barx, 0);
  const bool all_landed = !__syncthreads_or(!landed);
  if (!all_landed && tid == 0) set_status(st, MPCHOL_ERR_TIMEOUT, row0);
  // a finished pair: its tile's row sums (a chain of FMAs in column order; the
  // row's sum is the tiles' in order), magnitudes, MX codes and column sums
  const int mx = (qa.cand >> MXFP8) & 1u       ? MXFP8
                 : (qa.cand >> MXFP6E2M3) & 1u ? MXFP6E2M3
                 : (qa.cand >> MXFP6E3M2) & 1u ? MXFP6E3M2
                 : (qa.cand >> MXFP4) & 1u     ? MXFP4
                                               : -1;
  auto post = [&](int J, int t) {
    if (t < TR) {
      float v[32], sq = 0.0f, amax = 0.0f;
#pragma unroll
      for (int u = 0; u < 32; ++u) v[u] = Xs[xoff<TR>(t, 32 * J + u, bs)];
#pragma unroll
      for (int u = 0; u < 32; ++u) {
        sq = __fmaf_rn(v[u], v[u], sq);
        amax = fmaxf(amax, fabsf(v[u]));
      }
      s_sq[J][t] = sq;
      s_rmax[J][t] = amax;
      // an MX-family member of the candidates (at most one: they share the MX
      // code slot and scales)
      if (mx >= 0 && t < nrows) {
        if (mx == MXFP8) put_mx_block<MXFP8>(v, amax, qa, gi0 + t, J);
        else if (mx == MXFP6E2M3) put_mx_block<MXFP6E2M3>(v, amax, qa, gi0 + t, J);
        else if (mx == MXFP6E3M2) put_mx_block<MXFP6E3M2>(v, amax, qa, gi0 + t, J);
        else put_mx_block<MXFP4>(v, amax, qa, gi0 + t, J);
      }
    }
    // column sums (coherence rule): a thread sums column c over the slab's
    // rows, starting at row c % TR so that a warp's threads read different banks
    // (a fixed order per column), and adds it into copy slab % kColCopies of
    // colacc (the copies spread the CTAs' atomics over more L2 lines).  The
    // sums reach colacc as FP64 atomics of FP32 partials, which are exact while
    // a column's partials span less than 2^20 in magnitude; the order of the
    // atomics then does not change the result
    if (colacc != nullptr && t >= 32) {
      const int c = 32 * J + t - 32;
      float cs = 0.0f;
#pragma unroll 8
      for (int q = 0; q < TR; ++q) {
        const int r = (q + c) & (TR - 1);
        cs += (r < nrows) ? Xs[xoff<TR>(r, c, bs)] : 0.0f;
      }
      atomicAdd(colacc + (size_t)(slab % kColCopies) * bs + c, (double)cs);
    }
  };
  bool solved = all_landed && s_ok;
  if (solved) solved = slab_solve<TR>(Xs, bs, Lt, Wt, lrow, ready, tid, post);
  const bool gave_up = all_landed && s_ok && !solved;
  tc::fence_proxy_async_smem();                          // the slab, to the copies out
  solved = !__syncthreads_or(!solved);
  if (gave_up) set_status(st, MPCHOL_ERR_TIMEOUT, row0);
  if (!solved && tid == 0)                               // no copy in flight at the exit
    for (int J = 0; J < NT; ++J) tc::mbar_wait(&lrow[J], 0);
  if (solved && tid == NTHR - 1) {                       // the solved slab (rows past n are clipped)
    for (int q = 0; q < RPL; ++q)
      if (row0 + HR * q < n) tc::tma_store_2d(&tmapX, Xs + q * bs * HR, row0 + HR * q, s);
    tc::bulk_commit();
  }
  // Schur diagonal tracker and switching statistics of the slab, then the
  // ticket, by the warps that hold its rows
  if (warp < SW) {
    float bm = 0.0f, bmin = INFINITY;   // max d/dtilde, min dtilde and literal code
    int bl = 0;
    if (solved && tid < nrows) {
      const int gi = row0 + tid;
      const float sq = row_sq<TR>(s_sq, NT, tid);
      rowsq[gi] = sq;
      const float dt = dtilde[gi] - sq;
      dtilde[gi] = dt;
      const float di = d[gi];
      float ratio = dt > 0.0f ? di / dt : INFINITY;
      if (isnan(ratio)) ratio = INFINITY;
      bm = fmaxf(bm, ratio);
      bmin = dt > 0.0f ? fminf(bmin, dt) : 0.0f;
      // reference list {FP32, FP16, E4M3} with the reference's machine epsilons
      const float ref_eps[3] = {1.1920929e-7f, 0.0009765625f, 0.125f};
      int pick = 0;
#pragma unroll
      for (int p = 2; p >= 0; --p)
        if (ref_eps[p] * dt >= dp.eps_prime * di) pick = p;
      bl = max(bl, 2 - pick);
      if (next != nullptr && dp.floor_ratio > 0.0f && gi - (s + bs) < next_bs &&
          dt <= dp.floor_ratio * di)
        next->fp64_diag = 1;
    }
    bm = warp_max(bm);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      bl = max(bl, __shfl_xor_sync(0xffffffffu, bl, o));
      bmin = fminf(bmin, __shfl_xor_sync(0xffffffffu, bmin, o));
    }
    if (lane == 0) {
      atomicMax(&step->max_ratio_bits, __float_as_uint(bm));
      atomicMax(&step->literal_code, bl);
      if (bmin < INFINITY) atomicMax(&step->not_min_dt_bits, ~__float_as_uint(fmaxf(bmin, 0.0f)));
    }
    if (SW > 1) pair_sync(0);
    if (tid == 0) {
      __threadfence();
      s_last = atomicAdd(&step->grid_bar, 1) == (int)gridDim.x - 1;
    }
  }
  if (solved) quantize_rows_of_slab<TR>(Xs, bs, nrows, gi0, m, s_rmax, qa, tid);
  if (tid == NTHR - 1) tc::bulk_wait_read();             // the copies out have read the slab
  // the next kernel (the head of the trailing update) may be scheduled; it
  // waits for this grid before reading
  tc::grid_dep_trigger();
  __syncthreads();
  if (!s_last) return;
  __threadfence();                                       // every CTA's statistics
  // coherence ratio (||P^T 1||^2 / m) / min dtilde: the column sums' squares
  // summed in a fixed order (warp butterflies, then warps in order)
  if (colacc != nullptr) {
    double c2 = 0.0;
    if (tid < bs) {
      double cs = 0.0;
      for (int q = 0; q < kColCopies; ++q)
        cs += *reinterpret_cast<volatile double*>(colacc + (size_t)q * bs + tid);
      c2 = cs * cs;
    }
    c2 = warp_sum(c2);
    if ((tid & 31) == 0) red_coh[tid >> 5] = c2;
    __syncthreads();
  }
  if (tid != 0) return;
  if (*reinterpret_cast<volatile int*>(&st->code) != 0) return;
  StepState ss;
  ss.max_ratio_bits = *reinterpret_cast<volatile unsigned int*>(&step->max_ratio_bits);
  ss.literal_code = *reinterpret_cast<volatile int*>(&step->literal_code);
  float coh = 0.0f;
  if (colacc != nullptr) {
    double c2 = 0.0;
    for (int w = 0; w < NTHR / 32; ++w) c2 += red_coh[w];
    const float mind = __uint_as_float(~*reinterpret_cast<volatile unsigned int*>(&step->not_min_dt_bits));
    const double g = c2 / (double)m;
    coh = (mind > 0.0f) ? (float)(g / (double)mind) : INFINITY;
    if (isnan(coh)) coh = INFINITY;
    step->coh_bits = __float_as_uint(coh);
  }
  ss.coh_bits = __float_as_uint(coh);
  step->prec = resolve_precision(&ss, dp);
}

// Batched: blockIdx.y = system, blockIdx.x = 32-row slab.  Staging by
// cp.async (no per-system tensor maps), all of it in flight at once: with plain
// loads, two in flight per thread, staging took as long as the solve (128
// systems of 64 to 2048, all steps: 1354 -> 788 us).  The same slab solve; the
// epilogue keeps the row sums of squares (rounding-shift estimate) and the
// diagonal tracker.
__global__ void __launch_bounds__(NTHR, 2)
trsm_batched_kernel(BatchSys* __restrict__ sys, int s, int b) {
  constexpr int TR = 32;
  const BatchSys& S = sys[blockIdx.y];
  const int n = S.n;
  const int bs = min(b, n - s);
  const int row0 = s + bs + blockIdx.x * TR;
  const int nrows = min(TR, n - row0);
  if (bs <= 0 || nrows <= 0 || S.st->code != 0) return;
  extern __shared__ __align__(128) float sm[];
  const int NT = bs / 32;                     // bs == b: only the last block can be partial
  float* Xs = sm;
  float* Lt = Xs + (size_t)bs * TR;
  float* Wt = Lt + (size_t)(NT * (NT - 1) / 2) * TSZ;
  __shared__ __align__(8) uint64_t ready[MAXNT];
  __shared__ int s_ok;
  const int tid = threadIdx.x;
  const float* A = S.A;
  const int ld = S.ld;
  if (tid == 0) {
    s_ok = 1;
    for (int J = 0; J < NT; ++J) tc::mbar_init(&ready[J], 64);
    tc::fence_mbar_init();
  }
  // everything by 16-byte asynchronous copies, all in flight at once (columns of
  // the library's storage start on 128-byte boundaries at multiples of 32 rows;
  // slab rows past n are its padding, whose results are not stored)
  const int r4 = 4 * (tid & 7);
  for (int c = tid >> 3; c < bs; c += NTHR / 8)
    tc::cp_async16(Xs + c * TR + r4, A + (size_t)(s + c) * ld + row0 + r4);
  for (int q = tid >> 8; q < NT * (NT - 1) / 2; q += NTHR / 256) {   // half a CTA per tile
    int I = 1;
    while (tl(I + 1, 0) <= q) ++I;
    const int M = q - tl(I, 0), c = (tid & 255) >> 3;
    tc::cp_async16(Lt + q * TSZ + c * 32 + r4, A + (size_t)(s + 32 * M + c) * ld + s + 32 * I + r4);
  }
  for (int e = 4 * tid; e < NT * TSZ; e += 4 * NTHR) tc::cp_async16(Wt + e, S.winv + e);
  tc::cp_async_wait_all();
  __syncthreads();
  if (!slab_solve<TR>(Xs, bs, Lt, Wt, nullptr, ready, tid, [](int, int) {})) {
    s_ok = 0;
    set_status(S.st, MPCHOL_ERR_TIMEOUT, row0);
  }
  __syncthreads();
  if (!s_ok) return;
  for (int c = tid >> 3; c < bs; c += NTHR / 8) {
    const float4 v = *reinterpret_cast<const float4*>(Xs + c * TR + r4);
    float* g = S.A + (size_t)(s + c) * ld + row0 + r4;
    if (r4 + 3 < nrows) *reinterpret_cast<float4*>(g) = v;
    else {
      if (r4 < nrows) g[0] = v.x;
      if (r4 + 1 < nrows) g[1] = v.y;
      if (r4 + 2 < nrows) g[2] = v.z;
    }
  }
  __shared__ float s_sq[NTHR / TR][TR];
  slab_row_partials<TR>(Xs, bs, s_sq, tid);
  __syncthreads();
  if (tid < nrows) {
    const int gi = row0 + tid;
    const float sq = row_sq<TR>(s_sq, NT, tid);
    S.rowsq[gi] = sq;
    S.dtilde[gi] -= sq;
  }
}

int sm_count() {
  static int nsm = 0;
  if (nsm == 0) {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
      nsm = v;
    else
      return 148;
  }
  return nsm;
}

template <int TR>
cudaError_t launch_panel(const CUtensorMap& tmapX, const CUtensorMap& tmap32, float* A, int lda,
                         int n, int s, int bs, const float* winv, const float* d, float* dtilde,
                         float* rowsq, StepState* step, StepState* next, int next_bs,
                         const DecisionParams& dp, const QuantAll& qa, DevStatus* st,
                         cudaStream_t stream, const StepState* prev, double* colacc) {
  const int m = n - s - bs;
  const size_t smem = trsm_smem_floats(TR, bs) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(trsm_panel_kernel<TR>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(trsm_smem_floats(TR, 256) * sizeof(float)));
  if (e != cudaSuccess) return e;
  PdlLaunch L(dim3(ceil_div(m, TR)), dim3(NTHR), smem, stream);
  e = cudaLaunchKernelEx(&L.cfg, trsm_panel_kernel<TR>, tmapX, tmap32, A, lda, n, s, bs, winv, d,
                         dtilde, rowsq, step, next, next_bs, dp, st, qa, prev, colacc);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_trsm_panel(const CUtensorMap& tmapX, const CUtensorMap& tmapX16,
                              const CUtensorMap& tmap32, float* A,
                              int lda, int n, int s, int bs, const float* winv, const float* d,
                              float* dtilde, float* rowsq, StepState* step, StepState* next,
                              int next_bs, const DecisionParams& dp, const QuantAll& qa,
                              DevStatus* st, cudaStream_t stream, const StepState* prev,
                              double* colacc) {
  const int m = n - s - bs;
  if (m <= 0) return cudaSuccess;
  if (bs % 32 != 0 || bs > 32 * MAXNT) return cudaErrorInvalidValue;
  // 64-row slabs while the panel has more 32-row slabs than the GPU has SMs
  // (throughput: L11 staged once per 64 rows); below that the smallest slabs
  // that all run at once (latency: a CTA's work follows its rows).  B200, b =
  // 256, a panel solve inside a factorization: 35 us with 64-row slabs, 22 with 32,
  // 16 with 16.
  const int nsm = sm_count();
  if (ceil_div(m, 32) > nsm)
    return launch_panel<64>(tmapX, tmap32, A, lda, n, s, bs, winv, d, dtilde, rowsq, step, next,
                            next_bs, dp, qa, st, stream, prev, colacc);
  if (ceil_div(m, 16) > nsm)
    return launch_panel<32>(tmapX, tmap32, A, lda, n, s, bs, winv, d, dtilde, rowsq, step, next,
                            next_bs, dp, qa, st, stream, prev, colacc);
  return launch_panel<16>(tmapX16, tmap32, A, lda, n, s, bs, winv, d, dtilde, rowsq, step, next,
                          next_bs, dp, qa, st, stream, prev, colacc);
}

cudaError_t launch_trsm_batched(BatchSys* sys, int nact, int s, int b, int max_m,
                                cudaStream_t stream) {
  if (nact <= 0 || max_m <= 0) return cudaSuccess;
  if (b % 32 != 0 || b > 32 * MAXNT) return cudaErrorInvalidValue;
  const size_t smem = trsm_smem_floats(32, b) * sizeof(float);
  // the kernel's limit, not the launch's: the most any block needs
  cudaError_t e = cudaFuncSetAttribute(trsm_batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(trsm_smem_floats(32, 32 * MAXNT) * sizeof(float)));
  if (e != cudaSuccess) return e;
  trsm_batched_kernel<<<dim3(ceil_div(max_m, 32), nact), NTHR, smem, stream>>>(sys, s, b);
  return cudaGetLastError();
}

}  // namespace mpchol
