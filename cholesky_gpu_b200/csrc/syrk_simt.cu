// FP32 trailing update (SIMT FFMA), the "plain FP32" path.
//
// Replaces the reference's FP32 trailing GEMM LtSgemm (src/switching_chol.cuh:200-219,
// src/fp8_utils.cuh:231-302) and the CUTLASS FP32 GEMM of the uniform-precision
// prototype (src/sChol.cuh:284-306).  Unlike the reference it updates only the
// lower-triangle tiles (a SYRK, half the flops of the full GEMM it issues).
//
// C(i, j) -= sum_k P(i, k) P(j, k), each sum one fma chain over k from zero
// (both kernels, so a tile's values do not depend on which one ran).
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace mpchol {
namespace {

constexpr int BM = 128, BK = 16, NTH = 256;
constexpr int STAGES = 3;
constexpr int STRIP = BK * BM;                     // floats of one operand's chunk
constexpr int GROUP_SMEM = STAGES * 2 * STRIP;     // floats per tile group

__device__ __forceinline__ void group_sync(int group) {
  // named barrier of one 256-thread tile group (barrier 0 is __syncthreads)
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(NTH) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async(float* dst, const float* src, int valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(valid) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ROWS rows of P's columns [k0, k0 + KC) into dst (KC x ROWS, rows
// contiguous), zero past row m and column k, by NT threads.  vec: P's columns
// start on 16-byte boundaries.
template <int ROWS, int KC, int NT>
__device__ __forceinline__ void stage_strip(float* dst, const float* __restrict__ P, int ldp, int m, int k,
                                            int row0, int k0, bool vec, int tid) {
  if (vec) {
#pragma unroll
    for (int e = tid; e < KC * ROWS / 4; e += NT) {
      const int kk = e / (ROWS / 4), r = 4 * (e % (ROWS / 4));
      const int n = (k0 + kk < k) ? max(0, min(4, m - row0 - r)) : 0;
      cp_async<16>(dst + kk * ROWS + r, n > 0 ? P + (size_t)(k0 + kk) * ldp + row0 + r : P, 4 * n);
    }
  } else {
#pragma unroll 4
    for (int e = tid; e < KC * ROWS; e += NT) {
      const int kk = e / ROWS, r = e % ROWS;
      const bool in = k0 + kk < k && row0 + r < m;
      cp_async<4>(dst + e, in ? P + (size_t)(k0 + kk) * ldp + row0 + r : P, in ? 4 : 0);
    }
  }
}

// One 128 x 128 output tile (I, J) by the 256 threads of a tile group.  FFMA
// bound: 8 x 8 outputs per thread (rows 4 rg.. and 32 + 4 rg.. of the warp's
// 64, columns 4 cg.. and 16 + 4 cg.. of its 32), chunks of 16 k in three
// cp.async stages, one barrier per chunk.  The lane's bits interleave into rg
// and cg so that four neighbouring lanes read two different vectors of each
// operand (2.2 cycles of the SM's shared memory per 16-byte load, not 4).
__device__ __forceinline__ void syrk_f32_tile(float* __restrict__ C, int ldc, int m, int k,
                                              const float* __restrict__ P, int ldp, int I, int J, bool vec,
                                              float* sm, int tid, int group) {
  const int i0 = I * BM, j0 = J * BM;
  const bool diag = I == J;
  const int lane = tid & 31, warp = tid >> 5;
  const int rg = (lane & 1) | ((lane >> 1) & 6), cg = ((lane >> 1) & 1) | ((lane >> 3) & 2);
  const int r0 = 64 * (warp & 1) + 4 * rg, c0 = 32 * (warp >> 1) + 4 * cg;
  const int nch = ceil_div(k, BK);
  auto issue = [&](int ch) {
    if (ch < nch) {
      float* a = sm + (ch % STAGES) * 2 * STRIP;
      stage_strip<BM, BK, NTH>(a, P, ldp, m, k, i0, ch * BK, vec, tid);
      if (!diag) stage_strip<BM, BK, NTH>(a + STRIP, P, ldp, m, k, j0, ch * BK, vec, tid);
    }
    cp_commit();
  };
  float acc[8][8];                                 // [row][column]
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[a][b] = 0.0f;
  group_sync(group);                               // the previous tile's stages are free
#pragma unroll
  for (int q = 0; q < STAGES - 1; ++q) issue(q);
  for (int ch = 0; ch < nch; ++ch) {
    cp_wait<STAGES - 2>();
    group_sync(group);                             // chunk ch landed; chunk ch - 1 is used up
    issue(ch + STAGES - 1);
    const float* As = sm + (ch % STAGES) * 2 * STRIP + r0;
    const float* Bs = sm + (ch % STAGES) * 2 * STRIP + (diag ? 0 : STRIP) + c0;
#pragma unroll 8
    for (int kk = 0; kk < BK; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(As + kk * BM);
      const float4 a1 = *reinterpret_cast<const float4*>(As + kk * BM + 32);
      const float4 b0 = *reinterpret_cast<const float4*>(Bs + kk * BM);
      const float4 b1 = *reinterpret_cast<const float4*>(Bs + kk * BM + 16);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int b = 0; b < 8; ++b)
#pragma unroll
        for (int a = 0; a < 8; ++a) acc[a][b] = fmaf(av[a], bv[b], acc[a][b]);
    }
  }
  cp_wait<0>();
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int j = j0 + c0 + (b < 4 ? b : 12 + b);
    if (j >= m) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = i0 + r0 + 32 * h;
      float* c = C + (size_t)j * ldc + i;
      if (i >= j && i + 3 < m && (reinterpret_cast<uintptr_t>(c) & 15) == 0) {
        float4 v = *reinterpret_cast<const float4*>(c);
        v.x -= acc[4 * h][b];
        v.y -= acc[4 * h + 1][b];
        v.z -= acc[4 * h + 2][b];
        v.w -= acc[4 * h + 3][b];
        *reinterpret_cast<float4*>(c) = v;
      } else {
#pragma unroll
        for (int a = 0; a < 4; ++a)
          if (i + a < m && i + a >= j) c[a] -= acc[4 * h + a][b];
      }
    }
  }
}

// Two independent 256-thread tile groups per CTA (one CTA per SM by its
// register use), each walking the selected tiles with stride 2 * gridDim.x.
// n = 4100, K = 256: 109 us for 496 tiles (186 us with 8-deep chunks, two
// barriers each, and no prefetch).
__global__ void __launch_bounds__(2 * NTH, 1)
syrk_f32_kernel(float* __restrict__ C, int ldc, int m, int k, const float* __restrict__ P, int ldp,
                const int* prec_sel, DevStatus* st, TileSel sel, int vec) {
  if (st != nullptr && st->code != 0) return;
  if (prec_sel != nullptr && *prec_sel != FP32) return;
  extern __shared__ __align__(16) float sm_f32[];
  const int group = threadIdx.x / NTH, tid = threadIdx.x % NTH;
  const int T = ceil_div(m, BM);
  const int ntiles = sel_tile_count(T, sel);
  for (int t = 2 * blockIdx.x + group; t < ntiles; t += 2 * gridDim.x) {
    int I, J;
    sel_tile(t, sel, T, I, J);
    syrk_f32_tile(C, ldc, m, k, P, ldp, I, J, vec != 0, sm_f32 + group * GROUP_SMEM, tid, group);
  }
}

// The selected tiles as 32 x 32 tiles, 16 per 128-tile, by groups of four warps
// (G groups per CTA, each walking the 32-tiles with stride G * gridDim.x).  Few
// 128-tiles leave most SMs without one, and one of them takes an SM 25 us at K =
// 256; these take 3 us and spread.
//   G = 1: as many CTAs as there are 32-tiles; the tiles of the next diagonal
//          block, on the chain of the factorization (b = 256: 9 us for its
//          three 128-tiles, 57 us as such);
//   G = 8: one CTA per SM by its shared memory, for the concurrent part of an
//          update, which must leave an SM to the POTRF.
constexpr int SM = 32, SNT = 128;
template <int G> struct SmallCfg {
  static constexpr int SK = G == 1 ? 64 : 32, STG = G == 1 ? 4 : 3;
  static constexpr int STRIP32 = SK * SM;
  static constexpr size_t SMEM = (size_t)G * STG * 2 * STRIP32 * sizeof(float);
};
template <int G>
__global__ void __launch_bounds__(SNT * G)
syrk_f32_small_kernel(float* __restrict__ C, int ldc, int m, int k, const float* __restrict__ P, int ldp,
                      const int* prec_sel, DevStatus* st, TileSel sel, int vec) {
  using Cfg = SmallCfg<G>;
  constexpr int SK = Cfg::SK, STG = Cfg::STG;
  if (st != nullptr && st->code != 0) return;
  if (prec_sel != nullptr && *prec_sel != FP32) return;
  extern __shared__ __align__(16) float sm_f32[];
  const int group = threadIdx.x / SNT, tid = threadIdx.x % SNT, lane = tid & 31, warp = tid >> 5;
  float* const sm = sm_f32 + group * STG * 2 * Cfg::STRIP32;
  auto sync = [&]() {
    if constexpr (G == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(SNT) : "memory");
  };
  const int T = ceil_div(m, BM);
  const int nsub = 16 * sel_tile_count(T, sel);
  // warp: a 16 x 16 quarter; lane: rows 4 rg.., columns 2 cg..
  const int r0 = 16 * (warp & 1) + 4 * ((lane & 1) | ((lane >> 1) & 2));
  const int c0 = 16 * (warp >> 1) + 2 * (((lane >> 1) & 1) | ((lane >> 2) & 6));
  const int nch = ceil_div(k, SK);
  auto tile = [&](int u) {
    int I, J;
    sel_tile(u >> 4, sel, T, I, J);
    const int i0 = I * BM + SM * (u & 3), j0 = J * BM + SM * ((u >> 2) & 3);
    if (i0 >= m || j0 >= m || i0 < j0) return;       // uniform over the group
    const bool diag = i0 == j0;
    auto issue = [&](int ch) {
      if (ch < nch) {
        float* a = sm + (ch % STG) * 2 * Cfg::STRIP32;
        stage_strip<SM, SK, SNT>(a, P, ldp, m, k, i0, ch * SK, vec != 0, tid);
        if (!diag) stage_strip<SM, SK, SNT>(a + Cfg::STRIP32, P, ldp, m, k, j0, ch * SK, vec != 0, tid);
      }
      cp_commit();
    };
    float acc[4][2] = {};
    if (G > 1) sync();                               // the previous tile's stages are free
#pragma unroll
    for (int q = 0; q < STG - 1; ++q) issue(q);
    for (int ch = 0; ch < nch; ++ch) {
      cp_wait<STG - 2>();
      sync();
      issue(ch + STG - 1);
      const float* As = sm + (ch % STG) * 2 * Cfg::STRIP32 + r0;
      const float* Bs = sm + (ch % STG) * 2 * Cfg::STRIP32 + (diag ? 0 : Cfg::STRIP32) + c0;
#pragma unroll 16
      for (int kk = 0; kk < SK; ++kk) {
        const float4 a = *reinterpret_cast<const float4*>(As + kk * SM);
        const float2 b = *reinterpret_cast<const float2*>(Bs + kk * SM);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          acc[r][0] = fmaf(av[r], b.x, acc[r][0]);
          acc[r][1] = fmaf(av[r], b.y, acc[r][1]);
        }
      }
    }
    cp_wait<0>();
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int j = j0 + c0 + b;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = i0 + r0 + r;
        if (j < m && i < m && i >= j) C[(size_t)j * ldc + i] -= acc[r][b];
      }
    }
  };
  if constexpr (G == 1) tile(blockIdx.x);
  else
    for (int u = G * blockIdx.x + group; u < nsub; u += G * gridDim.x) tile(u);
}
// 128-tiles up to which the 32-tiles run: beyond, the larger tiles' reuse of
// what shared memory delivers wins.
// (K = 256, groups of eight: 27 us to 55 tiles, 50 to 136, 68 to 210; 128-tiles
// 57 us to 294, 109 to 496.)
constexpr int kSmallTiles = 136;
constexpr size_t kF32Smem = (size_t)2 * GROUP_SMEM * sizeof(float);

}  // namespace

cudaError_t launch_syrk_f32(float* C, int ldc, int m, int k, const float* P, int ldp,
                            const int* prec_sel, DevStatus* st, cudaStream_t stream, TileSel sel,
                            int max_sms) {
  if (m <= 0) return cudaSuccess;
  const int ntiles = sel_tile_count(ceil_div(m, BM), sel);
  if (ntiles <= 0) return cudaSuccess;
  const int vec = (reinterpret_cast<uintptr_t>(P) & 15) == 0 && ldp % 4 == 0;
  auto go = [&](auto kernel, int grid, int threads, size_t smem) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, threads, smem, stream>>>(C, ldc, m, k, P, ldp, prec_sel, st, sel, vec);
    return cudaGetLastError();
  };
  if (ntiles <= kSmallTiles)
    return max_sms > 0 ? go(syrk_f32_small_kernel<8>, std::min(max_sms, 2 * ntiles), 8 * SNT, SmallCfg<8>::SMEM)
                       : go(syrk_f32_small_kernel<1>, 16 * ntiles, SNT, SmallCfg<1>::SMEM);
  return go(syrk_f32_kernel, std::min(max_sms > 0 ? max_sms : 148, ceil_div(ntiles, 2)), 2 * NTH, kF32Smem);
}

}  // namespace mpchol
