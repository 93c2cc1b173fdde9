// FP64 lower-triangular rank-K update, the Schur-complement contraction of
// the numeric phase:
//
//     C[i, j] = fma(-W[i, c], L[j, c], C[i, j])   for c = 0 .. K-1 in order,
//     over rows i in [r0, r1), columns j in [c0, c1), only where i >= j.
//
// W = L * D (the pivot block applied); both W and L are column-major.  Used
// for the deferred trailing update of a two-level outer block
// (update_trailing, sparse/src/symmetric/factor.rs:1418-1526, applied once per
// 256-column outer block) and the NFS x NFS contribution block
// (compute_contribution_gemm, factor.rs:1590-1652).
//
// sm_100a has no FP64 tcgen05 kind: the kernel uses the FP64 tensor-core
// mma.sync (DMMA), K staged through shared memory in chunks of 16 by cp.async in
// a three-stage pipeline (8-byte copies: panel leading dimensions are odd in
// general; out-of-range elements are zero-filled by the copy itself).  Each
// 8x8x4 step adds a chain of four products to the accumulator in k order, so
// each output keeps one fma chain in K order and the result is bit-identical to
// the oracle's per-entry loop (checked on the device).  WR x WC warps of 32 x 32
// outputs (4 x 4 fragments of 8 x 8); W is negated when its fragments are read.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace rvg {

constexpr int G_BK = 16, G_STAGES = 3;

struct SyrkArgs {
  double* C;
  int64_t ldc;
  const double* W;  // W[i, c] = W[(i - r0) + c * ldw]
  int64_t ldw;
  const double* L;  // L[j, c] = L[j + c * ldl]   (j in C's column coordinates)
  int64_t ldl;
  int64_t r0, r1, c0, c1;
  int64_t K;
  const int32_t* Kdev;  // when set, *Kdev is added to K (columns counted on the device)
  // when set, the update runs only if *cond < cond_lt (decided on the device)
  const int32_t* cond;
  int32_t cond_lt;
  const int32_t* skip;  // when set and nonzero, the launch does nothing
};

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
  unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  int n = valid ? 8 : 0;  // 0 source bytes: the 8 destination bytes are zero-filled
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

template <int WR, int WC>
struct DmmaCfg {
  static constexpr int NT = 32 * WR * WC, BM = 32 * WR, BN = 32 * WC;
  static constexpr int LDW = BM + 8, LDL = BN + 8;  // k rows shifted 64 B apart: conflict-free fragment reads
  static constexpr size_t SMEM = (size_t)G_STAGES * G_BK * (LDW + LDL) * sizeof(double);
};

template <int WR, int WC, int MINB>
__global__ void __launch_bounds__(32 * WR * WC, MINB) k_syrk_dmma(SyrkArgs a) {
  using Cfg = DmmaCfg<WR, WC>;
  constexpr int NT = Cfg::NT, BM = Cfg::BM, BN = Cfg::BN, LDW = Cfg::LDW, LDL = Cfg::LDL;
  const int64_t i0 = a.r0 + (int64_t)blockIdx.y * BM;
  const int64_t j0 = a.c0 + (int64_t)blockIdx.x * BN;
  if (i0 >= a.r1 || j0 >= a.c1) return;
  if (i0 + BM - 1 < j0) return;
  if ((a.cond && *a.cond >= a.cond_lt) || (a.skip && *a.skip)) return;
  const int64_t K = (a.Kdev ? (int64_t)*a.Kdev : 0) + a.K;
  if (K <= 0) return;  // nothing eliminated: C unchanged
  extern __shared__ double gsm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = (warp % WR) * 32, wc = (warp / WR) * 32;
  const int nchunk = (int)((K + G_BK - 1) / G_BK);
  // A thread copies one row of W and one of L, every NT / BM-th (NT / BN-th)
  // column: its addresses advance by a constant.  (Indexed per element, the 64-bit
  // products and bounds were most of the instructions of a chunk: 27.2 -> 31.3
  // TFLOP/s on a 9600^2 rank-1024 update.)
  static_assert(NT % BM == 0 && NT % BN == 0, "a thread keeps its row");
  constexpr int SW = NT / BM, SL = NT / BN;  // columns between a thread's copies
  const int rw = tid % BM, kw = tid / BM, rl = tid % BN, kl = tid / BN;
  const bool okw = i0 + rw < a.r1, okl = j0 + rl < a.c1;
  const double* pw = a.W + (okw ? i0 + rw - a.r0 : 0) + (int64_t)kw * a.ldw;
  const double* pl = a.L + (okl ? j0 + rl : a.c0) + (int64_t)kl * a.ldl;
  const int64_t stw = SW * a.ldw, stl = SL * a.ldl;
  auto issue = [&](int ch) {
    double* sw = gsm + (ch % G_STAGES) * G_BK * (LDW + LDL);
    double* sl = sw + G_BK * LDW;
    const int64_t k0 = (int64_t)ch * G_BK;
    const bool full = k0 + G_BK <= K;
    const double* p = pw + k0 * a.ldw;
    const double* q = pl + k0 * a.ldl;
#pragma unroll
    for (int e = 0; e < G_BK / SW; ++e) {
      const bool v = okw && (full || k0 + kw + SW * e < K);
      cp_async8(sw + (kw + SW * e) * LDW + rw, v ? p : a.W, v);
      p += stw;
    }
#pragma unroll
    for (int e = 0; e < G_BK / SL; ++e) {
      const bool v = okl && (full || k0 + kl + SL * e < K);
      cp_async8(sl + (kl + SL * e) * LDL + rl, v ? q : a.L, v);
      q += stl;
    }
  };
#pragma unroll
  for (int s = 0; s < G_STAGES - 1; ++s) {
    if (s < nchunk) issue(s);
    cp_async_commit();
  }
  double acc[4][4][2];
  const int fr = lane >> 2, fc = (lane & 3) * 2;
#pragma unroll
  for (int mi = 0; mi < 4; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        // (clamped to the last row and column; what lies past them is not stored)
        const int64_t i = i0 + wr + mi * 8 + fr, j = j0 + wc + ni * 8 + fc + q;
        acc[mi][ni][q] = a.C[(i < a.r1 ? i : a.r1 - 1) + (j < a.c1 ? j : a.c1 - 1) * a.ldc];
      }
  for (int ch = 0; ch < nchunk; ++ch) {
    cp_async_wait<G_STAGES - 2>();
    __syncthreads();
    if (ch + G_STAGES - 1 < nchunk) issue(ch + G_STAGES - 1);
    cp_async_commit();
    const double* sw = gsm + (ch % G_STAGES) * G_BK * (LDW + LDL);
    const double* sl = sw + G_BK * LDW;
    // k beyond K is zero-filled in both operands: those steps add exact zeros
#pragma unroll
    for (int k4 = 0; k4 < G_BK; k4 += 4) {
      double af[4], bf[4];
      const int kk = k4 + (lane & 3);
#pragma unroll
      for (int mi = 0; mi < 4; ++mi) af[mi] = -sw[kk * LDW + wr + mi * 8 + fr];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) bf[ni] = sl[kk * LDL + wc + ni * 8 + fr];
#pragma unroll
      for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                       : "+d"(acc[mi][ni][0]), "+d"(acc[mi][ni][1])
                       : "d"(af[mi]), "d"(bf[ni]));
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int mi = 0; mi < 4; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int64_t i = i0 + wr + mi * 8 + fr, j = j0 + wc + ni * 8 + fc + q;
        if (i < a.r1 && j < a.c1 && i >= j) a.C[i + j * a.ldc] = acc[mi][ni][q];
      }
}


// the configuration used by the library: DMMA, 2 x 2 warps (64 x 64 tile),
// four CTAs per SM (the fastest of the measured shapes on a 9600^2 rank-1024
// update: 31.3 TFLOP/s; 128 x 64 with 4 or 8 warps 30.3 and 30.8, 64 x 128 29.4,
// 128 x 128 26.8; a fourth stage or tiles walked in groups of rows change nothing)
constexpr int SYRK_WR = 2, SYRK_WC = 2, SYRK_MINB = 4;
using SyrkMain = DmmaCfg<SYRK_WR, SYRK_WC>;
constexpr int G_T = SyrkMain::NT;
constexpr size_t G_SMEM = SyrkMain::SMEM;
constexpr auto k_syrk_lower = k_syrk_dmma<SYRK_WR, SYRK_WC, SYRK_MINB>;

inline dim3 syrk_grid(const SyrkArgs& a) {
  int64_t nr = (a.r1 - a.r0 + SyrkMain::BM - 1) / SyrkMain::BM, nc = (a.c1 - a.c0 + SyrkMain::BN - 1) / SyrkMain::BN;
  return dim3((unsigned)(nc > 0 ? nc : 0), (unsigned)(nr > 0 ? nr : 0));
}

}  // namespace rvg
