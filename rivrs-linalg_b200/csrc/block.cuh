// Complete pivoting on a diagonal block of up to 32 columns
// (factor_block_diagonal, sparse/src/symmetric/factor.rs:891-1153), by one CTA
// of 256 threads with the block in shared memory.
//
// The block is on the critical path of every 32 columns of a medium or large
// front, and it is 32 dependent pivot steps: bound by the latency of a step
// (two arg-max reductions, a reciprocal, the update), not by arithmetic.  So a
// step has one barrier and no section in which one warp works for the others:
//   * the trailing block is double-buffered (both triangles, so an entry needs
//     no row / column ordering): a step reads the old buffer through its
//     symmetric swap (positions sw(i)) and writes the updated entries at their
//     new positions; no warp swaps rows and columns first while others wait;
//   * every warp finds the pivot itself from the eight warps' candidates and
//     computes the reciprocal itself; a candidate's key carries the entry's
//     sign, so a 1x1 pivot needs no further load;
//   * each thread keeps the largest of its new entries (warps own the columns
//     j = warp mod 8, lanes rows), so the next arg-max takes one reduction per
//     warp instead of one per column;
//   * finished columns are stored by the row's original index (Lc), so later
//     swaps do not move them; they are put in position order once at the end.
// Every entry gets the operations of the reference's loops, in their order.
//
// Measured (clock64, one CTA, 32 columns): 55.5k -> 34.7k cycles where every
// pivot is 1x1 (a stencil's block), 41.3k -> 25.1k with mostly 2x2 pivots,
// against the version in which warp 0 searched, swapped and scaled while the
// others waited (three barrier-separated phases a step).  A step is ~1100
// cycles: barrier and candidate reduction ~300, decoding ~150, reciprocal ~90,
// update ~350, own reduction ~90.  Four warps (the repeated work issued once per
// scheduler: 41k / 29k), 16 warps with rows and columns kept in place and a
// position table (37k / 27k), and integer instead of FP64 compares (32.7k /
// 28.9k, slower over mixed pivots) were not better.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "dense.cuh"
#include "front.cuh"

namespace rvg {

constexpr int NT = APTP_THREADS;  // threads of the CTA APTP kernel
constexpr int IBMAX = 32;         // inner block size supported by the kernels

struct CtaShared {
  double T[IBMAX][IBMAX + 1];  // the block (lower triangle), in place
  int bperm[IBMAX];
  int8_t bdt[IBMAX];
  double bdd[IBMAX];
  double bdo[IBMAX];
  int bnelim, eff, n1, n2, end_pos, k;
  int tmpi;
  double dinv[IBMAX];
  unsigned two;  // bit c: a 2x2 pivot starts at c
  alignas(16) double TT[IBMAX][IBMAX + 2];  // the factored block transposed: TT[l][j] = L(j, l) (panel_row_t)
  // cta_block_factor only
  double Tb[IBMAX][IBMAX + 1];  // the other buffer of the trailing block
  double Lc[IBMAX][IBMAX + 1];  // Lc[c][r]: finished column c at the row of original index r
  double cand[2][NT / 32];      // per warp: largest magnitude of its new entries, and its key
  unsigned ckey[2][NT / 32];
};

// The largest magnitude (and, among equal ones, the smallest key) of the
// warp's lanes; magnitudes are >= 0, so their bits order like integers.
__device__ __forceinline__ void bf_argmax(double& v, unsigned& key) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  key = __reduce_min_sync(0xffffffffu, (hi == mh && lo == ml) ? key : 0xffffffffu);
  v = __hiloint2double((int)mh, (int)ml);
}

// A thread's running maximum: entries that are not > 0 in magnitude (NaN
// included) never count.  Key: (column, row) in the reference's scan order,
// then the sign.
struct BfMax {
  double v;
  unsigned key;
  __device__ __forceinline__ void take(double x, int j, int i) {
    const double a = fabs(x);
    if (a > v) {
      v = a;
      key = (unsigned)((j * 64 + i) * 2) | ((unsigned)__double2hiint(x) >> 31);
    }
  }
};

// Factors the bs x bs block in sh.T (lower triangle); leaves the factored
// block there (the D part of a 2x2 pivot included), the order in bperm, the
// pivots in bdt / bdd / bdo and the eliminated count in bnelim.
__device__ void cta_block_factor(CtaShared& sh, int bs, double small) {
  static_assert(NT == 256 && IBMAX == 32, "the update's column split assumes 8 warps and 32-column blocks");
  constexpr int Q = IBMAX / 8;  // columns of a warp
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (tid < IBMAX) { sh.bdt[tid] = PT_DELAYED; sh.bdd[tid] = 0; sh.bdo[tid] = 0; }
  int id = lane;  // original index of the row at position `lane`
  BfMax b{0.0, 0xffffffffu};
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int j = warp + 8 * q;
    if (lane >= j && lane < bs) {
      const double v = sh.T[lane][j];
      sh.T[j][lane] = v;
      b.take(v, j, lane);
    }
  }
  bf_argmax(b.v, b.key);
  if (lane == 0) { sh.cand[0][warp] = b.v; sh.ckey[0][warp] = b.key; }
  double(*T)[IBMAX + 1] = sh.T;
  double(*U)[IBMAX + 1] = sh.Tb;
  int cur = 0, ph = 0;
  for (; cur < bs; ph ^= 1) {
    __syncthreads();
    double mx = sh.cand[ph][lane & 7];
    unsigned key = sh.ckey[ph][lane & 7];
    bf_argmax(mx, key);
    if (!(mx >= small)) break;
    int mr = cur, mc = cur;
    double d;
    if (key != 0xffffffffu) {
      mc = (int)(key >> 7);
      mr = (int)(key >> 1) & 63;
      d = __hiloint2double(__double2hiint(mx) | (int)(key << 31), __double2loint(mx));
    } else {
      d = T[cur][cur];
    }
    int p1 = mr;  // 1x1: the pivot's position
    bool two = false;
    double amm = 0.0, att = 0.0, delta = 0.0;
    const double atm = d;
    if (mr != mc) {
      amm = T[mc][mc];
      att = T[mr][mr];
      delta = __dsub_rn(__dmul_rn(amm, att), __dmul_rn(atm, atm));
      two = fabs(delta) >= __dmul_rn(__dmul_rn(0.5, atm), atm);
      const bool m = fabs(amm) >= fabs(att);
      p1 = m ? mc : mr;
      d = m ? amm : att;
    }
    b = BfMax{0.0, 0xffffffffu};
    const int i = lane;
    if (!two) {  // T[i][j] -= L_i (L_j d), L = T[:, cur] / d, after the swap of cur and p1
      const double inv = __drcp_rn(d);
      const int si = i == cur ? p1 : (i == p1 ? cur : i);
      const double* Ti = T[si];
      const double ti = Ti[p1];
      double tj[Q], tij[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = warp + 8 * q;
        const int sj = j == cur ? p1 : (j == p1 ? cur : j);
        tj[q] = T[sj][p1];
        tij[q] = Ti[sj];
      }
      id = __shfl_sync(0xffffffffu, id, si);
      const double li = __dmul_rn(ti, inv);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = warp + 8 * q;
        const double nv = __dsub_rn(tij[q], __dmul_rn(li, __dmul_rn(__dmul_rn(tj[q], inv), d)));
        if (j > cur && j <= i && i < bs) {
          U[i][j] = nv;
          U[j][i] = nv;
          b.take(nv, j, i);
        }
      }
      if (warp == (cur & 7)) {
        if (i >= cur && i < bs) sh.Lc[cur][id] = i == cur ? d : li;
        if (i == cur) { sh.bdt[cur] = PT_1X1; sh.bdd[cur] = d; }
      }
      cur += 1;
    } else {  // rank 2: the swaps bring (mc, mr) to (cur, cur + 1); a11 = amm, a22 = att, a21 = atm, det = delta
      const double inv = __drcp_rn(delta);
      const int nt = mr == cur ? mc : mr;  // where the second swap finds mr
      auto sw = [&](int x) {
        const int y = x == cur + 1 ? nt : (x == nt ? cur + 1 : x);
        return y == cur ? mc : (y == mc ? cur : y);
      };
      const int si = sw(i);
      const double* Ti = T[si];
      const double x1 = Ti[mc], x2 = Ti[mr];
      double y1[Q], y2[Q], tij[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int sj = sw(warp + 8 * q);
        y1[q] = T[sj][mc];
        y2[q] = T[sj][mr];
        tij[q] = Ti[sj];
      }
      id = __shfl_sync(0xffffffffu, id, si);
      const double l1 = __dmul_rn(__dsub_rn(__dmul_rn(x1, att), __dmul_rn(x2, atm)), inv);
      const double l2 = __dmul_rn(__dsub_rn(__dmul_rn(x2, amm), __dmul_rn(x1, atm)), inv);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int j = warp + 8 * q;
        const double m1 = __dmul_rn(__dsub_rn(__dmul_rn(y1[q], att), __dmul_rn(y2[q], atm)), inv);
        const double m2 = __dmul_rn(__dsub_rn(__dmul_rn(y2[q], amm), __dmul_rn(y1[q], atm)), inv);
        const double w1 = __dadd_rn(__dmul_rn(m1, amm), __dmul_rn(m2, atm));
        const double w2 = __dadd_rn(__dmul_rn(m1, atm), __dmul_rn(m2, att));
        const double nv = __dsub_rn(tij[q], __dadd_rn(__dmul_rn(l1, w1), __dmul_rn(l2, w2)));
        if (j > cur + 1 && j <= i && i < bs) {
          U[i][j] = nv;
          U[j][i] = nv;
          b.take(nv, j, i);
        }
      }
      if (warp == (cur & 7) && i >= cur && i < bs) {
        sh.Lc[cur][id] = i == cur ? amm : (i == cur + 1 ? atm : l1);
        if (i > cur) sh.Lc[cur + 1][id] = i == cur + 1 ? att : l2;
        if (i == cur) {
          sh.bdt[cur] = PT_2X2; sh.bdt[cur + 1] = PT_2X2B;
          sh.bdd[cur] = amm; sh.bdd[cur + 1] = att; sh.bdo[cur] = atm;
        }
      }
      cur += 2;
    }
    bf_argmax(b.v, b.key);
    if (lane == 0) { sh.cand[ph ^ 1][warp] = b.v; sh.ckey[ph ^ 1][warp] = b.key; }
    double(*t)[IBMAX + 1] = T;
    T = U;
    U = t;
  }
  __syncthreads();
  // finished columns in position order; the trailing triangle is in the buffer T
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int j = warp + 8 * q;
    if (lane >= j && lane < bs) {
      if (j < cur) sh.T[lane][j] = sh.Lc[j][id];
      else if (T != sh.T) sh.T[lane][j] = T[lane][j];
    }
  }
  if (warp == 0) sh.bperm[lane] = id;
  if (tid == 0) sh.bnelim = cur;
  __syncthreads();
}

// The reciprocals each panel row's D^-1 step uses, 1 / d (1x1) or 1 / det
// (first column of a 2x2), by 32 threads (c = pivot).
__device__ __forceinline__ double pivot_inv(int c, int n, const int8_t* bdt, const double* bdd, const double* bdo) {
  if (c >= n) return 0.0;
  if (bdt[c] == PT_1X1) return 1.0 / bdd[c];
  if (bdt[c] == PT_2X2 && c + 1 < IBMAX)
    return 1.0 / __dsub_rn(__dmul_rn(bdd[c], bdd[c + 1]), __dmul_rn(bdo[c], bdo[c]));
  return 0.0;
}

// One panel row (apply_and_check, factor.rs:1295-1408) in registers, x[j] =
// its entry in the block's column j: x L11^-T over the n eliminated columns,
// then D^-1.  The outer loop is over the finished column l, the inner one
// over the later columns j: each x[j] still takes its terms in ascending l,
// but the n - l updates of a step are independent (the loop over j first is
// one dependent chain of n (n - 1) / 2 multiply-adds).  TT holds L11 by
// columns, so the inner loop reads two entries per shared-memory load.
// two: bit c set where a 2x2 pivot starts (a mask in a register: a type read
// from shared memory would put a load before every column's branch).  Returns
// the first pivot (1x1 or 2x2 start) with an entry at or above bound.
// FULL: n = 32, the usual block: no column is tested against n.
template <bool FULL>
__device__ __forceinline__ int panel_row_t(double (&x)[IBMAX], const double (*TT)[IBMAX + 2], unsigned two,
                                           const double* bdd, const double* bdo, const double* dinv, int n,
                                           double bound) {
#pragma unroll
  for (int l = 0; l + 1 < IBMAX; ++l) {
    if (!FULL && l + 1 >= n) break;
    const double nx = -x[l];
#pragma unroll
    for (int j = (l + 1) & ~1; j < IBMAX; j += 2) {
      const double2 t = *reinterpret_cast<const double2*>(&TT[l][j]);
      if (j > l && (FULL || j < n)) x[j] = __fma_rn(nx, t.x, x[j]);
      if (FULL || j + 1 < n) x[j + 1] = __fma_rn(nx, t.y, x[j + 1]);
    }
  }
  unsigned bad = 0;
#pragma unroll
  for (int c = 0; c < IBMAX; ++c) {
    if ((!FULL && c >= n) || (c > 0 && (two >> (c - 1)) & 1)) continue;  // (a second column goes with its first)
    const int d = c + 1 < IBMAX ? c + 1 : c;
    if ((two >> c) & 1) {
      const double A_ = bdd[c], B_ = bdo[c], C_ = bdd[d], inv_det = dinv[c];
      const double x1 = x[c], x2 = x[d];
      x[c] = __dmul_rn(__dsub_rn(__dmul_rn(x1, C_), __dmul_rn(x2, B_)), inv_det);
      x[d] = __dmul_rn(__dsub_rn(__dmul_rn(x2, A_), __dmul_rn(x1, B_)), inv_det);
      if (fabs(x[c]) >= bound || fabs(x[d]) >= bound) bad |= 1u << c;
    } else {
      x[c] = __dmul_rn(x[c], dinv[c]);
      if (fabs(x[c]) >= bound) bad |= 1u << c;
    }
  }
  return bad ? __ffs(bad) - 1 : n;
}

// The row's W = L D (compute_ld_into, factor.rs:1536-1563) in place of x, for
// its first n columns.
__device__ __forceinline__ void panel_row_w(double (&x)[IBMAX], unsigned two, const double* bdd, const double* bdo,
                                            int n) {
#pragma unroll
  for (int c = 0; c < IBMAX; ++c) {
    if (c >= n || (c > 0 && (two >> (c - 1)) & 1)) continue;
    const int d = c + 1 < IBMAX ? c + 1 : c;
    if ((two >> c) & 1) {
      const double l1 = x[c], l2 = x[d];
      x[c] = __dadd_rn(__dmul_rn(l1, bdd[c]), __dmul_rn(l2, bdo[c]));
      x[d] = __dadd_rn(__dmul_rn(l1, bdo[c]), __dmul_rn(l2, bdd[d]));
    } else {
      x[c] = __dmul_rn(x[c], bdd[c]);
    }
  }
}

}  // namespace rvg
