// Multi-kernel APTP for one large front (front order >= the large-front
// threshold): the same algorithm as the CTA kernel (factor_inner,
// factor.rs:1811-2095; two_level_factor, factor.rs:2108-2252) with every
// row-parallel step spread over the whole GPU and the pivot state kept on the
// device, so the host issues a fixed launch sequence:
//
//   per 256-column outer block, first:
//     lf_begin   1 CTA    checks the block's start column, then complete
//                         pivoting on its first 32-column diagonal block
//   per 32-column inner block (view-local position k), two launches:
//     lf_panel   grid     backup, column permutation, TRSM, D^-1 scaling,
//                         W = L D and the a-posteriori threshold scan of every
//                         panel row; the block's row permutation of the outer
//                         block's earlier columns
//     lf_update  grid     CTA 0: the NEXT inner block's 32 x 32 diagonal block
//                         takes this block's update and is factored at once; the
//                         other CTAs: the rank-32 update of the outer block's trailing columns
//                         on the FP64 tensor pipe.  The block is 32 dependent
//                         pivot steps on one SM, so it runs beside the update
//                         instead of after it (the block's own D entries are
//                         written by the last CTA).  When columns failed their
//                         threshold test, nothing is known of the next block
//                         yet: CTA 0 does the post-processing, the others also
//                         restore the failed panel columns and form their
//                         cross term, and the CTA that finishes last moves the
//                         delayed columns and factors the next block.
//   per 256-column outer block:
//     lf_prop    grid     row permutation of the front's earlier columns
//                         (W of the rows below the outer block is in the window
//                         of pending columns already: lf_panel wrote it)
//     Schur GEMM          the deferred update (update_trailing), split in
//                         two: the next outer block's columns take every
//                         pending column at once (near field); the columns
//                         after it (far field) only when the window is full
//                         (LF_WINDOW outer blocks, mixed_window in the mixed
//                         form) or when this block delayed
//                         a column (decided on the device), so each far-field
//                         entry is read and written once per window instead
//                         of once per block.  Each entry still takes one fma
//                         chain over the eliminated columns in order, so the
//                         result is bit-identical to the per-block update.
//     lf_outer   1 CTA    column order, delays to the end of the remaining
//                         fully-summed columns
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "dense.cuh"

namespace rvg {

// one inner block: its position, width, pivots found and eliminated, and the
// factored block
struct LFBlk {
  int32_t k, bs, bnelim, eff;
  uint32_t two;       // bit c: a 2x2 pivot starts at c
  int32_t bperm[32];
  int8_t bdt[32];
  double bdd[32], bdo[32], dinv[32];  // dinv: what the rows' D^-1 step multiplies by (pivot_inv)
  double T[32][33];   // factored block, 2x2 off-diagonals zeroed (the L11 of the TRSM)
  double Tb[32][33];  // the block before factorization
};

struct LFState {
  int32_t end_pos, gne, n1, n2, bne;
  // set when an outer block was launched for another start column than the
  // device reached (the host issues blocks ahead assuming no delays): every
  // later launch of the front returns at once until the host clears it
  int32_t spec_bad;
  int32_t done;  // CTAs of a k_lf_update with failed columns that have finished
  int32_t far_bne, far_skip;  // bne and spec_bad as they were when the far-field update on the far stream was forked
  int32_t valid[2];  // the outer block (its number + 1) that began last with each parity
  LFBlk b[2];    // inner block i is b[i & 1]: the update of block i factors block i + 1
};

struct LFArgs {
  double* a;        // front panel (m x p), ld m
  int64_t m, p;
  int32_t* perm;    // front pivot order (p)
  DRec D;           // front D (p)
  LFState* st;
  int32_t* lp;      // outer-block local column order (nb)
  double* pb;       // panel backup, rows x 32 (ld = bm)
  double* w;        // inner W, rows x 32 (column-major, ld = rows of the view)
  double* wo;       // pending W (column-major, ld wld): row i, pending column c at wo[(i - wrow0) + c * wld]
  int64_t wld, wrow0, wcol0;  // leading dimension, first row, this block's first pending column
  int64_t cs, bcols;  // outer block start, width
  int par;          // which of the state's two blocks is the current inner block
  int win;          // the rows below the outer block keep their W (the outer block joins the window)
  int outer;        // the outer block's number (lp is one of two arrays, by its parity)
  DevOpts o;
};

__global__ void k_lf_init(LFState* st, int32_t* perm, int64_t p) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->gne = 0; st->n1 = 0; st->n2 = 0; st->spec_bad = 0; st->done = 0;
    st->valid[0] = st->valid[1] = 0;
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < p; i += (int64_t)gridDim.x * blockDim.x)
    perm[i] = (int32_t)i;
}

// Complete pivoting on the diagonal block at view position k, into the state's
// block q (1 CTA).  n > 0: the n columns from position upd on (the block before,
// all of whose columns passed) are still to be applied: the entries first take
// that update, one fma chain per entry in column order, as the tensor-pipe
// tiles give the rest of the trailing columns.
__device__ void lf_block_cta(const LFArgs& A, CtaShared& sh, int q, int k, int end_pos, int upd, int n) {
  LFBlk& B = A.st->b[q];
  const int tid = threadIdx.x;
  PanelView V{A.a + A.cs + A.cs * A.m, A.m};
  const int bs = min(end_pos - k, A.o.ib);
  if (k >= end_pos) {  // no columns left in this outer block
    if (tid == 0) { B.k = k; B.bs = 0; B.bnelim = 0; B.eff = 0; B.two = 0; }
    return;
  }
  // 4 entries per thread, every load before the first store
  constexpr int PER = IBMAX * IBMAX / NT;
  const int i = tid % IBMAX, j0 = tid / IBMAX;
  double v[PER];
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int j = j0 + u * (NT / IBMAX);
    v[u] = (i < bs && j < bs && i >= j) ? V(k + i, k + j) : 0.0;
  }
  if (n > 0) {
    const int64_t bm = A.m - A.cs;
    double wv[PER], lv[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int c = j0 + u * (NT / IBMAX);
      const bool in = i < bs && c < n;
      wv[u] = in ? A.w[(k + i) + c * bm] : 0.0;
      lv[u] = in ? V(k + i, upd + c) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int c = j0 + u * (NT / IBMAX);
      sh.Tb[i][c] = wv[u];
      sh.Lc[i][c] = lv[u];
    }
    __syncthreads();
    for (int c = 0; c < n; ++c) {
      const double w = -sh.Tb[i][c];
#pragma unroll
      for (int u = 0; u < PER; ++u) v[u] = __fma_rn(w, sh.Lc[j0 + u * (NT / IBMAX)][c], v[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int j = j0 + u * (NT / IBMAX);
    if (i < bs && j < bs && i >= j) { sh.T[i][j] = v[u]; B.Tb[i][j] = v[u]; }
  }
  __syncthreads();
  cta_block_factor(sh, bs, A.o.small);
  const int bnelim = sh.bnelim;
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    const int j = j0 + u * (NT / IBMAX);
    if (i < bs && j < bs && i >= j) {
      // (the D off-diagonal of a 2x2 pivot is zeroed in L; where no pivot was found the panel stays as it is)
      const double t = (i == j + 1 && j < bnelim && sh.bdt[j] == PT_2X2) ? 0.0 : sh.T[i][j];
      if (bnelim > 0) V(k + i, k + j) = t;
      else if (n > 0) V(k + i, k + j) = v[u];
      B.T[i][j] = t;
    }
  }
  // (the row permutation of the view columns 0..k, step 5, is done by k_lf_panel's threads c < k)
  if (tid < 32) {
    if (bnelim > 0) {  // column order (step 6): lane i takes the entry of lane bperm[i]
      const int32_t ob = tid < bs ? A.lp[k + tid] : 0;
      const int32_t nbv = __shfl_sync(0xffffffffu, ob, sh.bperm[tid] & 31);
      if (tid < bs) A.lp[k + tid] = nbv;
    }
    B.bperm[tid] = sh.bperm[tid];
    B.bdt[tid] = sh.bdt[tid];
    B.bdd[tid] = sh.bdd[tid];
    B.bdo[tid] = sh.bdo[tid];
    B.dinv[tid] = pivot_inv(tid, bnelim, sh.bdt, sh.bdd, sh.bdo);
    const unsigned two = __ballot_sync(0xffffffffu, tid < bnelim && sh.bdt[tid] == PT_2X2);
    if (tid == 0) { B.k = k; B.bs = bs; B.bnelim = bnelim; B.eff = bnelim; B.two = two; }
  }
}

// Start of an outer block and its first inner block (1 CTA).
__global__ void __launch_bounds__(NT) k_lf_begin_outer(LFArgs A) {
  chain_enter();
  __shared__ CtaShared sh;
  LFState* st = A.st;
  if (st->spec_bad) return;
  if (st->gne != (int32_t)A.cs) {  // issued for a start column the factorization did not reach
    __syncthreads();               // every thread has read gne before it is flagged
    if (threadIdx.x == 0) st->spec_bad = 1;
    return;
  }
  if (threadIdx.x == 0) { st->end_pos = (int32_t)A.bcols; st->bne = 0; st->valid[A.outer & 1] = A.outer + 1; }
  for (int i = threadIdx.x; i < A.bcols; i += blockDim.x) A.lp[i] = i;
  __syncthreads();
  lf_block_cta(A, sh, 0, 0, (int)A.bcols, 0, 0);
}

// panel rows: backup, permute, TRSM, D^-1, threshold scan, W = L D (grid over
// rows, one row per thread, the row's 32 values in registers: every index into
// them is a compile-time constant).  W is formed for every pivot the block
// found, before the scan's result over all rows is known: the pivots that pass
// are a prefix, and the columns after them are written again by later blocks.
// Rows below the outer block also leave it in the window of pending columns.
// 8.5 us on a front of order 13,572, most of it latency: the launch, two trips
// to memory, the 31 dependent steps of the triangular solve.
constexpr int LF_PANEL_T = 64;

// One panel row; FULL: a 32-column block all of whose pivots were found, the
// usual one (nothing is tested against the block's width).  Returns the first
// failing pivot.
template <bool FULL>
__device__ __forceinline__ int lf_panel_row(const LFArgs& A, const PanelView& V, const double (*TT)[IBMAX + 2],
                                            const int* bperm, const double* bdd, const double* bdo,
                                            const double* dinv, unsigned two, int64_t r, int k, int bs, int bnelim,
                                            double bound) {
  const int64_t bm = A.m - A.cs;
  // every load of the row before the first store: the backup may alias the
  // panel as far as the compiler knows, so a load placed after a store
  // would wait for it (one memory round trip per column)
  double x[IBMAX];
  double* l = &V(r, k);
#pragma unroll
  for (int i = 0; i < IBMAX; ++i) x[i] = l[(int64_t)bperm[FULL ? i : min(i, bs - 1)] * A.m];
  double* pb = A.pb + r;  // the backup, in the block's column order
#pragma unroll
  for (int i = 0; i < IBMAX; ++i)
    if (FULL || i < bs) pb[i * bm] = x[i];
  const int fail = panel_row_t<FULL>(x, TT, two, bdd, bdo, dinv, bnelim, bound);
#pragma unroll
  for (int i = 0; i < IBMAX; ++i)
    if (FULL || i < bs) l[i * A.m] = x[i];
  panel_row_w(x, two, bdd, bdo, bnelim);
  double* w = A.w + r;
#pragma unroll
  for (int i = 0; i < IBMAX; ++i)
    if (FULL || i < bnelim) w[i * bm] = x[i];
  if (A.win && r >= A.bcols) {
    w = A.wo + (A.cs + r - A.wrow0) + (A.wcol0 + k) * A.wld;
#pragma unroll
    for (int i = 0; i < IBMAX; ++i)
      if (FULL || i < bnelim) w[i * A.wld] = x[i];
  }
  return fail;
}

__global__ void __launch_bounds__(LF_PANEL_T) k_lf_panel(LFArgs A) {
  chain_enter();
  __shared__ alignas(16) double TT[IBMAX][IBMAX + 2];  // TT[l][j] = L11(j, l)
  __shared__ int bperm[IBMAX];
  __shared__ double bdd[IBMAX], bdo[IBMAX], dinv[IBMAX];
  __shared__ int s_fail;
  // everything the state holds of the block in one round trip
  LFBlk* b = &A.st->b[A.par];
  const int spec_bad = A.st->spec_bad, bnelim = b->bnelim, bs = b->bs, k = b->k;
  const unsigned two = b->two;
  {
    // the factored block: thread t takes column t / 2 (rows of one half); entries past the block's width
    // are whatever an earlier block left and are never used
    const int j = threadIdx.x >> 1, h = threadIdx.x & 1;
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = b->T[h * 16 + u][j];
    const int c = threadIdx.x & 31;
    const int pc = b->bperm[c];
    const double d0 = b->bdd[c], d1 = b->bdo[c], d2 = b->dinv[c];
    if (spec_bad || bnelim == 0) return;  // a block issued past a mispredicted start column; nothing found
#pragma unroll
    for (int u = 0; u < 16; ++u) TT[j][h * 16 + u] = v[u];
    if (threadIdx.x < IBMAX) { bperm[c] = pc; bdd[c] = d0; bdo[c] = d1; dinv[c] = d2; }
    if (threadIdx.x == 0) s_fail = bnelim;
  }
  __syncthreads();
  const int64_t bm = A.m - A.cs;
  PanelView V{A.a + A.cs + A.cs * A.m, A.m};
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t be = k + bs;
  const double bound = 1.0 / A.o.threshold;
  if (r < k) {
    // the block's row permutation applied to the view's earlier column r (step 5 of the block, left to
    // the threads that have no panel row: they touch rows k .. be of columns before k, which no other
    // thread of this launch reads); all loads of the column before its stores
    double buf[IBMAX];
#pragma unroll
    for (int i = 0; i < IBMAX; ++i) buf[i] = i < bs ? V(k + bperm[i], r) : 0.0;
#pragma unroll
    for (int i = 0; i < IBMAX; ++i)
      if (i < bs) V(k + i, r) = buf[i];
  }
  if (r >= be && r < bm) {
    const int fail = (bs == IBMAX && bnelim == IBMAX)
                         ? lf_panel_row<true>(A, V, TT, bperm, bdd, bdo, dinv, two, r, k, bs, bnelim, bound)
                         : lf_panel_row<false>(A, V, TT, bperm, bdd, bdo, dinv, two, r, k, bs, bnelim, bound);
    if (fail < bnelim) atomicMin(&s_fail, fail);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_fail < bnelim) atomicMin(&b->eff, s_fail);
}

// Restore of the failed diagonal part, failed x failed term, D entries of
// block b, of whose pivots the first nelim passed: one CTA.  It writes only the
// block's own rows, the D entries and the counters.
__device__ __forceinline__ void lf_post_cta(const LFArgs& A, const LFBlk* b, int nelim) {
  LFState* st = A.st;
  const int bs = b->bs, k = b->k;
  const int tid = threadIdx.x;
  PanelView V{A.a + A.cs + A.cs * A.m, A.m};
  if (nelim < b->bnelim) {
    for (int t = tid; t < bs * bs; t += blockDim.x) {
      int i = t % bs, j = t / bs;
      if (i < nelim || j < nelim || i < j) continue;
      int c = b->bperm[j], r = b->bperm[i];
      V(k + i, k + j) = r >= c ? b->Tb[r][c] : b->Tb[c][r];
    }
    __syncthreads();
  }
  if (nelim > 0 && nelim < bs) {
    const int nf = bs - nelim;
    for (int t = tid; t < nf * nf; t += blockDim.x) {
      int i = t % nf, j = t / nf;
      if (i < j) continue;
      // sum over the eliminated columns c of (L D)(row i, c) * L(row j, c), each W entry formed as it is
      // added (no local array), in column order
      const double* l = &V(k + nelim + i, k);
      const double* lj = &V(k + nelim + j, k);
      double s = 0.0;
      int c = 0;
      while (c < nelim) {
        if (b->bdt[c] == PT_1X1) {
          s = __dadd_rn(s, __dmul_rn(__dmul_rn(l[c * A.m], b->bdd[c]), lj[c * A.m]));
          c += 1;
        } else {
          const double A_ = b->bdd[c], B_ = b->bdo[c], C_ = b->bdd[c + 1];
          const double l1 = l[c * A.m], l2 = l[(c + 1) * A.m];
          const double w0 = __dadd_rn(__dmul_rn(l1, A_), __dmul_rn(l2, B_));
          const double w1 = __dadd_rn(__dmul_rn(l1, B_), __dmul_rn(l2, C_));
          s = __dadd_rn(s, __dmul_rn(w0, lj[c * A.m]));
          s = __dadd_rn(s, __dmul_rn(w1, lj[(c + 1) * A.m]));
          c += 2;
        }
      }
      V(k + nelim + i, k + nelim + j) = __dsub_rn(V(k + nelim + i, k + nelim + j), s);
    }
  }
  if (tid < 32) {
    // D entries, one pivot column per lane (the adjusted nelim never splits a 2x2)
    DRec VD{A.D.type + A.cs, A.D.diag + A.cs, A.D.off + A.cs};
    const int c = tid;
    const int8_t t = c < nelim ? b->bdt[c] : (int8_t)PT_DELAYED;
    if (t != PT_DELAYED) {
      VD.type[k + c] = t;
      VD.diag[k + c] = b->bdd[c];
      VD.off[k + c] = t == PT_2X2 ? b->bdo[c] : 0.0;
    }
    const int n1 = __popc(__ballot_sync(0xffffffffu, t == PT_1X1));
    const int n2 = __popc(__ballot_sync(0xffffffffu, t == PT_2X2));
    if (tid == 0) { st->n1 += n1; st->n2 += n2; }
  }
}

// delayed columns of block b to the end of the outer block (1 CTA); returns the
// new end of the columns still to be tried
__device__ int lf_delay_cta(const LFArgs& A, const LFBlk* b, int nelim) {
  const int tid = threadIdx.x;
  const int k = b->k, bs = b->bs;
  int end_pos = A.st->end_pos;
  const int64_t bm = A.m - A.cs;
  PanelView V{A.a + A.cs + A.cs * A.m, A.m};
  __syncthreads();
  if (b->bnelim == 0) {
    for (int off = 0; off < bs; ++off) {
      end_pos -= 1;
      if (k + off < end_pos) {
        cta_swap(V, bm, k + off, end_pos);
        if (tid == 0) { int32_t t = A.lp[k + off]; A.lp[k + off] = A.lp[end_pos]; A.lp[end_pos] = t; }
      }
    }
  } else {
    for (int i = bs - nelim - 1; i >= 0; --i) {
      int dp = k + nelim + i;
      end_pos -= 1;
      if (dp < end_pos) {
        cta_swap(V, bm, dp, end_pos);
        if (tid == 0) { int32_t t = A.lp[dp]; A.lp[dp] = A.lp[end_pos]; A.lp[end_pos] = t; }
      }
    }
  }
  __syncthreads();
  if (tid == 0) A.st->end_pos = end_pos;
  return end_pos;
}

// The rank-nelim update of the outer block's trailing columns, and the next
// inner block (see the head of this file).  Grid: CTA 0, then CTAs whose warps
// take the 32 x 32 lower tiles of rows [ts, bm), columns [ts, bcols) in turn.
__global__ void __launch_bounds__(NT, 2) k_lf_update(LFArgs A, int next) {
  chain_enter();
  __shared__ CtaShared sh;
  __shared__ int s_last;
  LFState* st = A.st;
  const LFBlk* b = &st->b[A.par];
  const int tid = threadIdx.x;
  // the state in one round trip
  const int spec_bad = st->spec_bad, bs = b->bs, bnelim = b->bnelim, k = b->k, end_pos = st->end_pos;
  const unsigned two = b->two;
  int nelim = b->eff;
  if (spec_bad) return;  // a block issued past a mispredicted start column
  // the eliminated count: the panel's first failing column, one less where it would split a 2x2
  if (nelim > 0 && (two >> (nelim - 1)) & 1) nelim -= 1;
  const int ts = k + bs;
  const bool fail = nelim < bs;
  if (blockIdx.x == 0) {
    if (bs == 0) {  // nothing was left for this inner block
      if (next) lf_block_cta(A, sh, A.par ^ 1, k, end_pos, 0, 0);
      return;
    }
    if (!fail) {
      if (tid == 0) st->bne = ts;
      if (next) lf_block_cta(A, sh, A.par ^ 1, ts, end_pos, k, nelim);
      return;
    }
    if (bnelim > 0) lf_post_cta(A, b, nelim);
  } else if (nelim > 0 || (fail && bnelim > 0)) {
    const int bm = (int)(A.m - A.cs);
    double* v = A.a + A.cs + A.cs * A.m;
    PanelView V{v, A.m};
    if (nelim > 0) {
      const int bcols = (int)A.bcols;
      const int nrt = (bm - ts + 31) / 32, nct = (bcols - ts + 31) / 32;
      // the next diagonal block's entries are CTA 0's
      const int skip = (next && !fail) ? ts + min(end_pos - ts, A.o.ib) : ts;
      int ct = 0, rt = ((int)blockIdx.x - 1) * (NT / 32) + (tid >> 5);
      const int step = ((int)gridDim.x - 1) * (NT / 32);
      for (;; rt += step) {
        while (ct < nct && rt >= nrt - ct) { rt -= nrt - ct; ++ct; }
        if (ct >= nct) break;
        warp_tile_update(v, A.m, ts + (ct + rt) * 32, ts + ct * 32, bm, bcols, A.w, bm, v + (int64_t)k * A.m, A.m,
                         nelim, skip);
      }
    }
    if (!fail && blockIdx.x == gridDim.x - 1) lf_post_cta(A, b, nelim);  // (off CTA 0's path)
    if (fail) {
      // rows below the block: restore of the failed panel columns, the trailing x failed cross term
      const int nf = bs - nelim;
      for (int j = tid; j < nf * nelim; j += NT) sh.T[j % nf][j / nf] = V(k + nelim + j % nf, k + j / nf);
      __syncthreads();
      for (int64_t i = ts + (int64_t)(blockIdx.x - 1) * NT + tid; i < bm; i += (int64_t)(gridDim.x - 1) * NT) {
        if (nelim < bnelim)
          for (int j = nelim; j < bs; ++j) V(i, k + j) = A.pb[i + (int64_t)j * bm];
        for (int jj = 0; jj < nf && nelim > 0; ++jj) {
          double s = 0.0;
          for (int c = 0; c < nelim; ++c) s = __dadd_rn(s, __dmul_rn(A.w[i + (int64_t)c * bm], sh.T[jj][c]));
          V(i, k + nelim + jj) = __dsub_rn(V(i, k + nelim + jj), s);
        }
      }
    }
  }
  if (!fail || bs == 0) return;
  // columns failed: the last CTA to finish moves them to the end and factors the next block
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&st->done, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();  // the other CTAs' writes
  const int e2 = lf_delay_cta(A, b, nelim);
  if (tid == 0) { st->done = 0; st->bne = k + nelim; }
  if (next) lf_block_cta(A, sh, A.par ^ 1, k + nelim, e2, 0, 0);
}

// row permutation of the outer block applied to the front's earlier columns
// 0..cs (two_level_factor, factor.rs:2165-2181): 16 columns per CTA, fewer where
// blocks are so wide that 48 KB hold fewer (above 384 columns).  Nothing
// on the front's path reads those rows again, so it runs on a stream of its own
// beside the blocks that follow (12 to 17 us of ~290 per outer block of a
// 13,572 front); it acts if its outer block really began, whatever a later,
// mispredicted one has flagged meanwhile.
constexpr int LF_PROP_SMEM_MAX = 224 * 1024;  // one column of a block of 28,672
inline int lf_prop_cols(int64_t bcols) {
  const int64_t c = 48 * 1024 / (8 * bcols);
  return (int)(c < 1 ? 1 : c < 16 ? c : 16);
}
__global__ void __launch_bounds__(256) k_lf_prop(LFArgs A, int cols) {
  if (A.st->valid[A.outer & 1] != A.outer + 1) return;
  extern __shared__ double buf[];  // bcols x cols
  const int64_t c0 = (int64_t)blockIdx.x * cols;
  const int nc = (int)((A.cs - c0) < cols ? (A.cs - c0) : cols);
  if (nc <= 0) return;
  const int bc = (int)A.bcols;
  for (int t = threadIdx.x; t < nc * bc; t += blockDim.x) {
    int i = t % bc, c = t / bc;
    buf[t] = A.a[(A.cs + A.lp[i]) + (c0 + c) * A.m];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nc * bc; t += blockDim.x) {
    int i = t % bc, c = t / bc;
    A.a[(A.cs + i) + (c0 + c) * A.m] = buf[t];
  }
}

// end of an outer block: column order, delays to the end of the remaining
// fully-summed columns (two_level), eliminated total (1 CTA)
// The delayed columns of the outer block [cs, cs + bcols) (its last
// bcols - bne) swap places with the last columns of the remaining range
// [cs, cs + rem), so the next block starts on columns that were not tried
// (two_level_factor's swap, factor.rs:2108-2252).  One CTA.
__device__ __forceinline__ void lf_swap_delayed(const LFArgs& A, int64_t cs, int64_t bcols, int64_t rem, int bne) {
  const int tid = threadIdx.x;
  PanelView F{A.a, A.m};
  const int nf = (int)(bcols - bne);
  for (int i = 0; i < nf; ++i) {
    int64_t fp = cs + bne + i, e = cs + rem - 1 - i;
    if (fp < e) {
      cta_swap(F, A.m, fp, e);
      if (tid == 0) { int32_t t = A.perm[fp]; A.perm[fp] = A.perm[e]; A.perm[e] = t; }
    }
  }
}

// End of an outer block: its column order into the front's pivot order, the
// delay swap (unless `swap` is 0: a far-field update or the row permutation may
// still be running on another stream, and the host issues the swap itself,
// k_lf_swap, once it has seen the delay), the eliminated total, also into the
// host's (pinned) slot for this block when given.
__global__ void __launch_bounds__(NT) k_lf_outer(LFArgs A, int64_t rem, int two_level, int swap, int32_t* host_gne) {
  chain_enter();
  LFState* st = A.st;
  const int tid = threadIdx.x;
  if (st->spec_bad) {  // a block issued past a mispredicted start column
    if (tid == 0 && host_gne) *host_gne = st->gne;
    return;
  }
  const int bne = st->bne;
  const int64_t cs = A.cs, bcols = A.bcols;
  // perm[cs + i] = orig[lp[i]], via the inner W scratch as the copy buffer
  int32_t* orig = (int32_t*)A.w;
  for (int i = tid; i < bcols; i += NT) orig[i] = A.perm[cs + i];
  __syncthreads();
  for (int i = tid; i < bcols; i += NT) A.perm[cs + i] = orig[A.lp[i]];
  __syncthreads();
  if (swap && two_level && bne < bcols) lf_swap_delayed(A, cs, bcols, rem, bne);
  __syncthreads();
  if (tid == 0) {
    const int32_t g = st->gne + bne;
    st->gne = g;
    if (host_gne) *host_gne = g;
  }
}

// What a far-field update on the far stream reads of the state, taken on the
// front's stream before the fork: the chain goes on meanwhile, and the next
// block's k_lf_begin_outer clears bne and may set spec_bad while CTAs of the
// update have not started yet (another front's GEMM can hold their
// multiprocessors).  One far-field update runs at a time.
__global__ void k_lf_far(LFState* st) {
  st->far_bne = st->bne;
  st->far_skip = st->spec_bad;
}

// The delay swap of an outer block issued without it (k_lf_outer with swap =
// 0), with the block's start column, width, remaining range and eliminated
// count as the host read them.  One CTA.
__global__ void __launch_bounds__(NT) k_lf_swap(LFArgs A, int64_t cs, int64_t bcols, int64_t rem, int bne) {
  lf_swap_delayed(A, cs, bcols, rem, bne);
}

// TPP fallback on the leftover columns, then the front's results
__global__ void k_lf_finish(LFArgs A, DFront* F, int s) {
  LFState* st = A.st;
  __shared__ int cnt[2];
  const int lane = threadIdx.x;
  int gne = st->gne;
  if (lane == 0) { cnt[0] = 0; cnt[1] = 0; }
  __syncwarp();
  if (gne < A.p && A.o.failed_pivot_tpp) {
    WarpTpp T{PanelView{A.a, A.m}, A.m, A.p, lane};
    gne += (int)T.run(gne, A.p, A.perm, A.D, &cnt[0], &cnt[1], A.o);
  }
  __syncwarp();
  if (lane == 0) {
    F[s].ne = gne;
    F[s].n1 = st->n1 + cnt[0];
    F[s].n2 = st->n2 + cnt[1];
  }
}

}  // namespace rvg
