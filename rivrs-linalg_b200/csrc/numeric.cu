// B200 numeric phase: level-set multifrontal APTP factorization and the
// supernodal solve, behind the C ABI of include/rivrs_b200.h.
//
// Reference path (rivrs-linalg, sparse/src/symmetric/):
//   AptpNumeric::factor            numeric.rs:844-1023
//   factor_tree_levelset           numeric.rs:1957-2163
//   factor_single_supernode        numeric.rs:1226-1533
//   factor_small_leaf_subtree      numeric.rs:1562-1938
//   aptp_factor_in_place & kernels factor.rs:301-404, 891-3181
//   aptp_solve                     solve.rs:57-326
//   SparseLDLT::solve_in_place     solver.rs:370-428
//
// Layout in HBM (one handle):
//   panel arena   m x k column-major panel per front (the FS columns of the
//                 frontal matrix); after factorization it IS the factor:
//                 L11 in rows [0,ne), L21 in rows [ne,m), columns [0,ne).
//   index arena   per front: row list (m global indices: owned ++ delayed
//                 ++ pattern) followed by the local pivot order (k).
//   D arrays      per front k entries (type, diag, off).
//   contribution  the NFS x NFS Schur block of each non-root front, one
//                 stream-ordered allocation per wave, released once every
//                 parent that reads it has been assembled.
// Each wave (all fronts whose children are done) runs: row lists -> scatter
// of original entries -> extend-add, one pass per child ordinal so every
// destination receives its terms in the reference's order without atomics
// -> dense factorization (warp TPP or CTA APTP) -> contribution GEMM.  One
// small device->host copy per wave returns the eliminated counts that size
// the next wave (delays change front sizes at run time).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include <thread>

#include "block.cuh"
#include "dense.cuh"
#include "front.cuh"
#include "mlp.cuh"
#include "rvg_internal.h"
#include "tpp.cuh"

namespace rvg {

// ---------------------------------------------------------------------------
// error plumbing
// ---------------------------------------------------------------------------
thread_local std::string g_err;
void set_error(const std::string& s) { g_err = s; }

#define CK(call)                                                                                \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess) {                                                                    \
      set_error(std::string("CUDA error: ") + cudaGetErrorString(e_) + " at " #call);           \
      return e_ == cudaErrorMemoryAllocation ? RVG_ERR_OUT_OF_MEMORY : RVG_ERR_DEVICE;          \
    }                                                                                           \
  } while (0)

// ---------------------------------------------------------------------------
// assembly kernels
// ---------------------------------------------------------------------------

// Row list of each front: owned ++ delayed-from-children ++ pattern
// (numeric.rs:1239-1262), and the identity pivot order.
// dly: the children's delay offsets, in order (nullptr: those of their descriptors).
__device__ __forceinline__ void front_rows_cta(int s, const DFront& fr, const Statics& S, const Arenas& A,
                                               const DFront* F, const int32_t* dly, int32_t* rows) {
  int32_t* perm = rows + fr.m;
  int64_t o0 = S.own_ptr[s];
  for (int i = threadIdx.x; i < fr.nown; i += blockDim.x) rows[i] = S.own_idx[o0 + i];
  int64_t p0 = S.pat_ptr[s];
  for (int i = threadIdx.x; i < fr.nfs; i += blockDim.x) rows[fr.k + i] = S.pat_idx[p0 + i];
  for (int i = threadIdx.x; i < fr.k; i += blockDim.x) perm[i] = i;
  for (int64_t q = S.ch_ptr[s]; q < S.ch_ptr[s + 1]; ++q) {
    const DFront& c = F[S.ch_idx[q]];
    const int ne = c.ne, nd = c.k - ne;
    if (nd == 0) continue;
    const int32_t* crow = A.idx + c.idx;
    const int32_t* cperm = crow + c.m;
    const int off = fr.nown + (dly ? dly[q - S.ch_ptr[s]] : c.dly_off);
    for (int i = threadIdx.x; i < nd; i += blockDim.x) rows[off + i] = crow[cperm[ne + i]];
  }
}
__global__ void k_front_rows(const int32_t* ids, int n, DFront* F, Statics S, Arenas A) {
  if ((int)blockIdx.x >= n) return;
  const int s = ids[blockIdx.x];
  const DFront fr = F[s];
  front_rows_cta(s, fr, S, A, F, nullptr, A.idx + fr.idx);
}

struct ScatterItem { int32_t front; int32_t pad; int64_t e0; };

// Original entries (numeric.rs:1306-1344 amap path, 2376-2435 per-entry
// path); each destination receives at most one original entry.
__global__ void k_scatter(const ScatterItem* items, const DFront* F, Statics S, Arenas A, const double* vals,
                          const double* scal) {
  ScatterItem it = items[blockIdx.x];
  const DFront fr = F[it.front];
  int64_t e = it.e0 + threadIdx.x;
  if (e >= S.amap_ptr[it.front + 1]) return;
  const int32_t* q = S.amap + 5 * e;
  int32_t r = q[1], c = q[2];
  if (r >= fr.nown) r += fr.ndin;
  if (c >= fr.nown) c += fr.ndin;
  double v = vals[q[0]];
  if (scal) {
    if (fr.ndin == 0) v = __dmul_rn(__dmul_rn(v, scal[q[3]]), scal[q[4]]);
    else v = __dmul_rn(v, __dmul_rn(scal[q[3]], scal[q[4]]));
  }
  if (c < fr.k) {
    double* a = A.panel + fr.panel;
    a[r + (int64_t)c * fr.m] += v;
  } else if ((fr.flags & FF_HAS_CB) && r >= fr.k) {
    A.cbase[fr.cb + (r - fr.k) + (int64_t)(c - fr.k) * fr.nfs] += v;
  }
}

// Extend-add of one child's contribution into its parent
// (numeric.rs:2445-2559).  The child block is [delayed; NFS] x [delayed;
// NFS]: its delayed columns live in the child's panel (rows ne..k and k..m
// of columns ne..k), its NFS x NFS part in the child's contribution buffer.
// An item is a group of `width` columns [j0, j0 + width) of one child's block and
// a segment of its rows [i0, i0 + EA_ROWS), i >= j only: 32 columns where the
// items fill the GPU (a row's map is looked up once for all of them), 8 where
// they do not (a batch of 8 columns is two memory round trips, and four batches
// one after another are most of a small launch's 8.5 us).  Each CTA stages the group's destination
// columns in shared memory, then walks its rows in tiles of 256, one row per
// thread: the thread maps its row once, then handles the 32 columns in
// batches of 8 with all eight source loads, then all eight destination
// loads, in flight together (the one-entry-at-a-time loop kept too few bytes
// in flight per SM to reach HBM bandwidth).  Source reads are coalesced (a
// column of the child block is contiguous); each destination entry still
// receives exactly one term from this child, so the per-ordinal launches
// keep the reference's order of terms.
constexpr int EA_ROWS = 4096;  // rows per item
struct EaTile { int32_t parent; int32_t child; int32_t j0; int32_t i0; };

constexpr int EA_WIDE = 32, EA_NARROW = 8;
__global__ void __launch_bounds__(256, 3) k_extend_add_tiled(const EaTile* items, const DFront* F, Statics S, Arenas A,
                                                             int width) {
  const EaTile it = items[blockIdx.x];
  const DFront P = F[it.parent];
  const DFront C = F[it.child];
  const int nd = C.k - C.ne;
  const int sz = C.m - C.ne;
  const int32_t* __restrict__ ea = S.ea_map + S.ea_ptr[it.child];
  const double* __restrict__ cp = A.panel + C.panel;
  const double* __restrict__ cb = A.cbase + (C.cb < 0 ? 0 : C.cb);
  double* pp = A.panel + P.panel;
  double* pc = A.cbase + (P.cb < 0 ? 0 : P.cb);
  const bool pcb = (P.flags & FF_HAS_CB) != 0;
  auto map = [&](int i) -> int {
    if (i < nd) return P.nown + C.dly_off + i;
    int l = __ldg(ea + (i - nd));
    return l < P.nown ? l : l + P.ndin;
  };
  __shared__ int s_lj[32];
  const int jn = min(width, sz - it.j0);
  if (threadIdx.x < 32) s_lj[threadIdx.x] = threadIdx.x < jn ? map(it.j0 + threadIdx.x) : 0;
  __syncthreads();
  const int i1 = min(sz, it.i0 + EA_ROWS);
  for (int ib = it.i0; ib < i1; ib += 256) {
    const int i = ib + threadIdx.x;
    if (i >= i1) break;
    const int li = map(i);
    // rows of the child block: delayed rows live in the child's panel rows ne.., NFS rows at k..
    const int64_t prow = i < nd ? (int64_t)(C.ne + i) : (int64_t)(C.k + (i - nd));
#pragma unroll 1
    for (int jb = 0; jb < width; jb += 8) {
      double v[8];
      double* dst[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int jj = jb + q, j = it.j0 + jj;
        v[q] = 0.0;
        if (jj < jn && i >= j) {
          v[q] = j < nd ? cp[prow + (int64_t)(C.ne + j) * C.m] : cb[(i - nd) + (int64_t)(j - nd) * C.nfs];
        }
      }
      double old[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        dst[q] = nullptr;
        if (v[q] != 0.0) {
          const int lj = s_lj[jb + q];
          const int r = li >= lj ? li : lj, c = li >= lj ? lj : li;
          if (c < P.k) dst[q] = pp + r + (int64_t)c * P.m;
          else if (pcb && r >= P.k) dst[q] = pc + (r - P.k) + (int64_t)(c - P.k) * P.nfs;
        }
        old[q] = dst[q] ? *dst[q] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (dst[q]) *dst[q] = old[q] + v[q];
    }
  }
}

// Zeros the lower triangle (rows j..nfs of column j) of the contribution
// blocks of a wave: item = (front, first of 32 columns).  The upper
// triangle is never read.
struct CbZeroItem { int32_t front; int32_t j0; };
__global__ void __launch_bounds__(256) k_zero_cb_lower(const CbZeroItem* items, const DFront* F, Arenas A) {
  const CbZeroItem it = items[blockIdx.x];
  const DFront f = F[it.front];
  double* c = A.cbase + f.cb;
  const int jend = min(f.nfs, it.j0 + 32);
  for (int j = it.j0; j < jend; ++j) {
    double* col = c + (int64_t)j * f.nfs;
    for (int i = j + threadIdx.x; i < f.nfs; i += blockDim.x) col[i] = 0.0;
  }
}

// ---------------------------------------------------------------------------
// dense factorization kernels
// ---------------------------------------------------------------------------

// One warp per front: TPP on all k columns (small-leaf fronts, numeric.rs:
// 1805; fronts with k < ib, factor.rs:360-362).
// TPP on all k columns of front s by one warp; cnt: the warp's two shared counters.
__device__ void warp_tpp_front(int s, DFront* F, const Arenas& A, const DevOpts& o, int* cnt) {
  const int lane = threadIdx.x & 31;
  const DFront fr = F[s];
  if (lane == 0) { cnt[0] = 0; cnt[1] = 0; }
  __syncwarp();
  WarpTpp T{PanelView{A.panel + fr.panel, fr.m}, fr.m, fr.k, lane};
  int32_t* perm = A.idx + fr.idx + fr.m;
  DRec d{A.dtype + fr.dpos, A.ddiag + fr.dpos, A.doff + fr.dpos};
  int64_t ne = T.run(0, fr.k, perm, d, &cnt[0], &cnt[1], o);
  __syncwarp();
  if (lane == 0) { F[s].ne = (int32_t)ne; F[s].n1 = cnt[0]; F[s].n2 = cnt[1]; }
}

__global__ void k_tpp(const int32_t* ids, int n, DFront* F, Arenas A, DevOpts o) {
  int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= n) return;
  __shared__ int cnt[8][2];
  warp_tpp_front(ids[w], F, A, o, cnt[threadIdx.x >> 5]);
}

// Full symmetric swap of positions i, j inside a view of `rows` rows
// (swap_symmetric, factor.rs:458-461), all threads of the CTA.
__device__ void cta_swap(PanelView V, int64_t rows, int64_t i, int64_t j) {
  if (i == j) return;
  if (i > j) { int64_t t = i; i = j; j = t; }
  __syncthreads();
  int tid = threadIdx.x;
  if (tid == 0) { double t = V(i, i); V(i, i) = V(j, j); V(j, j) = t; }
  for (int64_t k = tid; k < i; k += NT) { double t = V(i, k); V(i, k) = V(j, k); V(j, k) = t; }
  for (int64_t k = i + 1 + tid; k < j; k += NT) { double t = V(k, i); V(k, i) = V(j, k); V(j, k) = t; }
  for (int64_t k = j + 1 + tid; k < rows; k += NT) { double t = V(k, i); V(k, i) = V(k, j); V(k, j) = t; }
  __syncthreads();
}

// One warp's 32 x 32 tile of a rank-n update, n <= 32:
//   V(i, j) = fma(-W(i, c), L(j, c), V(i, j)), c = 0 .. n - 1 in order,
// for i0 <= i < bm, j0 <= j < cmax, i >= j, with W(i, c) = W[i + c ldw] and
// L(j, c) = L[j + c ldl]; entries with i < skip and j < skip are left alone.  A
// contraction, so it runs on the FP64 tensor pipe (mma.sync m8n8k4, the fma
// chain per entry in order, as in gemm64.cuh), operands straight from L1 / L2:
// a tile's 8 x 16 DMMAs keep the pipe busy for ~2000 cycles against ~130 of
// loads (8 fragment loads per 16 DMMAs), so staging in shared memory and the
// barriers it would cost buy nothing.
__device__ __forceinline__ void warp_tile_update(double* V, int64_t ld, int i0, int j0, int bm, int cmax,
                                                 const double* W, int64_t ldw, const double* L, int64_t ldl, int n,
                                                 int skip) {
  const int lane = threadIdx.x & 31;
  const int fr = lane >> 2, fk = lane & 3, fc = fk * 2;
  // Offsets from the tile's corner (32 columns stay far below 2^31).  Rows and
  // columns past the region are clamped to its last one and dropped later, so
  // that every load is unconditional: a guarded load is a branch, and the
  // loads of a step then wait for one another.
  double* vt = V + i0 + (int64_t)j0 * ld;
  const double* wt = W + i0;
  const double* lt = L + j0;
  const int lv = (int)ld, lw = (int)ldw, ll = (int)ldl;
  const int ri = bm - 1 - i0, rj = cmax - 1 - j0;  // the last row and column
  int oi[4], oj[4];                                 // the lane's operand rows
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    oi[q] = min(8 * q + fr, ri);
    oj[q] = min(8 * q + fr, rj);
  }
  double acc[4][4][2];
#pragma unroll
  for (int ni = 0; ni < 4; ++ni)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double* col = vt + min(8 * ni + fc + q, rj) * lv;
#pragma unroll
      for (int mi = 0; mi < 4; ++mi) acc[mi][ni][q] = col[oi[mi]];
    }
  double af[2][4], bf[2][4];
  auto load = [&](int kk, double* x, double* y) {
    const int c = min(kk + fk, n - 1);
    const double* w = wt + c * lw;
    const double* l = lt + c * ll;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      x[q] = w[oi[q]];
      y[q] = l[oj[q]];
    }
  };
  auto mma = [&](int kk, const double* x, const double* y) {
    const bool in = kk + fk < n;  // columns past n: zeros, which add exact zeros
    double xn[4], yn[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      xn[q] = in ? -x[q] : 0.0;
      yn[q] = in ? y[q] : 0.0;
    }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                     : "+d"(acc[mi][ni][0]), "+d"(acc[mi][ni][1])
                     : "d"(xn[mi]), "d"(yn[ni]));
  };
  load(0, af[0], bf[0]);
#pragma unroll 1
  for (int kk = 0; kk < n; kk += 8) {
    load(kk + 4, af[1], bf[1]);
    mma(kk, af[0], bf[0]);
    load(kk + 8, af[0], bf[0]);
    if (kk + 4 < n) mma(kk + 4, af[1], bf[1]);
  }
#pragma unroll
  for (int ni = 0; ni < 4; ++ni)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int dj = 8 * ni + fc + q;
      double* col = vt + dj * lv;
#pragma unroll
      for (int mi = 0; mi < 4; ++mi) {
        const int di = 8 * mi + fr;
        if (di <= ri && dj <= rj && i0 + di >= j0 + dj && (i0 + di >= skip || j0 + dj >= skip)) col[di] = acc[mi][ni][q];
      }
    }
}

// The trailing update of one inner block inside a view, by the whole CTA
// (update_trailing, factor.rs:1418-1526): columns [ts, nfsb), rows [ts, bm),
// lower, W(i, c) = W[(i - ts) + c ldw], L = the view's columns k .. k + n - 1.
__device__ void cta_trailing_update(PanelView V, int k, int ts, int bm, int nfsb, int n, const double* W, int ldw) {
  const int nrt = (bm - ts + 31) / 32, nct = (nfsb - ts + 31) / 32;
  int ct = 0, rt = threadIdx.x >> 5;  // the warp's tile: column tile ct, the rt-th row tile from the diagonal down
  for (;; rt += NT / 32) {
    while (ct < nct && rt >= nrt - ct) { rt -= nrt - ct; ++ct; }
    if (ct >= nct) break;
    warp_tile_update(V.a, V.ld, ts + (ct + rt) * 32, ts + ct * 32, bm, nfsb, W - ts, ldw, V.a + (int64_t)k * V.ld, V.ld,
                     n, 0);
  }
}

// factor_inner (factor.rs:1811-2095) on the view V (rows `bm`, `pl` FS
// columns, NFS boundary `nfsb`), executed by the whole CTA.  D entries go to
// VD (view-relative), the view-local column order to lp.  Returns the number
// of eliminated columns.
//
// Per 32 columns: the block (latency bound, block.cuh), the panel rows (one
// row per thread in registers, W = L D formed while the row is there), the
// trailing update (FP64 tensor pipe).  A 368 x 368 front took 500 us per 32
// columns when the panel row lived in local memory (its loops had run-time
// bounds) and the update re-read W and L from global memory for every entry.
__device__ int cta_factor_inner(CtaShared& sh, PanelView V, int bm, int pl, int nfsb, DRec VD, int32_t* lp,
                                double* bk, int64_t ldb, double* W, const DevOpts& o) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ib = o.ib;
  const double bound = 1.0 / o.threshold;
  for (int i = tid; i < pl; i += NT) lp[i] = i;
  if (tid == 0) { sh.k = 0; sh.end_pos = pl; sh.n1 = 0; sh.n2 = 0; }
  __syncthreads();
  while (true) {
    int k = sh.k, end_pos = sh.end_pos;
    if (k >= end_pos) break;
    const int bs = min(end_pos - k, ib), be = k + bs;
    const int rows = bm - k;
    // 1. backup a[k..bm, k..k+bs] (the panel rows are read back from it), 2. load the diagonal block
    for (int i = tid; i < rows; i += NT) {
      const double* src = &V(k + i, k);
#pragma unroll 1
      for (int h = 0; h < bs; h += 16) {
        const double* s2 = src + (int64_t)h * V.ld;
        double* b2 = bk + i + h * ldb;
        const int lv = (int)V.ld, lb = (int)ldb;
        double v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = (h + j < bs && (i >= bs || i >= h + j)) ? s2[j * lv] : 0.0;
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (h + j < bs) {
            b2[j * lb] = v[j];
            if (i < bs) sh.T[i][h + j] = v[j];
          }
      }
    }
    __syncthreads();
    cta_block_factor(sh, bs, o.small);
    const int bnelim = sh.bnelim;
    if (bnelim == 0) {  // (the panel and the block are as they were)
      for (int off = 0; off < bs; ++off) {
        end_pos -= 1;
        if (k + off < end_pos) {
          cta_swap(V, bm, k + off, end_pos);
          if (tid == 0) { int32_t t = lp[k + off]; lp[k + off] = lp[end_pos]; lp[end_pos] = t; }
        }
      }
      __syncthreads();
      if (tid == 0) sh.end_pos = end_pos;
      __syncthreads();
      continue;
    }
    // the factored block back (lower triangle), the D off-diagonals of 2x2 pivots zeroed (step 4) both
    // there and in the L11 copy of the panel's rows
    for (int t = tid; t < IBMAX * IBMAX; t += NT) {
      const int i = t % IBMAX, j = t / IBMAX;
      if (i >= j && i < bs) {
        const double v = (i == j + 1 && j < bnelim && sh.bdt[j] == PT_2X2) ? 0.0 : sh.T[i][j];
        V(k + i, k + j) = v;
        sh.TT[j][i] = v;
      }
    }
    if (tid < IBMAX) {
      sh.dinv[tid] = pivot_inv(tid, bnelim, sh.bdt, sh.bdd, sh.bdo);
      // 6. column order: lane i takes the entry of lane bperm[i]
      const int32_t ob = tid < bs ? lp[k + tid] : 0;
      const int32_t nb = __shfl_sync(0xffffffffu, ob, sh.bperm[tid] & 31);
      if (tid < bs) lp[k + tid] = nb;
      const unsigned two = __ballot_sync(0xffffffffu, tid < bnelim && sh.bdt[tid] == PT_2X2);
      if (tid == 0) { sh.two = two; sh.eff = bnelim; }
    }
    // 5. row permutation of view columns 0..k: a warp per column
    {
      const int src = lane < bs ? sh.bperm[lane] : 0;
      for (int c0 = warp; c0 < k; c0 += 4 * (NT / 32)) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + u * (NT / 32);
          v[u] = (c < k && lane < bs) ? V(k + src, c) : 0.0;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + u * (NT / 32);
          if (c < k && lane < bs) V(k + lane, c) = v[u];
        }
      }
    }
    __syncthreads();
    // 3 + 7. each panel row permuted, TRSM with L11, D^-1 scaling, the threshold scan (apply_and_check,
    // factor.rs:1295-1408), and its W = L D for the update below (the pivots that pass keep theirs)
    const int tsz = bm - be;
    const unsigned two = sh.two;
    for (int r = tid; r < tsz; r += NT) {
      // leading dimensions the compiler may not see through: 32 column offsets each, hoisted out of this
      // loop, would not leave registers for the row
      int lb = (int)ldb, lv = (int)V.ld, lw = tsz;
      asm volatile("" : "+r"(lb), "+r"(lv), "+r"(lw));
      double x[IBMAX];
      const double* src = bk + bs + r;
#pragma unroll
      for (int i = 0; i < IBMAX; ++i) x[i] = i < bs ? src[sh.bperm[i] * lb] : 0.0;
      const int fail = panel_row_t<false>(x, sh.TT, two, sh.bdd, sh.bdo, sh.dinv, bnelim, bound);
      double* l = &V(be + r, k);
#pragma unroll
      for (int i = 0; i < IBMAX; ++i)
        if (i < bs) l[i * lv] = x[i];
      panel_row_w(x, two, sh.bdd, sh.bdo, bnelim);
#pragma unroll
      for (int i = 0; i < IBMAX; ++i)
        if (i < bnelim) W[r + i * lw] = x[i];
      if (fail < bnelim) atomicMin(&sh.eff, fail);
    }
    __syncthreads();
    int eff = sh.eff;
    // 8. adjust_for_2x2_boundary (factor.rs:1161-1174)
    if (eff > 0 && (two >> (eff - 1)) & 1) eff -= 1;
    // 9. partial restore of the failed columns
    if (eff < bnelim) {
      for (int t = tid; t < bs * bs; t += NT) {
        int i = t % bs, j = t / bs;
        if (i < eff || j < eff || i < j) continue;
        int c = sh.bperm[j], r = sh.bperm[i];
        V(k + i, k + j) = (r >= c) ? bk[r + (int64_t)c * ldb] : bk[c + (int64_t)r * ldb];
      }
      for (int j = eff; j < bs; ++j) {
        int c = sh.bperm[j];
        for (int i = bs + tid; i < rows; i += NT) V(k + i, k + j) = bk[i + (int64_t)c * ldb];
      }
      __syncthreads();
    }
    const int nelim = eff;
    // 10. Schur updates (update_trailing factor.rs:1418-1526, update_cross_terms 1669-1766)
    if (nelim > 0) {
      cta_trailing_update(V, k, be, bm, nfsb, nelim, W, tsz);
      if (nelim < bs) {
        const int nf = bs - nelim;
        // failed x failed: W of the failed rows formed entry by entry, in column order
        for (int t = tid; t < nf * nf; t += NT) {
          int i = t % nf, j = t / nf;
          if (i < j) continue;
          const double* l = &V(k + nelim + i, k);
          const double* lj = &V(k + nelim + j, k);
          double s = 0.0;
          int c = 0;
          while (c < nelim) {
            if (sh.bdt[c] == PT_1X1) {
              s = __dadd_rn(s, __dmul_rn(__dmul_rn(l[c * V.ld], sh.bdd[c]), lj[c * V.ld]));
              c += 1;
            } else {
              const double A_ = sh.bdd[c], B_ = sh.bdo[c], C_ = sh.bdd[c + 1];
              const double l1 = l[c * V.ld], l2 = l[(c + 1) * V.ld];
              s = __dadd_rn(s, __dmul_rn(__dadd_rn(__dmul_rn(l1, A_), __dmul_rn(l2, B_)), lj[c * V.ld]));
              s = __dadd_rn(s, __dmul_rn(__dadd_rn(__dmul_rn(l1, B_), __dmul_rn(l2, C_)), lj[(c + 1) * V.ld]));
              c += 2;
            }
          }
          V(k + nelim + i, k + nelim + j) = __dsub_rn(V(k + nelim + i, k + nelim + j), s);
        }
        // trailing x failed
        for (int j = 0; j < nf; ++j) {
          const double* lj = &V(k + nelim + j, k);
          for (int i = tid; i < tsz; i += NT) {
            double s = 0.0;
            for (int c = 0; c < nelim; ++c) s = __dadd_rn(s, __dmul_rn(W[i + (int64_t)c * tsz], lj[c * V.ld]));
            V(be + i, k + nelim + j) = __dsub_rn(V(be + i, k + nelim + j), s);
          }
        }
      }
    }
    // 11. D entries and counts for the passed columns (the adjusted nelim never splits a 2x2)
    if (tid < 32) {
      const int8_t t = lane < nelim ? sh.bdt[lane] : (int8_t)PT_DELAYED;
      if (t != PT_DELAYED) {
        VD.type[k + lane] = t;
        VD.diag[k + lane] = sh.bdd[lane];
        VD.off[k + lane] = t == PT_2X2 ? sh.bdo[lane] : 0.0;
      }
      const int c1 = __popc(__ballot_sync(0xffffffffu, t == PT_1X1));
      const int c2 = __popc(__ballot_sync(0xffffffffu, t == PT_2X2));
      if (lane == 0) { sh.n1 += c1; sh.n2 += c2; }
    }
    __syncthreads();
    // 12. delay the failed columns to end_pos
    if (nelim < bs) {
      int nd = bs - nelim;
      for (int i = nd - 1; i >= 0; --i) {
        int dp = k + nelim + i;
        end_pos -= 1;
        if (dp < end_pos) {
          cta_swap(V, bm, dp, end_pos);
          if (tid == 0) { int32_t t = lp[dp]; lp[dp] = lp[end_pos]; lp[end_pos] = t; }
        }
      }
    }
    __syncthreads();
    if (tid == 0) { sh.k = k + nelim; sh.end_pos = end_pos; }
    __syncthreads();
  }
  return sh.k;
}

// One CTA per front: aptp_factor_in_place (factor.rs:301-404) for fronts with
// k >= ib outside small-leaf subtrees: factor_inner (k <= nb) or
// two_level_factor (k > nb), then the TPP fallback on the leftover columns.
// One front by the whole CTA (aptp_factor_in_place, factor.rs:301-404).
// Every thread reaches every barrier; the CTA's shared state is free again
// when it returns.
__device__ __forceinline__ void cta_aptp_front(CtaShared& sh, int* tpp_cnt, int s, DFront* F, const Arenas& A,
                                               const DevOpts& o) {
  const int tid = threadIdx.x;
  const DFront fr = F[s];
  const int64_t m = fr.m;
  const int p = fr.k;
  PanelView Av{A.panel + fr.panel, m};
  int32_t* perm = A.idx + fr.idx + m;
  DRec D{A.dtype + fr.dpos, A.ddiag + fr.dpos, A.doff + fr.dpos};
  double* bk = A.scratch + fr.scratch;            // m x ib
  double* W = bk + m * IBMAX;                     // m x IBMAX (row-major)
  int32_t* lp = (int32_t*)(W + m * IBMAX);        // nb ints
  int n1 = 0, n2 = 0;
  int gne = 0;
  if (p <= o.nb) {
    gne = cta_factor_inner(sh, Av, (int)m, p, p, D, lp, bk, m, W, o);
    n1 = sh.n1; n2 = sh.n2;
    for (int i = tid; i < p; i += NT) perm[i] = lp[i];
    __syncthreads();
  } else {
    // two_level_factor (factor.rs:2108-2252)
    int rem = p;
    while (rem > 0) {
      int cs = gne, bcols = min(rem, o.nb);
      PanelView V{&Av(cs, cs), m};
      DRec VD{D.type + cs, D.diag + cs, D.off + cs};
      int bne = cta_factor_inner(sh, V, (int)m - cs, bcols, p - cs, VD, lp, bk, m, W, o);
      n1 += sh.n1; n2 += sh.n2;
      // propagate the row permutation to columns 0..cs
      if (cs > 0) {
        // two-pass propagation through the backup buffer: gather, then write
        for (int64_t c0 = 0; c0 < cs; c0 += IBMAX) {
          int nc = (int)(cs - c0 < IBMAX ? cs - c0 : IBMAX);
          for (int t = tid; t < nc * bcols; t += NT) {
            int i = t % bcols, cc = t / bcols;
            bk[i + (int64_t)cc * m] = Av(cs + lp[i], c0 + cc);
          }
          __syncthreads();
          for (int t = tid; t < nc * bcols; t += NT) {
            int i = t % bcols, cc = t / bcols;
            Av(cs + i, c0 + cc) = bk[i + (int64_t)cc * m];
          }
          __syncthreads();
        }
      }
      // column order of the outer block
      if (tid == 0) {
        for (int i = 0; i < bcols; ++i) ((int32_t*)W)[i] = perm[cs + i];
        for (int i = 0; i < bcols; ++i) perm[cs + i] = ((int32_t*)W)[lp[i]];
      }
      __syncthreads();
      // delayed columns to the end of the unprocessed region
      if (bne < bcols) {
        int nf = bcols - bne;
        for (int i = 0; i < nf; ++i) {
          int fp = cs + bne + i, e = cs + rem - 1 - i;
          if (fp < e) {
            cta_swap(Av, m, fp, e);
            if (tid == 0) { int32_t t = perm[fp]; perm[fp] = perm[e]; perm[e] = t; }
          }
        }
      }
      __syncthreads();
      gne += bne;
      rem -= bcols;
    }
  }
  // TPP fallback on columns gne..p (factor.rs:376-401)
  if (gne < p && o.failed_pivot_tpp) {
    if (tid < 32) {
      if (tid == 0) { tpp_cnt[0] = 0; tpp_cnt[1] = 0; }
      __syncwarp();
      WarpTpp T{Av, m, p, tid};
      int64_t add = T.run(gne, p, perm, D, &tpp_cnt[0], &tpp_cnt[1], o);
      if (tid == 0) sh.tmpi = (int)add;
    }
    __syncthreads();
    gne += sh.tmpi;
    n1 += tpp_cnt[0];
    n2 += tpp_cnt[1];
  }
  if (tid == 0) { F[s].ne = gne; F[s].n1 = n1; F[s].n2 = n2; }
  __syncthreads();
}

__global__ void __launch_bounds__(NT) k_aptp(const int32_t* ids, int n, DFront* F, Arenas A, DevOpts o) {
  if ((int)blockIdx.x >= n) return;
  __shared__ CtaShared sh;
  __shared__ int tpp_cnt[2];
  cta_aptp_front(sh, tpp_cnt, ids[blockIdx.x], F, A, o);
}

// The medium fronts of a wave (across every system of a union) as one
// persistent launch: a grid of at most the resident CTAs, each taking the
// next front from a work queue (*next, zero at launch) until the list is
// done.  The host lists the fronts largest first, so the long ones start
// early and the short ones fill in behind them.  Which CTA factors a front
// changes nothing in its result.  Two CTAs per SM: one's block and panel
// latency runs under the other's tensor-pipe update.
__global__ void __launch_bounds__(NT, 2) k_front_queue(const int32_t* ids, int na, int32_t* next, DFront* F, Arenas A,
                                                       DevOpts o) {
  __shared__ CtaShared sh;
  __shared__ int tpp_cnt[2];
  __shared__ int s_i;
  wave_kernel_enter();
  for (;;) {
    if (threadIdx.x == 0) s_i = atomicAdd(next, 1);
    __syncthreads();
    const int i = s_i;
    __syncthreads();  // every thread has read s_i before thread 0 takes the next item
    if (i >= na) break;
    cta_aptp_front(sh, tpp_cnt, ids[i], F, A, o);
  }
  wave_kernel_exit();
}

}  // namespace rvg

#include "gemm64.cuh"
#include "umma.cuh"
#include "large.cuh"
#include "solve_sf.cuh"

namespace rvg {

// ---------------------------------------------------------------------------
// contribution GEMM: CB -= (L21_NFS D) L21_NFS^T, lower triangle
// (compute_contribution_gemm, factor.rs:1590-1652)
// ---------------------------------------------------------------------------
struct TileItem { int32_t front; int32_t ti; int32_t tj; int32_t pad; };

// W = L21_NFS * D into scratch (nfs x ne, column-major) for the fronts whose
// contribution GEMM reads it (launch_syrk): 256 rows x CBW_COLS columns per
// CTA, one row per thread, every load of the chunk before its first store.  (A
// thread that walks all of a front's columns pays one memory round trip per
// column: 339 us for 12,882 x 648.)  A 2x2 pair belongs to the chunk of its
// first column.
constexpr int CBW_COLS = 32;
__global__ void __launch_bounds__(256) k_cb_w(const TileItem* items, const DFront* F, Arenas A) {
  const TileItem it = items[blockIdx.x];
  const DFront fr = F[it.front];
  const int8_t* dt = A.dtype + fr.dpos;
  const double* dd = A.ddiag + fr.dpos;
  const double* dof = A.doff + fr.dpos;
  const int64_t i = (int64_t)it.ti * 256 + threadIdx.x;
  const int c0 = it.tj * CBW_COLS, n = fr.ne - c0;
  if (i >= fr.nfs || n <= 0) return;
  const double* l = A.panel + fr.panel + fr.k + i + (int64_t)c0 * fr.m;
  double* W = A.scratch + fr.scratch + i + (int64_t)c0 * fr.nfs;
  dt += c0;
  dd += c0;
  dof += c0;
  double lv[CBW_COLS + 1];
#pragma unroll
  for (int c = 0; c <= CBW_COLS; ++c) lv[c] = c < n ? l[(int64_t)c * fr.m] : 0.0;
#pragma unroll
  for (int c = 0; c < CBW_COLS; ++c) {
    if (c >= n) break;
    const int8_t t = dt[c];
    if (t == PT_1X1) {
      W[(int64_t)c * fr.nfs] = __dmul_rn(lv[c], dd[c]);
    } else if (t == PT_2X2) {
      W[(int64_t)c * fr.nfs] = __dadd_rn(__dmul_rn(lv[c], dd[c]), __dmul_rn(lv[c + 1], dof[c]));
      W[(int64_t)(c + 1) * fr.nfs] = __dadd_rn(__dmul_rn(lv[c], dof[c]), __dmul_rn(lv[c + 1], dd[c + 1]));
    }
  }
}

constexpr int GT = 64;  // output tile of k_cb_gemm

// Contribution blocks of the small and medium fronts:
// C[i,j] = fma(-W[i,c], L[j,c], C[i,j]) for c ascending (each output entry an
// fma chain in the oracle's order), W = L D formed as it is loaded: a W entry is
// one or two products, so it costs less than a pass that writes W and a second
// one that reads it.  64 x 64 outputs per CTA, 32 x 32 per warp on the FP64
// tensor pipe (as warp_tile_update); the next step's operands load while this
// one's 16 DMMAs run.
__global__ void __launch_bounds__(128) k_cb_gemm(const TileItem* items, const DFront* F, Arenas A) {
  const TileItem it = items[blockIdx.x];
  const DFront fr = F[it.front];
  const int nfs = fr.nfs, ne = fr.ne, m = fr.m;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fr_ = lane >> 2, fk = lane & 3, fc = fk * 2;
  const int i0 = it.ti * GT + (warp & 1) * 32, j0 = it.tj * GT + (warp >> 1) * 32;
  if (ne <= 0 || i0 >= nfs || j0 >= nfs || i0 + 31 < j0) return;
  const double* L = A.panel + fr.panel + fr.k;  // L21_NFS(j, c) = L[j + c m]
  const int8_t* dt = A.dtype + fr.dpos;
  const double* dd = A.ddiag + fr.dpos;
  const double* dof = A.doff + fr.dpos;
  double* C = A.cbase + fr.cb + i0 + (int64_t)j0 * nfs;
  const double* la = L + i0;
  const double* lb = L + j0;
  const int ri = nfs - 1 - i0, rj = nfs - 1 - j0;  // loads clamped to the last row and column (warp_tile_update)
  int oi[4], oj[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    oi[q] = min(8 * q + fr_, ri);
    oj[q] = min(8 * q + fr_, rj);
  }
  double acc[4][4][2];
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const double* col = C + min(8 * y + fc + q, rj) * nfs;
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[x][y][q] = col[oi[x]];
    }
  // a step's operands: the lane's column of L for its W entries (the pair's first column and its second;
  // equal ones for a 1x1), their coefficients, the column of L for the other side
  struct Op { double v0[4], v1[4], b[4], e0, e1; int kind; };
  auto load = [&](int kk, Op& o) {
    const int c = min(kk + fk, ne - 1);
    const int8_t t = dt[c];
    const int cf = t == PT_2X2B ? c - 1 : c, cs = t == PT_2X2 ? c + 1 : c;
    o.kind = kk + fk >= ne ? 0 : (t == PT_1X1 ? 1 : 2);
    const double d = dd[c], off = dof[cf];
    o.e0 = t == PT_2X2B ? off : d;
    o.e1 = t == PT_2X2B ? d : off;
    const double* l0 = la + (int64_t)cf * m;
    const double* l1 = la + (int64_t)cs * m;
    const double* l2 = lb + (int64_t)c * m;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      o.v0[q] = l0[oi[q]];
      o.v1[q] = l1[oi[q]];
      o.b[q] = l2[oj[q]];
    }
  };
  auto mma = [&](const Op& o) {
    double a[4], b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double w0 = __dmul_rn(o.v0[q], o.e0);
      const double w = o.kind == 2 ? __dadd_rn(w0, __dmul_rn(o.v1[q], o.e1)) : w0;
      a[q] = o.kind ? -w : 0.0;
      b[q] = o.kind ? o.b[q] : 0.0;
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y)
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                     : "+d"(acc[x][y][0]), "+d"(acc[x][y][1])
                     : "d"(a[x]), "d"(b[y]));
  };
  Op p0, p1;
  load(0, p0);
#pragma unroll 1
  for (int kk = 0; kk < ne; kk += 8) {  // columns past ne are zeros: they add exact zeros
    load(kk + 4, p1);
    mma(p0);
    load(kk + 8, p0);
    if (kk + 4 < ne) mma(p1);
  }
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int dj = 8 * y + fc + q;
      double* col = C + (int64_t)dj * nfs;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int di = 8 * x + fr_;
        if (di <= ri && dj <= rj && i0 + di >= j0 + dj) col[di] = acc[x][y][q];
      }
    }
}

// ---------------------------------------------------------------------------
// solve kernels (aptp_solve, solve.rs:57-326; SparseLDLT::solve_in_place,
// solver.rs:396-425)
// ---------------------------------------------------------------------------
__global__ void k_perm_scale_in(const double* rhs, int64_t ldb, int64_t nrhs, double* x, int64_t n,
                                const int64_t* pfwd, const double* scal) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * nrhs) return;
  int64_t i = t % n, r = t / n;
  double v = rhs[pfwd[i] + r * ldb];
  if (scal) v = __dmul_rn(v, scal[i]);
  x[i + r * n] = v;
}
__global__ void k_perm_scale_out(double* rhs, int64_t ldb, int64_t nrhs, const double* x, int64_t n,
                                 const int64_t* pfwd, const double* scal) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * nrhs) return;
  int64_t i = t % n, r = t / n;
  double v = x[i + r * n];
  if (scal) v = __dmul_rn(v, scal[i]);
  rhs[pfwd[i] + r * ldb] = v;
}

// ---------------------------------------------------------------------------
// FP64 iterative refinement (residual of the unfactored matrix)
// ---------------------------------------------------------------------------
// r = b - A x; A full symmetric CSC, so column i is also row i
// right-hand side j = blockIdx.y of columns at stride ldx (x, b) and ldr (r)
__global__ void k_residual(const int64_t* colptr, const int32_t* rowidx, const double* val, const double* x,
                           const double* b, double* r, int64_t n, int64_t ldx, int64_t ldr) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x += blockIdx.y * ldx;
  b += blockIdx.y * ldx;
  r += blockIdx.y * ldr;
  double s = 0.0;
  for (int64_t p = colptr[i]; p < colptr[i + 1]; ++p) s = __fma_rn(val[p], x[rowidx[p]], s);
  r[i] = b[i] - s;
}
// out[3j] += ||r_j||^2, out[3j + 1] += ||x_j||^2, out[3j + 2] += ||b_j||^2 for j = blockIdx.y
__global__ void k_norms3(const double* r, const double* x, const double* b, int64_t n, double* out, int64_t ldx,
                         int64_t ldr) {
  x += blockIdx.y * ldx;
  b += blockIdx.y * ldx;
  r += blockIdx.y * ldr;
  out += 3 * blockIdx.y;
  double s0 = 0, s1 = 0, s2 = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    s0 += r[i] * r[i]; s1 += x[i] * x[i]; s2 += b[i] * b[i];
  }
  for (int o = 16; o > 0; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if ((threadIdx.x & 31) == 0) { atomicAdd(out, s0); atomicAdd(out + 1, s1); atomicAdd(out + 2, s2); }
}
// One read of the n values before a factorization: *flag is raised when any of
// them is NaN or infinite, and their sum of squares (||A||_F^2 for the
// refinement) is added to *sum when given.
struct ScanOut { double sum; int32_t bad, pad; };
__global__ void k_scan_values(const double* v, int64_t n, ScanOut* out, int want_sum) {
  double s = 0;
  bool bad = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double x = v[i];
    bad |= !isfinite(x);
    s += x * x;
  }
  if (bad) atomicExch(&out->bad, 1);
  if (!want_sum) return;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(&out->sum, s);
}

__global__ void k_sumsq(const double* v, int64_t n, double* out) {
  double s = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) s += v[i] * v[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}
// GMRES building blocks (one right-hand side): y = A x over the full symmetric CSC
__global__ void k_spmv(const int64_t* colptr, const int32_t* rowidx, const double* val, const double* x, double* y,
                       int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int64_t p = colptr[i]; p < colptr[i + 1]; ++p) s = __fma_rn(val[p], x[rowidx[p]], s);
  y[i] = s;
}
// out[i] += V_i . w for the basis vectors i = blockIdx.y (columns of V at stride n)
__global__ void k_dots(const double* V, const double* w, int64_t n, double* out) {
  const double* v = V + blockIdx.y * n;
  double s = 0.0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    s = __fma_rn(v[k], w[k], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out + blockIdx.y, s);
}
// w -= sum_{i < cnt} c_i V_i   (c on the device)
__global__ void k_sub_comb(double* w, const double* V, const double* c, int cnt, int64_t n) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double s = w[k];
  for (int i = 0; i < cnt; ++i) s = __fma_rn(-c[i], V[(int64_t)i * n + k], s);
  w[k] = s;
}
// x += sum_{i < cnt} c_i Z_i
__global__ void k_add_comb(double* x, const double* Z, const double* c, int cnt, int64_t n) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double s = x[k];
  for (int i = 0; i < cnt; ++i) s = __fma_rn(c[i], Z[(int64_t)i * n + k], s);
  x[k] = s;
}
__global__ void k_scale_to(double* v, const double* w, double a, int64_t n) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) v[k] = w[k] * a;
}

__global__ void k_axpy1(double* x, const double* d, int64_t n, int64_t ldx, int64_t ldd) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[blockIdx.y * ldx + i] += d[blockIdx.y * ldd + i];
}

}  // namespace rvg

// ===========================================================================
// host driver
// ===========================================================================
namespace rvg {

// Start of a wave, one CTA per front: its descriptor, its children's delay
// offsets (dly_vals: the wave's children in order, front i's from dly0[i] on),
// its row list (k_front_rows) and, for blocks of order <= WB_ZERO, the zeroed
// lower triangle of its contribution block (larger ones: k_zero_cb_lower).  Four
// kernels of a few microseconds each otherwise, and as many launches, in every
// wave.
constexpr int WB_ZERO = 256;
__global__ void __launch_bounds__(128) k_wave_begin(const DFront* staged, const int32_t* ids, const int32_t* dly0,
                                                    const int32_t* dly_vals, DFront* F, Statics S, Arenas A) {
  const int i = blockIdx.x, s = ids[i];
  const DFront fr = staged[i];
  if (threadIdx.x == 0) F[s] = fr;
  int32_t* rows = A.idx + fr.idx;
  front_rows_cta(s, fr, S, A, F, dly_vals + dly0[i], rows);
  const int64_t q0 = S.ch_ptr[s], nq = S.ch_ptr[s + 1] - q0;
  __syncthreads();  // (the children's descriptors have been read)
  for (int64_t q = threadIdx.x; q < nq; q += blockDim.x) F[S.ch_idx[q0 + q]].dly_off = dly_vals[dly0[i] + q];
  if ((fr.flags & FF_HAS_CB) && fr.nfs <= WB_ZERO) {
    double* c = A.cbase + fr.cb;
    for (int j = threadIdx.x >> 5; j < fr.nfs; j += (int)(blockDim.x >> 5))
      for (int r = j + (threadIdx.x & 31); r < fr.nfs; r += 32) c[r + (int64_t)j * fr.nfs] = 0.0;
  }
}
// eliminated counts of a wave's fronts, and behind them the device error word
__global__ void k_get_counts(const int32_t* ids, int n, const DFront* F, int32_t* out, const int32_t* err) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (err && i == 0) out[3 * n] = *err;
  if (i < n) { const DFront& f = F[ids[i]]; out[3 * i] = f.ne; out[3 * i + 1] = f.n1; out[3 * i + 2] = f.n2; }
}
// The factorization's D by sign (MixedDiagonal::compute_inertia,
// diagonal.rs:391-461), out[0..2] = positive, negative, zero eigenvalues, and
// out[3] = its zero pivots (numeric.rs:987-1009).  One warp per front at a
// time; counting here leaves four numbers to copy instead of the D arrays.
__global__ void __launch_bounds__(256) k_d_counts(const DFront* F, int64_t ns, Arenas A, unsigned long long* out) {
  const int lane = threadIdx.x & 31;
  int64_t c[4] = {0, 0, 0, 0};
  for (int64_t s = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); s < ns; s += (int64_t)gridDim.x * 8) {
    const DFront f = F[s];
    for (int i = lane; i < f.ne; i += 32) {
      const int64_t q = f.dpos + i;
      const int8_t t = A.dtype[q];
      const double a = A.ddiag[q];
      if (t == PT_1X1) {
        c[a > 0 ? 0 : (a < 0 ? 1 : 2)]++;
        if (a == 0.0) c[3]++;
      } else if (t == PT_2X2) {
        const double b = A.doff[q], cc = A.ddiag[q + 1];
        const double det = a * cc - b * b, tr = a + cc;
        if (det > 0) c[tr > 0 ? 0 : 1] += 2;
        else if (det < 0) { c[0]++; c[1]++; }
        else if (tr > 0) { c[0]++; c[2]++; }
        else if (tr < 0) { c[1]++; c[2]++; }
        else c[2] += 2;
      }
    }
    if (lane == 0 && f.parent < 0 && f.ne < f.m) c[3] += f.k - f.ne;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int64_t v = c[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0 && v) atomicAdd(out + q, (unsigned long long)v);
  }
}

// Refactorization replay checks: the counts (and a large front's progress)
// the captured schedule assumed.  On a difference the flag is raised and the
// recorded value put in place of the computed one, so that every later launch
// of the graph indexes the fronts exactly as the recorded factorization did
// (the parents' sizes and delayed-row offsets were laid out from the record);
// the factor is then discarded and recomputed dynamically.
__global__ void k_check_counts(const int32_t* ids, int n, DFront* F, const int32_t* rec, int32_t* mismatch) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = ids[i];
  DFront& f = F[s];
  const int32_t* r = rec + 3 * (int64_t)s;
  if (f.ne != r[0] || f.n1 != r[1] || f.n2 != r[2]) {
    atomicExch(mismatch, 1);
    f.ne = r[0]; f.n1 = r[1]; f.n2 = r[2];
  }
}
__global__ void k_check_gne(LFState* st, int32_t expect, int32_t* mismatch) {
  if (threadIdx.x == 0 && st->gne != expect) {
    atomicExch(mismatch, 1);
    st->gne = expect;
  }
}

// ---------------------------------------------------------------------------
// learned precision (precision = 2): per large front, features of the
// assembled front, the selector's decision, and the observed pivot growth.
// Row of a front in the feature table (FEAT_STRIDE 32-bit words):
//   0 max |a| over the fully-summed columns (lower part), 1 max |a_jj|,
//   2 min |a_jj|, 3 min over columns of |a_jj| / max_{i>j} |a_ij|, 4 columns
//   with that ratio < u, 5 negative diagonals, 6 zero diagonals (as counts),
//   7 max |D| after the factorization; 8..19 the 12 features; 20 the
//   selector's probability that the mixed form is safe; 21 the route (1 =
//   mixed).  Maxima, minima and counts combine by atomics whose result does
//   not depend on their order, so features and routes are reproducible.
// ---------------------------------------------------------------------------
constexpr int FEAT_STRIDE = 32;
constexpr unsigned F_POS_INF = 0x7f800000u;

__global__ void k_feat_init(const int32_t* ids, int n, unsigned* feat) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    unsigned* r = feat + (size_t)ids[i] * FEAT_STRIDE;
    r[0] = 0u; r[1] = 0u; r[2] = F_POS_INF; r[3] = F_POS_INF; r[4] = 0u; r[5] = 0u; r[6] = 0u; r[7] = 0u;
  }
}

__device__ __forceinline__ unsigned fbits(double v) { return __float_as_uint((float)v); }

// grid (column chunks of 8, fronts): warp w of chunk x reads column 8x + w
// of the front's fully-summed block from its diagonal down.
__global__ void __launch_bounds__(256) k_front_features(const int32_t* ids, const DFront* F, Arenas A, double u,
                                                        unsigned* feat) {
  const int s = ids[blockIdx.y];
  const DFront f = F[s];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t j = (int64_t)blockIdx.x * 8 + warp;
  __shared__ unsigned sv[8][7];
  unsigned v[7] = {0u, 0u, F_POS_INF, F_POS_INF, 0u, 0u, 0u};
  if (j < f.k) {
    const double* col = A.panel + f.panel + j * (int64_t)f.m;
    double cm = 0.0;
    for (int64_t i = j + 1 + lane; i < f.m; i += 32) cm = fmax(cm, fabs(col[i]));
    for (int o = 16; o > 0; o >>= 1) cm = fmax(cm, __shfl_xor_sync(0xffffffffu, cm, o));
    const double d = col[j], ad = fabs(d);
    v[0] = fbits(fmax(cm, ad));
    v[1] = fbits(ad);
    v[2] = fbits(ad);
    const double ratio = cm > 0.0 ? ad / cm : INFINITY;
    v[3] = fbits(ratio);
    v[4] = ratio < u ? 1u : 0u;
    v[5] = d < 0.0 ? 1u : 0u;
    v[6] = d == 0.0 ? 1u : 0u;
  }
  if (lane == 0)
    for (int q = 0; q < 7; ++q) sv[warp][q] = v[q];
  __syncthreads();
  if (threadIdx.x == 0) {
    if ((int64_t)blockIdx.x * 8 >= f.k) return;
    unsigned r[7] = {0u, 0u, F_POS_INF, F_POS_INF, 0u, 0u, 0u};
    for (int w = 0; w < 8; ++w) {
      r[0] = max(r[0], sv[w][0]); r[1] = max(r[1], sv[w][1]);
      r[2] = min(r[2], sv[w][2]); r[3] = min(r[3], sv[w][3]);
      r[4] += sv[w][4]; r[5] += sv[w][5]; r[6] += sv[w][6];
    }
    unsigned* row = feat + (size_t)s * FEAT_STRIDE;
    atomicMax(row + 0, r[0]); atomicMax(row + 1, r[1]);
    atomicMin(row + 2, r[2]); atomicMin(row + 3, r[3]);
    if (r[4]) atomicAdd(row + 4, r[4]);
    if (r[5]) atomicAdd(row + 5, r[5]);
    if (r[6]) atomicAdd(row + 6, r[6]);
  }
}

// One warp per front: the 12 features, the network, the route.
__global__ void k_mlp_route(const int32_t* ids, int n, const DFront* F, const float* P, float thresh, int force_fp64,
                            unsigned* feat, int32_t* route_out) {
  __shared__ MlpAct act;
  __shared__ float fx[MLP_IN];
  const int i = blockIdx.x, lane = threadIdx.x;
  if (i >= n) return;
  const int s = ids[i];
  const DFront f = F[s];
  unsigned* row = feat + (size_t)s * FEAT_STRIDE;
  if (lane == 0) {
    const float lo = 1e-30f;
    const float mx = fmaxf(__uint_as_float(row[0]), lo);
    const float k = (float)max(f.k, 1), m = (float)max(f.m, 1);
    fx[0] = log2f(m);
    fx[1] = log2f(k);
    fx[2] = k / m;
    fx[3] = log2f(1.f + (float)f.ndin);
    fx[4] = (float)f.ndin / k;
    fx[5] = log10f(mx);
    fx[6] = log10f(fmaxf(__uint_as_float(row[1]) / mx, lo));
    fx[7] = log10f(fmaxf(__uint_as_float(row[2]) / mx, lo));
    fx[8] = log10f(fminf(fmaxf(__uint_as_float(row[3]), lo), 1e10f));
    fx[9] = (float)row[4] / k;
    fx[10] = (float)row[5] / k;
    fx[11] = (float)row[6] / k;
  }
  __syncwarp();
  const float xin = lane < MLP_IN ? fx[lane] : 0.f;
  const float z = mlp_forward_warp(P, xin, act);
  if (lane < MLP_IN) row[8 + lane] = __float_as_uint(fx[lane]);
  if (lane == 0) {
    const float pr = mlp_sigmoid(z);
    const int r = (!force_fp64 && pr >= thresh) ? 1 : 0;
    row[20] = __float_as_uint(pr);
    row[21] = __float_as_uint((float)r);
    route_out[i] = r;
  }
}

// After the wave's factorization: max |D| of each large front; a front that
// took the mixed form and whose max |D| exceeds bound * max |a| raises flag.
__global__ void k_front_growth(const int32_t* ids, const DFront* F, Arenas A, double bound, unsigned* feat,
                               int32_t* flag, int32_t* route) {
  const int s = ids[blockIdx.x];
  const DFront f = F[s];
  __shared__ double sm[8];
  double mx = 0.0;
  for (int c = threadIdx.x; c < f.ne; c += blockDim.x) {
    const int64_t q = f.dpos + c;
    mx = fmax(mx, A.dtype[q] == PT_2X2 ? fmax(fabs(A.ddiag[q]), fabs(A.doff[q])) : fabs(A.ddiag[q]));
  }
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) mx = fmax(mx, sm[w]);
    unsigned* row = feat + (size_t)s * FEAT_STRIDE;
    row[7] = fbits(mx);
    const double amax = (double)__uint_as_float(row[0]);
    if (__uint_as_float(row[21]) == 1.f && mx > bound * amax) {
      atomicAdd(flag, 1);
      route[blockIdx.x] = 2;  // refactored in FP64 once the wave is done
    }
  }
}

}  // namespace rvg

using namespace rvg;

// One large front in flight: the stream its launches go to, its pivot state
// on the device and the packed window of its mixed-form updates.  Context 0 is
// on the handle's own stream, or on one of its own while the wave's other fronts
// are queued there; the others let the large fronts of one wave run side by side
// (one host thread each).
constexpr int LF_AHEAD = 8;  // outer blocks of a large front issued ahead of the host's check of their start
struct LfCtx {
  cudaStream_t st = nullptr;
  LFState* lf = nullptr;
  float* wpack = nullptr; size_t wpack_cap = 0;
  bool own = false;        // stream and state created for this context
  bool marks = false;      // profiling marks (only one front in flight, on the handle's stream)
  int64_t launches = 0;
  double sync_ms = 0, syrk_flops = 0;
  // issue-ahead of outer blocks: the device's eliminated total after each
  // issued block lands in a pinned slot, with an event behind it
  int32_t* h_gne = nullptr;
  cudaEvent_t ring_ev[LF_AHEAD] = {};
  double wait_ms = 0;     // host waits on blocks issued ahead (the stream still holds later blocks)
  int64_t misses = 0;     // blocks issued for a start column the factorization did not reach
  // far-field part of a full window's update, beside the next outer blocks (mixed form)
  cudaStream_t far_st = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_far = nullptr;
  // row permutations of the outer blocks, beside the blocks that follow (one event per parity)
  cudaStream_t prop_st = nullptr;
  cudaEvent_t ev_prop_fork = nullptr, ev_prop[2] = {};
  int64_t far_launches = 0;
  int id = 0;  // position in the handle's contexts (its window buffer's address-stable arena)
};
// A full window's far field (the columns after the next window's blocks but
// its last) is updated on a second stream while those blocks are factored;
// the GEMM leaves LF_FAR_SMS multiprocessors to their latency-bound kernels.
constexpr int LF_FAR_SMS = 24;  // the default of rvg_options::far_field_sms
constexpr int LF_CONCURRENT = 8;  // large fronts of a wave in flight at once

struct VmArenas;

struct rvg_handle {
  Plan P;
  rvg_options opt;
  VmArenas* vm = nullptr;  // address-stable arenas (graph_refactor = 2), else nullptr
  int device = 0;
  cudaStream_t st = nullptr;
  cudaEvent_t ev[8] = {};
  cudaEvent_t ev_large = nullptr, ev_beside = nullptr;  // forks and joins of the large fronts' streams
  int64_t nnz = 0;
  // static device data
  int64_t *d_own_ptr = nullptr, *d_pat_ptr = nullptr, *d_amap_ptr = nullptr, *d_ea_ptr = nullptr, *d_ch_ptr = nullptr;
  int32_t *d_own_idx = nullptr, *d_pat_idx = nullptr, *d_amap = nullptr, *d_ea_map = nullptr, *d_ch_idx = nullptr;
  int64_t* d_pfwd = nullptr;
  // per-factor device data
  DFront* d_fronts = nullptr;
  std::vector<DFront> h_fronts;
  double* panel = nullptr; size_t panel_cap = 0;
  int32_t* idx = nullptr; size_t idx_cap = 0;
  int8_t* dtype = nullptr; double* ddiag = nullptr; double* doff = nullptr; size_t d_cap = 0;
  double* d_vals = nullptr; double* d_scal = nullptr; bool has_scaling = false;
  double* d_x = nullptr; size_t x_cap = 0;
  double* solve_work = nullptr; size_t solve_work_cap = 0;
  char* d_stage = nullptr; size_t stage_cap = 0;   // per-wave packed launch data
  char* h_stage = nullptr; size_t h_stage_cap = 0; // pinned host mirror
  int32_t* h_counts = nullptr; size_t h_counts_cap = 0;
  LFState* d_lf = nullptr;                          // state of the large-front path
  std::vector<LfCtx> lfx;                            // concurrent large-front contexts 1.. (0 = the handle's)
  cudaStream_t lf_st = nullptr;                      // context 0's stream beside the small and medium fronts
  int64_t* d_colptr = nullptr;                      // matrix pattern (full symmetric CSC = its own CSR)
  int32_t* d_rowidx = nullptr;
  double a_fro = 0;                                 // ||A||_F of the last factored values
  double* d_ref = nullptr; size_t ref_cap = 0;      // refinement vectors r, d, b (3n) and norms
  double* d_gm = nullptr; size_t gm_cap = 0;        // GMRES-IR: Krylov basis, preconditioned basis, work
  double* h_norms = nullptr;
  char* h_norms_m = nullptr; size_t h_norms_m_cap = 0;  // pinned per-column norms of the refinement
  double* scratch = nullptr; size_t scratch_cap = 0; // per-wave scratch, persistent across factors
  double* cb_arena = nullptr; size_t cb_cap = 0;     // contribution blocks, first-fit by wave
  float* pack = nullptr; size_t pack_cap = 0;        // TF32 hi/lo operand tiles of the mixed-form updates
  float* wpack = nullptr; size_t wpack_cap = 0;      // the same for a large front's window of pending columns
  int32_t* d_err = nullptr;                          // set by a device wait that timed out
  int32_t* sf_sync = nullptr; size_t sf_sync_cap = 0; // solve: ticket counters and block flags of all waves
  // solve: block layout of the factored fronts, made by the first solve after a factorization
  struct SfLayout {
    bool ok = false;
    struct Wave { size_t fwd, bwd, mfwd, mbwd; int32_t nbf, nbb; int64_t tf, tb; };  // offsets in the buffer and sf_sync
    std::vector<Wave> w;
    int64_t nsync = 0, slots = 1, rows = 0;  // sf_sync words, partial-sum slots, rows of all fronts
  } sf;
  char* sf_lay = nullptr; size_t sf_lay_cap = 0;
  double* sf_part = nullptr; size_t sf_part_cap = 0;   // backward solve: partial sums of one wave
  int nsm = 0;                                       // SMs of the device (persistent grids)
  bool chain_pdl = true;                             // large-front chain kernels by programmatic dependent launch
  std::map<int64_t, int64_t> cb_free;                // offset -> length of the free ranges
  bool factored = false;
  bool need_presize = false;                         // arenas released by rvg_trim
  // refactorization replay (graph_refactor): the host's decisions in the last dynamic factorization
  bool rec_ok = false;                               // a complete record is available
  std::vector<int32_t> rec_cnt;                      // per front: eliminated, 1x1 and 2x2 counts
  std::vector<std::vector<int32_t>> rec_g;           // per large front: eliminated count after each outer block
  std::vector<size_t> rec_stage;                     // per wave: bytes of the packed launch data
  int64_t rec_d_used = 0;                            // D entries used
  bool replay = false;                               // run_factor is being captured into the graph
  int32_t* d_rec = nullptr; size_t d_rec_cap = 0;    // rec_cnt on the device (for the checks)
  int32_t* d_mismatch = nullptr;                     // set by a check that sees another decision
  char* h_stage_all = nullptr; size_t h_stage_all_cap = 0;  // pinned launch data of every wave (replay)
  std::vector<size_t> stage_off;                     // per wave: its offset in h_stage_all
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t gexec = nullptr;
  const double* graph_ds = nullptr;                  // the scaling pointer the graph reads
  // learned precision (precision = 2)
  float* d_sel = nullptr;                            // selector parameters (MLP_NPARAM floats)
  float sel_thresh = 0.5f;                           // probability at or above which a front takes the mixed form
  double sel_bound = 1e6;                            // growth bound: max |D| <= bound * max |a| for a mixed front
  unsigned* d_feat = nullptr; size_t d_feat_cap = 0; // feature table, FEAT_STRIDE words per front
  int32_t* d_sel_flag = nullptr;                     // mixed fronts over the growth bound in the last run
  std::vector<int8_t> route;                         // per front: 1 = mixed form (decided on the device)
  std::vector<int32_t> sel_large;                    // the large fronts of the last factorization
  bool sel_force_fp64 = false;                       // the FP64 refactorization after a growth flag
  int aptp_ctas = 0;                                 // resident CTAs of the medium fronts' queue kernel
  ScanOut* d_scan = nullptr;                         // the scan of the values and the scaling before a factorization
  unsigned long long* d_dcount = nullptr;            // k_d_counts: D entries by sign, zero pivots
  int64_t inertia[3] = {0, 0, 0};                    // of the last factorization
  int64_t sel_routed = 0, sel_flagged = 0, sel_fallback = 0;
  // measurement
  bool profiling = false;
  std::vector<cudaEvent_t> ev_pool;
  size_t ev_used = 0;
  double syrk_flops = 0, syrk_ms = 0;
  std::vector<cudaEvent_t> mk_pool;                  // per-kind marks (profiling): event, kind
  std::vector<int> mk_kind;
  size_t mk_used = 0;
  double part_ms[RVG_PARTS] = {};
  int64_t syrk_launches = 0, launches = 0, factor_launches = 0, solve_launches = 0;
  int64_t arena_bytes = 0, peak_bytes = 0;
  double host_alloc_ms = 0, host_sync_ms = 0, host_total_ms = 0;
  double host_wait_ms = 0;  // waits on large-front blocks issued ahead (later blocks still queued)
  double host_gap_ms = 0;   // host time between a wave's synchronisation and the next wave's first launch
  bool sf_attr = false;     // the backward solve kernels' shared-memory limit raised
  char* d_stage2 = nullptr; size_t stage2_cap = 0;  // launch data of FP64 refactorizations of single fronts
  char* h_stage2 = nullptr; size_t h_stage2_cap = 0;
  int64_t sel_refactored = 0;                       // fronts refactored in FP64 after their growth check
  int64_t lf_misses = 0;    // large-front blocks issued past a delay (returned at once, issued again)
  int64_t lf_far = 0;       // far-field window updates run on a large front's second stream
  // results
  int64_t tot1 = 0, tot2 = 0, totdel = 0, zero_piv = 0, max_front = 0;
  double t_assembly = 0, t_kernel = 0, t_gemm = 0, t_factor = 0, t_solve = 0, t_dom = 0, n_dom = 0;
};

namespace {

double now_ms() {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// Profiling marks: the time between a mark and the one before it is charged
// to the later mark's kind (a kind < 0 starts a new segment).  Read back
// after each stream synchronisation.
void mark(rvg_handle* h, int kind) {
  if (!h->profiling || h->replay) return;
  if (h->mk_used == h->mk_pool.size()) {
    cudaEvent_t e;
    if (cudaEventCreate(&e) != cudaSuccess) return;
    h->mk_pool.push_back(e);
    h->mk_kind.push_back(-1);
  }
  cudaEventRecord(h->mk_pool[h->mk_used], h->st);
  h->mk_kind[h->mk_used++] = kind;
}
void mark_flush(rvg_handle* h) {
  for (size_t i = 1; i < h->mk_used; ++i) {
    float ms = 0;
    if (h->mk_kind[i] >= 0 && cudaEventElapsedTime(&ms, h->mk_pool[i - 1], h->mk_pool[i]) == cudaSuccess)
      h->part_ms[h->mk_kind[i]] += ms;
  }
  h->mk_used = 0;
}

// Set while a refactorization graph is captured: every buffer must already be
// large enough (the capture replays the sizes of the last factorization), so a
// growth request aborts the capture and the factorization runs dynamically.
thread_local bool tl_no_alloc = false;
static int no_alloc_fail() {
  set_error("refactorization replay would allocate");
  return RVG_ERR_DEVICE;
}

template <class T>
int ensure(T*& p, size_t& cap, size_t need, cudaStream_t st) {
  if (need <= cap && p) return RVG_OK;
  if (tl_no_alloc) return no_alloc_fail();
  size_t nc = std::max(need, cap + cap / 2);
  if (nc == 0) nc = 1;
  T* np = nullptr;
  CK(cudaMallocAsync((void**)&np, nc * sizeof(T), st));
  if (p) {
    if (cap) CK(cudaMemcpyAsync(np, p, cap * sizeof(T), cudaMemcpyDeviceToDevice, st));
    CK(cudaFreeAsync(p, st));
  }
  p = np;
  cap = nc;
  return RVG_OK;
}

int ensure_host(char*& p, size_t& cap, size_t need) {
  if (need <= cap && p) return RVG_OK;
  if (tl_no_alloc) return no_alloc_fail();
  size_t nc = std::max(need, cap + cap / 2);
  if (p) CK(cudaFreeHost(p));
  p = nullptr;
  CK(cudaMallocHost((void**)&p, nc));
  cap = nc;
  return RVG_OK;
}

int vm_d_arrays(rvg_handle* h, size_t need);
int ensure_d_arrays(rvg_handle* h, size_t need) {  // type / diag / off share one capacity
  if (h->vm) return vm_d_arrays(h, need);
  if (need <= h->d_cap && h->dtype) return RVG_OK;
  if (tl_no_alloc) return no_alloc_fail();
  size_t nc = std::max(need, h->d_cap + h->d_cap / 2);
  int8_t* t; double *a, *b;
  CK(cudaMallocAsync((void**)&t, nc, h->st));
  CK(cudaMallocAsync((void**)&a, nc * 8, h->st));
  CK(cudaMallocAsync((void**)&b, nc * 8, h->st));
  if (h->dtype) {
    CK(cudaMemcpyAsync(t, h->dtype, h->d_cap, cudaMemcpyDeviceToDevice, h->st));
    CK(cudaMemcpyAsync(a, h->ddiag, h->d_cap * 8, cudaMemcpyDeviceToDevice, h->st));
    CK(cudaMemcpyAsync(b, h->doff, h->d_cap * 8, cudaMemcpyDeviceToDevice, h->st));
    CK(cudaFreeAsync(h->dtype, h->st)); CK(cudaFreeAsync(h->ddiag, h->st)); CK(cudaFreeAsync(h->doff, h->st));
  }
  h->dtype = t; h->ddiag = a; h->doff = b; h->d_cap = nc;
  return RVG_OK;
}

template <class T>
int ensure_nocopy(T*& p, size_t& cap, size_t need, cudaStream_t st) {
  if (need <= cap && p) return RVG_OK;
  if (tl_no_alloc) return no_alloc_fail();
  size_t nc = std::max(need, cap + cap / 4);
  if (nc == 0) nc = 1;
  if (p) CK(cudaFreeAsync(p, st));
  p = nullptr;
  CK(cudaMallocAsync((void**)&p, nc * sizeof(T), st));
  cap = nc;
  return RVG_OK;
}

// ---------------------------------------------------------------------------
// Address-stable arenas (graph_refactor = 2).  A captured refactorization
// graph holds the addresses of the factorization's arenas, and rvg_trim
// releases their memory so that many handles can take turns on one device.
// In this mode each arena is a range of virtual addresses reserved once for
// the handle's life (as large as the device's memory); physical memory is
// mapped into it in chunks as the arena grows (contents and address kept),
// unmapped by rvg_trim, and mapped again by the next factorization up to the
// largest size the arena reached, so the graph's addresses stay valid.
enum VmSlotId {
  VM_PANEL = 0, VM_IDX, VM_DTYPE, VM_DDIAG, VM_DOFF, VM_SCRATCH, VM_CB, VM_PACK, VM_STAGE,
  VM_WPACK0,  // + context id
  VM_NSLOTS = VM_WPACK0 + LF_CONCURRENT
};
}  // namespace (the arenas' types complete the handle's forward declaration, at file scope)
struct VmSlot {
  CUdeviceptr va = 0;
  size_t reserved = 0, mapped = 0, high = 0;
  std::vector<std::pair<size_t, CUmemGenericAllocationHandle>> chunks;  // (bytes, physical memory) from va on
};
struct VmArenas {
  size_t gran = 0, reserve = 0;  // reserve: the device's memory, the most any range grows to
  CUmemAllocationProp prop = {};
  CUmemAccessDesc access = {};
  VmSlot slot[VM_NSLOTS];
};
namespace {

// The driver's virtual-memory calls, looked up through the runtime
// (cudaGetDriverEntryPoint) so that the library does not link the driver
// library itself and still loads on a machine without one.
struct VmApi {
  decltype(&cuGetErrorString) err = nullptr;
  decltype(&cuMemGetAllocationGranularity) gran = nullptr;
  decltype(&cuMemAddressReserve) reserve = nullptr;
  decltype(&cuMemAddressFree) free = nullptr;
  decltype(&cuMemCreate) create = nullptr;
  decltype(&cuMemRelease) release = nullptr;
  decltype(&cuMemMap) map = nullptr;
  decltype(&cuMemUnmap) unmap = nullptr;
  decltype(&cuMemSetAccess) access = nullptr;
};
VmApi g_vm;

int vm_api() {
  if (g_vm.access) return RVG_OK;
  VmApi a;
  bool ok = true;
  auto get = [&](const char* name, auto& fp) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess ||
        !f)
      ok = false;
    fp = reinterpret_cast<std::remove_reference_t<decltype(fp)>>(f);
  };
  get("cuGetErrorString", a.err);
  get("cuMemGetAllocationGranularity", a.gran);
  get("cuMemAddressReserve", a.reserve);
  get("cuMemAddressFree", a.free);
  get("cuMemCreate", a.create);
  get("cuMemRelease", a.release);
  get("cuMemMap", a.map);
  get("cuMemUnmap", a.unmap);
  get("cuMemSetAccess", a.access);
  if (!ok) {
    cudaGetLastError();
    set_error("the driver's virtual-memory calls are not available (graph_refactor = 2)");
    return RVG_ERR_DEVICE;
  }
  g_vm = a;
  return RVG_OK;
}

int cu_fail(CUresult r, const char* what) {
  const char* msg = nullptr;
  if (g_vm.err) g_vm.err(r, &msg);
  set_error(std::string("CUDA driver error: ") + (msg ? msg : "unknown") + " at " + what);
  return r == CUDA_ERROR_OUT_OF_MEMORY ? RVG_ERR_OUT_OF_MEMORY : RVG_ERR_DEVICE;
}
#define CU(x)                                  \
  do {                                         \
    const CUresult cu_r_ = (x);                \
    if (cu_r_ != CUDA_SUCCESS) return cu_fail(cu_r_, #x); \
  } while (0)

int vm_create(rvg_handle* h) {
  if (int rc = vm_api()) return rc;
  std::unique_ptr<VmArenas> v(new VmArenas);
  v->prop.type = CU_MEM_ALLOCATION_TYPE_PINNED;
  v->prop.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
  v->prop.location.id = h->device;
  CU(g_vm.gran(&v->gran, &v->prop, CU_MEM_ALLOC_GRANULARITY_RECOMMENDED));
  size_t fr = 0, tot = 0;
  CK(cudaMemGetInfo(&fr, &tot));
  v->reserve = (tot + v->gran - 1) / v->gran * v->gran;
  v->access.location = v->prop.location;
  v->access.flags = CU_MEM_ACCESS_FLAGS_PROT_READWRITE;
  h->vm = v.release();
  return RVG_OK;
}

void vm_unmap(VmSlot& s);

// backs at least `bytes` of slot `id` (at least its largest earlier size).
// A range is reserved at four times its first size (256 MB at least); one that
// must grow past its reservation moves to a larger one (contents copied, the
// replay graph dropped: it held the old addresses).
int vm_map(rvg_handle* h, int id, size_t bytes) {
  VmArenas* v = h->vm;
  VmSlot& s = v->slot[id];
  const size_t want = std::max((bytes + v->gran - 1) / v->gran * v->gran, s.high);
  if (want <= s.mapped) return RVG_OK;
  if (want > v->reserve) {
    set_error("an arena would exceed the device's memory");
    return RVG_ERR_OUT_OF_MEMORY;
  }
  if (!s.va || want > s.reserved) {
    const size_t r = std::min(v->reserve, std::max<size_t>(4 * want, (size_t)256 << 20) / v->gran * v->gran);
    CUdeviceptr nva = 0;
    CU(g_vm.reserve(&nva, r, v->gran, 0, 0));
    if (s.va) {  // move: map the new range, copy what the old one held, release the old one
      VmSlot old = s;
      s = VmSlot();
      s.va = nva;
      s.reserved = r;
      int rc = vm_map(h, id, old.mapped);
      if (rc) {  // the old range stays the arena; the new one goes
        vm_unmap(s);
        g_vm.free(nva, r);
        s = old;
        return rc;
      }
      CK(cudaDeviceSynchronize());
      CK(cudaMemcpy((void*)s.va, (const void*)old.va, old.mapped, cudaMemcpyDeviceToDevice));
      vm_unmap(old);
      g_vm.free(old.va, old.reserved);
      s.high = std::max(s.high, old.high);
      if (h->gexec) cudaGraphExecDestroy(h->gexec);  // the replay graph held the old addresses
      if (h->graph) cudaGraphDestroy(h->graph);
      h->gexec = nullptr;
      h->graph = nullptr;
    } else {
      s.va = nva;
      s.reserved = r;
    }
  }
  size_t add = std::max(want - s.mapped, (s.mapped / 4 + v->gran - 1) / v->gran * v->gran);  // fewer, larger chunks
  add = std::min(add, s.reserved - s.mapped);
  CUmemGenericAllocationHandle m = 0;
  CUresult r = g_vm.create(&m, add, &v->prop, 0);
  if (r == CUDA_ERROR_OUT_OF_MEMORY) {  // memory kept by the stream-ordered pool: hand it back, try again
    cudaDeviceSynchronize();
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, h->device) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
    r = g_vm.create(&m, add, &v->prop, 0);
  }
  if (r != CUDA_SUCCESS) return cu_fail(r, "cuMemCreate");
  r = g_vm.map(s.va + s.mapped, add, 0, m, 0);
  if (r != CUDA_SUCCESS) {
    g_vm.release(m);
    return cu_fail(r, "cuMemMap");
  }
  r = g_vm.access(s.va + s.mapped, add, &v->access, 1);
  if (r != CUDA_SUCCESS) {
    g_vm.unmap(s.va + s.mapped, add);
    g_vm.release(m);
    return cu_fail(r, "cuMemSetAccess");
  }
  s.chunks.emplace_back(add, m);
  s.mapped += add;
  s.high = std::max(s.high, s.mapped);
  return RVG_OK;
}

// releases a slot's physical memory, keeping its addresses (the device must
// be done with it: the callers synchronise the device first)
void vm_unmap(VmSlot& s) {
  size_t off = 0;
  for (auto& c : s.chunks) {
    g_vm.unmap(s.va + off, c.first);
    g_vm.release(c.second);
    off += c.first;
  }
  s.chunks.clear();
  s.mapped = 0;
}

void vm_destroy(rvg_handle* h) {
  if (!h->vm) return;
  cudaDeviceSynchronize();
  for (VmSlot& s : h->vm->slot) {
    vm_unmap(s);
    if (s.va) g_vm.free(s.va, s.reserved);
  }
  delete h->vm;
  h->vm = nullptr;
}

// The arena of slot `id` with room for `need` elements: address-stable in the
// graph_refactor = 2 mode (growth maps more memory behind the contents), else
// ensure()'s stream-ordered reallocation (`copy`: the contents move along).
template <class T>
int arena_ensure(rvg_handle* h, int id, T*& p, size_t& cap, size_t need, cudaStream_t st, bool copy) {
  if (!h->vm) return copy ? ensure(p, cap, need, st) : ensure_nocopy(p, cap, need, st);
  if (need <= cap && p) return RVG_OK;
  if (tl_no_alloc) return no_alloc_fail();
  int rc = vm_map(h, id, std::max<size_t>(need, 1) * sizeof(T));
  if (rc) return rc;
  p = reinterpret_cast<T*>(h->vm->slot[id].va);
  cap = h->vm->slot[id].mapped / sizeof(T);
  return RVG_OK;
}

// Every arena mapped again up to its largest size and bound to its pointer:
// a replayed graph touches them all without the host's ensure calls.
int vm_restore(rvg_handle* h) {
  for (int id = 0; id < VM_NSLOTS; ++id) {
    VmSlot& sl = h->vm->slot[id];
    if (sl.high > sl.mapped) {
      int rc = vm_map(h, id, sl.high);
      if (rc) return rc;
    }
  }
  auto bind = [&](int id, auto*& p, size_t& cap) {
    const VmSlot& sl = h->vm->slot[id];
    if (sl.mapped && !p) {
      p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(sl.va);
      cap = sl.mapped / sizeof(*p);
    }
  };
  bind(VM_PANEL, h->panel, h->panel_cap);
  bind(VM_IDX, h->idx, h->idx_cap);
  bind(VM_SCRATCH, h->scratch, h->scratch_cap);
  bind(VM_CB, h->cb_arena, h->cb_cap);
  bind(VM_PACK, h->pack, h->pack_cap);
  bind(VM_STAGE, h->d_stage, h->stage_cap);
  bind(VM_WPACK0, h->wpack, h->wpack_cap);
  for (size_t t = 1; t < h->lfx.size(); ++t) bind(VM_WPACK0 + (int)t, h->lfx[t].wpack, h->lfx[t].wpack_cap);
  if (!h->dtype && h->vm->slot[VM_DTYPE].mapped) {
    size_t ct = 0, ca = 0, cb = 0;
    bind(VM_DTYPE, h->dtype, ct);
    bind(VM_DDIAG, h->ddiag, ca);
    bind(VM_DOFF, h->doff, cb);
    h->d_cap = std::min(ct, std::min(ca, cb));
  }
  return RVG_OK;
}

int vm_d_arrays(rvg_handle* h, size_t need) {
  if (need <= h->d_cap && h->dtype) return RVG_OK;
  if (tl_no_alloc) return no_alloc_fail();
  size_t ct = 0, ca = 0, cb = 0;
  int rc;
  if ((rc = arena_ensure(h, VM_DTYPE, h->dtype, ct, need, h->st, true)) ||
      (rc = arena_ensure(h, VM_DDIAG, h->ddiag, ca, need, h->st, true)) ||
      (rc = arena_ensure(h, VM_DOFF, h->doff, cb, need, h->st, true)))
    return rc;
  h->d_cap = std::min(ct, std::min(ca, cb));
  return RVG_OK;
}

// first-fit allocation of `len` doubles in the CB arena; grows (with a copy of
// the live contents) when no free range fits
int cb_alloc(rvg_handle* h, int64_t len, int64_t* off) {
  for (auto it = h->cb_free.begin(); it != h->cb_free.end(); ++it) {
    if (it->second >= len) {
      *off = it->first;
      int64_t rest = it->second - len, start = it->first + len;
      h->cb_free.erase(it);
      if (rest > 0) h->cb_free[start] = rest;
      return RVG_OK;
    }
  }
  if (tl_no_alloc) return no_alloc_fail();
  // grow: new capacity covers the old one plus the request
  size_t old = h->cb_cap;
  size_t nc = std::max(old + (size_t)len, old + old / 4);
  if (h->vm) {  // more memory behind the same addresses
    size_t cap = old;
    int rc = arena_ensure(h, VM_CB, h->cb_arena, cap, nc, h->st, true);
    if (rc) return rc;
    nc = cap;
  } else {
    double* np = nullptr;
    CK(cudaMallocAsync((void**)&np, nc * sizeof(double), h->st));
    if (h->cb_arena) {
      if (old) CK(cudaMemcpyAsync(np, h->cb_arena, old * sizeof(double), cudaMemcpyDeviceToDevice, h->st));
      CK(cudaFreeAsync(h->cb_arena, h->st));
    }
    h->cb_arena = np;
  }
  h->cb_cap = nc;
  // the tail [old, nc) is free; merge with a free range ending at `old`
  int64_t start = (int64_t)old, length = (int64_t)(nc - old);
  auto it = h->cb_free.lower_bound(start);
  if (it != h->cb_free.begin()) {
    auto pv = std::prev(it);
    if (pv->first + pv->second == start) { start = pv->first; length += pv->second; h->cb_free.erase(pv); }
  }
  h->cb_free[start] = length;
  return cb_alloc(h, len, off);
}

void cb_release(rvg_handle* h, int64_t off, int64_t len) {
  if (len <= 0) return;
  auto it = h->cb_free.emplace(off, len).first;
  auto nx = std::next(it);
  if (nx != h->cb_free.end() && it->first + it->second == nx->first) { it->second += nx->second; h->cb_free.erase(nx); }
  if (it != h->cb_free.begin()) {
    auto pv = std::prev(it);
    if (pv->first + pv->second == it->first) { pv->second += it->second; h->cb_free.erase(it); }
  }
}

template <class T>
int upload(T*& d, const std::vector<T>& h, cudaStream_t st) {
  size_t n = std::max<size_t>(h.size(), 1);
  CK(cudaMallocAsync((void**)&d, n * sizeof(T), st));
  if (!h.empty()) CK(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, st));
  return RVG_OK;
}

// Packs the typed arrays of one wave into one buffer (16-byte aligned
// sections) so the whole wave is a single host->device copy.
struct Packer {
  std::vector<char> buf;
  template <class T>
  size_t add(const std::vector<T>& v) {
    size_t off = (buf.size() + 15) & ~size_t(15);
    buf.resize(off + v.size() * sizeof(T));
    if (!v.empty()) std::memcpy(buf.data() + off, v.data(), v.size() * sizeof(T));
    return off;
  }
};

Statics statics(rvg_handle* h) {
  return Statics{h->d_own_ptr, h->d_own_idx, h->d_pat_ptr, h->d_pat_idx, h->d_amap_ptr,
                 h->d_amap, h->d_ea_ptr, h->d_ea_map, h->d_ch_ptr, h->d_ch_idx};
}

DevOpts devopts(const rvg_options& o) {
  return DevOpts{o.threshold, o.small, (int)o.outer_block_size, (int)o.inner_block_size, o.failed_pivot_tpp};
}

unsigned blocks_for(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// Columns of the pending window of a large front's deferred updates: LF_WINDOW
// outer blocks, or rvg_options::mixed_window of them in the mixed form (a full
// window's update reads and writes every trailing entry once in FP64 for K =
// window columns of BF16 or TF32 products: at K = 1024 that C stream already
// asks for most of the HBM bandwidth at the tensor cores' rate, so a deeper
// window is faster, and less accurate), except in the mixed form when the
// outer block is not a whole number of 128-row tiles (its packed operands are
// appended tile- and chunk-aligned): then one block (every block's update
// applied at once).
constexpr int64_t LF_WINDOW = 4;
constexpr int64_t LF_WINDOW_MAX = 8;
int64_t lf_mixed_window(const rvg_handle* h) { return h->opt.mixed_window > 0 ? h->opt.mixed_window : LF_WINDOW; }
int64_t lf_window_cols(const rvg_handle* h, int64_t nb, bool mixed) {
  return !mixed ? LF_WINDOW * nb : (nb % 128 == 0 ? lf_mixed_window(h) * nb : nb);
}
// outer blocks of window storage a large front's scratch holds (any front of the handle may take the mixed
// form unless the precision is plain FP64)
int64_t lf_window_blocks(const rvg_handle* h) {
  return h->opt.precision == 0 ? LF_WINDOW : std::max(LF_WINDOW, lf_mixed_window(h));
}

// Which fronts of a wave take the multi-kernel path (the whole GPU, one front
// after another) instead of one CTA each: every front of order >= T, and
// those of order >= T / 2 when the wave holds at most LF_FEW of them (a few
// such fronts leave most SMs idle on the CTA path; many keep them busy).
// Results do not depend on the choice: both paths perform the same
// arithmetic.  mid = the wave's count of non-TPP fronts with T/2 <= m < T.
constexpr int64_t LF_FEW = 16;
inline bool front_is_large(int64_t m, bool tpp, int64_t T, int64_t mid) {
  return !tpp && (m >= T || (m >= T / 2 && mid <= LF_FEW));
}

// Medium fronts that would hold a wave up on one CTA go to the large fronts'
// path (results do not depend on it).  One CTA's time grows with the front's
// trailing tiles, the whole GPU's hardly.  Measured for one dense front (us on
// one CTA / on the whole GPU; in brackets what the two models below give):
//   order 128   152 / 130   (125 / 185)      384    803 / 378   (692 / 505)
//         192   248 / 185   (213 / 243)      512   1415 / 481  (1288 / 661)
//         256   363 / 236   (330 / 306)     1000   6884 / 1027 (7088 / 1561)
// The second model is on the safe side, by 1.3 to 1.5 times: a dense front moves
// from order 320 or so on (as routed: 320 570 us, 384 376), where alone it would
// gain from 192 on already.  The queue runs all its fronts at once, the large
// path up to `ctx` at a time beside it, each further one with a host thread to
// start: the j longest fronts move where that makes the longer of the two
// shortest, and only if it saves a tenth.  (That the queue's CTAs may have to
// take turns, above two fronts a multiprocessor, is left out: the large path then
// gets the multiprocessors as the queue empties: 1500 fronts of order 300 take 4.5
// ms, with one of order 600 beside them 4.7.)  Only fronts of order >= T / 16 (128
// at the default threshold) count, so the threshold still turns the path off; they
// keep the FP64 updates in every precision.
constexpr int LF_ROUTED_MAX = 16;
double cta_front_us(double m, double k) {
  double t = 0;
  for (double c = 32; c < k + 32; c += 32) {
    const double cols = std::max(0.0, k - c), rows = std::max(0.0, m - c);
    t += 28 + rows / 40 + 1.2 * cols * (rows - cols / 2) / 1024;
  }
  return t;
}
double lf_front_us(double m, double k, double nb) {
  return std::ceil(k / 32) * (24 + m / 60) + 60 * std::ceil(k / nb) + 20;
}
// the positions in mk (order, fully-summed columns) of the fronts to move
std::vector<int> route_medium(const std::vector<std::pair<int64_t, int64_t>>& mk, int64_t T, int64_t nb) {
  std::vector<std::pair<double, int>> c;
  for (int i = 0; i < (int)mk.size(); ++i) c.emplace_back(cta_front_us((double)mk[i].first, (double)mk[i].second), i);
  const int top = (int)std::min<size_t>(c.size(), LF_ROUTED_MAX + 1);
  std::partial_sort(c.begin(), c.begin() + top, c.end(), [](const auto& a, const auto& b) {
    return a.first > b.first || (a.first == b.first && a.second < b.second);
  });
  const int ctx = LF_CONCURRENT;
  int best = 0;
  double best_t = c.empty() ? 0 : 0.9 * c[0].first, sum = 0, longest = 0;
  for (int j = 1; j <= (int)std::min<size_t>(c.size(), LF_ROUTED_MAX); ++j) {
    const auto& f = mk[c[j - 1].second];
    if (f.first < T / 16) break;
    const double l = lf_front_us((double)f.first, (double)f.second, (double)nb);
    sum += l;
    longest = std::max(longest, l);
    const double lf = std::max(longest, sum / std::min(j, ctx)) + 15 + 25 * (std::min(j, ctx) - 1);
    const double t = std::max(lf, j < (int)c.size() ? c[j].first : 0.0);
    if (t < best_t) { best_t = t; best = j; }
  }
  std::vector<int> out;
  for (int j = 0; j < best; ++j) out.push_back(c[j].second);
  return out;
}

// Arena sizes of the delay-free schedule, computed from the pattern alone
// (delays can only add to them; the arenas grow in that case).
int presize_arenas(rvg_handle* h) {
  Plan& P = h->P;
  const int64_t nb = h->opt.outer_block_size, ib = h->opt.inner_block_size;
  int64_t panel = 0, idx = 0, dsz = 0, scratch = 0;
  std::vector<int64_t> cbw(P.waves.size(), 0), rel(P.waves.size(), -1);
  const int64_t T = h->opt.large_front_threshold;
  for (size_t w = 0; w < P.waves.size(); ++w) {
    int64_t sc_w = 0, mid = 0;
    for (int64_t s : P.waves[w]) {
      const Snode& x = P.sn[s];
      const int64_t k = x.n_owned(), m = k + (int64_t)x.pattern.size();
      if (!(x.in_small_leaf || k < ib) && m >= T / 2 && m < T) ++mid;
    }
    std::vector<std::pair<int64_t, int64_t>> med;
    std::vector<int64_t> med_s;
    for (int64_t s : P.waves[w]) {
      const Snode& x = P.sn[s];
      const int64_t k = x.n_owned(), m = k + (int64_t)x.pattern.size();
      const bool tpp = x.in_small_leaf || k < ib;
      if (!tpp && !front_is_large(m, tpp, T, mid)) { med.emplace_back(m, k); med_s.push_back(s); }
    }
    std::vector<int64_t> routed;
    for (int i : route_medium(med, T, nb)) routed.push_back(med_s[i]);
    for (int64_t s : P.waves[w]) {
      const Snode& x = P.sn[s];
      int64_t k = x.n_owned(), nfs = (int64_t)x.pattern.size(), m = k + nfs;
      panel += m * k;
      idx += m + k;
      dsz += k;
      bool has_cb = x.parent >= 0 && nfs > 0;
      if (has_cb) cbw[w] += nfs * nfs;
      bool tpp = x.in_small_leaf || k < ib;
      bool large = front_is_large(m, tpp, T, mid);
      int64_t sc = tpp ? 0 : (2 * IBMAX * m + nb);
      if (large || std::find(routed.begin(), routed.end(), s) != routed.end())
        sc = m * (2 * IBMAX + lf_window_blocks(h) * nb) + nb;
      if (has_cb && large) sc = std::max<int64_t>(sc, nfs * k);  // k_cb_w
      sc_w += sc;
      if (x.parent >= 0) rel[w] = std::max<int64_t>(rel[w], P.height[x.parent]);
    }
    scratch = std::max(scratch, sc_w);
  }
  // first-fit simulation of the contribution arena
  std::map<int64_t, int64_t> fr;
  int64_t hw = 0;
  std::vector<int64_t> off(P.waves.size(), -1);
  auto sim_free = [&](int64_t o, int64_t l) {
    auto it = fr.emplace(o, l).first;
    auto nx = std::next(it);
    if (nx != fr.end() && it->first + it->second == nx->first) { it->second += nx->second; fr.erase(nx); }
    if (it != fr.begin()) {
      auto pv = std::prev(it);
      if (pv->first + pv->second == it->first) { pv->second += it->second; fr.erase(it); }
    }
  };
  for (size_t w = 0; w < P.waves.size(); ++w) {
    // same order as run_factor: this wave's block is allocated before the
    // blocks its assembly consumed are released
    if (w > 0)
      for (size_t w2 = 0; w2 + 1 < w; ++w2)
        if (off[w2] >= 0 && rel[w2] == (int64_t)(w - 1)) { sim_free(off[w2], cbw[w2]); off[w2] = -1; }
    if (!cbw[w]) continue;
    bool placed = false;
    for (auto it = fr.begin(); it != fr.end(); ++it)
      if (it->second >= cbw[w]) {
        off[w] = it->first;
        int64_t rest = it->second - cbw[w], st = it->first + cbw[w];
        fr.erase(it);
        if (rest > 0) fr[st] = rest;
        placed = true;
        break;
      }
    if (!placed) {
      // extend at the end (merging a free tail)
      int64_t start = hw;
      auto it = fr.end();
      if (!fr.empty()) {
        auto last = std::prev(it);
        if (last->first + last->second == hw) { start = last->first; fr.erase(last); }
      }
      off[w] = start;
      hw = start + cbw[w];
    }
  }
  int rc;
  cudaStream_t st = h->st;
  if ((rc = arena_ensure(h, VM_PANEL, h->panel, h->panel_cap, (size_t)(panel + panel / 16 + 1024), st, true)))
    return rc;
  if ((rc = arena_ensure(h, VM_IDX, h->idx, h->idx_cap, (size_t)(idx + idx / 16 + 1024), st, true))) return rc;
  if ((rc = ensure_d_arrays(h, (size_t)(dsz + dsz / 8 + 1024)))) return rc;
  if ((rc = arena_ensure(h, VM_SCRATCH, h->scratch, h->scratch_cap, (size_t)(scratch + 1024), st, false)))
    return rc;
  if (hw > 0 && !h->cb_arena) {
    const size_t want = (size_t)(hw + hw / 16 + 1024);
    if (h->vm) {
      size_t cap = 0;
      if ((rc = arena_ensure(h, VM_CB, h->cb_arena, cap, want, st, false))) return rc;
      h->cb_cap = cap;
    } else {
      h->cb_cap = want;
      CK(cudaMallocAsync((void**)&h->cb_arena, h->cb_cap * sizeof(double), st));
    }
  }
  return RVG_OK;
}

double lower_entries(int64_t r0, int64_t r1, int64_t c0, int64_t c1) {
  double e = 0;
  for (int64_t j = c0; j < c1; ++j) {
    int64_t lo = j > r0 ? j : r0;
    if (r1 > lo) e += (double)(r1 - lo);
  }
  return e;
}

// CUDA events around each Schur GEMM launch (profiling): their sum is the
// GEMM time the measured rate is based on.
int syrk_ev(rvg_handle* h, bool on = true) {
  if (!h->profiling || !on || h->replay) return RVG_OK;
  if (h->ev_used + 1 > h->ev_pool.size()) {
    for (int i = 0; i < 64; ++i) {
      cudaEvent_t e;
      CK(cudaEventCreate(&e));
      h->ev_pool.push_back(e);
    }
  }
  CK(cudaEventRecord(h->ev_pool[h->ev_used++], h->st));
  return RVG_OK;
}

// The tensor-core Schur GEMM over a.ntiles 128 x 128 lower tiles: the flush
// depth picks the k_syrk_tc instance; without flushing, 256-column CTA tiles
// (k_syrk_tc_pair, over column-tile pairs) unless 128 is asked for.
template <int FMT>
static void launch_tc_fmt(rvg_handle* h, cudaStream_t st, TcArgs ta, int max_ctas) {
  const int64_t cap = max_ctas > 0 ? std::min<int64_t>(max_ctas, h->nsm) : h->nsm;
  if (h->opt.mixed_flush == 0 && h->opt.mixed_tile_cols == 256) {
    ta.ntiles = tp_count_tiles(ta.nr, ta.nc, ta.r0, ta.c0);
    const unsigned grid = (unsigned)std::min<int64_t>(ta.ntiles, cap);
    k_syrk_tc_pair<FMT><<<grid, TC_THREADS, TP_SMEM, st>>>(ta);
    return;
  }
  const unsigned grid = (unsigned)std::min<int64_t>(ta.ntiles, cap);
  switch (h->opt.mixed_flush) {
    case 1: k_syrk_tc<1, FMT><<<grid, TC_THREADS, TC_SMEM, st>>>(ta); break;
    case 2: k_syrk_tc<2, FMT><<<grid, TC_THREADS, TC_SMEM, st>>>(ta); break;
    case 4: k_syrk_tc<4, FMT><<<grid, TC_THREADS, TC_SMEM, st>>>(ta); break;
    case 8: k_syrk_tc<8, FMT><<<grid, TC_THREADS, TC_SMEM, st>>>(ta); break;
    default: k_syrk_tc<TC_NO_FLUSH, FMT><<<grid, TC_THREADS, TC_SMEM, st>>>(ta); break;
  }
}
static void launch_tc(rvg_handle* h, cudaStream_t st, TcArgs ta, int max_ctas = 0) {
  if (h->opt.mixed_operands == 1) launch_tc_fmt<TC_BF16>(h, st, ta, max_ctas);
  else launch_tc_fmt<TC_TF32>(h, st, ta, max_ctas);
}
// the operand split of the mixed form (TF32 or BF16 parts)
static void launch_pack(rvg_handle* h, cudaStream_t st, dim3 grid, const PackArgs& pa) {
  if (h->opt.mixed_operands == 1) k_pack_bf16x3<<<grid, 256, 0, st>>>(pa);
  else k_pack_tf32x3<<<grid, 256, 0, st>>>(pa);
}

// The Schur update C -= W L^T (lower) of one contribution block.  kmax bounds
// the device-side K (columns eliminated).
// Whether front s takes the mixed form's tensor-core updates: every large
// front with precision = 1, the selector's choice with precision = 2.
bool front_mixed(const rvg_handle* h, int64_t s) {
  if (h->h_fronts[s].flags & FF_ROUTED) return false;
  if (h->opt.precision == 1) return true;
  if (h->opt.precision != 2 || h->sel_force_fp64) return false;
  return s >= 0 && s < (int64_t)h->route.size() && h->route[s] != 0;
}

// A kernel of the large-front chain: with programmatic stream serialization
// it may start while the previous kernel of the stream still runs (each chain
// kernel waits for its predecessor in chain_enter() before any memory access),
// which hides the launch gap between the chain's short dependent kernels.
template <typename... KP, typename... AP>
static void launch_chain(const rvg_handle* h, void (*kern)(KP...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t st, AP... args) {
  if (!h->chain_pdl) {
    kern<<<grid, block, smem, st>>>(args...);
    return;
  }
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kern, args...);  // a failure stays the thread's last error, checked as for <<<>>>
}

// The launches of a wave's small and medium fronts touch different fronts, so
// all but the first may start while the one before still runs (programmatic
// stream serialization; wave_kernel_enter / _exit).  Together they are complete
// when the last one is.
template <typename... KP, typename... AP>
static void launch_beside(bool beside, void (*kern)(KP...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                          AP... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = beside ? 1 : 0;
  (void)cudaLaunchKernelEx(&cfg, kern, args...);  // a failure stays the thread's last error
}

int launch_syrk(rvg_handle* h, const SyrkArgs& ga, int64_t kmax, bool mixed) {
  cudaStream_t st = h->st;
  if (mixed) {
    const int64_t nr = (ga.r1 - ga.r0 + TC_BM - 1) / TC_BM, nc = (ga.c1 - ga.c0 + TC_BN - 1) / TC_BN;
    const int64_t Q = (kmax + TC_BK - 1) / TC_BK;
    const int64_t ntiles = (nr > 0 && nc > 0) ? tc_count_tiles(nr, nc, ga.r0, ga.c0) : 0;
    if (ntiles > 0 && Q > 0) {
      int rc = arena_ensure(h, VM_PACK, h->pack, h->pack_cap, (size_t)(nr + nc) * Q * TC_BLOCK, st, false);
      if (rc) return rc;
      float* pl = h->pack + (size_t)nr * Q * TC_BLOCK;
      PackArgs aw{ga.W, ga.ldw, ga.r1 - ga.r0, Q, ga.Kdev, ga.K, h->pack};
      PackArgs al{ga.L + ga.c0, ga.ldl, ga.c1 - ga.c0, Q, ga.Kdev, ga.K, pl};
      launch_pack(h, st, dim3((unsigned)Q, (unsigned)nr), aw);
      launch_pack(h, st, dim3((unsigned)Q, (unsigned)nc), al);
      TcArgs ta{ga.C, ga.ldc, ga.r0, ga.r1, ga.c0, ga.c1, h->pack, pl, Q, ga.Kdev, ga.K, nr, nc, ntiles, h->d_err};
      if ((rc = syrk_ev(h))) return rc;
      launch_tc(h, st, ta);
      if ((rc = syrk_ev(h))) return rc;
      h->launches += 3;
      h->syrk_launches++;
    }
  } else {
    int rc = syrk_ev(h);
    if (rc) return rc;
    k_syrk_lower<<<syrk_grid(ga), G_T, G_SMEM, st>>>(ga);
    if ((rc = syrk_ev(h))) return rc;
    h->launches++;
    h->syrk_launches++;
  }
  return RVG_OK;
}

// Deferred update of a large front's columns [c0, c1) (rows [c0, m)) by the
// window of pending columns [wd, wd + kadd + *kdev): W rows start at wrow
// (ld m - wrow), L is the panel itself; the mixed form reads the packed
// window (tile 0 = rows [wrow, wrow + 128), F / 32 chunks per tile).  With
// cond set the launch only acts if *cond < cond_lt.
int launch_window_gemm(rvg_handle* h, LfCtx& cx, const LFArgs& a, int64_t m, int64_t c0, int64_t c1, int64_t wd,
                       int64_t wrow, int64_t F, const float* pk_w, const float* pk_l, int64_t kadd,
                       const int32_t* kdev, const int32_t* cond, int32_t cond_lt, bool mixed,
                       const int32_t* skip = nullptr, cudaStream_t on = nullptr, int max_ctas = 0) {
  cudaStream_t st = on ? on : cx.st;
  if (c1 <= c0) return RVG_OK;
  int rc = syrk_ev(h, cx.marks);
  if (rc) return rc;
  if (mixed) {
    const int64_t Fq = F / TC_BK;
    const int64_t nr = (m - c0 + TC_BM - 1) / TC_BM, nc = (c1 - c0 + TC_BN - 1) / TC_BN;
    const int64_t ntiles = tc_count_tiles(nr, nc, c0, c0);
    const int64_t t0 = (c0 - wrow) / TC_BM;
    TcArgs ta{a.a, m, c0, m, c0, c1, pk_w + (size_t)t0 * Fq * TC_BLOCK, pk_l + (size_t)t0 * Fq * TC_BLOCK, Fq, kdev,
              kadd, nr, nc, ntiles, h->d_err, cond, cond_lt, 0, skip};
    launch_tc(h, st, ta, max_ctas);
  } else {
    SyrkArgs ga{};
    ga.C = a.a;
    ga.ldc = m;
    ga.W = a.wo + (c0 - wrow);
    ga.ldw = m - wrow;
    ga.L = a.a + wd * m;
    ga.ldl = m;
    ga.r0 = c0;
    ga.r1 = m;
    ga.c0 = c0;
    ga.c1 = c1;
    ga.K = kadd;
    ga.Kdev = kdev;
    ga.cond = cond;
    ga.cond_lt = cond_lt;
    ga.skip = skip;
    k_syrk_lower<<<syrk_grid(ga), G_T, G_SMEM, st>>>(ga);
  }
  if ((rc = syrk_ev(h, cx.marks))) return rc;
  cx.launches++;
  if (cx.marks) h->syrk_launches++;
  return RVG_OK;
}

// One large front on the whole GPU: the launch sequence of large.cuh, with
// one host synchronisation per 256-column outer block (its start column
// depends on the delays of the previous block).
int factor_large_front(rvg_handle* h, LfCtx& cx, int32_t s, const Arenas& Ar, const DevOpts& dop) {
  cudaStream_t st = cx.st;
  auto mk = [&](int kind) { if (cx.marks) mark(h, kind); };
  const DFront& f = h->h_fronts[s];
  const int64_t m = f.m, p = f.k, nb = h->opt.outer_block_size, ib = h->opt.inner_block_size;
  LFArgs a{};
  a.a = Ar.panel + f.panel;
  a.m = m;
  a.p = p;
  a.perm = Ar.idx + f.idx + m;
  a.D = DRec{Ar.dtype + f.dpos, Ar.ddiag + f.dpos, Ar.doff + f.dpos};
  a.st = cx.lf;
  double* sc = Ar.scratch + f.scratch;
  a.pb = sc;
  a.w = sc + m * IBMAX;
  a.wo = sc + 2 * m * IBMAX;
  const bool mixed = front_mixed(h, s);
  const int64_t F = lf_window_cols(h, nb, mixed);
  int32_t* const lp2 = (int32_t*)(sc + m * (2 * IBMAX + lf_window_blocks(h) * nb));  // two arrays of nb
  a.o = dop;
  const int two_level = p > nb;
  const int64_t Fq = F / TC_BK;
  // the packed window (W and L parts), twice: a full window's far-field update may still read one
  // buffer on the far stream while the next blocks pack into the other
  float* pk_wb[2] = {nullptr, nullptr};
  float* pk_lb[2] = {nullptr, nullptr};
  if (mixed && two_level) {
    const int64_t tiles = (m + TC_BM - 1) / TC_BM;
    const size_t one = (size_t)tiles * Fq * TC_BLOCK;
    int rc = arena_ensure(h, VM_WPACK0 + cx.id, cx.wpack, cx.wpack_cap, 4 * one, st, false);
    if (rc) return rc;
    pk_wb[0] = cx.wpack; pk_lb[0] = cx.wpack + one;
    pk_wb[1] = cx.wpack + 2 * one; pk_lb[1] = cx.wpack + 3 * one;
  }
  // far-field updates beside the next blocks: the mixed form in the dynamic schedule (not while
  // recording profiling marks, not inside a captured graph)
  const bool profiling_marks = cx.marks && h->profiling;  // this front's launches carry the profiling events
  // (the far part starts far_ahead blocks after the window's first W row: a whole number of the packed
  // window's 128-row tiles only when the block width is a multiple of 128).  The far part of a flush
  // runs beside every block of the next window but its last, whose near-field update writes the first
  // far-field columns and so waits for it.
  const int64_t far_ahead = std::max<int64_t>(1, F / nb - 1);
  const int far_sms = h->opt.far_field_sms < 0 ? LF_FAR_SMS : h->opt.far_field_sms;
  const bool async_far = mixed && two_level && !profiling_marks && !h->replay && nb % TC_BM == 0 && far_sms > 0 &&
                         far_sms < h->nsm;
  if (async_far && !cx.far_st) {
    if (tl_no_alloc) return no_alloc_fail();
    CK(cudaStreamCreateWithFlags(&cx.far_st, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&cx.ev_fork, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&cx.ev_far, cudaEventDisableTiming));
  }
  // The row permutations on their own stream, and the delay swap (which touches the same rows) left to the
  // host, in the dynamic schedule; in order on the front's stream in a captured graph or with the marks on.
  const bool side_prop = two_level && !profiling_marks && !h->replay;
  if (side_prop && !cx.prop_st) {
    if (tl_no_alloc) return no_alloc_fail();
    CK(cudaStreamCreateWithFlags(&cx.prop_st, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&cx.ev_prop_fork, cudaEventDisableTiming));
    for (auto& e : cx.ev_prop) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  bool prop_due[2] = {false, false};  // a permutation of that parity's lp may still run
  const bool host_swap = async_far || side_prop;
  mk(-1);
  k_lf_init<<<blocks_for(p, 256), 256, 0, st>>>(a.st, a.perm, p);
  cx.launches++;
  if (!h->replay) h->rec_g[s].clear();
  const int32_t* skip = &a.st->spec_bad;
  int irc = RVG_OK;  // first error of a launch helper inside issue()
  // Host view of the loop before an outer block: start column (eliminated so far), remaining
  // columns, the window of pending columns [wd, gne) whose W rows start at wrow, the block's index,
  // the packed-window buffer in use, and the block at which a far-field update running on the far
  // stream must be waited for (-1: none running).
  struct HostLF { int64_t gne, rem, wd, wrow; size_t outer; int par; int64_t far_due; };
  // what the host decided when it issued a block
  struct Issued { HostLF before; int64_t cs, bcols, oe, kadd, ncol; bool flush, window, far, waited; int slot; };
  // a CUDA call inside issue(): its failure becomes issue()'s error
  auto ck = [&](cudaError_t e, const char* what) {
    if (e != cudaSuccess && !irc) {
      set_error(std::string("CUDA error: ") + cudaGetErrorString(e) + " at " + what);
      irc = RVG_ERR_DEVICE;
    }
  };
  auto far_wait = [&]() {  // the stream takes up after the running far-field update
    ck(cudaStreamWaitEvent(st, cx.ev_far, 0), "cudaStreamWaitEvent (far-field update)");
    return irc;
  };
  // Launches one outer block for start column S.gne (1 + 2 per inner block + the outer-block steps).
  auto issue = [&](const HostLF& S, int slot) -> Issued {
    Issued I{};
    I.before = S;
    I.slot = slot;
    const int64_t rem = S.rem, cs = S.gne, wd = S.wd, wrow = S.wrow;
    const int64_t bcols = std::min(rem, nb), bm = m - cs, oe = cs + bcols;
    float* pk_w = pk_wb[S.par];
    float* pk_l = pk_lb[S.par];
    I.cs = cs; I.bcols = bcols; I.oe = oe;
    a.cs = cs;
    a.bcols = bcols;
    a.outer = (int)S.outer;
    const int opar = a.outer & 1;
    a.lp = lp2 + opar * nb;
    if (prop_due[opar]) {
      ck(cudaStreamWaitEvent(st, cx.ev_prop[opar], 0), "cudaStreamWaitEvent (row permutation)");
      prop_due[opar] = false;
    }
    I.window = two_level && oe < p;
    a.win = I.window;
    if (I.window) {  // this block's W joins the window [wd, gne + bne)
      I.kadd = cs - wd;
      a.wld = m - wrow;
      a.wrow0 = wrow;
      a.wcol0 = I.kadd;
    }
    launch_chain(h, k_lf_begin_outer, 1, NT, 0, st, a);
    mk(RVG_PART_LF_BLOCK);
    const int64_t ninner = (bcols + ib - 1) / ib;
    // per inner block: the panel rows, then its update beside the next inner block
    for (int64_t it = 0; it < ninner; ++it) {
      a.par = (int)(it & 1);
      launch_chain(h, k_lf_panel, blocks_for(bm, LF_PANEL_T), LF_PANEL_T, 0, st, a);
      mk(RVG_PART_LF_PANEL);
      // CTAs for the lower tiles right of column (it + 1) ib, where the trailing columns start if none was
      // delayed (they take more tiles each otherwise), two per SM at most
      const int64_t ts = std::min((it + 1) * ib, bcols), nrt = (bm - ts + 31) / 32, nct = (bcols - ts + 31) / 32;
      const int64_t tiles = nct * nrt - nct * (nct - 1) / 2;
      const int64_t ctas = std::max<int64_t>(1, std::min<int64_t>((tiles + NT / 32 - 1) / (NT / 32), 2 * h->nsm));
      launch_chain(h, k_lf_update, (unsigned)(1 + ctas), NT, 0, st, a, (int)(it + 1 < ninner));
      mk(RVG_PART_LF_UPDATE);
    }
    cx.launches += 1 + 2 * ninner;
    if (two_level) {
      if (cs > 0) {
        const cudaStream_t ps = side_prop ? cx.prop_st : st;
        if (side_prop) {
          ck(cudaEventRecord(cx.ev_prop_fork, st), "cudaEventRecord (row permutation fork)");
          ck(cudaStreamWaitEvent(ps, cx.ev_prop_fork, 0), "cudaStreamWaitEvent (row permutation fork)");
        }
        const int pc = lf_prop_cols(bcols);
        k_lf_prop<<<(unsigned)((cs + pc - 1) / pc), 256, (size_t)bcols * pc * 8, ps>>>(a, pc);
        if (side_prop) {
          ck(cudaEventRecord(cx.ev_prop[opar], ps), "cudaEventRecord (row permutation)");
          prop_due[opar] = true;
        }
        cx.launches++;
        mk(RVG_PART_LF_PROP);
      }
      if (I.window) {
        const int64_t kadd = I.kadd;
        // The next outer block is [g, g + min(rem - bcols, nb)); columns past
        // rem (delayed ones parked at the end) belong to no later block.  The
        // window is applied everywhere when it is full, or when the next block
        // is the last one (so no column is left pending for the end of the front).
        I.flush = kadd + bcols >= F || rem - bcols < nb;
        I.ncol = nb;
        const int32_t* bne_dev = &a.st->bne;
        if (mixed) {
          // append this block's chunks of W (rows [oe, m)) and L (rows [oe, p))
          const int64_t q0 = kadd / TC_BK, nqb = (bcols + TC_BK - 1) / TC_BK, t0 = (oe - wrow) / TC_BM;
          PackArgs pw{a.wo + (oe - wrow), a.wld, m - oe, Fq, bne_dev, kadd, pk_w, q0, t0, nullptr, 0, skip};
          PackArgs pl{a.a + wd * m + oe, m, p - oe, Fq, bne_dev, kadd, pk_l, q0, t0, nullptr, 0, skip};
          launch_pack(h, st, dim3((unsigned)nqb, blocks_for(m - oe, TC_BM)), pw);
          launch_pack(h, st, dim3((unsigned)nqb, blocks_for(p - oe, TC_BM)), pl);
          cx.launches += 2;
        }
        // columns of a far-field update still running: the next block's (the near field) from the
        // block it was launched for on, every trailing column at a flush
        if (S.far_due >= 0 && ((int64_t)S.outer >= S.far_due || I.flush)) {
          irc = irc ? irc : far_wait();
          I.waited = true;
        }
        if (I.flush) {
          const int64_t split = oe + far_ahead * nb;
          if (async_far && p - split >= 2 * nb) {
            // the next far_ahead blocks' columns now, the rest on the far stream beside them (both
            // after the packs; they touch different columns).  The far part takes its counts from k_lf_far:
            // the state itself moves on with the next blocks
            k_lf_far<<<1, 1, 0, st>>>(a.st);
            ck(cudaEventRecord(cx.ev_fork, st), "cudaEventRecord (far-field fork)");
            ck(cudaStreamWaitEvent(cx.far_st, cx.ev_fork, 0), "cudaStreamWaitEvent (far-field fork)");
            irc = irc ? irc : launch_window_gemm(h, cx, a, m, oe, split, wd, wrow, F, pk_w, pk_l, kadd, bne_dev,
                                                 nullptr, 0, mixed, skip);
            irc = irc ? irc : launch_window_gemm(h, cx, a, m, split, p, wd, wrow, F, pk_w, pk_l, kadd, &a.st->far_bne,
                                                 nullptr, 0, mixed, &a.st->far_skip, cx.far_st, h->nsm - far_sms);
            ck(cudaEventRecord(cx.ev_far, cx.far_st), "cudaEventRecord (far-field join)");
            cx.launches++;
            cx.far_launches++;
            I.far = true;
          } else {
            // the window is full: every trailing column takes it (one GEMM)
            irc = irc ? irc : launch_window_gemm(h, cx, a, m, oe, p, wd, wrow, F, pk_w, pk_l, kadd, bne_dev,
                                                 nullptr, 0, mixed, skip);
          }
        } else {
          // near field: the next outer block's columns (oe + nb <= p here) take the whole window
          irc = irc ? irc : launch_window_gemm(h, cx, a, m, oe, oe + I.ncol, wd, wrow, F, pk_w, pk_l, kadd, bne_dev,
                                               nullptr, 0, mixed, skip);
          // far field: only if this block delayed columns (decided on the device); with far-field
          // updates on the far stream the host issues it once it has seen the delay
          if (oe + nb < p && !async_far)
            irc = irc ? irc : launch_window_gemm(h, cx, a, m, oe + nb, p, wd, wrow, F, pk_w, pk_l, kadd, bne_dev,
                                                 bne_dev, (int32_t)bcols, mixed, skip);
        }
        mk(RVG_PART_LF_SYRK);
      }
    }
    launch_chain(h, k_lf_outer, 1, NT, 0, st, a, rem, (int)two_level, host_swap ? 0 : 1,
                 h->replay ? (int32_t*)nullptr : cx.h_gne + slot);
    cx.launches++;
    mk(RVG_PART_LF_OUTER);
    return I;
  };
  // The state after block I if it eliminated up to column g (no side effects).
  auto next_state = [&](const Issued& I, int32_t g) -> HostLF {
    HostLF S = I.before;
    const int64_t bne = g - I.cs;
    if (two_level && I.window && (I.flush || bne < I.bcols)) {  // every column is up to date: a new, empty window
      S.wd = g;
      S.wrow = g + std::min(S.rem - I.bcols, nb);
    }
    if (I.flush) S.par ^= 1;
    S.far_due = I.far ? (int64_t)I.before.outer + far_ahead : (I.waited ? -1 : I.before.far_due);
    S.gne = g;
    S.rem -= I.bcols;
    S.outer += 1;
    return S;
  };
  // The Schur-GEMM flops of block I (where the GEMM's events are recorded: the front carrying the marks).
  auto account = [&](const Issued& I, int32_t g) {
    if (!(two_level && I.window) || !cx.marks) return;
    const int64_t bne = g - I.cs;
    const double K = (double)(I.kadd + bne);
    if (I.flush) {
      cx.syrk_flops += 2.0 * K * lower_entries(I.oe, m, I.oe, p);
    } else {
      cx.syrk_flops += 2.0 * K * lower_entries(I.oe, m, I.oe, I.oe + I.ncol);
      if (I.oe + nb < p && bne < I.bcols) cx.syrk_flops += 2.0 * K * lower_entries(I.oe + nb, m, I.oe + nb, p);
    }
  };
  HostLF S{0, p, 0, std::min(p, nb), 0, 0, -1};
  if (h->replay) {
    // the progress of the recorded factorization, checked on the device
    const std::vector<int32_t>& rg = h->rec_g[s];
    while (S.rem > 0) {
      Issued I = issue(S, 0);
      if (irc) return irc;
      if (S.outer >= rg.size()) { set_error("refactorization replay: record too short"); return RVG_ERR_DEVICE; }
      const int32_t g = rg[S.outer];
      k_check_gne<<<1, 32, 0, st>>>(a.st, g, h->d_mismatch);
      CK(cudaGetLastError());
      account(I, g);
      S = next_state(I, g);
    }
  } else {
    // Blocks go out ahead on the guess that none delays a column (the next
    // start column is then this one plus its width); the device checks each
    // guess when the block begins (k_lf_begin_outer), and a wrong one turns
    // every later launch of the front into a no-op.  The host reads the
    // device's eliminated total after each block in issue order, at most
    // LF_AHEAD blocks behind; at the first one that differs it waits for the
    // streams, issues what that block's delay asks for (with far-field
    // updates on the far stream: the far field's update by the window and the
    // delay swap), clears the flag and issues again from the true start column.
    if (!cx.h_gne) {
      if (tl_no_alloc) return no_alloc_fail();
      CK(cudaHostAlloc((void**)&cx.h_gne, LF_AHEAD * sizeof(int32_t), cudaHostAllocDefault));
      for (int i = 0; i < LF_AHEAD; ++i) CK(cudaEventCreateWithFlags(&cx.ring_ev[i], cudaEventDisableTiming));
    }
    std::deque<Issued> q;
    int next_slot = 0;
    // with the profiling marks on, one block at a time: the marks are read back after each block
    const int ahead = profiling_marks ? 1 : LF_AHEAD;
    while (S.rem > 0 || !q.empty()) {
      if (S.rem > 0 && (int)q.size() < ahead) {
        const int slot = next_slot;
        next_slot = (next_slot + 1) % LF_AHEAD;
        Issued I = issue(S, slot);
        if (irc) return irc;
        CK(cudaEventRecord(cx.ring_ev[slot], st));
        CK(cudaGetLastError());
        q.push_back(I);
        S = next_state(I, (int32_t)(I.cs + I.bcols));  // the guess: no delayed column in this block
        continue;
      }
      const Issued I = q.front();
      q.pop_front();
      const double t0 = now_ms();
      CK(cudaEventSynchronize(cx.ring_ev[I.slot]));
      const double waited = now_ms() - t0;
      const int32_t g = *(volatile int32_t*)(cx.h_gne + I.slot);  // written by the block's k_lf_outer
      h->rec_g[s].push_back(g);
      if (profiling_marks) {
        mark_flush(h);
        mk(-1);
      }
      account(I, g);
      // the device worked on this and the queued blocks meanwhile
      cx.wait_ms += waited;
      if (g == I.cs + I.bcols) continue;  // as guessed
      // a block delayed columns: the blocks issued after it did nothing; the
      // streams run dry while the host issues them again
      const double t1 = now_ms();
      CK(cudaStreamSynchronize(st));
      if (cx.far_st) CK(cudaStreamSynchronize(cx.far_st));
      if (cx.prop_st) CK(cudaStreamSynchronize(cx.prop_st));
      prop_due[0] = prop_due[1] = false;
      cx.sync_ms += now_ms() - t1;
      cx.misses += (int64_t)q.size();
      q.clear();
      HostLF T = next_state(I, g);
      T.far_due = -1;  // nothing runs on the far stream any more
      if (host_swap) {
        const int64_t bne = g - I.cs;
        a.cs = I.cs;
        a.bcols = I.bcols;
        if (async_far && I.window && !I.flush && I.oe + nb < p) {
          // the far field takes the window, this block's eliminated columns included
          irc = launch_window_gemm(h, cx, a, m, I.oe + nb, p, I.before.wd, I.before.wrow, F, pk_wb[I.before.par],
                                   pk_lb[I.before.par], I.kadd + bne, nullptr, nullptr, 0, mixed);
          if (irc) return irc;
        }
        if (two_level && bne < I.bcols)
          k_lf_swap<<<1, NT, 0, st>>>(a, I.cs, I.bcols, I.before.rem, (int)bne);
        cx.launches += 2;
      }
      CK(cudaMemsetAsync(&a.st->spec_bad, 0, sizeof(int32_t), st));
      CK(cudaGetLastError());
      S = T;
    }
  }
  if (S.far_due >= 0) CK(cudaStreamWaitEvent(st, cx.ev_far, 0));  // a far-field update still running
  for (int q = 0; q < 2; ++q)
    if (prop_due[q]) CK(cudaStreamWaitEvent(st, cx.ev_prop[q], 0));
  k_lf_finish<<<1, 32, 0, st>>>(a, h->d_fronts, s);
  cx.launches++;
  mk(RVG_PART_LF_SETUP);
  CK(cudaGetLastError());
  return RVG_OK;
}

// The large fronts of one wave: one after another on the handle's stream when
// there is one (profiling marks on), otherwise up to LF_CONCURRENT at a time,
// each context's fronts in turn on its own host thread and stream, ordered
// after the wave's assembly and before what follows by events.  beside: the
// event behind the assembly when the wave's small and medium fronts are queued
// on the handle's stream meanwhile; context 0 then has a stream of its own too
// and the large ones run beside them.  counted: ids[0] is the wave's only large
// front, the others medium ones on its path: its GEMMs are counted as if it
// were alone.
int factor_large_fronts(rvg_handle* h, const std::vector<int32_t>& ids, const Arenas& A, const DevOpts& dop,
                        cudaEvent_t beside = nullptr, bool counted = false) {
  if (ids.empty()) return RVG_OK;
  if (h->lfx.empty()) {
    h->lfx.resize(1);
    h->lfx[0].lf = h->d_lf;
  }
  if (beside && !h->lf_st) {
    if (tl_no_alloc) return no_alloc_fail();
    CK(cudaStreamCreateWithFlags(&h->lf_st, cudaStreamNonBlocking));
  }
  auto fold = [&](LfCtx& c) {
    h->launches += c.launches;
    h->host_sync_ms += c.sync_ms;
    h->host_wait_ms += c.wait_ms;
    h->lf_misses += c.misses;
    h->lf_far += c.far_launches;
    h->syrk_flops += c.syrk_flops;
    c.launches = 0; c.sync_ms = 0; c.syrk_flops = 0; c.wait_ms = 0; c.misses = 0; c.far_launches = 0;
  };
  // (a capture forks into the same contexts with the fronts dealt the same way:
  // the replayed graph runs them concurrently on the buffers the dynamic run sized)
  const int nc = (int)std::min<size_t>(ids.size(), LF_CONCURRENT);
  while ((int)h->lfx.size() < nc) {  // grown before any reference into lfx is taken
    if (tl_no_alloc) return no_alloc_fail();
    LfCtx c;
    c.own = true;
    c.id = (int)h->lfx.size();
    CK(cudaStreamCreateWithFlags(&c.st, cudaStreamNonBlocking));
    CK(cudaMalloc((void**)&c.lf, sizeof(LFState)));
    h->lfx.push_back(c);
  }
  LfCtx& c0 = h->lfx[0];
  c0.st = beside ? h->lf_st : h->st;
  c0.wpack = h->wpack; c0.wpack_cap = h->wpack_cap;
  int rc = RVG_OK;
  if (nc == 1 && !beside) {
    c0.marks = true;
    for (int32_t s : ids)
      if ((rc = factor_large_front(h, c0, s, A, dop))) break;
    h->wpack = c0.wpack; h->wpack_cap = c0.wpack_cap;
    fold(c0);
    return rc;
  }
  mark(h, -1);
  cudaEvent_t ready = h->ev_large;
  if (!ready) {
    CK(cudaEventCreateWithFlags(&h->ev_large, cudaEventDisableTiming));
    ready = h->ev_large;
  }
  if (!beside) CK(cudaEventRecord(ready, h->st));
  const int first = beside ? 0 : 1;  // the first context not on the handle's stream
  for (int t = first; t < nc; ++t) CK(cudaStreamWaitEvent(h->lfx[t].st, beside ? beside : ready, 0));
  std::vector<int> rcs(nc, RVG_OK);
  std::vector<std::string> errs(nc);
  const bool no_alloc = tl_no_alloc;
  auto work = [&](int t) {
    cudaSetDevice(h->device);
    const bool was = tl_no_alloc;
    tl_no_alloc = no_alloc;
    LfCtx& c = h->lfx[t];
    for (size_t i = t; i < ids.size(); i += nc) {
      c.marks = counted && i == 0;
      if ((rcs[t] = factor_large_front(h, c, ids[i], A, dop))) { errs[t] = g_err; break; }
    }
    tl_no_alloc = was;
  };
  std::vector<std::thread> th;
  for (int t = 1; t < nc; ++t) th.emplace_back(work, t);
  work(0);
  for (auto& x : th) x.join();
  h->wpack = c0.wpack; h->wpack_cap = c0.wpack_cap;
  for (int t = first; t < nc; ++t) {
    CK(cudaEventRecord(ready, h->lfx[t].st));
    CK(cudaStreamWaitEvent(h->st, ready, 0));
  }
  mark(h, RVG_PART_OTHER);
  for (int t = 0; t < nc; ++t) {
    fold(h->lfx[t]);
    if (rcs[t] && !rc) { rc = rcs[t]; set_error(errs[t]); }
  }
  return rc;
}

int finish_factor(rvg_handle* h, int64_t d_used);

// k_cb_w's items of front s (columns that were delayed are found on the device)
void add_cb_w(std::vector<TileItem>& items, int32_t s, const DFront& f) {
  for (int tj = 0; tj * CBW_COLS < f.k; ++tj)
    for (int ti = 0; ti * 256 < f.nfs; ++ti) items.push_back(TileItem{s, ti, tj, 0});
}

// Learned precision: large fronts of the wave just factored whose mixed-form
// D grew past the bound (k_front_growth) are factored again in FP64, alone.
// Each is assembled again from scratch -- original entries and its children's
// contribution blocks, which the wave released to the allocator but which no
// allocation overwrites before the next wave -- then factored on the
// large-front path with FP64 updates, and its contribution block is formed
// again with the FP64 GEMM.  The results are those a plain FP64 factorization
// gives the front from the same children.
int refactor_fp64(rvg_handle* h, const std::vector<int32_t>& redo, const Arenas& A, const DevOpts& dop,
                  const double* d_vals, const double* d_scal) {
  cudaStream_t st = h->st;
  const Plan& P = h->P;
  int rc;
  for (int32_t s : redo) h->route[s] = 0;
  h->sel_refactored += (int64_t)redo.size();
  for (int32_t s : redo) {
    const DFront& f = h->h_fronts[s];
    CK(cudaMemsetAsync(A.panel + f.panel, 0, (size_t)f.m * f.k * 8, st));
    if (f.flags & FF_HAS_CB) CK(cudaMemsetAsync(A.cbase + f.cb, 0, (size_t)f.nfs * f.nfs * 8, st));
  }
  const int n = (int)redo.size();
  std::vector<ScatterItem> sitems;
  for (int32_t s : redo)
    for (int64_t e = P.amap_ptr[s]; e < P.amap_ptr[s + 1]; e += 256) sitems.push_back(ScatterItem{s, 0, e});
  size_t maxch = 0;
  for (int32_t s : redo) maxch = std::max(maxch, P.children[s].size());
  std::vector<std::vector<EaTile>> eitems(maxch);
  for (size_t q = 0; q < maxch; ++q)
    for (int32_t s : redo) {
      if (q >= P.children[s].size()) continue;
      const int64_t c = P.children[s][q];
      const DFront& cf = h->h_fronts[c];
      if (!(cf.flags & FF_HAS_PARENT) || cf.ne >= cf.m) continue;
      const int sz = cf.m - cf.ne;
      for (int j0 = 0; j0 < sz; j0 += 32)
        for (int i0 = j0; i0 < sz; i0 += EA_ROWS) eitems[q].push_back(EaTile{s, (int32_t)c, j0, i0});
    }
  std::vector<TileItem> witems, gitems;
  std::vector<int32_t> big_cb;
  for (int32_t s : redo) {
    const DFront& f = h->h_fronts[s];
    if (!(f.flags & FF_HAS_CB) || f.k == 0) continue;
    if (f.nfs >= 256) {  // GEMM by launch_syrk
      add_cb_w(witems, s, f);
      big_cb.push_back(s);
      continue;
    }
    const int nt = (f.nfs + GT - 1) / GT;
    for (int tj = 0; tj < nt; ++tj)
      for (int ti = tj; ti < nt; ++ti) gitems.push_back(TileItem{s, ti, tj, 0});
  }
  Packer pk;
  const size_t o_ids = pk.add(redo), o_s = pk.add(sitems), o_w = pk.add(witems), o_g = pk.add(gitems);
  std::vector<size_t> o_e(maxch);
  for (size_t q = 0; q < maxch; ++q) o_e[q] = pk.add(eitems[q]);
  const size_t o_cnt = pk.add(std::vector<int32_t>(3 * (size_t)n, 0));
  if ((rc = ensure(h->d_stage2, h->stage2_cap, pk.buf.size(), st))) return rc;
  if ((rc = ensure_host(h->h_stage2, h->h_stage2_cap, std::max(pk.buf.size(), (size_t)3 * n * 4)))) return rc;
  std::memcpy(h->h_stage2, pk.buf.data(), pk.buf.size());
  CK(cudaMemcpyAsync(h->d_stage2, h->h_stage2, pk.buf.size(), cudaMemcpyHostToDevice, st));
  char* D = h->d_stage2;
  const int32_t* d_ids = (const int32_t*)(D + o_ids);
  k_front_rows<<<n, 128, 0, st>>>(d_ids, n, h->d_fronts, statics(h), A);
  if (!sitems.empty())
    k_scatter<<<(unsigned)sitems.size(), 256, 0, st>>>((const ScatterItem*)(D + o_s), h->d_fronts, statics(h), A,
                                                       d_vals, d_scal);
  for (size_t q = 0; q < maxch; ++q)
    if (!eitems[q].empty())
      k_extend_add_tiled<<<(unsigned)eitems[q].size(), 256, 0, st>>>((const EaTile*)(D + o_e[q]), h->d_fronts,
                                                                      statics(h), A, EA_WIDE);
  CK(cudaGetLastError());
  if ((rc = factor_large_fronts(h, redo, A, dop))) return rc;
  if (!witems.empty())
    k_cb_w<<<(unsigned)witems.size(), 256, 0, st>>>((const TileItem*)(D + o_w), h->d_fronts, A);
  if (!gitems.empty())
    k_cb_gemm<<<(unsigned)gitems.size(), 128, 0, st>>>((const TileItem*)(D + o_g), h->d_fronts, A);
  for (int32_t s : big_cb) {
    const DFront& f = h->h_fronts[s];
    SyrkArgs ga{A.cbase + f.cb, f.nfs, A.scratch + f.scratch, f.nfs, A.panel + f.panel + f.k, f.m,
                0, f.nfs, 0, f.nfs, 0, &h->d_fronts[s].ne};
    if ((rc = launch_syrk(h, ga, f.k, false))) return rc;
  }
  k_get_counts<<<blocks_for(n, 128), 128, 0, st>>>(d_ids, n, h->d_fronts, (int32_t*)(D + o_cnt), nullptr);
  int32_t* hc = (int32_t*)h->h_stage2;
  CK(cudaMemcpyAsync(hc, D + o_cnt, (size_t)3 * n * 4, cudaMemcpyDeviceToHost, st));
  const double ts0 = now_ms();
  CK(cudaStreamSynchronize(st));
  h->host_sync_ms += now_ms() - ts0;
  for (int i = 0; i < n; ++i) {
    DFront& f = h->h_fronts[redo[i]];
    f.ne = hc[3 * i]; f.n1 = hc[3 * i + 1]; f.n2 = hc[3 * i + 2];
  }
  h->launches += 4 + (int64_t)maxch + (sitems.empty() ? 0 : 1);
  return RVG_OK;
}

// Launches of a wave's TPP fronts (one CTA each, k_tpp_cta), which sorts them
// by size, largest first.  A launch's CTAs all reserve the shared memory of its
// largest front, so the fronts are split where 8, 4, 2 or 1 of them fit on a
// multiprocessor (larger ones stay in global memory), and a smaller class joins
// the launch above it while that still runs in one go: a launch less, the same
// device time (100 fronts of order 80 and 300 of order 24: 113 us together, 110
// apart; 50 of 110 and 200 of 24: 171 and 171).
//
// Threads: 256.  A front's steps are latency bound, and where 4 CTAs or fewer
// share a multiprocessor its issue slots are not (us, 256 / 128 / 64 threads: 600
// fronts of order 80 236 / 281 / 419, 600 of 160 1449 / 2188 / 3843, in global
// memory 600 of 200 1930 / 2409 / 4222).  Small fronts (27 KB) fit 8 to a
// multiprocessor but their registers only at 128 threads, and fewer warps waste
// fewer issue slots on the decisions every warp repeats: 128 above two CTAs a
// multiprocessor (order 24: 296 fronts 40 / 42 / 50 and 600 64 / 46 / 52; order
// 55: 296 81 / 91 / 124, 600 145 / 112 / 136), 64 where they come in several
// rounds and are short (1800 of 40 212 / 149 / 130, of 55 306 / 224 / 261).
struct TppLaunch { int first, count, threads; size_t smem; };

// classes of at most `bytes` per front, of which `ctas` fit on a multiprocessor
struct TppClass { size_t bytes; int ctas; };
constexpr TppClass TPP_CLASS[4] = {{TPP_SMEM_MAX, 1}, {112 * 1024, 2}, {55 * 1024, 4}, {27 * 1024, 8}};
constexpr bool tpp_class_fits(const TppClass& c, int threads) {  // 228 KB, of which 1 KB a CTA is the system's
  return (c.bytes + 1024 + 128) * c.ctas <= 228 * 1024 && c.ctas * threads <= TPP_CTAS * TPP_MAX_T;
}
static_assert(tpp_class_fits(TPP_CLASS[0], 256) && tpp_class_fits(TPP_CLASS[1], 256) &&
                  tpp_class_fits(TPP_CLASS[2], 256) && tpp_class_fits(TPP_CLASS[3], 128),
              "TPP classes by the CTAs that fit");

std::vector<TppLaunch> plan_tpp(const rvg_handle* h, std::vector<int32_t>& ids) {
  std::vector<TppLaunch> out;
  if (ids.empty()) return out;
  auto bytes = [&](int32_t s) {
    const DFront& f = h->h_fronts[s];
    return (size_t)tpp_ld(f.m) * f.k * 8 + (size_t)f.k * 4;
  };
  std::stable_sort(ids.begin(), ids.end(), [&](int32_t a, int32_t b) { return bytes(a) > bytes(b); });
  const int n = (int)ids.size();
  int i = 0;
  while (i < n) {
    const size_t b = bytes(ids[i]);
    int c = 3;  // -1: global memory
    while (c >= 0 && b > TPP_CLASS[c].bytes) --c;
    int e = i;
    while (e < n && (c == 3 || bytes(ids[e]) > TPP_CLASS[c + 1].bytes)) ++e;
    if (c >= 0 && n - i <= TPP_CLASS[c].ctas * h->nsm) e = n;  // the rest fits beside it
    TppLaunch t{i, e - i, 256, c < 0 ? 0 : b};
    if (c == 3 && t.count > 2 * h->nsm)
      t.threads = t.count > TPP_CLASS[c].ctas * h->nsm && b <= 18 * 1024 ? 64 : 128;
    out.push_back(t);
    i = e;
  }
  return out;
}

// The numeric factorization proper: the level-set schedule of
// factor_tree_levelset (numeric.rs:1957-2163) with every front of a wave
// processed by the same launches.
int run_factor(rvg_handle* h, const double* d_vals, const double* d_scal) {
  Plan& P = h->P;
  cudaStream_t st = h->st;
  const int64_t ns = (int64_t)P.sn.size();
  h->factored = false;
  h->h_fronts.assign(ns, DFront());
  int64_t panel_used = 0, idx_used = 0, d_used = 0;
  std::vector<int64_t> cb_block(P.waves.size(), -1), cb_len(P.waves.size(), 0);
  std::vector<int64_t> cb_release_at(P.waves.size(), -1);
  h->cb_free.clear();
  if (h->cb_cap) h->cb_free[0] = (int64_t)h->cb_cap;
  const DevOpts dop = devopts(h->opt);
  const int ib = (int)h->opt.inner_block_size;
  double t_asm = 0, t_ker = 0, t_gem = 0;
  int rc;
  const double t_start = now_ms();
  h->host_alloc_ms = 0;
  h->host_sync_ms = 0;
  h->host_wait_ms = 0;
  h->host_gap_ms = 0;
  h->lf_misses = 0;
  h->lf_far = 0;
  h->ev_used = 0;
  h->mk_used = 0;
  for (double& v : h->part_ms) v = 0;
  h->syrk_flops = 0;
  h->syrk_ms = 0;
  h->syrk_launches = 0;
  h->launches = 0;
  h->peak_bytes = 0;
  if (h->opt.precision == 2) {
    if (!h->d_sel) { set_error("precision = 2 (learned) needs a selector: call rvg_set_selector first"); return RVG_ERR_INVALID_INPUT; }
    if ((rc = ensure(h->d_feat, h->d_feat_cap, (size_t)std::max<int64_t>(ns, 1) * FEAT_STRIDE, st))) return rc;
    if (!h->d_sel_flag) CK(cudaMalloc((void**)&h->d_sel_flag, sizeof(int32_t)));
    CK(cudaMemsetAsync(h->d_sel_flag, 0, sizeof(int32_t), st));
    h->route.assign(ns, 0);
    h->sel_large.clear();
    h->sel_routed = 0;
    h->sel_refactored = 0;
  }
  if (!h->replay) {
    h->rec_ok = false;
    h->rec_g.assign(ns, {});
    h->rec_stage.assign(P.waves.size(), 0);
  }
  CK(cudaEventRecord(h->ev[0], st));
  double t_ret = -1;  // host time the last wave synchronisation returned, until the next wave's first launch
  for (size_t w = 0; w < P.waves.size(); ++w) {
    const std::vector<int64_t>& wave = P.waves[w];
    const int nw = (int)wave.size();
    // ---- sizes from the children's eliminated counts (numeric.rs:1239-1262)
    int64_t panel_need = 0, idx_need = 0, d_need = 0, cb_need = 0, scratch_need = 0;
    std::vector<int32_t> dly0, dly_vals;  // the children's delay offsets, and each front's first
    for (int64_t s : wave) {
      DFront& f = h->h_fronts[s];
      dly0.push_back((int32_t)dly_vals.size());
      int64_t nown = P.sn[s].n_owned(), ndin = 0;
      for (int64_t c : P.children[s]) {
        DFront& cf = h->h_fronts[c];
        cf.dly_off = (int32_t)ndin;
        dly_vals.push_back((int32_t)ndin);
        ndin += cf.k - cf.ne;
      }
      int64_t k = nown + ndin, nfs = (int64_t)P.sn[s].pattern.size(), m = k + nfs;
      f.m = (int32_t)m; f.k = (int32_t)k; f.nown = (int32_t)nown; f.ndin = (int32_t)ndin; f.nfs = (int32_t)nfs;
      f.ne = 0; f.n1 = 0; f.n2 = 0;
      f.parent = (int32_t)P.sn[s].parent;
      f.flags = (P.sn[s].in_small_leaf ? FF_SMALL_LEAF : 0) | (f.parent >= 0 ? FF_HAS_PARENT : 0) |
                ((f.parent >= 0 && nfs > 0) ? FF_HAS_CB : 0);
      f.panel = panel_used + panel_need; panel_need += m * k;
      f.idx = idx_used + idx_need; idx_need += m + k;
      f.dpos = d_used + d_need; d_need += k;
      if (f.flags & FF_HAS_CB) cb_need += nfs * nfs;
    }
    {
      const int64_t T = h->opt.large_front_threshold;
      int64_t mid = 0;
      for (int64_t s : wave) {
        const DFront& f = h->h_fronts[s];
        if (!((f.flags & FF_SMALL_LEAF) || f.k < ib) && f.m >= T / 2 && f.m < T) ++mid;
      }
      std::vector<std::pair<int64_t, int64_t>> med;
      std::vector<int64_t> med_s;
      for (int64_t s : wave) {
        DFront& f = h->h_fronts[s];
        const bool tpp = (f.flags & FF_SMALL_LEAF) || f.k < ib;
        if (front_is_large(f.m, tpp, T, mid)) f.flags |= FF_LARGE;
        else if (!tpp) { med.emplace_back(f.m, f.k); med_s.push_back(s); }
      }
      for (int i : route_medium(med, T, h->opt.outer_block_size)) h->h_fronts[med_s[i]].flags |= FF_ROUTED;
      for (int64_t s : wave) {
        DFront& f = h->h_fronts[s];
        const int64_t m = f.m, k = f.k, nfs = f.nfs;
        const bool tpp = (f.flags & FF_SMALL_LEAF) || k < ib;
        const bool large = (f.flags & FF_LARGE) != 0;
        int64_t sc = tpp ? 0 : (2 * IBMAX * m + h->opt.outer_block_size);
        if (large || (f.flags & FF_ROUTED))
          sc = m * (2 * IBMAX + lf_window_blocks(h) * h->opt.outer_block_size) + h->opt.outer_block_size;
        if ((f.flags & FF_HAS_CB) && large) sc = std::max<int64_t>(sc, nfs * k);  // k_cb_w
        f.scratch = scratch_need; scratch_need += sc;
      }
    }
    double ta = now_ms();
    if (t_ret >= 0) {  // the stream has been empty since the last wave's synchronisation returned
      h->host_gap_ms += ta - t_ret;
      t_ret = -1;
    }
    if ((rc = arena_ensure(h, VM_PANEL, h->panel, h->panel_cap, (size_t)(panel_used + panel_need), st, true)))
      return rc;
    if ((rc = arena_ensure(h, VM_IDX, h->idx, h->idx_cap, (size_t)(idx_used + idx_need), st, true))) return rc;
    if ((rc = ensure_d_arrays(h, (size_t)(d_used + d_need)))) return rc;
    if ((rc = arena_ensure(h, VM_SCRATCH, h->scratch, h->scratch_cap, (size_t)std::max<int64_t>(scratch_need, 1), st,
                           false)))
      return rc;
    double* scratch = h->scratch;
    if (cb_need) {
      if ((rc = cb_alloc(h, cb_need, &cb_block[w]))) return rc;
      cb_len[w] = cb_need;
    }
    h->host_alloc_ms += now_ms() - ta;
    {
      int64_t off = cb_block[w];
      for (int64_t s : wave) {
        DFront& f = h->h_fronts[s];
        if (f.flags & FF_HAS_CB) { f.cb = off; off += (int64_t)f.nfs * f.nfs; }
        else f.cb = -1;
      }
    }
    if (panel_need) CK(cudaMemsetAsync(h->panel + panel_used, 0, (size_t)panel_need * 8, st));
    const Arenas A{h->panel, h->idx, h->dtype, h->ddiag, h->doff, scratch, h->cb_arena};
    // ---- launch data of the whole wave, packed into one upload
    std::vector<int32_t> ids(wave.begin(), wave.end()), tpp_ids, aptp_ids, large_ids, routed_ids;
    std::vector<DFront> staged;
    staged.reserve(nw);
    for (int64_t s : wave) {
      staged.push_back(h->h_fronts[s]);
      const DFront& f = h->h_fronts[s];
      if ((f.flags & FF_SMALL_LEAF) || f.k < ib) tpp_ids.push_back((int32_t)s);
      else if (f.flags & FF_LARGE) large_ids.push_back((int32_t)s);
      else if (f.flags & FF_ROUTED) routed_ids.push_back((int32_t)s);
      else aptp_ids.push_back((int32_t)s);
    }
    // medium fronts largest first (dense work ~ k m^2): the persistent launch starts the long ones early
    std::stable_sort(aptp_ids.begin(), aptp_ids.end(), [&](int32_t a, int32_t b) {
      const DFront &fa = h->h_fronts[a], &fb = h->h_fronts[b];
      return (double)fa.k * fa.m * fa.m > (double)fb.k * fb.m * fb.m;
    });
    const std::vector<TppLaunch> tpp_launches = plan_tpp(h, tpp_ids);
    int n_small_launches = 0;
    std::vector<ScatterItem> sitems;
    for (int64_t s : wave)
      for (int64_t e = P.amap_ptr[s]; e < P.amap_ptr[s + 1]; e += 256) sitems.push_back(ScatterItem{(int32_t)s, 0, e});
    size_t maxch = 0;
    for (int64_t s : wave) maxch = std::max(maxch, P.children[s].size());
    std::vector<std::vector<EaTile>> eitems(maxch);
    std::vector<int> ewidth(maxch, EA_WIDE);
    auto ea_items = [&](size_t q, int width) {
      eitems[q].clear();
      for (int64_t s : wave) {
        if (q >= P.children[s].size()) continue;
        int64_t c = P.children[s][q];
        const DFront& cf = h->h_fronts[c];
        if (!(cf.flags & FF_HAS_PARENT) || cf.ne >= cf.m) continue;
        int sz = cf.m - cf.ne;
        for (int j0 = 0; j0 < sz; j0 += width)
          for (int i0 = j0; i0 < sz; i0 += EA_ROWS) eitems[q].push_back(EaTile{(int32_t)s, (int32_t)c, j0, i0});
      }
    };
    for (size_t q = 0; q < maxch; ++q) {
      ea_items(q, EA_WIDE);
      if (eitems[q].size() < (size_t)h->nsm) ea_items(q, ewidth[q] = EA_NARROW);  // (up to 4 times as many: 4 per SM)
    }
    std::vector<CbZeroItem> zitems;
    for (int64_t s : wave) {
      const DFront& f = h->h_fronts[s];
      if ((f.flags & FF_HAS_CB) && f.nfs > WB_ZERO)
        for (int j0 = 0; j0 < f.nfs; j0 += 32) zitems.push_back(CbZeroItem{(int32_t)s, j0});
    }
    std::vector<TileItem> witems, gitems;
    std::vector<int64_t> cb_syrk_fronts;
    for (int64_t s : wave) {
      const DFront& f = h->h_fronts[s];
      if (!(f.flags & FF_HAS_CB) || f.k == 0) continue;
      if ((f.flags & FF_LARGE) && f.nfs >= 256) {  // GEMM by launch_syrk
        add_cb_w(witems, (int32_t)s, f);
        continue;
      }
      int nt = (f.nfs + GT - 1) / GT;
      for (int tj = 0; tj < nt; ++tj)
        for (int ti = tj; ti < nt; ++ti) gitems.push_back(TileItem{(int32_t)s, ti, tj, 0});
    }
    Packer pk;
    size_t o_staged = pk.add(staged), o_ids = pk.add(ids), o_dly0 = pk.add(dly0), o_dly_vals = pk.add(dly_vals);
    size_t o_tpp = pk.add(tpp_ids), o_aptp = pk.add(aptp_ids), o_s = pk.add(sitems);
    std::vector<size_t> o_e(maxch);
    for (size_t q = 0; q < maxch; ++q) o_e[q] = pk.add(eitems[q]);
    size_t o_w = pk.add(witems), o_g = pk.add(gitems), o_z = pk.add(zitems);
    size_t o_cnt = pk.add(std::vector<int32_t>(3 * (size_t)nw + 4, 0));
    size_t o_q = pk.add(std::vector<int32_t>(4, 0));  // work-queue counter of the medium fronts' launch
    const bool learned = h->opt.precision == 2 && !large_ids.empty();
    size_t o_lg = 0, o_rt = 0;
    if (learned) {
      o_lg = pk.add(large_ids);
      o_rt = pk.add(std::vector<int32_t>(large_ids.size(), 0));
    }
    if ((rc = arena_ensure(h, VM_STAGE, h->d_stage, h->stage_cap, pk.buf.size(), st, true))) return rc;
    char* hs;
    if (h->replay) {  // a slice of its own: the graph copies from it at every replay
      if (pk.buf.size() != h->rec_stage[w]) { set_error("refactorization replay: launch data differ"); return RVG_ERR_DEVICE; }
      hs = h->h_stage_all + h->stage_off[w];
    } else {
      if ((rc = ensure_host(h->h_stage, h->h_stage_cap, pk.buf.size()))) return rc;
      hs = h->h_stage;
      h->rec_stage[w] = pk.buf.size();
    }
    std::memcpy(hs, pk.buf.data(), pk.buf.size());
    CK(cudaMemcpyAsync(h->d_stage, hs, pk.buf.size(), cudaMemcpyHostToDevice, st));
    char* D = h->d_stage;
    const int32_t* d_ids = (const int32_t*)(D + o_ids);
    // ---- descriptors, row lists, small contribution blocks
    k_wave_begin<<<nw, 128, 0, st>>>((const DFront*)(D + o_staged), d_ids, (const int32_t*)(D + o_dly0),
                                     (const int32_t*)(D + o_dly_vals), h->d_fronts, statics(h), A);
    // the larger contribution blocks of this wave: zero lower triangles (the extend-add adds into them)
    if (!zitems.empty())
      k_zero_cb_lower<<<(unsigned)zitems.size(), 256, 0, st>>>((const CbZeroItem*)(D + o_z), h->d_fronts, A);
    CK(cudaEventRecord(h->ev[1], st));
    // ---- assembly
    if (!sitems.empty())
      k_scatter<<<(unsigned)sitems.size(), 256, 0, st>>>((const ScatterItem*)(D + o_s), h->d_fronts, statics(h), A,
                                                         d_vals, d_scal);
    for (size_t q = 0; q < maxch; ++q)
      if (!eitems[q].empty())
        k_extend_add_tiled<<<(unsigned)eitems[q].size(), 256, 0, st>>>((const EaTile*)(D + o_e[q]), h->d_fronts,
                                                                        statics(h), A, ewidth[q]);
    CK(cudaEventRecord(h->ev[2], st));
    // contribution blocks whose parents are now all assembled
    for (size_t w2 = 0; w2 < w; ++w2)
      if (cb_block[w2] >= 0 && cb_release_at[w2] == (int64_t)w) { cb_release(h, cb_block[w2], cb_len[w2]); cb_block[w2] = -1; }
    // ---- learned precision: features of the assembled large fronts, the
    // selector's route for each (read back: it picks the launches below)
    if (learned) {
      const int nl = (int)large_ids.size();
      const int32_t* d_lg = (const int32_t*)(D + o_lg);
      int32_t* d_rt = (int32_t*)(D + o_rt);
      int64_t kmax = 0;
      for (int32_t s : large_ids) kmax = std::max<int64_t>(kmax, h->h_fronts[s].k);
      k_feat_init<<<1, 256, 0, st>>>(d_lg, nl, h->d_feat);
      k_front_features<<<dim3((unsigned)((kmax + 7) / 8), (unsigned)nl), 256, 0, st>>>(d_lg, h->d_fronts, A,
                                                                                     h->opt.threshold, h->d_feat);
      k_mlp_route<<<nl, 32, 0, st>>>(d_lg, nl, h->d_fronts, h->d_sel, h->sel_thresh, h->sel_force_fp64 ? 1 : 0,
                                    h->d_feat, d_rt);
      CK(cudaGetLastError());
      if ((rc = ensure_host((char*&)h->h_counts, h->h_counts_cap, (size_t)(std::max(3 * nw + 4, nl)) * 4))) return rc;
      CK(cudaMemcpyAsync(h->h_counts, d_rt, (size_t)nl * 4, cudaMemcpyDeviceToHost, st));
      CK(cudaEventRecord(h->ev[6], st));  // read below, once the wave's small and medium fronts are queued
      h->launches += 3;
    }
    // ---- dense factorization
    mark(h, -1);
    // large fronts beside the small and medium ones (one after the other while the profiling marks are on).
    // Beside: up to two medium fronts a multiprocessor, which all run from the start; the queue's CTAs fill
    // the GPU then, and of a longer queue the large fronts see the end only (one of order 1500 with 296 fronts of
    // order 300: 2.5 ms; 1500 such fronts alone 4.5, with it 5.7)
    std::vector<int32_t> lf_ids(large_ids);
    lf_ids.insert(lf_ids.end(), routed_ids.begin(), routed_ids.end());
    const bool beside = !lf_ids.empty() && !(aptp_ids.empty() && tpp_ids.empty()) && !h->profiling;
    if (beside) {
      if (!h->ev_beside) CK(cudaEventCreateWithFlags(&h->ev_beside, cudaEventDisableTiming));
      CK(cudaEventRecord(h->ev_beside, st));
    }
    // the wave's small and medium fronts (profiling: part "aptp")
    bool group = false;  // a launch of the group has gone out: the next ones may start beside it
    if (!aptp_ids.empty()) {
      if (!h->aptp_ctas) {  // resident CTAs of the queue kernel on this device
        int occ = 0;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_front_queue, NT, 0));
        h->aptp_ctas = std::max(1, occ) * std::max(1, h->nsm);
      }
      const int na = (int)aptp_ids.size();
      k_front_queue<<<(unsigned)std::min(na, h->aptp_ctas), NT, 0, st>>>((const int32_t*)(D + o_aptp), na,
                                                                          (int32_t*)(D + o_q), h->d_fronts, A, dop);
      group = true;
      n_small_launches++;
    }
    for (const TppLaunch& t : tpp_launches) {
      launch_beside(group, t.smem ? k_tpp_cta<true> : k_tpp_cta<false>, (unsigned)t.count, (unsigned)t.threads, t.smem,
                    st, (const int32_t*)(D + o_tpp) + t.first, h->d_fronts, A, dop);
      group = true;
      n_small_launches++;
    }
    mark(h, RVG_PART_APTP);
    if (learned) {  // the routes of the large fronts (the device is busy with the fronts queued above)
      const int nl = (int)large_ids.size();
      const double ts0 = now_ms();
      CK(cudaEventSynchronize(h->ev[6]));
      h->host_wait_ms += now_ms() - ts0;
      for (int i = 0; i < nl; ++i) {
        h->route[large_ids[i]] = (int8_t)(h->h_counts[i] != 0);
        h->sel_routed += h->h_counts[i] != 0;
      }
      h->sel_large.insert(h->sel_large.end(), large_ids.begin(), large_ids.end());
    }
    const bool counted = large_ids.size() == 1;
    if (counted && !routed_ids.empty() && h->profiling) {  // the large front alone: it carries the profiling marks
      if ((rc = factor_large_fronts(h, large_ids, A, dop)) || (rc = factor_large_fronts(h, routed_ids, A, dop)))
        return rc;
    } else if ((rc = factor_large_fronts(h, lf_ids, A, dop, beside ? h->ev_beside : nullptr, counted))) {
      return rc;
    }
    CK(cudaEventRecord(h->ev[3], st));
    // ---- contribution GEMM (fronts with nothing eliminated skip inside)
    mark(h, -1);
    if (!witems.empty())
      k_cb_w<<<(unsigned)witems.size(), 256, 0, st>>>((const TileItem*)(D + o_w), h->d_fronts, A);
    mark(h, RVG_PART_CB_W);
    if (!gitems.empty())
      k_cb_gemm<<<(unsigned)gitems.size(), 128, 0, st>>>((const TileItem*)(D + o_g), h->d_fronts, A);
    mark(h, RVG_PART_CB_GEMM);
    for (int64_t s : wave) {
      const DFront& f = h->h_fronts[s];
      if (!(f.flags & FF_HAS_CB) || f.k == 0 || !((f.flags & FF_LARGE) && f.nfs >= 256)) continue;
      SyrkArgs ga{A.cbase + f.cb, f.nfs, A.scratch + f.scratch, f.nfs, A.panel + f.panel + f.k, f.m,
                  0, f.nfs, 0, f.nfs, 0, &h->d_fronts[s].ne};
      if ((rc = launch_syrk(h, ga, f.k, front_mixed(h, s)))) return rc;
      mark(h, RVG_PART_CB_SYRK);
      cb_syrk_fronts.push_back(s);
    }
    if (learned) {
      k_front_growth<<<(unsigned)large_ids.size(), 256, 0, st>>>((const int32_t*)(D + o_lg), h->d_fronts, A,
                                                                 h->sel_bound, h->d_feat, h->d_sel_flag,
                                                                 (int32_t*)(D + o_rt));
      h->launches++;
    }
    CK(cudaEventRecord(h->ev[4], st));
    CK(cudaGetLastError());
    // ---- eliminated counts back to the host (replay: the recorded ones, checked on the device)
    if (h->replay) {
      k_check_counts<<<blocks_for(nw, 128), 128, 0, st>>>(d_ids, nw, h->d_fronts, h->d_rec, h->d_mismatch);
      CK(cudaGetLastError());
      for (int i = 0; i < nw; ++i) {
        DFront& f = h->h_fronts[wave[i]];
        const int32_t* r = &h->rec_cnt[3 * (size_t)wave[i]];
        f.ne = r[0]; f.n1 = r[1]; f.n2 = r[2];
      }
      for (int64_t s : cb_syrk_fronts) {
        const DFront& f = h->h_fronts[s];
        h->syrk_flops += 2.0 * (double)f.ne * (double)f.nfs * (double)(f.nfs + 1) / 2.0;
      }
      int64_t last = -1;
      for (int64_t s : wave) if (P.sn[s].parent >= 0) last = std::max(last, P.height[P.sn[s].parent]);
      cb_release_at[w] = last;
      panel_used += panel_need; idx_used += idx_need; d_used += d_need;
      continue;
    }
    k_get_counts<<<blocks_for(nw, 128), 128, 0, st>>>(d_ids, nw, h->d_fronts, (int32_t*)(D + o_cnt), h->d_err);
    const size_t nlr = learned ? large_ids.size() : 0;  // the large fronts' routes after the growth check
    if ((rc = ensure_host((char*&)h->h_counts, h->h_counts_cap, (size_t)(3 * nw + 4 + nlr) * 4))) return rc;
    CK(cudaMemcpyAsync(h->h_counts, D + o_cnt, (size_t)(3 * nw + 1) * 4, cudaMemcpyDeviceToHost, st));
    if (nlr) CK(cudaMemcpyAsync(h->h_counts + 3 * nw + 4, D + o_rt, nlr * 4, cudaMemcpyDeviceToHost, st));
    {
      double ts0 = now_ms();
      CK(cudaStreamSynchronize(st));
      t_ret = now_ms();
      h->host_sync_ms += t_ret - ts0;
    }
    mark_flush(h);
    if (h->h_counts[3 * nw]) {
      CK(cudaMemsetAsync(h->d_err, 0, sizeof(int32_t), st));
      set_error("a tensor-core Schur update gave up waiting on its pipeline (device timeout)");
      return RVG_ERR_DEVICE_TIMEOUT;
    }
    for (int i = 0; i < nw; ++i) {
      DFront& f = h->h_fronts[wave[i]];
      f.ne = h->h_counts[3 * i]; f.n1 = h->h_counts[3 * i + 1]; f.n2 = h->h_counts[3 * i + 2];
    }
    if (nlr) {
      std::vector<int32_t> redo;
      for (size_t i = 0; i < nlr; ++i)
        if (h->h_counts[3 * nw + 4 + i] == 2) redo.push_back(large_ids[i]);
      if (!redo.empty() && (rc = refactor_fp64(h, redo, A, dop, d_vals, d_scal))) return rc;
    }
    for (int64_t s : cb_syrk_fronts) {
      const DFront& f = h->h_fronts[s];
      h->syrk_flops += 2.0 * (double)f.ne * (double)f.nfs * (double)(f.nfs + 1) / 2.0;
    }
    h->launches += 1 + (int64_t)eitems.size() * 0 + (sitems.empty() ? 0 : 1) +
                   n_small_launches + (witems.empty() ? 0 : 1) + (gitems.empty() ? 0 : 1) + 2 +
                   (zitems.empty() ? 0 : 1);
    for (size_t q = 0; q < maxch; ++q) h->launches += eitems[q].empty() ? 0 : 1;
    if (h->profiling) {  // the device memory in use (profiling runs only: the query costs host time)
      size_t fb = 0, tb = 0;
      cudaMemGetInfo(&fb, &tb);
      h->peak_bytes = std::max<int64_t>(h->peak_bytes, (int64_t)(tb - fb));
    }
    int64_t last = -1;
    for (int64_t s : wave) if (P.sn[s].parent >= 0) last = std::max(last, P.height[P.sn[s].parent]);
    cb_release_at[w] = last;
    float a1 = 0, a2 = 0, a3 = 0;
    cudaEventElapsedTime(&a1, h->ev[1], h->ev[2]);
    cudaEventElapsedTime(&a2, h->ev[2], h->ev[3]);
    cudaEventElapsedTime(&a3, h->ev[3], h->ev[4]);
    t_asm += a1; t_ker += a2; t_gem += a3;
    panel_used += panel_need; idx_used += idx_need; d_used += d_need;
  }
  for (size_t w = 0; w < cb_block.size(); ++w)
    if (cb_block[w] >= 0) { cb_release(h, cb_block[w], cb_len[w]); cb_block[w] = -1; }
  CK(cudaEventRecord(h->ev[5], st));
  if (h->replay) {
    if (d_used != h->rec_d_used) { set_error("refactorization replay: sizes differ"); return RVG_ERR_DEVICE; }
    return RVG_OK;  // captured; the statistics follow each replay (finish_factor)
  }
  h->factor_launches = h->launches;
  h->host_total_ms = now_ms() - t_start;
  h->rec_cnt.assign(3 * ns, 0);
  for (int64_t s = 0; s < ns; ++s) {
    const DFront& f = h->h_fronts[s];
    h->rec_cnt[3 * s] = f.ne; h->rec_cnt[3 * s + 1] = f.n1; h->rec_cnt[3 * s + 2] = f.n2;
  }
  h->rec_d_used = d_used;
  h->t_assembly = t_asm; h->t_kernel = t_ker; h->t_gemm = t_gem;
  rc = finish_factor(h, d_used);
  if (rc) return rc;
  h->rec_ok = true;
  return RVG_OK;
}

// Host side of the end of a factorization (dynamic or replayed): the total
// time, the Schur GEMM time of the profiling events, the aggregate statistics.
int finish_factor(rvg_handle* h, int64_t d_used) {
  cudaStream_t st = h->st;
  const int64_t ns = (int64_t)h->P.sn.size();
  // aggregate stats (numeric.rs:929-1009)
  h->tot1 = h->tot2 = h->totdel = h->zero_piv = h->max_front = 0;
  h->inertia[0] = h->inertia[1] = h->inertia[2] = 0;
  unsigned long long* hc = (unsigned long long*)h->h_norms;
  if (d_used) {
    if (!h->d_dcount) CK(cudaMalloc((void**)&h->d_dcount, 4 * sizeof(unsigned long long)));
    CK(cudaMemsetAsync(h->d_dcount, 0, 4 * sizeof(unsigned long long), st));
    const Arenas A{h->panel, h->idx, h->dtype, h->ddiag, h->doff, nullptr, h->cb_arena};
    k_d_counts<<<(unsigned)std::min<int64_t>((ns + 7) / 8, 4 * h->nsm), 256, 0, st>>>(h->d_fronts, ns, A, h->d_dcount);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(hc, h->d_dcount, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
  }
  CK(cudaStreamSynchronize(st));
  if (d_used) {
    for (int q = 0; q < 3; ++q) h->inertia[q] = (int64_t)hc[q];
    h->zero_piv = (int64_t)hc[3];
  }
  float tot = 0;
  cudaEventElapsedTime(&tot, h->ev[0], h->ev[5]);
  h->t_factor = tot;
  if (h->profiling)
    for (size_t e = 0; e + 1 < h->ev_used; e += 2) {
      float ms = 0;
      cudaEventElapsedTime(&ms, h->ev_pool[e], h->ev_pool[e + 1]);
      h->syrk_ms += ms;
    }
  for (int64_t s = 0; s < ns; ++s) {
    const DFront& f = h->h_fronts[s];
    h->tot1 += f.n1; h->tot2 += f.n2; h->totdel += f.k - f.ne;
    h->max_front = std::max<int64_t>(h->max_front, f.m);
  }
  h->factored = true;
  return RVG_OK;
}

}  // namespace

// ===========================================================================
// C ABI (numeric part)
// ===========================================================================
extern "C" {

const char* rvg_last_error(void) { return g_err.c_str(); }

void rvg_default_options(rvg_options* o) {
  o->threshold = 0.01;
  o->small = 1e-20;
  o->outer_block_size = 256;
  o->inner_block_size = 32;
  o->nemin = 32;
  o->small_leaf_threshold = 256;
  o->failed_pivot_tpp = 1;
  o->fallback_bk = 1;
  o->large_front_threshold = 2048;
  o->precision = 0;
  o->mixed_flush = 4;
  o->mixed_tile_cols = 256;
  o->mixed_operands = 0;
  o->graph_refactor = 0;
  o->far_field_sms = -1;
  o->mixed_window = 0;
}

static int check_opts(const rvg_options& o) {  // factor.rs:307-347 (precision and below: no counterpart)
  if (!(o.threshold > 0.0 && o.threshold <= 1.0)) { set_error("threshold must be in (0, 1]"); return RVG_ERR_INVALID_INPUT; }
  if (!(o.small >= 0.0)) { set_error("small must be >= 0.0"); return RVG_ERR_INVALID_INPUT; }
  if (o.outer_block_size <= 0) { set_error("outer_block_size must be > 0"); return RVG_ERR_INVALID_INPUT; }
  if (o.inner_block_size <= 0) { set_error("inner_block_size must be > 0"); return RVG_ERR_INVALID_INPUT; }
  if (o.inner_block_size > o.outer_block_size) {
    set_error("inner_block_size must be <= outer_block_size");
    return RVG_ERR_INVALID_INPUT;
  }
  if (o.inner_block_size > IBMAX) { set_error("inner_block_size above 32 is not supported by the B200 kernels"); return RVG_ERR_INVALID_INPUT; }
  if (o.nemin < 1) { set_error("nemin must be >= 1"); return RVG_ERR_INVALID_INPUT; }
  if (o.large_front_threshold < 1) { set_error("large_front_threshold must be >= 1"); return RVG_ERR_INVALID_INPUT; }
  if (o.precision < 0 || o.precision > 2) { set_error("precision must be 0 (FP64), 1 (mixed) or 2 (learned)"); return RVG_ERR_INVALID_INPUT; }
  if (o.mixed_flush != 0 && o.mixed_flush != 1 && o.mixed_flush != 2 && o.mixed_flush != 4 && o.mixed_flush != 8) {
    set_error("mixed_flush must be 0, 1, 2, 4 or 8");
    return RVG_ERR_INVALID_INPUT;
  }
  if (o.mixed_operands != 0 && o.mixed_operands != 1) {
    set_error("mixed_operands must be 0 (TF32) or 1 (BF16)");
    return RVG_ERR_INVALID_INPUT;
  }
  if (o.mixed_tile_cols != 128 && o.mixed_tile_cols != 256) {
    set_error("mixed_tile_cols must be 128 or 256");
    return RVG_ERR_INVALID_INPUT;
  }
  if (o.far_field_sms < -1) { set_error("far_field_sms must be -1 (default), 0 (no split) or a count"); return RVG_ERR_INVALID_INPUT; }
  if (o.mixed_window < 0 || o.mixed_window > LF_WINDOW_MAX) {
    set_error("mixed_window must be 0 (default) or 1 to 8 outer blocks");
    return RVG_ERR_INVALID_INPUT;
  }
  if (o.graph_refactor < 0 || o.graph_refactor > 2) {
    set_error("graph_refactor must be 0 (off), 1 (replay) or 2 (replay, arenas kept at their addresses across rvg_trim)");
    return RVG_ERR_INVALID_INPUT;
  }
  return RVG_OK;
}

rvg_status rvg_create(int64_t n, int64_t nsup, const int64_t* sup_begin, const int64_t* sup_end, const int64_t* pat_ptr,
                      const int64_t* pat_idx, const int64_t* sup_parent, const int64_t* perm_fwd, const int64_t* colptr,
                      const int64_t* rowidx, const rvg_options* opt, rvg_handle** out) {
  if (!out) { set_error("null output handle"); return RVG_ERR_INVALID_INPUT; }
  *out = nullptr;
  rvg_options o;
  rvg_default_options(&o);
  if (opt) o = *opt;
  int rc = check_opts(o);
  if (rc) return (rvg_status)rc;
  if (n < 0 || nsup < 0) { set_error("negative size"); return RVG_ERR_INVALID_INPUT; }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    set_error("no CUDA device available (the numeric phase has no CPU fallback)");
    return RVG_ERR_DEVICE;
  }
  std::unique_ptr<rvg_handle> h(new rvg_handle());
  h->opt = o;
  h->nnz = n ? colptr[n] : 0;
  std::string err;
  rc = build_plan(nullptr, n, nsup, sup_begin, sup_end, pat_ptr, pat_idx, sup_parent, perm_fwd, colptr, rowidx, o, h->P, &err);
  if (rc) { set_error(err); return (rvg_status)rc; }
  CK(cudaGetDevice(&h->device));
  CK(cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking));
  for (auto& e : h->ev) CK(cudaEventCreate(&e));
  {
    cudaMemPool_t pool;
    CK(cudaDeviceGetDefaultMemPool(&pool, h->device));
    uint64_t thr = UINT64_MAX;
    CK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr));
  }
  Plan& P = h->P;
  const int64_t ns = (int64_t)P.sn.size();
  std::vector<int64_t> chp(ns + 1, 0);
  std::vector<int32_t> chi;
  for (int64_t s = 0; s < ns; ++s) {
    chp[s + 1] = chp[s] + (int64_t)P.children[s].size();
    for (int64_t c : P.children[s]) chi.push_back((int32_t)c);
  }
  cudaStream_t st = h->st;
  if ((rc = upload(h->d_own_ptr, P.own_ptr, st)) || (rc = upload(h->d_own_idx, P.own_idx, st)) ||
      (rc = upload(h->d_pat_ptr, P.pat_ptr, st)) || (rc = upload(h->d_pat_idx, P.pat_idx, st)) ||
      (rc = upload(h->d_amap_ptr, P.amap_ptr, st)) || (rc = upload(h->d_amap, P.amap, st)) ||
      (rc = upload(h->d_ea_ptr, P.ea_ptr, st)) || (rc = upload(h->d_ea_map, P.ea_map, st)) ||
      (rc = upload(h->d_ch_ptr, chp, st)) || (rc = upload(h->d_ch_idx, chi, st)) ||
      (rc = upload(h->d_pfwd, P.perm_fwd, st)))
    return (rvg_status)rc;
  CK(cudaMallocAsync((void**)&h->d_fronts, std::max<int64_t>(ns, 1) * sizeof(DFront), st));
  CK(cudaMallocAsync((void**)&h->d_lf, sizeof(LFState), st));
  {
    std::vector<int64_t> cp(colptr, colptr + n + 1);
    std::vector<int32_t> ri(rowidx, rowidx + h->nnz);
    if ((rc = upload(h->d_colptr, cp, st)) || (rc = upload(h->d_rowidx, ri, st))) return (rvg_status)rc;
  }
  CK(cudaMallocHost((void**)&h->h_norms, 4 * sizeof(double)));
  if (o.graph_refactor == 2 && (rc = vm_create(h.get()))) return (rvg_status)rc;  // address-stable arenas
  if ((rc = presize_arenas(h.get()))) return (rvg_status)rc;
  CK(cudaFuncSetAttribute(k_lf_prop, cudaFuncAttributeMaxDynamicSharedMemorySize, LF_PROP_SMEM_MAX));
  CK(cudaFuncSetAttribute(k_tpp_cta<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TPP_SMEM_MAX));
  CK(cudaFuncSetAttribute(k_syrk_lower, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<1, TC_TF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<2, TC_TF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<4, TC_TF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<8, TC_TF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<TC_NO_FLUSH, TC_TF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc_pair<TC_TF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TP_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<1, TC_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<2, TC_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<4, TC_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<8, TC_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc<TC_NO_FLUSH, TC_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
  CK(cudaFuncSetAttribute(k_syrk_tc_pair<TC_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TP_SMEM));
  CK(cudaDeviceGetAttribute(&h->nsm, cudaDevAttrMultiProcessorCount, h->device));
  {  // RVG_CHAIN_PDL=0 launches the large-front chain kernels plainly (same results; for timing comparisons)
    const char* e = std::getenv("RVG_CHAIN_PDL");
    h->chain_pdl = !(e && e[0] == '0');
  }

  CK(cudaMallocAsync((void**)&h->d_err, sizeof(int32_t), st));
  CK(cudaMemsetAsync(h->d_err, 0, sizeof(int32_t), st));
  CK(cudaMallocAsync((void**)&h->d_vals, std::max<int64_t>(h->nnz, 1) * 8, st));
  CK(cudaMallocAsync((void**)&h->d_scal, std::max<int64_t>(n, 1) * 8, st));
  CK(cudaStreamSynchronize(st));
  *out = h.release();
  return RVG_OK;
}

static int device_wait_status(rvg_handle* h);

static void drop_graph(rvg_handle* h) {
  if (h->gexec) cudaGraphExecDestroy(h->gexec);
  if (h->graph) cudaGraphDestroy(h->graph);
  h->gexec = nullptr;
  h->graph = nullptr;
}

// Refactorization as one CUDA graph launch.  The first call after a dynamic
// factorization captures run_factor with every host decision taken from that
// factorization's record (front sizes, eliminated counts, the large fronts'
// progress per outer block) and the launch data of each wave in a pinned slice
// of its own; device checks compare what the replayed factorization actually
// eliminated with the record.  Later calls launch the graph.  *done = false
// (and the graph dropped) when the checks saw another decision, when a buffer
// would have to grow, or when capture fails: the caller then factors
// dynamically, which records again.  The results are the dynamic path's.
static int replay_factor(rvg_handle* h, const double* ds, bool* done) {
  *done = false;
  cudaStream_t st = h->st;
  if (h->gexec && h->graph_ds != ds) drop_graph(h);
  if (!h->gexec) {
    // device copy of the recorded counts, the mismatch word, the pinned launch data
    const size_t nc = h->rec_cnt.size();
    int rc;
    if ((rc = ensure(h->d_rec, h->d_rec_cap, std::max<size_t>(nc, 1), st))) return rc;
    if (!h->d_mismatch) CK(cudaMalloc((void**)&h->d_mismatch, sizeof(int32_t)));
    if (nc) CK(cudaMemcpyAsync(h->d_rec, h->rec_cnt.data(), nc * 4, cudaMemcpyHostToDevice, st));
    h->stage_off.assign(h->rec_stage.size(), 0);
    size_t tot = 0;
    for (size_t w = 0; w < h->rec_stage.size(); ++w) { h->stage_off[w] = tot; tot += (h->rec_stage[w] + 255) & ~size_t(255); }
    if ((rc = ensure_host(h->h_stage_all, h->h_stage_all_cap, std::max<size_t>(tot, 1)))) return rc;
    CK(cudaStreamSynchronize(st));
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    h->replay = true;
    tl_no_alloc = true;
    rc = run_factor(h, h->d_vals, ds);
    tl_no_alloc = false;
    h->replay = false;
    const cudaError_t ec = cudaStreamEndCapture(st, &g);
    if (rc || ec != cudaSuccess || !g) {
      if (g) cudaGraphDestroy(g);
      cudaGetLastError();
      h->rec_ok = false;
      return RVG_OK;  // not replayable: factor dynamically
    }
    if (cudaGraphInstantiate(&h->gexec, g, 0) != cudaSuccess) {
      cudaGraphDestroy(g);
      cudaGetLastError();
      h->gexec = nullptr;
      h->rec_ok = false;
      return RVG_OK;
    }
    h->graph = g;
    h->graph_ds = ds;
  }
  CK(cudaMemsetAsync(h->d_mismatch, 0, sizeof(int32_t), st));
  const double t0 = now_ms();
  h->ev_used = 0;  // no per-launch events inside the graph
  CK(cudaEventRecord(h->ev[0], st));  // (the records inside the capture only ordered the capture)
  CK(cudaGraphLaunch(h->gexec, st));
  CK(cudaEventRecord(h->ev[5], st));
  int32_t mis = 0;
  CK(cudaMemcpyAsync(&mis, h->d_mismatch, 4, cudaMemcpyDeviceToHost, st));
  int rc = finish_factor(h, h->rec_d_used);  // synchronises
  if (rc) return rc;
  if ((rc = device_wait_status(h))) return rc;
  h->host_total_ms = now_ms() - t0;
  for (double& v : h->part_ms) v = 0;
  if (mis) {  // another decision than the recorded one: this factor is not valid
    h->factored = false;
    drop_graph(h);
    h->rec_ok = false;
    return RVG_OK;
  }
  h->factor_launches = 1;
  h->host_sync_ms = 0;
  h->host_wait_ms = 0;
  h->host_gap_ms = 0;
  h->lf_misses = 0;
  h->lf_far = 0;
  *done = true;
  return RVG_OK;
}

static int factor_common(rvg_handle* h, const double* dv, const double* ds) {
  int rc;
  h->sf.ok = false;  // the solve's layout is the last factorization's
  if (h->need_presize) {  // after rvg_trim: the arenas at their delay-free size again
    if ((rc = presize_arenas(h))) return rc;
    if (h->vm && (rc = vm_restore(h))) return rc;  // (address-stable: up to their largest size, all of them)
    h->need_presize = false;
  }
  // the refinement needs the unfactored values and ||A||_F
  if (dv != h->d_vals && h->nnz) CK(cudaMemcpyAsync(h->d_vals, dv, h->nnz * 8, cudaMemcpyDeviceToDevice, h->st));
  // NaN or Inf in the values or the scaling: a clean InvalidInput before any factor kernel runs (the
  // reference rejects them in its MC64 scaling, ordering/matching.rs:143-157)
  // (and ||A||_F from the same read)
  h->a_fro = 0;
  if (h->nnz || (ds && h->P.n)) {
    if (!h->d_scan) CK(cudaMalloc((void**)&h->d_scan, sizeof(ScanOut)));
    CK(cudaMemsetAsync(h->d_scan, 0, sizeof(ScanOut), h->st));
    if (h->nnz) k_scan_values<<<296, 256, 0, h->st>>>(h->d_vals, h->nnz, h->d_scan, 1);
    if (ds && h->P.n) k_scan_values<<<296, 256, 0, h->st>>>(ds, h->P.n, h->d_scan, 0);
    CK(cudaGetLastError());
    const ScanOut* sc = (const ScanOut*)h->h_norms;
    CK(cudaMemcpyAsync(h->h_norms, h->d_scan, sizeof(ScanOut), cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
    if (sc->bad) {
      h->factored = false;
      set_error("the matrix values or the scaling contain NaN or Inf");
      return RVG_ERR_INVALID_INPUT;
    }
    h->a_fro = std::sqrt(sc->sum);
  }
  bool done = false;
  if (h->opt.graph_refactor && h->rec_ok && h->opt.precision != 2) {
    if ((rc = replay_factor(h, ds, &done))) return rc;
  }
  if (!done) {
    drop_graph(h);  // a dynamic run may move buffers: the next refactorization captures anew
    rc = run_factor(h, h->d_vals, ds);
    if (rc) return rc;
  }
  if (h->opt.precision == 2) {
    // fronts that took the mixed form and grew past the bound were factored
    // again in FP64 at the end of their wave (refactor_fp64)
    int32_t flagged = 0;
    CK(cudaMemcpyAsync(&flagged, h->d_sel_flag, 4, cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
    h->sel_flagged = flagged;
    h->sel_fallback = h->sel_refactored;
  }
  return RVG_OK;
}

rvg_status rvg_factor(rvg_handle* h, const double* values, const double* scaling) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (h->P.n > 0 && !values) { set_error("null values"); return RVG_ERR_INVALID_INPUT; }
  CK(cudaSetDevice(h->device));
  if (h->nnz) CK(cudaMemcpyAsync(h->d_vals, values, h->nnz * 8, cudaMemcpyHostToDevice, h->st));
  h->has_scaling = scaling != nullptr;
  if (scaling && h->P.n) CK(cudaMemcpyAsync(h->d_scal, scaling, h->P.n * 8, cudaMemcpyHostToDevice, h->st));
  return (rvg_status)factor_common(h, h->d_vals, h->has_scaling ? h->d_scal : nullptr);
}

rvg_status rvg_factor_device(rvg_handle* h, const double* d_values, const double* d_scaling) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  CK(cudaSetDevice(h->device));
  h->has_scaling = d_scaling != nullptr;
  if (d_scaling && h->P.n) CK(cudaMemcpyAsync(h->d_scal, d_scaling, h->P.n * 8, cudaMemcpyDeviceToDevice, h->st));
  return (rvg_status)factor_common(h, d_values, h->has_scaling ? h->d_scal : nullptr);
}

// Status of the bounded device waits (mixed-form GEMM pipeline, solve
// dependencies) since the last check; resets the word.  Synchronises.
static int device_wait_status(rvg_handle* h) {
  int32_t e = 0;
  CK(cudaMemcpyAsync(&e, h->d_err, 4, cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  if (e) {
    CK(cudaMemsetAsync(h->d_err, 0, 4, h->st));
    set_error(e == 2 ? "a solve block gave up waiting for the blocks it depends on (device timeout)"
                     : "a tensor-core Schur update gave up waiting on its pipeline (device timeout)");
    return RVG_ERR_DEVICE_TIMEOUT;
  }
  return RVG_OK;
}

// The block layout of the factored fronts for the solve kernels: per wave, the
// forward blocks (diagonal, then L21, per front) and the backward tickets
// (gathers, partial sums, column blocks), the front of every ticket, and the
// fronts' offsets in the solve workspace (DFront::scratch: rows before it).
// Valid until the next factorization or rvg_trim.
static int sf_make_layout(rvg_handle* h) {
  const Plan& P = h->P;
  cudaStream_t st = h->st;
  rvg_handle::SfLayout& Y = h->sf;
  Y = rvg_handle::SfLayout();
  std::vector<DFront> fr = h->h_fronts;
  for (auto& f : fr) { f.scratch = Y.rows; Y.rows += f.m; }
  Packer pk;
  const size_t o_fr = pk.add(fr);
  for (size_t w = 0; w < P.waves.size(); ++w) {
    std::vector<SfFront> vf, vb;
    std::vector<int32_t> mf, mb;
    int32_t slots = 0;
    rvg_handle::SfLayout::Wave v{};
    for (int64_t s : P.waves[w]) {
      const DFront& f = fr[s];
      if (f.ne == 0) continue;
      const int32_t nbd = (f.ne + SF_B - 1) / SF_B, nbr = (f.m - f.ne + SF_B - 1) / SF_B;
      const int32_t ngrp = (nbr + SF_PG - 1) / SF_PG;
      const int32_t at = (int32_t)vf.size();
      vf.push_back(SfFront{(int32_t)s, v.nbf, nbd, nbr, 0, 0});
      vb.push_back(SfFront{(int32_t)s, v.nbb, nbd, nbr, ngrp, slots});
      v.nbf += nbd + nbr;
      v.nbb += nbr + nbd * ngrp + nbd;  // gathers, partial sums, column blocks
      mf.resize(v.nbf, at);
      mb.resize(v.nbb, at);
      slots += nbd * ngrp;
    }
    Y.slots = std::max<int64_t>(Y.slots, slots);
    v.fwd = pk.add(vf);
    v.bwd = pk.add(vb);
    v.mfwd = pk.add(mf);
    v.mbwd = pk.add(mb);
    v.tf = Y.nsync;
    Y.nsync += 1;  // the forward blocks need a ticket counter only
    v.tb = Y.nsync;
    Y.nsync += 1 + v.nbb;
    Y.w.push_back(v);
  }
  int rc;
  if ((rc = ensure_nocopy(h->sf_lay, h->sf_lay_cap, pk.buf.size() + 16, st))) return rc;
  // through the pinned buffer when it is large enough as it is: growing it would cost more than the copy
  const char* src = pk.buf.data();
  if (pk.buf.size() <= h->h_stage_cap && h->h_stage) {
    std::memcpy(h->h_stage, src, pk.buf.size());
    src = h->h_stage;
  }
  CK(cudaMemcpyAsync(h->sf_lay, src, pk.buf.size(), cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(h->d_fronts, h->sf_lay + o_fr, fr.size() * sizeof(DFront), cudaMemcpyDeviceToDevice, st));
  CK(cudaStreamSynchronize(st));  // the source is free again
  Y.ok = true;
  return RVG_OK;
}

// aptp_solve (solve.rs:57-326) with the permutation and scaling of
// SparseLDLT::solve_in_place (solver.rs:396-425): per wave one forward launch
// (leaves first) and, in reverse, one backward launch of solve_sf.cuh.
static int solve_common(rvg_handle* h, double* d_rhs, int64_t nrhs, int64_t ldb) {
  const int64_t n = h->P.n;
  cudaStream_t st = h->st;
  if (n == 0 || nrhs == 0) return RVG_OK;
  // right-hand sides per pass: 8, 4, 2 or 1.  A pass costs the factor's read
  // and the chain of its diagonal blocks whatever its width, so the last
  // columns go through one pass of the next width up (5 to 7 as 8, 3 as 4)
  // beside columns of zeros, not through several narrow ones.  Passes of 1 / 2 /
  // 4 / 8 columns take 2.45 / 3.36 / 3.76 / 5.37 ms on a KKT 36^3, 3.03 / 4.01 /
  // 4.49 / 6.37 on a 64^3 Laplacian and 0.25 / 0.31 / 0.34 / 0.44 on a 16^3 one:
  // 4 is less than 2 + 1 (5.81, 7.04, 0.55), 8 less than 4 + 1 (6.21, 7.53, 0.58)
  auto pass = [](int64_t left) { return left > 4 ? 8 : left > 2 ? 4 : (int)left; };
  const int rmax = pass(nrhs);
  const int64_t npad = nrhs / 8 * 8 + pass(nrhs % 8);
  int rc = ensure(h->d_x, h->x_cap, (size_t)(n * npad), st);
  if (rc) return rc;
  if (!h->sf.ok && (rc = sf_make_layout(h))) return rc;
  const rvg_handle::SfLayout& Y = h->sf;
  const size_t nw = Y.w.size();
  // the per-front solve workspace: forward results, then final values (R x m each)
  const int64_t wneed = 2 * (int64_t)rmax * Y.rows;
  if ((rc = ensure(h->solve_work, h->solve_work_cap, (size_t)std::max<int64_t>(wneed, 1), st))) return rc;
  if ((rc = ensure(h->sf_sync, h->sf_sync_cap, (size_t)std::max<int64_t>(Y.nsync, 1), st))) return rc;
  if ((rc = ensure_nocopy(h->sf_part, h->sf_part_cap, (size_t)Y.slots * 8 * SF_B, st))) return rc;
  Arenas A{h->panel, h->idx, h->dtype, h->ddiag, h->doff, nullptr, h->cb_arena};
  CK(cudaEventRecord(h->ev[6], st));
  int64_t launches = 0;
  int64_t tot = n * nrhs;
  k_perm_scale_in<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(d_rhs, ldb, nrhs, h->d_x, n, h->d_pfwd,
                                                                 h->has_scaling ? h->d_scal : nullptr);
  launches++;
  if (npad > nrhs) CK(cudaMemsetAsync(h->d_x + n * nrhs, 0, (size_t)(n * (npad - nrhs)) * 8, st));
  auto wave = [&](size_t w, bool fwd, int64_t rh) {
    const rvg_handle::SfLayout::Wave& v = Y.w[w];
    SfWave sw;
    sw.part = h->sf_part;
    sw.fr = (const SfFront*)(h->sf_lay + (fwd ? v.fwd : v.bwd));
    sw.fmap = (const int32_t*)(h->sf_lay + (fwd ? v.mfwd : v.mbwd));
    sw.nblk = fwd ? v.nbf : v.nbb;
    sw.ticket = h->sf_sync + (fwd ? v.tf : v.tb);
    sw.flags = sw.ticket + 1;
    sw.x = h->d_x + rh * n;
    sw.ldx = n;
    sw.work = h->solve_work;
    sw.err = h->d_err;
    return sw;
  };
  auto fwd = [&](int r, const SfWave& sw) {
    const dim3 g((unsigned)std::min<int64_t>(sw.nblk, 16LL * h->nsm));
    switch (r) {
      case 8: launch_chain(h, k_sf_fwd<8>, g, SF_B, 0, st, sw, (const DFront*)h->d_fronts, A); break;
      case 4: launch_chain(h, k_sf_fwd<4>, g, SF_B, 0, st, sw, (const DFront*)h->d_fronts, A); break;
      case 2: launch_chain(h, k_sf_fwd<2>, g, SF_B, 0, st, sw, (const DFront*)h->d_fronts, A); break;
      default: launch_chain(h, k_sf_fwd<1>, g, SF_B, 0, st, sw, (const DFront*)h->d_fronts, A); break;
    }
  };
  if (!h->sf_attr) {  // the backward kernels' static + dynamic shared memory exceeds the default 48 KB
    CK(cudaFuncSetAttribute(k_sf_bwd<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SF_BWD_DYN));
    CK(cudaFuncSetAttribute(k_sf_bwd<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, SF_BWD_DYN));
    CK(cudaFuncSetAttribute(k_sf_bwd<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, SF_BWD_DYN));
    CK(cudaFuncSetAttribute(k_sf_bwd<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, SF_BWD_DYN));
    h->sf_attr = true;
  }
  auto bwd = [&](int r, const SfWave& sw) {
    const dim3 g((unsigned)std::min<int64_t>(sw.nblk, 6LL * h->nsm));
    switch (r) {
      case 8: launch_chain(h, k_sf_bwd<8>, g, SF_B, SF_BWD_DYN, st, sw, (const DFront*)h->d_fronts, A); break;
      case 4: launch_chain(h, k_sf_bwd<4>, g, SF_B, SF_BWD_DYN, st, sw, (const DFront*)h->d_fronts, A); break;
      case 2: launch_chain(h, k_sf_bwd<2>, g, SF_B, SF_BWD_DYN, st, sw, (const DFront*)h->d_fronts, A); break;
      default: launch_chain(h, k_sf_bwd<1>, g, SF_B, SF_BWD_DYN, st, sw, (const DFront*)h->d_fronts, A); break;
    }
  };
  for (int64_t rh = 0; rh < nrhs;) {
    const int r = pass(nrhs - rh);
    CK(cudaMemsetAsync(h->solve_work, 0xff, (size_t)(2 * (int64_t)r * Y.rows) * 8, st));  // SF_EMPTY
    CK(cudaMemsetAsync(h->sf_sync, 0, (size_t)Y.nsync * 4, st));
    for (size_t w = 0; w < nw; ++w) {
      if (!Y.w[w].nbf) continue;
      fwd(r, wave(w, true, rh));
      launches++;
    }
    for (size_t w = nw; w-- > 0;) {
      if (!Y.w[w].nbb) continue;
      bwd(r, wave(w, false, rh));
      launches++;
    }
    rh += r;
  }
  k_perm_scale_out<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(d_rhs, ldb, nrhs, h->d_x, n, h->d_pfwd,
                                                                  h->has_scaling ? h->d_scal : nullptr);
  launches++;
  h->solve_launches = launches;
  CK(cudaEventRecord(h->ev[7], st));
  CK(cudaGetLastError());
  return RVG_OK;
}

rvg_status rvg_solve_device(rvg_handle* h, double* d_rhs, int64_t nrhs, int64_t ldb) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  if (nrhs < 0 || (nrhs > 0 && ldb < h->P.n)) { set_error("RHS length must match matrix dimension"); return RVG_ERR_DIMENSION_MISMATCH; }
  CK(cudaSetDevice(h->device));
  int rc = solve_common(h, d_rhs, nrhs, ldb);
  if (rc) return (rvg_status)rc;
  CK(cudaStreamSynchronize(h->st));
  float ms = 0;
  cudaEventElapsedTime(&ms, h->ev[6], h->ev[7]);
  h->t_solve = ms;
  return RVG_OK;
}

rvg_status rvg_solve(rvg_handle* h, double* rhs, int64_t nrhs, int64_t ldb) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  if (nrhs < 0 || (nrhs > 0 && ldb < h->P.n)) { set_error("RHS length must match matrix dimension"); return RVG_ERR_DIMENSION_MISMATCH; }
  if (h->P.n == 0 || nrhs == 0) return RVG_OK;
  CK(cudaSetDevice(h->device));
  double* d = nullptr;
  size_t bytes = (size_t)ldb * (size_t)(nrhs - 1) * 8 + (size_t)h->P.n * 8;
  CK(cudaMallocAsync((void**)&d, bytes, h->st));
  CK(cudaMemcpyAsync(d, rhs, bytes, cudaMemcpyHostToDevice, h->st));
  int rc = solve_common(h, d, nrhs, ldb);
  if (rc) return (rvg_status)rc;
  CK(cudaMemcpyAsync(rhs, d, bytes, cudaMemcpyDeviceToHost, h->st));
  CK(cudaFreeAsync(d, h->st));
  if ((rc = device_wait_status(h))) return (rvg_status)rc;
  float ms = 0;
  cudaEventElapsedTime(&ms, h->ev[6], h->ev[7]);
  h->t_solve = ms;
  return RVG_OK;
}

// nrhs right-hand sides at once (columns at stride ld of b and x): the blocked
// solve, then residuals, norms and corrections of every column until each
// column's scaled backward error is <= tol (or max_iter corrections); bwd[j]
// is column j's final error.
static int refine_common(rvg_handle* h, const double* d_b, double* d_x, int64_t nrhs, int64_t ld, double tol,
                         int32_t max_iter, int32_t* iters, double* bwd, bool* stalled = nullptr) {
  const int64_t n = h->P.n;
  cudaStream_t st = h->st;
  int rc = ensure(h->d_ref, h->ref_cap, (size_t)((nrhs + 1) * n + 3 * nrhs + 8), st);
  if (rc) return rc;
  double* r = h->d_ref;                  // n x nrhs, ld n
  double* nrm = h->d_ref + nrhs * n;     // 3 per column
  if ((rc = ensure_host((char*&)h->h_norms_m, h->h_norms_m_cap, (size_t)(3 * nrhs + 1) * 8))) return rc;
  double* hn = (double*)h->h_norms_m;
  if (ld == n) CK(cudaMemcpyAsync(d_x, d_b, (size_t)(n * nrhs) * 8, cudaMemcpyDeviceToDevice, st));
  else CK(cudaMemcpy2DAsync(d_x, ld * 8, d_b, ld * 8, n * 8, nrhs, cudaMemcpyDeviceToDevice, st));
  if ((rc = solve_common(h, d_x, nrhs, ld))) return rc;
  int it = 0;
  double prev_worst = 0;
  if (stalled) *stalled = false;
  const dim3 g((unsigned)blocks_for(n, 256), (unsigned)nrhs), gn(64, (unsigned)nrhs);
  for (;;) {
    k_residual<<<g, 256, 0, st>>>(h->d_colptr, h->d_rowidx, h->d_vals, d_x, d_b, r, n, ld, n);
    CK(cudaMemsetAsync(nrm, 0, (size_t)(3 * nrhs) * 8, st));
    k_norms3<<<gn, 256, 0, st>>>(r, d_x, d_b, n, nrm, ld, n);
    CK(cudaMemcpyAsync(hn, nrm, (size_t)(3 * nrhs) * 8, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    bool done = true;
    double worst = 0;
    for (int64_t j = 0; j < nrhs; ++j) {
      const double denom = h->a_fro * std::sqrt(hn[3 * j + 1]) + std::sqrt(hn[3 * j + 2]);
      const double e = denom == 0 ? 0.0 : std::sqrt(hn[3 * j]) / denom;
      if (bwd) bwd[j] = e;
      if (!(e <= tol)) done = false;
      worst = std::max(worst, e);
    }
    if (done || it >= max_iter) break;
    // with `stalled` given: stop once a correction no longer halves the error
    if (stalled && it > 0 && !(worst <= 0.5 * prev_worst)) { *stalled = true; break; }
    prev_worst = worst;
    if ((rc = solve_common(h, r, nrhs, n))) return rc;
    k_axpy1<<<g, 256, 0, st>>>(d_x, r, n, ld, n);
    ++it;
  }
  CK(cudaGetLastError());
  if ((rc = device_wait_status(h))) return rc;
  if (iters) *iters = it;
  return RVG_OK;
}

// GMRES-IR: restarted flexible GMRES in FP64 on A x = b with the factor as
// right preconditioner (z_j = solve(v_j), w = A z_j, Gram-Schmidt applied
// twice, Givens rotations on the host, x += Z y at every restart).  It stops
// when the scaled backward error of the true residual, checked at every
// restart and when the rotated residual estimate reaches tol, is <= tol, or
// after max_iter preconditioned products; *iters counts them (one solve each).
static int gmres_common(rvg_handle* h, const double* d_b, double* d_x, double tol, int32_t max_iter, int32_t restart,
                        int32_t* iters, double* bwd, bool x_given = false) {
  const int64_t n = h->P.n;
  cudaStream_t st = h->st;
  const int m = restart;
  // V (m + 1 basis vectors), Z (m preconditioned ones), r / w, coefficients
  int rc = ensure(h->d_gm, h->gm_cap, (size_t)((2 * m + 2) * n + 4 * (m + 2) + 8), st);
  if (rc) return rc;
  double* V = h->d_gm;
  double* Z = V + (int64_t)(m + 1) * n;
  double* w = Z + (int64_t)m * n;
  double* dc = w + n;          // m + 1 coefficients
  double* dn = dc + (m + 2);   // norms
  if ((rc = ensure_host((char*&)h->h_norms_m, h->h_norms_m_cap, (size_t)(4 * (m + 2) + 8) * 8))) return rc;
  double* hn = (double*)h->h_norms_m;
  const unsigned nb = blocks_for(n, 256);
  const dim3 gd(64, 1);
  auto sync_read = [&](const double* src, int cnt) -> int {
    CK(cudaMemcpyAsync(hn, src, (size_t)cnt * 8, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return RVG_OK;
  };
  // true residual r = b - A x into w; its backward error and ||r||
  auto residual = [&](double& e, double& rn) -> int {
    k_residual<<<dim3(nb, 1), 256, 0, st>>>(h->d_colptr, h->d_rowidx, h->d_vals, d_x, d_b, w, n, n, n);
    CK(cudaMemsetAsync(dn, 0, 3 * 8, st));
    k_norms3<<<dim3(64, 1), 256, 0, st>>>(w, d_x, d_b, n, dn, n, n);
    int r2 = sync_read(dn, 3);
    if (r2) return r2;
    const double denom = h->a_fro * std::sqrt(hn[1]) + std::sqrt(hn[2]);
    rn = std::sqrt(hn[0]);
    e = denom == 0 ? 0.0 : rn / denom;
    return RVG_OK;
  };
  if (!x_given) {
    CK(cudaMemcpyAsync(d_x, d_b, n * 8, cudaMemcpyDeviceToDevice, st));
    if ((rc = solve_common(h, d_x, 1, n))) return rc;  // x0 = M^-1 b
  }
  int it = 0;
  double e = 0, beta = 0;
  std::vector<double> H((size_t)(m + 1) * m), cs(m), sn(m), g(m + 1), y(m);
  for (;;) {
    if ((rc = residual(e, beta))) return rc;
    if (e <= tol || it >= max_iter || beta == 0) break;
    // target for the residual estimate: the backward error with the current ||x||
    const double xnorm = std::sqrt(hn[1]), bnorm = std::sqrt(hn[2]);
    const double target = 0.5 * tol * (h->a_fro * xnorm + bnorm);
    k_scale_to<<<nb, 256, 0, st>>>(V, w, 1.0 / beta, n);
    std::fill(g.begin(), g.end(), 0.0);
    g[0] = beta;
    int j = 0;
    for (; j < m && it < max_iter; ++j) {
      double* z = Z + (int64_t)j * n;
      CK(cudaMemcpyAsync(z, V + (int64_t)j * n, n * 8, cudaMemcpyDeviceToDevice, st));
      if ((rc = solve_common(h, z, 1, n))) return rc;
      ++it;
      k_spmv<<<nb, 256, 0, st>>>(h->d_colptr, h->d_rowidx, h->d_vals, z, w, n);
      // Gram-Schmidt twice against v_0..v_j
      for (int pass = 0; pass < 2; ++pass) {
        CK(cudaMemsetAsync(dc, 0, (size_t)(j + 1) * 8, st));
        k_dots<<<dim3(64, (unsigned)(j + 1)), 256, 0, st>>>(V, w, n, dc);
        k_sub_comb<<<nb, 256, 0, st>>>(w, V, dc, j + 1, n);
        if ((rc = sync_read(dc, j + 1))) return rc;
        for (int i = 0; i <= j; ++i) H[(size_t)i * m + j] = (pass ? H[(size_t)i * m + j] : 0.0) + hn[i];
      }
      CK(cudaMemsetAsync(dn, 0, 8, st));
      k_sumsq<<<64, 256, 0, st>>>(w, n, dn);
      if ((rc = sync_read(dn, 1))) return rc;
      const double hn1 = std::sqrt(hn[0]);
      H[(size_t)(j + 1) * m + j] = hn1;
      if (hn1 > 0) k_scale_to<<<nb, 256, 0, st>>>(V + (int64_t)(j + 1) * n, w, 1.0 / hn1, n);
      // Givens rotations
      for (int i = 0; i < j; ++i) {
        const double a = H[(size_t)i * m + j], b2 = H[(size_t)(i + 1) * m + j];
        H[(size_t)i * m + j] = cs[i] * a + sn[i] * b2;
        H[(size_t)(i + 1) * m + j] = -sn[i] * a + cs[i] * b2;
      }
      const double a = H[(size_t)j * m + j], b2 = H[(size_t)(j + 1) * m + j];
      const double rr = std::hypot(a, b2);
      cs[j] = rr == 0 ? 1.0 : a / rr;
      sn[j] = rr == 0 ? 0.0 : b2 / rr;
      H[(size_t)j * m + j] = rr;
      H[(size_t)(j + 1) * m + j] = 0.0;
      g[j + 1] = -sn[j] * g[j];
      g[j] = cs[j] * g[j];
      if (std::fabs(g[j + 1]) <= target || hn1 == 0) { ++j; break; }
    }
    // y = H^-1 g on the leading j x j triangle, x += Z y
    for (int i = j - 1; i >= 0; --i) {
      double s2 = g[i];
      for (int k = i + 1; k < j; ++k) s2 -= H[(size_t)i * m + k] * y[k];
      y[i] = H[(size_t)i * m + i] == 0 ? 0.0 : s2 / H[(size_t)i * m + i];
    }
    if (j > 0) {
      CK(cudaMemcpyAsync(dc, y.data(), (size_t)j * 8, cudaMemcpyHostToDevice, st));
      k_add_comb<<<nb, 256, 0, st>>>(d_x, Z, dc, j, n);
    }
  }
  CK(cudaGetLastError());
  if ((rc = device_wait_status(h))) return rc;
  if (iters) *iters = it;
  if (bwd) *bwd = e;
  return RVG_OK;
}

// Iterative refinement while every correction at least halves the backward
// error, then GMRES-IR from the refined x: the cheap method when it converges,
// the robust one when the factor's error times the condition number is too
// large for it.  *method: 0 refinement alone, 1 escalated to GMRES-IR;
// *iters: the solves after the first one (corrections + GMRES products).
static int auto_common(rvg_handle* h, const double* d_b, double* d_x, double tol, int32_t max_iter, int32_t* iters,
                       double* bwd, int32_t* method) {
  bool stalled = false;
  int32_t it1 = 0, it2 = 0;
  double e = 0;
  int rc = refine_common(h, d_b, d_x, 1, h->P.n, tol, std::min<int32_t>(max_iter, 10), &it1, &e, &stalled);
  if (rc) return rc;
  if (method) *method = 0;
  if (!(e <= tol) && it1 < max_iter) {
    if ((rc = gmres_common(h, d_b, d_x, tol, max_iter - it1, 30, &it2, &e, true))) return rc;
    if (method) *method = 1;
  }
  if (iters) *iters = it1 + it2;
  if (bwd) *bwd = e;
  return RVG_OK;
}

rvg_status rvg_solve_auto_device(rvg_handle* h, const double* d_rhs, double* d_x, double tol, int32_t max_iter,
                                 int32_t* iters, double* bwd_err, int32_t* method) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  if (h->P.n == 0) { if (iters) *iters = 0; if (bwd_err) *bwd_err = 0; if (method) *method = 0; return RVG_OK; }
  CK(cudaSetDevice(h->device));
  double t0 = now_ms();
  int rc = auto_common(h, d_rhs, d_x, tol, max_iter, iters, bwd_err, method);
  h->t_solve = now_ms() - t0;
  return (rvg_status)rc;
}

rvg_status rvg_solve_auto(rvg_handle* h, const double* rhs, double* x, double tol, int32_t max_iter, int32_t* iters,
                          double* bwd_err, int32_t* method) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  const int64_t n = h->P.n;
  if (n == 0) { if (iters) *iters = 0; if (bwd_err) *bwd_err = 0; if (method) *method = 0; return RVG_OK; }
  CK(cudaSetDevice(h->device));
  double t0 = now_ms();
  double* d = nullptr;
  CK(cudaMallocAsync((void**)&d, 2 * n * 8, h->st));
  CK(cudaMemcpyAsync(d, rhs, n * 8, cudaMemcpyHostToDevice, h->st));
  int rc = auto_common(h, d, d + n, tol, max_iter, iters, bwd_err, method);
  if (rc) return (rvg_status)rc;
  CK(cudaMemcpyAsync(x, d + n, n * 8, cudaMemcpyDeviceToHost, h->st));
  CK(cudaFreeAsync(d, h->st));
  CK(cudaStreamSynchronize(h->st));
  h->t_solve = now_ms() - t0;
  return RVG_OK;
}

rvg_status rvg_solve_gmres_device(rvg_handle* h, const double* d_rhs, double* d_x, double tol, int32_t max_iter,
                                  int32_t restart, int32_t* iters, double* bwd_err) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  if (restart < 1 || restart > 200) { set_error("restart must be in [1, 200]"); return RVG_ERR_INVALID_INPUT; }
  if (h->P.n == 0) { if (iters) *iters = 0; if (bwd_err) *bwd_err = 0; return RVG_OK; }
  CK(cudaSetDevice(h->device));
  double t0 = now_ms();
  int rc = gmres_common(h, d_rhs, d_x, tol, max_iter, restart, iters, bwd_err);
  h->t_solve = now_ms() - t0;
  return (rvg_status)rc;
}

rvg_status rvg_solve_gmres(rvg_handle* h, const double* rhs, double* x, double tol, int32_t max_iter, int32_t restart,
                           int32_t* iters, double* bwd_err) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  if (restart < 1 || restart > 200) { set_error("restart must be in [1, 200]"); return RVG_ERR_INVALID_INPUT; }
  const int64_t n = h->P.n;
  if (n == 0) { if (iters) *iters = 0; if (bwd_err) *bwd_err = 0; return RVG_OK; }
  CK(cudaSetDevice(h->device));
  double t0 = now_ms();
  double* d = nullptr;
  CK(cudaMallocAsync((void**)&d, 2 * n * 8, h->st));
  CK(cudaMemcpyAsync(d, rhs, n * 8, cudaMemcpyHostToDevice, h->st));
  int rc = gmres_common(h, d, d + n, tol, max_iter, restart, iters, bwd_err);
  if (rc) return (rvg_status)rc;
  CK(cudaMemcpyAsync(x, d + n, n * 8, cudaMemcpyDeviceToHost, h->st));
  CK(cudaFreeAsync(d, h->st));
  CK(cudaStreamSynchronize(h->st));
  h->t_solve = now_ms() - t0;
  return RVG_OK;
}

rvg_status rvg_solve_refine_device(rvg_handle* h, const double* d_rhs, double* d_x, double tol, int32_t max_iter,
                                   int32_t* iters, double* bwd_err) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  if (h->P.n == 0) { if (iters) *iters = 0; if (bwd_err) *bwd_err = 0; return RVG_OK; }
  CK(cudaSetDevice(h->device));
  double t0 = now_ms();
  int rc = refine_common(h, d_rhs, d_x, 1, h->P.n, tol, max_iter, iters, bwd_err);
  h->t_solve = now_ms() - t0;
  return (rvg_status)rc;
}

rvg_status rvg_solve_refine(rvg_handle* h, const double* rhs, double* x, double tol, int32_t max_iter, int32_t* iters,
                            double* bwd_err) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  const int64_t n = h->P.n;
  if (n == 0) { if (iters) *iters = 0; if (bwd_err) *bwd_err = 0; return RVG_OK; }
  CK(cudaSetDevice(h->device));
  double t0 = now_ms();
  double* d = nullptr;
  CK(cudaMallocAsync((void**)&d, 2 * n * 8, h->st));
  CK(cudaMemcpyAsync(d, rhs, n * 8, cudaMemcpyHostToDevice, h->st));
  int rc = refine_common(h, d, d + n, 1, n, tol, max_iter, iters, bwd_err);
  if (rc) return (rvg_status)rc;
  CK(cudaMemcpyAsync(x, d + n, n * 8, cudaMemcpyDeviceToHost, h->st));
  CK(cudaFreeAsync(d, h->st));
  CK(cudaStreamSynchronize(h->st));
  h->t_solve = now_ms() - t0;
  return RVG_OK;
}

rvg_status rvg_solve_refine_nrhs_device(rvg_handle* h, const double* d_rhs, double* d_x, int64_t nrhs, int64_t ldb,
                                        double tol, int32_t max_iter, int32_t* iters, double* bwd_err) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  const int64_t n = h->P.n;
  if (nrhs < 1 || ldb < n || (n > 0 && (!d_rhs || !d_x))) { set_error("need nrhs >= 1, ldb >= n and both vectors"); return RVG_ERR_INVALID_INPUT; }
  if (n == 0) { if (iters) *iters = 0; if (bwd_err) for (int64_t j = 0; j < nrhs; ++j) bwd_err[j] = 0; return RVG_OK; }
  CK(cudaSetDevice(h->device));
  double t0 = now_ms();
  int rc = refine_common(h, d_rhs, d_x, nrhs, ldb, tol, max_iter, iters, bwd_err);
  h->t_solve = now_ms() - t0;
  return (rvg_status)rc;
}

rvg_status rvg_solve_refine_nrhs(rvg_handle* h, const double* rhs, double* x, int64_t nrhs, int64_t ldb, double tol,
                                 int32_t max_iter, int32_t* iters, double* bwd_err) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called before solve()"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  const int64_t n = h->P.n;
  if (nrhs < 1 || ldb < n || (n > 0 && (!rhs || !x))) { set_error("need nrhs >= 1, ldb >= n and both arrays"); return RVG_ERR_INVALID_INPUT; }
  if (n == 0) { if (iters) *iters = 0; if (bwd_err) for (int64_t j = 0; j < nrhs; ++j) bwd_err[j] = 0; return RVG_OK; }
  CK(cudaSetDevice(h->device));
  double t0 = now_ms();
  double* d = nullptr;
  CK(cudaMallocAsync((void**)&d, 2 * (size_t)(n * nrhs) * 8, h->st));
  CK(cudaMemcpy2DAsync(d, n * 8, rhs, ldb * 8, n * 8, nrhs, cudaMemcpyHostToDevice, h->st));
  int rc = refine_common(h, d, d + n * nrhs, nrhs, n, tol, max_iter, iters, bwd_err);
  if (rc) return (rvg_status)rc;
  CK(cudaMemcpy2DAsync(x, ldb * 8, d + n * nrhs, n * 8, n * 8, nrhs, cudaMemcpyDeviceToHost, h->st));
  CK(cudaFreeAsync(d, h->st));
  CK(cudaStreamSynchronize(h->st));
  h->t_solve = now_ms() - t0;
  return RVG_OK;
}

rvg_status rvg_inertia(rvg_handle* h, int64_t out3[3]) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called first"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  for (int q = 0; q < 3; ++q) out3[q] = h->inertia[q];
  return RVG_OK;
}

rvg_status rvg_get_stats(rvg_handle* h, rvg_stats* o) {
  if (!h || !o) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called first"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  o->total_1x1_pivots = h->tot1;
  o->total_2x2_pivots = h->tot2;
  o->total_delayed = h->totdel;
  o->zero_pivots = h->zero_piv;
  o->max_front_size = h->max_front;
  o->supernodes_before_amalgamation = h->P.nsup_before;
  o->supernodes_after_amalgamation = (int64_t)h->P.sn.size();
  o->merges_performed = h->P.merges;
  o->small_leaf_subtrees = h->P.sl_subtrees;
  o->small_leaf_nodes = h->P.sl_nodes;
  return RVG_OK;
}

rvg_status rvg_pivot_record(rvg_handle* h, int64_t* col, int8_t* code, double* d_diag, double* d_off, int64_t* count) {
  if (!h || !count) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored) { set_error("factor() must be called first"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  int64_t tot = 0, isz = 0;
  for (auto& f : h->h_fronts) { tot = std::max<int64_t>(tot, f.dpos + f.k); isz = std::max<int64_t>(isz, f.idx + f.m + f.k); }
  std::vector<int8_t> dt(tot);
  std::vector<double> dd(tot), dof(tot);
  std::vector<int32_t> ix(isz);
  if (tot) {
    CK(cudaMemcpy(dt.data(), h->dtype, tot, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(dd.data(), h->ddiag, tot * 8, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(dof.data(), h->doff, tot * 8, cudaMemcpyDeviceToHost));
  }
  if (isz) CK(cudaMemcpy(ix.data(), h->idx, isz * 4, cudaMemcpyDeviceToHost));
  int64_t t = 0;
  for (auto& f : h->h_fronts) {
    const int32_t* rows = ix.data() + f.idx;
    const int32_t* perm = rows + f.m;
    for (int c = 0; c < f.ne; ++c) {
      int64_t q = f.dpos + c;
      if (col) col[t] = rows[perm[c]];
      int8_t cd = dt[q];
      if (code) code[t] = cd;
      if (d_diag) d_diag[t] = dd[q];
      if (d_off) d_off[t] = cd == 2 ? dof[q] : 0.0;
      ++t;
    }
  }
  *count = t;
  return RVG_OK;
}

rvg_status rvg_front_info(rvg_handle* h, int64_t* out9, int64_t* nsup) {
  if (!h || !nsup) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  *nsup = (int64_t)h->P.sn.size();
  if (!out9) return RVG_OK;
  for (size_t s = 0; s < h->P.sn.size(); ++s) {
    const DFront& f = h->factored ? h->h_fronts[s] : DFront();
    int64_t* o = out9 + 9 * s;
    o[0] = f.m; o[1] = f.k; o[2] = f.ne; o[3] = f.n1; o[4] = f.n2; o[5] = h->P.sn[s].parent;
    o[6] = h->P.sn[s].n_owned(); o[7] = h->P.sn[s].in_small_leaf ? 1 : 0; o[8] = h->P.height[s];
  }
  return RVG_OK;
}

rvg_status rvg_work(rvg_handle* h, double out6[6]) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  Plan& P = h->P;
  double solve_bytes = 0;
  for (auto& s : P.sn) {
    double k = (double)s.n_owned(), r = (double)s.pattern.size();
    double stored = k * (k + 1) / 2 + r * k;
    solve_bytes += 2 * 8 * stored + 8 * k + 2 * 4 * (k + r) + 2 * 2 * 8 * (k + r);
  }
  out6[0] = P.flops_factor; out6[1] = P.flops_schur; out6[2] = P.bytes_assembly; out6[3] = solve_bytes;
  out6[4] = (double)P.nnz_l; out6[5] = (double)P.max_front;
  return RVG_OK;
}

rvg_status rvg_timings(rvg_handle* h, double out7[7]) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  out7[0] = h->t_assembly; out7[1] = h->t_kernel; out7[2] = h->t_gemm; out7[3] = h->t_factor; out7[4] = h->t_solve;
  out7[5] = h->t_dom; out7[6] = h->n_dom;
  return RVG_OK;
}

rvg_status rvg_set_profiling(rvg_handle* h, int32_t enable) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  h->profiling = enable != 0;
  return RVG_OK;
}

// The solve's waits on what nothing delivers: a flag, and a block's values for 8 right-hand sides.
__global__ void k_wait_probe(const int32_t* flag, int32_t* err) { sf_wait(flag, err); }
__global__ void __launch_bounds__(SF_B) k_take_probe(const double* values, int32_t* err) {
  __shared__ double dst[8][SF_B];
  sf_take_block<8>(values, SF_B, SF_B, true, dst, err);
}

rvg_status rvg_selftest_waits(rvg_handle* h, int32_t which) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (which != 0 && which != 1) { set_error("which must be 0 (solve waits) or 1 (tensor-core pipeline)"); return RVG_ERR_INVALID_INPUT; }
  CK(cudaSetDevice(h->device));
  cudaStream_t st = h->st;
  int rc = device_wait_status(h);  // start from a clean error word
  if (rc) return (rvg_status)rc;
  if ((rc = ensure(h->sf_sync, h->sf_sync_cap, 2, st))) return (rvg_status)rc;
  CK(cudaMemsetAsync(h->sf_sync, 0, 2 * sizeof(int32_t), st));
  if (which == 0) {
    k_wait_probe<<<1, 1, 0, st>>>(h->sf_sync, h->d_err);
    CK(cudaGetLastError());
    if ((rc = device_wait_status(h)) != RVG_ERR_DEVICE_TIMEOUT) return (rvg_status)rc;
    if ((rc = ensure(h->solve_work, h->solve_work_cap, 8 * SF_B, st))) return (rvg_status)rc;
    CK(cudaMemsetAsync(h->solve_work, 0xff, 8 * SF_B * sizeof(double), st));  // SF_EMPTY
    k_take_probe<<<1, SF_B, 0, st>>>(h->solve_work, h->d_err);
  } else {
    // one 128 x 128 tile, K = 32, operands never copied in: the MMA warp's wait runs out
    double* c = nullptr;
    float* p = nullptr;
    CK(cudaMallocAsync((void**)&c, 128 * 128 * sizeof(double), st));
    CK(cudaMallocAsync((void**)&p, 2 * (size_t)TC_BLOCK * sizeof(float), st));
    TcArgs ta{c, 128, 0, 128, 0, 128, p, p + TC_BLOCK, 1, nullptr, 32, 1, 1, 1, h->d_err, nullptr, 0, 1};
    k_syrk_tc<4, TC_TF32><<<1, TC_THREADS, TC_SMEM, st>>>(ta);
    CK(cudaFreeAsync(c, st));
    CK(cudaFreeAsync(p, st));
  }
  CK(cudaGetLastError());
  return (rvg_status)device_wait_status(h);
}

rvg_status rvg_get_profile(rvg_handle* h, rvg_profile* o) {
  if (!h || !o) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  o->factor_ms = h->t_factor;
  o->solve_ms = h->t_solve;
  o->assembly_ms = h->t_assembly;
  o->dense_ms = h->t_kernel;
  o->cbgemm_ms = h->t_gemm;
  o->syrk_ms = h->syrk_ms;
  o->syrk_flops = h->syrk_flops;
  o->syrk_launches = h->syrk_launches;
  o->factor_launches = h->factor_launches;
  o->solve_launches = h->solve_launches;
  o->peak_bytes = h->peak_bytes;
  o->host_total_ms = h->host_total_ms;
  o->host_alloc_ms = h->host_alloc_ms;
  o->host_sync_ms = h->host_sync_ms;
  for (int i = 0; i < RVG_PARTS; ++i) o->part_ms[i] = h->part_ms[i];
  o->host_wait_ms = h->host_wait_ms;
  o->lf_misses = h->lf_misses;
  o->host_gap_ms = h->host_gap_ms;
  o->lf_far_updates = h->lf_far;
  return RVG_OK;
}

static int trim_buf(void* p, cudaStream_t st) {
  if (p) CK(cudaFreeAsync(p, st));
  return RVG_OK;
}

static float ubits(unsigned u) {
  float f;
  std::memcpy(&f, &u, 4);
  return f;
}

rvg_status rvg_set_selector(rvg_handle* h, const float* params, int64_t nparams, float threshold,
                            double growth_bound) {
  if (!h || !params) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  if (nparams != MLP_NPARAM) { set_error("selector parameters: expected rvg_mlp_param_count() floats"); return RVG_ERR_DIMENSION_MISMATCH; }
  for (int c = 0; c < MLP_IN; ++c)
    if (!(params[MLP_SD + c] > 0.f)) { set_error("selector normalisation: standard deviations must be positive"); return RVG_ERR_INVALID_INPUT; }
  if (!(growth_bound > 0)) { set_error("growth bound must be positive"); return RVG_ERR_INVALID_INPUT; }
  CK(cudaSetDevice(h->device));
  if (!h->d_sel) CK(cudaMalloc((void**)&h->d_sel, MLP_NPARAM * sizeof(float)));
  CK(cudaMemcpyAsync(h->d_sel, params, MLP_NPARAM * sizeof(float), cudaMemcpyHostToDevice, h->st));
  CK(cudaStreamSynchronize(h->st));
  h->sel_thresh = threshold;
  h->sel_bound = growth_bound;
  return RVG_OK;
}

rvg_status rvg_front_features(rvg_handle* h, double* out, int64_t cap_rows, int64_t* nrows) {
  if (!h || !nrows) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  if (!h->factored || h->opt.precision != 2) { set_error("no learned-precision factorization to report"); return RVG_ERR_SOLVE_BEFORE_FACTOR; }
  *nrows = (int64_t)h->sel_large.size();
  if (!out) return RVG_OK;
  if (cap_rows < *nrows) { set_error("feature table: too few rows"); return RVG_ERR_DIMENSION_MISMATCH; }
  std::vector<unsigned> rows((size_t)h->P.sn.size() * FEAT_STRIDE);
  if (!rows.empty()) CK(cudaMemcpy(rows.data(), h->d_feat, rows.size() * 4, cudaMemcpyDeviceToHost));
  for (size_t i = 0; i < h->sel_large.size(); ++i) {
    const int32_t s = h->sel_large[i];
    const DFront& f = h->h_fronts[s];
    const unsigned* r = rows.data() + (size_t)s * FEAT_STRIDE;
    double* o = out + i * RVG_FRONT_FEATURE_COLS;
    o[0] = s; o[1] = f.m; o[2] = f.k; o[3] = f.ne; o[4] = f.n1; o[5] = f.n2;
    o[6] = ubits(r[21]);  // route
    o[7] = ubits(r[20]);  // probability
    o[8] = ubits(r[0]);   // max |a|
    o[9] = ubits(r[7]);   // max |D|
    for (int c = 0; c < MLP_IN; ++c) o[10 + c] = ubits(r[8 + c]);
  }
  return RVG_OK;
}

rvg_status rvg_selector_stats(rvg_handle* h, int64_t out4[4]) {
  if (!h || !out4) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  out4[0] = (int64_t)h->sel_large.size();
  out4[1] = h->sel_routed;
  out4[2] = h->sel_flagged;
  out4[3] = h->sel_fallback;
  return RVG_OK;
}

rvg_status rvg_trim(rvg_handle* h, int32_t what) {
  if (!h) { set_error("null handle"); return RVG_ERR_INVALID_INPUT; }
  if (what & ~3) { set_error("what: bit 0 = workspace, bit 1 = factor"); return RVG_ERR_INVALID_INPUT; }
  CK(cudaSetDevice(h->device));
  cudaStream_t st = h->st;
  int rc;
#define RVG_TRIM(p, cap)                              \
  do {                                                \
    if ((rc = trim_buf(p, st))) return (rvg_status)rc; \
    p = nullptr;                                      \
    cap = 0;                                          \
  } while (0)
  if (h->vm && what) CK(cudaDeviceSynchronize());  // nothing may use an arena whose memory goes
  auto vm_trim = [&](int id, auto*& p, size_t& cap) {  // address-stable arenas: the memory goes, the addresses stay
    vm_unmap(h->vm->slot[id]);
    p = nullptr;
    cap = 0;
  };
  if ((what & 1) && h->vm) {
    vm_trim(VM_SCRATCH, h->scratch, h->scratch_cap);
    vm_trim(VM_CB, h->cb_arena, h->cb_cap);
    vm_trim(VM_PACK, h->pack, h->pack_cap);
    vm_trim(VM_WPACK0, h->wpack, h->wpack_cap);
    for (size_t t = 1; t < h->lfx.size(); ++t) vm_trim(VM_WPACK0 + (int)t, h->lfx[t].wpack, h->lfx[t].wpack_cap);
    if (!h->lfx.empty()) { h->lfx[0].wpack = nullptr; h->lfx[0].wpack_cap = 0; }
    vm_trim(VM_STAGE, h->d_stage, h->stage_cap);
  } else if (what & 1) {
    RVG_TRIM(h->scratch, h->scratch_cap);
    RVG_TRIM(h->cb_arena, h->cb_cap);
    RVG_TRIM(h->pack, h->pack_cap);
    RVG_TRIM(h->wpack, h->wpack_cap);
    for (size_t t = 1; t < h->lfx.size(); ++t) RVG_TRIM(h->lfx[t].wpack, h->lfx[t].wpack_cap);
    if (!h->lfx.empty()) { h->lfx[0].wpack = nullptr; h->lfx[0].wpack_cap = 0; }
    RVG_TRIM(h->d_stage, h->stage_cap);
  }
  if (what & 1) {
    RVG_TRIM(h->solve_work, h->solve_work_cap);
    RVG_TRIM(h->sf_part, h->sf_part_cap);
    RVG_TRIM(h->sf_lay, h->sf_lay_cap);
    h->sf.ok = false;
    RVG_TRIM(h->d_x, h->x_cap);
    RVG_TRIM(h->d_ref, h->ref_cap);
    RVG_TRIM(h->d_gm, h->gm_cap);
    RVG_TRIM(h->d_stage2, h->stage2_cap);
    h->cb_free.clear();
  }
  if ((what & 2) && h->vm) {
    vm_trim(VM_PANEL, h->panel, h->panel_cap);
    vm_trim(VM_IDX, h->idx, h->idx_cap);
    size_t c1 = 0, c2 = 0;
    vm_trim(VM_DTYPE, h->dtype, h->d_cap);
    vm_trim(VM_DDIAG, h->ddiag, c1);
    vm_trim(VM_DOFF, h->doff, c2);
    h->factored = false;
  } else if (what & 2) {
    RVG_TRIM(h->panel, h->panel_cap);
    RVG_TRIM(h->idx, h->idx_cap);
    if ((rc = trim_buf(h->dtype, st)) || (rc = trim_buf(h->ddiag, st)) || (rc = trim_buf(h->doff, st)))
      return (rvg_status)rc;
    h->dtype = nullptr; h->ddiag = nullptr; h->doff = nullptr; h->d_cap = 0;
    h->factored = false;
  }
#undef RVG_TRIM
  if (what) {
    h->need_presize = true;
    if (!h->vm) drop_graph(h);  // it holds the addresses of the released buffers (kept in the vm mode)
  }
  CK(cudaStreamSynchronize(st));  // the memory is back in the pool when this returns
  return RVG_OK;
}

rvg_status rvg_mem_info(int64_t out2[2]) {
  if (!out2) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  size_t f = 0, t = 0;
  CK(cudaMemGetInfo(&f, &t));
  out2[0] = (int64_t)f;
  out2[1] = (int64_t)t;
  return RVG_OK;
}

rvg_status rvg_stream(rvg_handle* h, void** s) {
  if (!h || !s) { set_error("null argument"); return RVG_ERR_INVALID_INPUT; }
  *s = (void*)h->st;
  return RVG_OK;
}

void rvg_destroy(rvg_handle* h) {
  if (!h) return;
  cudaSetDevice(h->device);
  cudaStream_t st = h->st;
  auto fr = [&](void* p) { if (p) cudaFreeAsync(p, st); };
  fr(h->d_own_ptr); fr(h->d_own_idx); fr(h->d_pat_ptr); fr(h->d_pat_idx); fr(h->d_amap_ptr); fr(h->d_amap);
  fr(h->d_ea_ptr); fr(h->d_ea_map); fr(h->d_ch_ptr); fr(h->d_ch_idx); fr(h->d_pfwd); fr(h->d_fronts);
  if (!h->vm) {  // (address-stable arenas are released by vm_destroy below)
    fr(h->panel); fr(h->idx); fr(h->dtype); fr(h->ddiag); fr(h->doff);
    fr(h->d_stage); fr(h->scratch); fr(h->cb_arena); fr(h->pack); fr(h->wpack);
  }
  fr(h->d_vals); fr(h->d_scal);
  fr(h->d_x); fr(h->solve_work); fr(h->d_stage2); fr(h->d_lf); fr(h->sf_sync); fr(h->sf_part); fr(h->sf_lay); fr(h->d_gm);
  drop_graph(h);
  fr(h->d_rec);
  if (h->d_sel) cudaFree(h->d_sel);
  fr(h->d_feat);
  if (h->d_sel_flag) cudaFree(h->d_sel_flag);
  if (h->d_scan) cudaFree(h->d_scan);
  if (h->d_dcount) cudaFree(h->d_dcount);
  if (h->d_mismatch) cudaFree(h->d_mismatch);
  if (h->h_stage_all) cudaFreeHost(h->h_stage_all);
  for (size_t t = 0; t < h->lfx.size(); ++t) {
    LfCtx& c = h->lfx[t];
    if (c.h_gne) cudaFreeHost(c.h_gne);
    for (auto& e : c.ring_ev) if (e) cudaEventDestroy(e);
    if (c.far_st) { cudaStreamSynchronize(c.far_st); cudaStreamDestroy(c.far_st); }
    if (c.ev_fork) cudaEventDestroy(c.ev_fork);
    if (c.ev_far) cudaEventDestroy(c.ev_far);
    if (c.prop_st) { cudaStreamSynchronize(c.prop_st); cudaStreamDestroy(c.prop_st); }
    if (c.ev_prop_fork) cudaEventDestroy(c.ev_prop_fork);
    for (auto& e : c.ev_prop) if (e) cudaEventDestroy(e);
    if (t == 0) continue;  // the handle's own stream, state and window buffer
    if (!h->vm) fr(c.wpack);
    if (c.lf) cudaFree(c.lf);
    if (c.own && c.st) { cudaStreamSynchronize(c.st); cudaStreamDestroy(c.st); }
  }
  if (h->lf_st) { cudaStreamSynchronize(h->lf_st); cudaStreamDestroy(h->lf_st); }
  fr(h->d_err);
  fr(h->d_colptr); fr(h->d_rowidx); fr(h->d_ref);
  if (st) { cudaStreamSynchronize(st); cudaStreamDestroy(st); }
  vm_destroy(h);
  if (h->h_stage) cudaFreeHost(h->h_stage);
  if (h->h_stage2) cudaFreeHost(h->h_stage2);
  if (h->h_counts) cudaFreeHost(h->h_counts);
  if (h->h_norms) cudaFreeHost(h->h_norms);
  if (h->h_norms_m) cudaFreeHost(h->h_norms_m);
  for (auto e : h->ev_pool) cudaEventDestroy(e);
  for (auto e : h->mk_pool) cudaEventDestroy(e);
  for (auto& e : h->ev) if (e) cudaEventDestroy(e);
  if (h->ev_large) cudaEventDestroy(h->ev_large);
  if (h->ev_beside) cudaEventDestroy(h->ev_beside);
  delete h;
  cudaGetLastError();  // nothing of this handle's teardown is left for the caller's next call to report
}

}  // extern "C"
