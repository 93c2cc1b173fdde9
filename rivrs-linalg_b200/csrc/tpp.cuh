// Threshold partial pivoting (factor.rs:2268-2947) of one small front by one
// CTA: the small-leaf fronts (numeric.rs:1805) and the fronts with k < ib
// (factor.rs:360-362).
//
// Such a front is a few kilobytes and a chain of up to k dependent pivot
// decisions, so it is bound by the latency of a decision, not by arithmetic or
// bandwidth: the front is brought into shared memory once, and a step is two
// CTA barriers.  Warps own columns (j = warp mod W) and lanes rows; the warps
// that update the next two columns also leave their column maxima, so the
// usual decision (2x2 on the next two columns, or 1x1 on the second) reads two
// maxima and three entries.  Other candidates (p > ne + 1) are scanned by
// every warp for itself, with the routines of WarpTpp.  Every entry gets the
// operations of the reference's loops, in their order.
//
// Measured: ~1.2 us a pivot (an 81 x 81 front 100 us), ~8 us with one warp per
// front in global memory; the small fronts of an 8^3 Laplacian 1.31 -> 0.30 ms,
// of a 16^3 one ~3.5 -> 0.51 ms.  What is left is the decision (the 2x2 test's
// divisions) and the barriers: holding 256 rows of L in registers for the update
// was slower (0.35 ms, 124 registers).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "dense.cuh"
#include "front.cuh"

namespace rvg {

constexpr int TPP_MAX_T = 256;               // threads of a CTA at most
constexpr int TPP_CTAS = 4;                  // such CTAs on a multiprocessor: 64 registers a thread
constexpr size_t TPP_SMEM_MAX = 226 * 1024;  // dynamic shared memory of a CTA at most

// Off: int where the front is in shared memory, int64_t where it is in global
// memory (with a raised small_leaf_threshold, m k is not bounded by 2^31 there).
template <class Off>
struct CtaTpp {
  double* a;
  Off ld;
  int m, n;  // n = k: all stored columns are candidates
  int32_t* perm;
  DRec d;
  double* mx;  // [0] max |a(r, ne)| over r > ne, r != ne + 1; [1] max |a(r, ne + 1)| over r > ne + 1
  int tid, nt, lane, warp, nw;

  __device__ __forceinline__ double& at(int i, int j) const { return a[i + j * ld]; }

  // largest of the lanes' magnitudes (>= 0, NaN left out by fmax)
  __device__ __forceinline__ static double warp_absmax(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    return __hiloint2double((int)mh, (int)ml);
  }

  // column maxima of columns c and c + 1 into mx
  __device__ void scan(int c) const {
    for (int q = 0; q < 2; ++q)
      if (warp == (nw > 1 ? q : 0)) {
        const int j = c + q;
        double v = 0.0;
        if (j < n)
          for (int i = j + 1 + lane; i < m; i += 32)
            if (q == 1 || i != c + 1) v = fmax(v, fabs(at(i, j)));
        v = warp_absmax(v);
        if (lane == 0) mx[q] = v;
      }
  }

  // a(i, j) -= L_i . (D L_j) for the columns j in [c, n), the new maxima of columns c and c + 1 into mx;
  // f(i, wj...) gives the entry's update
  template <class W, class U>
  __device__ __forceinline__ void update(int c, W wof, U upd) const {
    for (int j = c + warp; j < n; j += nw) {
      const auto w = wof(j);
      double* col = a + (int64_t)j * ld;
      if (j < c + 2) {  // uniform over the warp
        double v = 0.0;
        for (int i = j + lane; i < m; i += 32) {
          const double x = upd(col[i], i, w);
          col[i] = x;
          if (i > j && (j > c || i != c + 1)) v = fmax(v, fabs(x));
        }
        v = warp_absmax(v);
        if (lane == 0) mx[j - c] = v;
      } else {
        int i = j + lane;
        for (; i + 96 < m; i += 128) {
          double x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) x[u] = upd(col[i + 32 * u], i + 32 * u, w);
#pragma unroll
          for (int u = 0; u < 4; ++u) col[i + 32 * u] = x[u];
        }
        for (; i < m; i += 32) col[i] = upd(col[i], i, w);
      }
    }
    // maxima of columns that do not exist
    if (tid == 0) {
      if (c >= n) mx[0] = 0.0;
      if (c + 1 >= n) mx[1] = 0.0;
    }
  }

  // (2616-2641)
  __device__ void apply_1x1(int ne) const {
    const double dv = at(ne, ne), inv = 1.0 / dv;
    double* l = a + (int64_t)ne * ld;
    for (int i = ne + 1 + tid; i < m; i += nt) l[i] = l[i] * inv;
    if (tid == 0) { d.type[ne] = PT_1X1; d.diag[ne] = dv; d.off[ne] = 0.0; }
    __syncthreads();
    update(ne + 1, [&](int j) { return l[j] * dv; }, [&](double x, int i, double w) { return x - l[i] * w; });
    __syncthreads();
  }
  // (2649-2683)
  __device__ void apply_2x2(int ne) const {
    const double a11 = at(ne, ne), a21 = at(ne + 1, ne), a22 = at(ne + 1, ne + 1);
    const double det = a11 * a22 - a21 * a21, inv_det = 1.0 / det;
    double* l = a + (int64_t)ne * ld;
    double* l2 = l + ld;
    for (int i = ne + 2 + tid; i < m; i += nt) {
      const double ai1 = l[i], ai2 = l2[i];
      l[i] = (ai1 * a22 - ai2 * a21) * inv_det;
      l2[i] = (ai2 * a11 - ai1 * a21) * inv_det;
    }
    __syncthreads();
    if (tid == 0) {  // (every thread has read a21)
      l[ne + 1] = 0.0;
      d.type[ne] = PT_2X2; d.type[ne + 1] = PT_2X2B;
      d.diag[ne] = a11; d.diag[ne + 1] = a22; d.off[ne] = a21; d.off[ne + 1] = 0.0;
    }
    struct W2 { double w1, w2; };
    update(ne + 2, [&](int j) { return W2{l[j] * a11 + l2[j] * a21, l[j] * a21 + l2[j] * a22}; },
           [&](double x, int i, W2 w) { return x - (l[i] * w.w1 + l2[i] * w.w2); });
    __syncthreads();
  }
  // swap_rect (2528-2580) by the whole CTA; the caller's reads are done before it starts
  __device__ void swap(int i, int j) const {
    if (i == j) return;
    if (i > j) { int t = i; i = j; j = t; }
    __syncthreads();
    if (tid == 0) {
      double t = at(i, i); at(i, i) = at(j, j); at(j, j) = t;
      int32_t q = perm[i]; perm[i] = perm[j]; perm[j] = q;
    }
    for (int k = tid; k < i; k += nt) { double t = at(i, k); at(i, k) = at(j, k); at(j, k) = t; }
    for (int k = i + 1 + tid; k < j; k += nt) { double t = at(k, i); at(k, i) = at(j, k); at(j, k) = t; }
    for (int k = j + 1 + tid; k < m; k += nt) { double t = at(k, i); at(k, i) = at(k, j); at(k, j) = t; }
    __syncthreads();
  }
  // a zero pivot at ne: no update
  __device__ void zero_pivot(int ne) const {
    __syncthreads();
    if (tid == 0) { d.type[ne] = PT_1X1; d.diag[ne] = 0.0; d.off[ne] = 0.0; }
    for (int r = ne + 1 + tid; r < m; r += nt) at(r, ne) = 0.0;
    __syncthreads();
  }

  // The TPP loop (tpp_factor, 2335-2506); every decision is taken by every thread from the same values.
  __device__ int run(const DevOpts& o, int* n1, int* n2) const {
    const double u = o.threshold, small = o.small;
    const WarpTpp T{PanelView{a, ld}, m, n, lane};
    // (with no limit, 0, the maxima cannot tell a column of zeros from one without a number: scan it)
    const bool limit = small > 0.0;
    int ne = 0, c1 = 0, c2 = 0;
    scan(0);
    __syncthreads();
    while (ne < n) {
      const double mt = mx[0], mp = mx[1];
      const double ann = fabs(at(ne, ne)), sub = ne + 1 < m ? fabs(at(ne + 1, ne)) : 0.0;
      if (limit ? !(ann >= small || mt >= small || sub >= small) : T.col_small(ne, ne, m, small)) {
        zero_pivot(ne);
        ++c1;
        ne += 1;
        scan(ne);
        __syncthreads();
        continue;
      }
      bool found = false;
      for (int p = ne + 1; p < n; ++p) {
        int t = ne;
        double maxt = mt, maxp = mp;
        bool tiny;
        if (p == ne + 1) {
          tiny = limit ? !(sub >= small || fabs(at(p, p)) >= small || mp >= small) : T.col_small(p, ne, m, small);
        } else {
          tiny = T.col_small(p, ne, m, small);
          if (!tiny) {
            t = (int)T.row_abs_max(p, ne, p);
            maxt = T.rc_abs_max_excl(t, ne, p);
            maxp = T.rc_abs_max_excl(p, ne, t);
          }
        }
        if (!limit && p == ne + 1) __syncthreads();  // every warp has scanned the columns that apply_2x2 writes
        if (tiny) {
          swap(p, ne);
          zero_pivot(ne);
          ++c1;
          ne += 1;
          scan(ne);
          __syncthreads();
          found = true;
          break;
        }
        if (T.test_2x2(t, p, maxt, maxp, u, small)) {
          swap(t, ne);
          const int np = p == ne ? t : p;
          swap(np, ne + 1);
          apply_2x2(ne);
          ++c2;
          ne += 2;
          found = true;
          break;
        }
        const double maxp_t = fmax(maxp, fabs(T.sym(p, t)));
        if (fabs(at(p, p)) >= u * maxp_t) {
          swap(p, ne);
          apply_1x1(ne);
          ++c1;
          ne += 1;
          found = true;
          break;
        }
      }
      if (!found) {
        const double maxp = ne + 1 < m ? fmax(mt, sub) : mt;
        if (!(fabs(at(ne, ne)) >= u * maxp)) break;
        __syncthreads();  // every warp is done scanning the candidates' rows, column ne among them
        apply_1x1(ne);
        ++c1;
        ne += 1;
      }
    }
    *n1 = c1;
    *n2 = c2;
    return ne;
  }
};

// One CTA per front.  SMEM: the front (its lower trapezoid, leading dimension
// m | 1: row scans hit different banks) and its pivot order live in dynamic
// shared memory meanwhile; else it stays in global memory.  Two kernels of 64
// registers: one that holds both kinds of offsets takes 78, with which 3 instead
// of 4 CTAs of 256 threads fit on a multiprocessor.
__host__ __device__ __forceinline__ int tpp_ld(int m) { return m | 1; }

template <bool SMEM>
__global__ void __launch_bounds__(TPP_MAX_T, TPP_CTAS) k_tpp_cta(const int32_t* ids, DFront* F, Arenas A, DevOpts o) {
  extern __shared__ double tsm[];
  __shared__ double s_mx[2];
  wave_kernel_enter();
  const int s = ids[blockIdx.x];
  const DFront fr = F[s];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int nw = nt >> 5, m = fr.m, k = fr.k;
  double* g = A.panel + fr.panel;
  int32_t* gperm = A.idx + fr.idx + m;
  const DRec d{A.dtype + fr.dpos, A.ddiag + fr.dpos, A.doff + fr.dpos};
  int n1 = 0, n2 = 0, ne;
  if constexpr (SMEM) {
    const int ld = tpp_ld(m);
    int32_t* perm = (int32_t*)(tsm + (size_t)ld * k);
    for (int j = warp; j < k; j += nw) {
      const double* src = g + (int64_t)j * m;
      double* dst = tsm + j * ld;
#pragma unroll 4
      for (int i = j + lane; i < m; i += 32) dst[i] = src[i];
    }
    for (int i = tid; i < k; i += nt) perm[i] = i;
    __syncthreads();
    const CtaTpp<int> T{tsm, ld, m, k, perm, d, s_mx, tid, nt, lane, warp, nw};
    ne = T.run(o, &n1, &n2);
    __syncthreads();
    for (int j = warp; j < k; j += nw) {
      double* dst = g + (int64_t)j * m;
      const double* src = tsm + j * ld;
#pragma unroll 4
      for (int i = j + lane; i < m; i += 32) dst[i] = src[i];
    }
    for (int i = tid; i < k; i += nt) gperm[i] = perm[i];
  } else {
    const CtaTpp<int64_t> T{g, m, m, k, gperm, d, s_mx, tid, nt, lane, warp, nw};
    ne = T.run(o, &n1, &n2);
  }
  if (tid == 0) { F[s].ne = ne; F[s].n1 = n1; F[s].n2 = n2; }
  wave_kernel_exit();
}

}  // namespace rvg
