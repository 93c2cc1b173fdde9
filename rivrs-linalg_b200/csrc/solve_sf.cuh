// Supernodal solve (aptp_solve, sparse/src/symmetric/solve.rs:57-326) as one
// launch per wave and direction: forward_solve_supernode (solve.rs:161-230)
// with the diagonal solve (solve.rs:232-252) folded into the backward pass,
// and backward_solve_supernode (solve.rs:254-326).
//
// Every front of the wave is cut into 64-row blocks; CTAs take blocks in
// ticket order from one atomic counter (front by front, and inside a front in
// dependency order), so a block only ever waits for blocks with a smaller
// ticket, which are held by CTAs that are already running: no deadlock, and
// no co-residency assumption beyond that.  Waits are bounded by the global
// timer; one that runs out sets *err and the solve goes on (the caller gets
// RVG_ERR_DEVICE_TIMEOUT).
//
// forward, per front (y kept in the front's work vector v, rows < ne):
//   diagonal block r (rows [64r, 64r + 64) of L11): y = x[col] - sum over the
//     finished column blocks b < r of L[rows, b] y_b (each as soon as it is
//     there), then the unit lower solve of the 64 x 64 diagonal block;
//     publish y_r;
//   L21 block (rows >= ne): -sum over all column blocks of L[rows, b] y_b,
//     added atomically into x at the parent's rows (siblings share rows).
// backward, per front, in ticket order:
//   gather tickets: the parent's final values at 64 rows of L21 into v + m
//     (rows >= ne);
//   partial-sum tickets: for a column block and a group of up to 8 L21 row
//     blocks, the sums L[rows, cols]^T x[rows] over the group, into a slot of
//     the wave's partial-sum buffer (the L21 reduction of one column block is
//     spread over CTAs, as the forward pass spreads its rows);
//   column blocks, descending (x_final in v + m): z = D^-1 y on the block's
//     columns (2x2 pairs may straddle blocks: y is still intact in v), minus
//     the block's partial sums in group order, minus L[rows of later blocks,
//     cols]^T x_final of those blocks (each once it is there), then the unit
//     upper solve (L11^T) of the diagonal block; x[col] = x_final.
//
// The chain of diagonal blocks bounds a large front (213 blocks for order
// 13,572), so what a block does between its predecessor's values and its own
// is kept short:
//   * the values are their own flags: the work vectors are filled with a
//     pattern no value takes (SF_EMPTY; NaN results are stored as the
//     canonical NaN), and a reader takes a value once it differs.  The next
//     block of the chain polls the values themselves (one trip through L2
//     instead of fence, flag, flag read and value read); the many blocks
//     further away watch one value with one thread, to keep the traffic on
//     those lines low;
//   * the sums over 64 columns run as interleaved chains (forward four with up to
//     two right-hand sides, two with more; backward four);
//   * the diagonal block is solved by eights (sf_diag): 8 or 16 short barriers
//     instead of 64 warp-serial steps, all right-hand sides side by side.
// What a solve needs to know of the factor (block layout, the front of each
// ticket) is uploaded once per factorization; ticket counters and flags of all
// waves are cleared together.
// Up to 8 right-hand sides go through one launch (template R), each L value
// read once for all of them.  Measured per block of the chain (order 13,572):
// forward 4.1 -> 3.3 us with one right-hand side, 32 -> 8.6 us with eight.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "front.cuh"

namespace rvg {

constexpr int SF_B = 64;                            // block rows / columns
constexpr uint64_t SF_TIMEOUT_NS = 1000000000ull;   // 1 s until the first wait gives up,
constexpr uint64_t SF_GIVEN_UP_NS = 1000000ull;     // 1 ms for each wait after that
constexpr int SF_PG = 8;  // backward: L21 row blocks per partial-sum ticket (512 rows)
constexpr int SF_BWD_DYN = SF_B * (SF_B + 1) * 8;  // k_sf_bwd's dynamic shared memory

// one front of a wave: its first ticket and its block counts
struct SfFront {
  int32_t s;      // supernode
  int32_t blk0;   // first ticket of the front
  int32_t nbd;    // diagonal blocks (ceil(ne / 64))
  int32_t nbr;    // L21 blocks (ceil((m - ne) / 64)): forward row blocks, backward gather tickets
  int32_t ngrp;   // backward: partial-sum tickets per column block (ceil(nbr / SF_PG))
  int32_t pslot;  // backward: the front's first partial-sum slot (R x 64 values each)
};

struct SfWave {
  const SfFront* fr;
  const int32_t* fmap;  // the position in fr of each ticket's front
  double* part;     // backward partial sums: slot q at part + q R 64
  int32_t nblk;
  int32_t* ticket;  // zeroed before the launch
  int32_t* flags;   // nblk entries, zeroed before the launch (backward: gathers and partial sums)
  double* x;        // solution vectors, permuted order: right-hand side r at x + r ldx
  int64_t ldx;
  double* work;     // per-front work at 2 R DFront::scratch: y (R x m) then x_final (R x m); SF_EMPTY before the pass
  int32_t* err;
};

__device__ __forceinline__ int32_t sf_ld_acquire(const int32_t* p) {
  int32_t v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void sf_st_release(int32_t* p, int32_t v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint64_t sf_timer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// A work value not written yet (all bits set).
constexpr unsigned long long SF_EMPTY = ~0ull;
__device__ __forceinline__ unsigned long long sf_peek(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void sf_publish(double* p, double v) {
  const unsigned long long b = v != v ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(v);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}
// Whether a wait that began at t0 has run out: after SF_TIMEOUT_NS, or after SF_GIVEN_UP_NS when another one has
// (a block may have to wait 1 + R times, and all that depends on it again: the limits must not add up).
__device__ __forceinline__ bool sf_run_out(uint64_t t0, int32_t* err) {
  const uint64_t dt = sf_timer() - t0;
  if (dt <= SF_GIVEN_UP_NS) return false;
  if (dt > SF_TIMEOUT_NS) {
    atomicExch(err, 2);
    return true;
  }
  return sf_ld_acquire(err) != 0;
}
// bounded wait for a published value
__device__ __forceinline__ double sf_take(const double* p, int32_t* err) {
  unsigned long long v = sf_peek(p);
  if (v == SF_EMPTY) {
    const uint64_t t0 = sf_timer();
    while ((v = sf_peek(p)) == SF_EMPTY)
      if (sf_run_out(t0, err)) return 0.0;
  }
  return __longlong_as_double((long long)v);
}
// The R values of a block's column t (at src + r m, t < n) into dst[r][t], by the whole CTA.  far: one
// thread watches the block's last column first.
template <int R>
__device__ __forceinline__ void sf_take_block(const double* src, int64_t m, int n, bool far, double (*dst)[SF_B],
                                              int32_t* err) {
  const int t = threadIdx.x;
  if (far) {
    if (t == 0) (void)sf_take(src + (R - 1) * m + n - 1, err);
    __syncthreads();
  }
  if (t < n) {
    unsigned long long v[R];  // every right-hand side's value in flight before the first is looked at
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = sf_peek(src + r * m + t);
#pragma unroll
    for (int r = 0; r < R; ++r)
      dst[r][t] = v[r] != SF_EMPTY ? __longlong_as_double((long long)v[r]) : sf_take(src + r * m + t, err);
  }
  __syncthreads();
}

// bounded wait for a published block (thread 0 of the CTA)
__device__ __forceinline__ void sf_wait(const int32_t* flag, int32_t* err) {
  if (sf_ld_acquire(flag)) return;
  const uint64_t t0 = sf_timer();
  while (!sf_ld_acquire(flag))
    if (sf_run_out(t0, err)) return;
}

__device__ __forceinline__ int32_t sf_col(const int32_t* rows, const int32_t* perm, int64_t i) { return rows[perm[i]]; }
__device__ __forceinline__ int32_t sf_row(const int32_t* rows, const int32_t* perm, int64_t ne, int64_t k,
                                          int64_t t) {
  const int64_t q = ne + t;
  return q < k ? rows[perm[q]] : rows[q];
}

// One row of a 64-column strip (columns at stride m) into dst[0, nc), 16
// loads in flight per thread (the loads are independent; issuing them before
// the first use keeps the row's memory latency from serialising).
__device__ __forceinline__ void sf_load_strip(const double* src, int64_t m, int nc, double* dst) {
#pragma unroll
  for (int c0 = 0; c0 < SF_B; c0 += 16) {
    double r[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) r[u] = c0 + u < nc ? __ldg(src + (int64_t)(c0 + u) * m) : 0.0;
#pragma unroll
    for (int u = 0; u < 16; ++u) dst[c0 + u] = r[u];
  }
}

// acc[r] -= sum_c l[c] y[r][c] over a 64-column strip: W interleaved chains per right-hand side
// (columns past the block hold l = 0, y is finite or the front's result is not)
template <int R>
__device__ __forceinline__ void sf_strip(const double (&l)[SF_B], int n, const double (*y)[SF_B], double (&acc)[R]) {
  constexpr int W = R <= 2 ? 4 : 2;  // chains: enough right-hand sides fill the pipe by themselves
#pragma unroll
  for (int r = 0; r < R; ++r) {
    double s[W];
#pragma unroll
    for (int u = 0; u < W; ++u) s[u] = 0.0;
#pragma unroll
    for (int c = 0; c < SF_B; ++c)
      if (c < n) s[c % W] = __fma_rn(-l[c], y[r][c], s[c % W]);
#pragma unroll
    for (int u = 0; u < W; ++u) acc[r] += s[u];
  }
}

// Unit triangular solve of a diagonal block of n <= 64 rows held in shared
// memory, row t of the R right-hand sides in acc of thread t; y is scratch.
// Lower: L(t, j) = Ld[t][j], from the top; upper (the transpose): Ld[j][t],
// from the bottom.  By eights: the 8 unknowns are solved (by thread r for
// right-hand side r, or by every thread for itself), then every remaining row
// takes their update.
template <int R, bool UPPER>
__device__ __forceinline__ void sf_diag(const double (*Ld)[SF_B + 1], int n, double (*y)[SF_B], double (&acc)[R]) {
  const int t = threadIdx.x;
  const int nb = (n + 7) / 8;
  if constexpr (R <= 2) {
    // few right-hand sides: every thread solves the 8 unknowns itself, from coefficients read before the
    // barrier, so a step is one barrier and one shared-memory trip
    for (int q = 0; q < nb; ++q) {
      const int j0 = (UPPER ? nb - 1 - q : q) * 8;
      const bool own = t >= j0 && t < j0 + 8;
      const bool later = UPPER ? t < j0 : (t >= j0 + 8 && t < n);
      if (own) {
#pragma unroll
        for (int r = 0; r < R; ++r) y[r][t] = t < n ? acc[r] : 0.0;
      }
      double cf[8][8], l[8];
#pragma unroll
      for (int a = 1; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < a; ++b) cf[a][b] = j0 + a < n ? Ld[j0 + a][j0 + b] : 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j) l[j] = later && j0 + j < n ? (UPPER ? Ld[j0 + j][t] : Ld[t][j0 + j]) : 0.0;
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = y[r][j0 + i];
        if (!UPPER) {
#pragma unroll
          for (int j = 0; j < 7; ++j)
#pragma unroll
            for (int i = j + 1; i < 8; ++i) v[i] = __fma_rn(-cf[i][j], v[j], v[i]);
        } else {
#pragma unroll
          for (int j = 7; j > 0; --j)
#pragma unroll
            for (int i = 0; i < j; ++i) v[i] = __fma_rn(-cf[j][i], v[j], v[i]);
        }
        if (own) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (t == j0 + i) acc[r] = v[i];
        } else {
          double e = 0.0, o = 0.0;
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            e = __fma_rn(-l[j], v[j], e);
            o = __fma_rn(-l[j + 1], v[j + 1], o);
          }
          if (later) acc[r] += e + o;
        }
      }
    }
    return;
  }
  for (int q = 0; q < nb; ++q) {
    const int j0 = (UPPER ? nb - 1 - q : q) * 8, j1 = j0 + 8 < n ? j0 + 8 : n;
    if (t >= j0 && t < j0 + 8) {
#pragma unroll
      for (int r = 0; r < R; ++r) y[r][t] = t < n ? acc[r] : 0.0;
    }
    __syncthreads();
    if (t < R) {
      double v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = y[t][j0 + i];
      if (!UPPER) {
#pragma unroll
        for (int j = 0; j < 7; ++j)
#pragma unroll
          for (int i = j + 1; i < 8; ++i)
            if (j0 + i < n) v[i] = __fma_rn(-Ld[j0 + i][j0 + j], v[j], v[i]);
      } else {
#pragma unroll
        for (int j = 7; j > 0; --j)
          if (j0 + j < n) {
#pragma unroll
            for (int i = 0; i < j; ++i) v[i] = __fma_rn(-Ld[j0 + j][j0 + i], v[j], v[i]);
          }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) y[t][j0 + i] = v[i];
    }
    __syncthreads();
    if (t >= j0 && t < j1) {
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = y[r][t];
    } else if (UPPER ? t < j0 : (t >= j1 && t < n)) {
      double l[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) l[j] = j0 + j < n ? (UPPER ? Ld[j0 + j][t] : Ld[t][j0 + j]) : 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = __fma_rn(-l[j], y[r][j0 + j], acc[r]);
    }
  }
}

// R right-hand sides at once: every L value is read once for all of them.
template <int R>
__global__ void __launch_bounds__(SF_B) k_sf_fwd(SfWave w, const DFront* F, Arenas A) {
  __shared__ int s_blk;
  __shared__ double yb[R][SF_B];
  __shared__ double Ls[SF_B][SF_B + 1];
  const int t = threadIdx.x;
  chain_enter();  // (launched while the wave before still runs)
  for (;;) {
    if (t == 0) s_blk = atomicAdd(w.ticket, 1);
    __syncthreads();
    const int blk = s_blk;
    __syncthreads();
    if (blk >= w.nblk) break;
    const SfFront sf = w.fr[w.fmap[blk]];
    const DFront fr = F[sf.s];
    const int64_t m = fr.m, ne = fr.ne;
    const double* L = A.panel + fr.panel;
    const int32_t* rows = A.idx + fr.idx;
    const int32_t* perm = rows + m;
    double* v = w.work + 2 * R * fr.scratch;  // y of right-hand side r at v + r m
    const int b = blk - sf.blk0;
    const bool diag = b < sf.nbd;
    const int64_t r0 = diag ? (int64_t)b * SF_B : ne + (int64_t)(b - sf.nbd) * SF_B;
    const int64_t r1 = diag ? (r0 + SF_B < ne ? r0 + SF_B : ne) : (r0 + SF_B < m ? r0 + SF_B : m);
    const int64_t i = r0 + t;
    const bool row = i < r1;
    double acc[R];
    if (diag && row) {
      const int32_t g = sf_col(rows, perm, i);
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = w.x[r * w.ldx + g];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = 0.0;
    }
    // The factor is final: the L strips are read before the waits on the
    // blocks they multiply, so only the y values are on the chain.
    const int nr = (int)(r1 - r0);
    if (diag && row) sf_load_strip(L + i + r0 * m, m, nr, &Ls[t][0]);  // the diagonal block, staged early
    const int ncb = diag ? b : sf.nbd;
    for (int cb = 0; cb < ncb; ++cb) {
      const int64_t c0 = (int64_t)cb * SF_B;
      const int nc = (int)((c0 + SF_B < ne ? c0 + SF_B : ne) - c0);
      double lr[SF_B];
      if (row) sf_load_strip(L + i + c0 * m, m, nc, lr);
      sf_take_block<R>(v + c0, m, nc, !(diag && cb == b - 1), yb, w.err);
      if (row) sf_strip<R>(lr, nc, yb, acc);
      __syncthreads();
    }
    if (diag) {
      __syncthreads();  // the staged diagonal block
      sf_diag<R, false>(Ls, nr, yb, acc);
      if (row) {
#pragma unroll
        for (int r = 0; r < R; ++r) sf_publish(&v[r * m + i], acc[r]);
      }
      __syncthreads();  // Ls and yb are free again
    } else if (row) {
      const int32_t g = sf_row(rows, perm, ne, fr.k, i - ne);
#pragma unroll
      for (int r = 0; r < R; ++r) atomicAdd(&w.x[r * w.ldx + g], acc[r]);
    }
  }
}

// z = D^-1 y for column c of a front (MixedDiagonal::solve_in_place,
// diagonal.rs:312-360: zero pivots give 0, 2x2 blocks by Cramer's rule)
__device__ __forceinline__ double sf_dinv(const DFront& fr, const Arenas& A, const double* y, int64_t c) {
  const int8_t* dt = A.dtype + fr.dpos;
  const double* dd = A.ddiag + fr.dpos;
  const double* dof = A.doff + fr.dpos;
  if (dt[c] == PT_1X1) {
    const double d = dd[c];
    return d == 0.0 ? 0.0 : __ddiv_rn(y[c], d);
  }
  const int64_t c0 = dt[c] == PT_2X2 ? c : c - 1;
  const double a = dd[c0], b = dof[c0], cc = dd[c0 + 1];
  const double det = __dsub_rn(__dmul_rn(a, cc), __dmul_rn(b, b));
  const double r1 = y[c0], r2 = y[c0 + 1];
  if (det == 0.0) return 0.0;
  return c == c0 ? __ddiv_rn(__dsub_rn(__dmul_rn(cc, r1), __dmul_rn(b, r2)), det)
                 : __ddiv_rn(__dsub_rn(__dmul_rn(a, r2), __dmul_rn(b, r1)), det);
}

template <int R>
__global__ void __launch_bounds__(SF_B) k_sf_bwd(SfWave w, const DFront* F, Arenas A) {
  __shared__ int s_blk;
  __shared__ double Ls[SF_B][SF_B + 1];
  // a column block's diagonal block, staged before its waits (dynamic shared memory: SF_BWD_DYN bytes)
  extern __shared__ double sf_dyn[];
  double(*Ld)[SF_B + 1] = reinterpret_cast<double(*)[SF_B + 1]>(sf_dyn);
  __shared__ double xs[R][SF_B];
  const int t = threadIdx.x;
  chain_enter();  // (launched while the wave before still runs)
  for (;;) {
    if (t == 0) s_blk = atomicAdd(w.ticket, 1);
    __syncthreads();
    const int blk = s_blk;
    __syncthreads();
    if (blk >= w.nblk) break;
    const SfFront sf = w.fr[w.fmap[blk]];
    const DFront fr = F[sf.s];
    const int64_t m = fr.m, ne = fr.ne;
    const double* L = A.panel + fr.panel;
    const int32_t* rows = A.idx + fr.idx;
    const int32_t* perm = rows + m;
    const double* y = w.work + 2 * R * fr.scratch;  // forward results of right-hand side r at y + r m
    double* xf = w.work + 2 * R * fr.scratch + R * m;  // final values of this front's columns, at xf + r m
    int32_t* flags = w.flags + sf.blk0;
    const int nbr = sf.nbr, ngrp = sf.ngrp;
    const int lt = blk - sf.blk0;  // ticket within the front
    const int npart = sf.nbd * ngrp;
    if (lt < nbr) {
      // gather ticket: the parent's final values at 64 rows of L21 into xf
      const int64_t i = ne + (int64_t)lt * SF_B + t;
      if (i < m) {
        const int32_t g = sf_row(rows, perm, ne, fr.k, i - ne);
#pragma unroll
        for (int r = 0; r < R; ++r) xf[r * m + i] = w.x[r * w.ldx + g];
      }
      __threadfence();
      __syncthreads();
      if (t == 0) sf_st_release(&flags[lt], 1);
      continue;
    }
    if (lt < nbr + npart) {
      // partial-sum ticket (column blocks descending, groups ascending)
      const int pq = lt - nbr;
      const int b = sf.nbd - 1 - pq / ngrp, gi = pq % ngrp;
      const int64_t c0 = (int64_t)b * SF_B;
      const int nc = (int)((c0 + SF_B < ne ? c0 + SF_B : ne) - c0);
      double ps[R];
#pragma unroll
      for (int r = 0; r < R; ++r) ps[r] = 0.0;
      const int rb1 = (gi + 1) * SF_PG < nbr ? (gi + 1) * SF_PG : nbr;
      for (int rb = gi * SF_PG; rb < rb1; ++rb) {
        if (t == 0) sf_wait(&flags[rb], w.err);
        const int64_t i0 = ne + (int64_t)rb * SF_B;
        const int nr = (int)((i0 + SF_B < m ? i0 + SF_B : m) - i0);
        __syncthreads();
        if (t < nr) {
#pragma unroll
          for (int r = 0; r < R; ++r) xs[r][t] = __ldcg(&xf[r * m + i0 + t]);
          sf_load_strip(L + i0 + t + c0 * m, m, nc, &Ls[t][0]);
        }
        __syncthreads();
        if (t < nc)
          for (int rr = 0; rr < nr; ++rr) {
            const double l = Ls[rr][t];
#pragma unroll
            for (int r = 0; r < R; ++r) ps[r] = __fma_rn(l, xs[r][rr], ps[r]);
          }
      }
      double* slot = w.part + ((int64_t)sf.pslot + pq) * R * SF_B;
#pragma unroll
      for (int r = 0; r < R; ++r) slot[r * SF_B + t] = ps[r];
      __threadfence();
      __syncthreads();
      if (t == 0) sf_st_release(&flags[lt], 1);
      continue;
    }
    const int q = lt - nbr - npart;  // column blocks, descending
    const int b = sf.nbd - 1 - q;
    const int64_t c0 = (int64_t)b * SF_B;
    const int nc = (int)((c0 + SF_B < ne ? c0 + SF_B : ne) - c0);
    const bool col = t < nc;
    if (col) sf_load_strip(L + (c0 + t) + c0 * m, m, nc, &Ld[t][0]);  // Ld[row][col]; the factor is final
    double acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = col ? sf_dinv(fr, A, y + r * m, c0 + t) : 0.0;
    // the block's L21 partial sums, in group order
    for (int gi = 0; gi < ngrp; ++gi) {
      const int pq = q * ngrp + gi;
      if (t == 0) sf_wait(&flags[nbr + pq], w.err);
      __syncthreads();
      const double* slot = w.part + ((int64_t)sf.pslot + pq) * R * SF_B;
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = __dsub_rn(acc[r], __ldcg(&slot[r * SF_B + t]));
    }
    // rows of later diagonal blocks, from the last one down, as they finish; each strip is in shared memory
    // before the wait on its block
    for (int rblk = sf.nbd - 1; rblk > b; --rblk) {
      const int64_t i0 = (int64_t)rblk * SF_B;
      const int nr = (int)((i0 + SF_B < ne ? i0 + SF_B : ne) - i0);
      __syncthreads();  // the strip before it has been used
      if (t < nr) sf_load_strip(L + i0 + t + c0 * m, m, nc, &Ls[t][0]);
      sf_take_block<R>(xf + i0, m, nr, rblk != b + 1, xs, w.err);
      if (col) {
        double s[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r) s[r][0] = s[r][1] = s[r][2] = s[r][3] = 0.0;
        int rr = 0;
        for (; rr + 4 <= nr; rr += 4)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const double l = Ls[rr + u][t];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r][u] = __fma_rn(-l, xs[r][rr + u], s[r][u]);
          }
        for (; rr < nr; ++rr) {
          const double l = Ls[rr][t];
#pragma unroll
          for (int r = 0; r < R; ++r) s[r][0] = __fma_rn(-l, xs[r][rr], s[r][0]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] += (s[r][0] + s[r][1]) + (s[r][2] + s[r][3]);
      }
    }
    // the diagonal block: x_c = acc_c - sum_{c < i < c0 + nc} L(i, c) x_i, from the bottom
    __syncthreads();
    sf_diag<R, true>(Ld, nc, xs, acc);
    if (col) {
      const int32_t g = sf_col(rows, perm, c0 + t);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        sf_publish(&xf[r * m + c0 + t], acc[r]);
        w.x[r * w.ldx + g] = acc[r];
      }
    }
    __syncthreads();  // Ld and xs are free again
  }
}

}  // namespace rvg
