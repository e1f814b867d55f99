// Bunch-Kaufman building blocks shared by the level-scheduled factorization
// (numeric.cu) and the batched QP solver (batch.cu): the Bunch-Kaufman
// factorization of one supernode diagonal block (LAPACK dsytrf('L') pivot rule,
// alpha = (1+sqrt(17))/8) with explicit interchanges, the inverse of its D, and
// the solve of the rows below the block.
#pragma once
#include <cuda_runtime.h>

#include "plan.hpp"

namespace nqg {
namespace {

constexpr int BK_SMALL = 64;       // diagonal blocks up to this width live in shared memory
constexpr int BK_SMALL_ROWS = 64;  // rows below that their kernel stages at a time

__device__ __forceinline__ void flag_status(int *st, int bits) { atomicOr(st, bits); }

// Magnitude, the sign bit cleared also for -0 and NaN: the searches below order
// its bits.
[[maybe_unused]] __device__ __forceinline__ float tabs(float v) { return fabsf(v); }
[[maybe_unused]] __device__ __forceinline__ double tabs(double v) { return fabs(v); }

// Warp-wide argmax of |value| with the smallest index winning ties (the
// LAPACK idamax convention) over the lanes that have one (idx >= 0); every
// lane returns the winner.  The bits of a floating-point number with a clear
// sign (v comes from tabs; with its sign bit -0.0 would beat every value) order
// like an integer: two integer reductions and a vote instead of a tree of
// compares (an FP64 compare holds the FP64 pipe of the SM quarter for 64
// cycles).
[[maybe_unused]] __device__ __forceinline__ void warp_argmax(float &v, int &idx) {
  const unsigned FULL = 0xffffffffu;
  const unsigned key = idx >= 0 ? __float_as_uint(v) + 1u : 0u;
  const unsigned best = __reduce_max_sync(FULL, key);
  const int win = __reduce_min_sync(FULL, best && key == best ? idx : 0x7fffffff);
  const unsigned who = __ballot_sync(FULL, idx == win);
  v = __shfl_sync(FULL, v, who ? __ffs(who) - 1 : 0);
  idx = best ? win : -1;
}
[[maybe_unused]] __device__ __forceinline__ void warp_argmax(double &v, int &idx) {
  const unsigned FULL = 0xffffffffu;
  const bool has = idx >= 0;
  const unsigned hi = has ? (unsigned)__double2hiint(v) + 1u : 0u;
  const unsigned bh = __reduce_max_sync(FULL, hi);
  const bool top = has && hi == bh;
  const unsigned lo = top ? (unsigned)__double2loint(v) : 0u;
  const unsigned bl = __reduce_max_sync(FULL, lo);
  const int win = __reduce_min_sync(FULL, top && lo == bl ? idx : 0x7fffffff);
  const unsigned who = __ballot_sync(FULL, idx == win);
  v = __shfl_sync(FULL, v, who ? __ffs(who) - 1 : 0);
  idx = bh ? win : -1;
}

// Lanes (rows of 32, two rows deep) to one candidate each: the larger, the
// smaller index on ties.
template <class T> __device__ __forceinline__ void take_larger(T &v, int &i, T v2, int i2) {
  if (i2 >= 0 && (i < 0 || v2 > v)) {
    v = v2;
    i = i2;
  }
}

// Bunch-Kaufman (alpha = (1+sqrt(17))/8, the LAPACK dsytf2('L') pivot rule
// and the reference's reorder_after_sytrf form: explicit interchanges, L with
// unit diagonal, D / E the diagonal and 2x2 sub-diagonals, perm[m] = original
// local column at position m) on a lower-stored block of at most 64 columns.
// Every warp of the group finds the pivot by itself from the shared block (no
// broadcast to wait for), and the trailing columns are dealt to the warps, a
// lane per row.  wi of nw: this warp's place in the group that calls together;
// nw = 1 synchronizes the warp only.  Returns whether any interchange happened.
// A 22-column FP64 block took about 100k cycles by one warp whose lanes walked
// their rows' columns one after another (w^2 / 2 multiply-adds of 64 cycles).
template <class T>
__device__ __forceinline__ bool bk_block(T *a, int lda, int w, T *D, T *E, int *perm, int *status, int wi, int nw) {
  const unsigned FULL = 0xffffffffu;
  const T alpha = (T)((1.0 + sqrt(17.0)) / 8.0);
  const int lane = threadIdx.x & 31;
  auto sync = [&]() {
    if (nw > 1) __syncthreads();
    else __syncwarp();
  };
  bool pivoted = false;
  if (wi == 0)
#pragma unroll 1
    for (int m = lane; m < w; m += 32) perm[m] = m;
  int k = 0;
  while (k < w) {
    const T akk = a[k + k * lda], absakk = tabs(akk);
    // rows k+1+lane and k+33+lane of column k
    const int i0 = k + 1 + lane, i1 = i0 + 32;
    T c0 = i0 < w ? a[i0 + k * lda] : T(0), c1 = i1 < w ? a[i1 + k * lda] : T(0);
    T cv = tabs(c0);
    int ci = i0 < w ? i0 : -1;
    warp_argmax(cv, ci);
    if (w - k > 33) {
      T v2 = tabs(c1);
      int j2 = i1 < w ? i1 : -1;
      warp_argmax(v2, j2);
      take_larger(cv, ci, v2, j2);
    }
    const T colmax = ci >= 0 ? cv : T(0);
    const int imax = ci;
    int kp = k, kstep = 1, zero = 0;
    if ((absakk >= colmax ? absakk : colmax) == T(0) || absakk != absakk) {
      zero = 1;
    } else if (!(absakk >= alpha * colmax)) {
      T rv = T(-1);
      int ri = -1;
#pragma unroll 1
      for (int b = k; b < w; b += 32) {
        const int j = b + lane;
        int jj = j < w && j != imax ? j : -1;
        T v = jj < 0 ? T(0) : (j < imax ? tabs(a[imax + j * lda]) : tabs(a[j + imax * lda]));
        warp_argmax(v, jj);
        take_larger(rv, ri, v, jj);
      }
      const T rowmax = rv;
      if (!(absakk >= alpha * colmax * (colmax / rowmax))) {
        kp = imax;
        if (!(tabs(a[imax + imax * lda]) >= alpha * rowmax)) kstep = 2;
      }
    }
    const int kk = k + kstep - 1;
    if (zero && wi == 0 && lane == 0) atomicOr(status, absakk == absakk ? ST_ZERO_PIVOT : ST_NONFINITE);
    sync();
    if (kp != kk) {  // symmetric interchange of kk and kp (kp > kk), by the first warp
      pivoted = true;
      if (wi == 0) {
#pragma unroll 1
        for (int i = kp + 1 + lane; i < w; i += 32) {
          const T t = a[i + kk * lda];
          a[i + kk * lda] = a[i + kp * lda];
          a[i + kp * lda] = t;
        }
#pragma unroll 1
        for (int j = kk + 1 + lane; j < kp; j += 32) {
          const T t = a[j + kk * lda];
          a[j + kk * lda] = a[kp + j * lda];
          a[kp + j * lda] = t;
        }
        const int ncols_left = kstep == 2 ? k + 1 : k;
#pragma unroll 1
        for (int cc = lane; cc < ncols_left; cc += 32) {
          const T t = a[kk + cc * lda];
          a[kk + cc * lda] = a[kp + cc * lda];
          a[kp + cc * lda] = t;
        }
        if (lane == 0) {
          const T t = a[kk + kk * lda];
          a[kk + kk * lda] = a[kp + kp * lda];
          a[kp + kp * lda] = t;
          const int pt = perm[kk];
          perm[kk] = perm[kp];
          perm[kp] = pt;
        }
      }
      sync();
    }
    if (kstep == 1) {
      const T d = kp != kk ? a[k + k * lda] : akk;
      if (kp != kk) {
        c0 = i0 < w ? a[i0 + k * lda] : T(0);
        c1 = i1 < w ? a[i1 + k * lda] : T(0);
      }
      if (!zero) {
        const T r1 = T(1) / d;
        const T m0 = r1 * c0;  // multipliers, row i0 (and i1)
        T m1 = T(0);
        if (w - k > 33) m1 = r1 * c1;
        // column j by warp (j - k - 1) mod nw: rows i >= j, four columns at a time
#pragma unroll 1
        for (int j = k + 1 + wi; j < w; j += 4 * nw) {
          T v[4], mj[4];
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int jj = j + h * nw, q = jj - k - 1;
            v[h] = i0 >= jj && i0 < w ? a[i0 + jj * lda] : T(0);
            mj[h] = q < 32 ? __shfl_sync(FULL, m0, q & 31) : __shfl_sync(FULL, m1, q & 31);
          }
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int jj = j + h * nw;
            if (jj < w) v[h] -= mj[h] * c0;
            if (i0 >= jj && i0 < w) a[i0 + jj * lda] = v[h];
          }
          if (w - k > 33)
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int jj = j + h * nw;
              if (i1 >= jj && i1 < w) a[i1 + jj * lda] -= mj[h] * c1;
            }
        }
        sync();  // every warp has read column k
        if (wi == 0) {
          if (i0 < w) a[i0 + k * lda] = m0;
          if (i1 < w) a[i1 + k * lda] = m1;
        }
      }
      if (wi == 0 && lane == 0) {
        D[k] = d;
        E[k] = T(0);
      }
    } else {
      // 2x2 pivot on rows/cols k, k+1
      const T a11 = a[k + k * lda], a21 = a[k + 1 + k * lda], a22 = a[k + 1 + (k + 1) * lda];
      const T i21 = T(1) / a21;
      const T d11 = a22 * i21, d22 = a11 * i21;
      const T d21 = (T(1) / (d11 * d22 - T(1))) * i21;
      const int p0 = k + 2 + lane, p1 = p0 + 32;
      T x0 = T(0), y0 = T(0), x1 = T(0), y1 = T(0);
      if (p0 < w) {
        x0 = a[p0 + k * lda];
        y0 = a[p0 + (k + 1) * lda];
      }
      if (p1 < w) {
        x1 = a[p1 + k * lda];
        y1 = a[p1 + (k + 1) * lda];
      }
      const T u0 = d21 * (d11 * x0 - y0), v0 = d21 * (d22 * y0 - x0);
      T u1 = T(0), v1 = T(0);
      if (w - k > 34) {
        u1 = d21 * (d11 * x1 - y1);
        v1 = d21 * (d22 * y1 - x1);
      }
#pragma unroll 2
      for (int j = k + 2 + wi; j < w; j += nw) {
        const int q = j - k - 2;
        const T uj = q < 32 ? __shfl_sync(FULL, u0, q & 31) : __shfl_sync(FULL, u1, q & 31);
        const T vj = q < 32 ? __shfl_sync(FULL, v0, q & 31) : __shfl_sync(FULL, v1, q & 31);
        if (p0 >= j && p0 < w) a[p0 + j * lda] -= x0 * uj + y0 * vj;
        if (w - k > 34 && p1 >= j && p1 < w) a[p1 + j * lda] -= x1 * uj + y1 * vj;
      }
      sync();
      if (wi == 0) {
        if (p0 < w) {
          a[p0 + k * lda] = u0;
          a[p0 + (k + 1) * lda] = v0;
        }
        if (p1 < w) {
          a[p1 + k * lda] = u1;
          a[p1 + (k + 1) * lda] = v1;
        }
        if (lane == 0) {
          D[k] = a11;
          D[k + 1] = a22;
          E[k] = a21;
          E[k + 1] = T(0);
          a[k + 1 + k * lda] = T(0);
        }
      }
    }
    sync();
    k += kstep;
  }
  if (wi == 0)
#pragma unroll 1
    for (int m = lane; m < w; m += 32) a[m + m * lda] = T(1);
  sync();
  return pivoted;
}

// The same of a block of any width (and of blocks in global memory), by the
// whole CTA: every warp finds the pivot by itself, the trailing columns are
// dealt to the warps, a step's multipliers wait in the strict upper triangle
// (its rows k, k + 1, which are zeroed again).  Three barriers a step.
// Columns before k0 are final (bk_blocked).
template <class T>
__device__ void bk_factor(T *a, int lda, int w, T *D, T *E, int *perm, int *status, bool *pivoted_out, int k0 = 0) {
  const T alpha = (T)((1.0 + sqrt(17.0)) / 8.0);
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wi = tid >> 5, nw = nt >> 5;
  bool pivoted = false;
  for (int m = tid; m < w; m += nt) perm[m] = m;
  __syncthreads();
  auto at = [&](int i, int j) -> T & { return a[i + (size_t)j * lda]; };
  int k = k0;
#pragma unroll 1
  while (k < w) {
    const T akk = at(k, k), absakk = tabs(akk);
    T cv = T(0);
    int ci = -1;
#pragma unroll 1
    for (int i = k + 1 + lane; i < w; i += 32) take_larger(cv, ci, tabs(at(i, k)), i);
    warp_argmax(cv, ci);
    const T colmax = ci >= 0 ? cv : T(0);
    const int imax = ci;
    int kp = k, kstep = 1, zero = 0;
    if ((absakk >= colmax ? absakk : colmax) == T(0) || absakk != absakk) {
      zero = 1;
    } else if (!(absakk >= alpha * colmax)) {
      // rowmax: off-diagonal max of row/column imax inside the trailing block
      T rv = T(0);
      int ri = -1;
#pragma unroll 1
      for (int j = k + lane; j < w; j += 32)
        if (j != imax) take_larger(rv, ri, j < imax ? tabs(at(imax, j)) : tabs(at(j, imax)), j);
      warp_argmax(rv, ri);
      const T rowmax = rv;
      if (!(absakk >= alpha * colmax * (colmax / rowmax))) {
        kp = imax;
        if (!(tabs(at(imax, imax)) >= alpha * rowmax)) kstep = 2;
      }
    }
    const int kk = k + kstep - 1;
    // a NaN pivot is reported by the non-finite check, not as a zero pivot
    if (zero && tid == 0 && absakk == absakk) flag_status(status, ST_ZERO_PIVOT);
    __syncthreads();
    if (kp != kk) {  // symmetric interchange of kk and kp (kp > kk)
      pivoted = true;
      for (int i = kp + 1 + tid; i < w; i += nt) {
        const T t = at(i, kk);
        at(i, kk) = at(i, kp);
        at(i, kp) = t;
      }
      for (int j = kk + 1 + tid; j < kp; j += nt) {
        const T t = at(j, kk);
        at(j, kk) = at(kp, j);
        at(kp, j) = t;
      }
      // rows kk and kp of the columns to the left of the current pivot
      // (for a 2x2 pivot this includes column k: LAPACK swaps A(k+1,k), A(kp,k))
      const int ncols_left = kstep == 2 ? k + 1 : k;
      for (int c = tid; c < ncols_left; c += nt) {
        const T t = at(kk, c);
        at(kk, c) = at(kp, c);
        at(kp, c) = t;
      }
      if (tid == 0) {
        const T t = at(kk, kk);
        at(kk, kk) = at(kp, kp);
        at(kp, kp) = t;
        const int pt = perm[kk];
        perm[kk] = perm[kp];
        perm[kp] = pt;
      }
      __syncthreads();
    }
    if (kstep == 1) {
      const T d = at(k, k);
      if (!zero) {
        const T r1 = T(1) / d;
        for (int i = k + 1 + tid; i < w; i += nt) at(k, i) = r1 * at(i, k);
        __syncthreads();
#pragma unroll 1
        for (int j = k + 1 + wi; j < w; j += nw) {
          const T mj = at(k, j);
#pragma unroll 2
          for (int i = j + lane; i < w; i += 32) at(i, j) -= mj * at(i, k);
        }
        __syncthreads();
        for (int i = k + 1 + tid; i < w; i += nt) {
          at(i, k) = at(k, i);
          at(k, i) = T(0);
        }
      }
      if (tid == 0) {
        D[k] = d;
        E[k] = T(0);
      }
    } else {
      // 2x2 pivot on rows/cols k, k+1
      const T a11 = at(k, k), a21 = at(k + 1, k), a22 = at(k + 1, k + 1);
      const T i21 = T(1) / a21;
      const T d11 = a22 * i21, d22 = a11 * i21;
      const T d21 = (T(1) / (d11 * d22 - T(1))) * i21;
      for (int j = k + 2 + tid; j < w; j += nt) {
        const T x = at(j, k), y = at(j, k + 1);
        at(k, j) = d21 * (d11 * x - y);
        at(k + 1, j) = d21 * (d22 * y - x);
      }
      __syncthreads();
#pragma unroll 1
      for (int j = k + 2 + wi; j < w; j += nw) {
        const T uj = at(k, j), vj = at(k + 1, j);
#pragma unroll 2
        for (int i = j + lane; i < w; i += 32) at(i, j) -= at(i, k) * uj + at(i, k + 1) * vj;
      }
      __syncthreads();
      for (int j = k + 2 + tid; j < w; j += nt) {
        at(j, k) = at(k, j);
        at(j, k + 1) = at(k + 1, j);
        at(k, j) = T(0);
        at(k + 1, j) = T(0);
      }
      if (tid == 0) {
        D[k] = a11;
        D[k + 1] = a22;
        E[k] = a21;
        E[k + 1] = T(0);
        at(k + 1, k) = T(0);
      }
    }
    // the next search reads columns from k + kstep on: final since the last barrier
    k += kstep;
  }
  __syncthreads();
  for (int m = tid; m < w; m += nt) at(m, m) = T(1);
  __syncthreads();
  if (pivoted_out) *pivoted_out = pivoted;
}

// The leading columns of bk_factor's block that need no interchange, eight at a
// time: one warp factors the 8 x 8 diagonal, a thread per row solves the rows
// below against it and tests the Bunch-Kaufman rule for its entries, and only
// if all pass is the step stored and the rest of the block updated.  Returns the
// columns done (a multiple of 8); entries get the same multiply-adds in the same
// order as in bk_factor, which takes over from there.  A column at a time costs
// three barriers, a search and an update of 8 dependent reads, 6700 cycles at 130
// columns of FP64.  256 threads, at most that many columns.
template <class T> __device__ int bk_blocked(T *a, int lda, int w, T *D, T *E) {
  constexpr int B = 8, CAP = 256;
  __shared__ T Ls[B][CAP], Ld[B][B], rinv[B], dv[B];
  if (w > CAP || blockDim.x != CAP) return 0;
  const T alpha = (T)((1.0 + sqrt(17.0)) / 8.0);
  const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5, nw = CAP / 32;
  int b = 0;
#pragma unroll 1
  for (; b + B <= w; b += B) {
    T *ab = a + b + (size_t)b * lda;
    const int m = w - b - B;
    bool ok = true;
    if (wi == 0) {
      T v[B];
      const int q = min(lane, B - 1);
#pragma unroll
      for (int c = 0; c < B; ++c) v[c] = ab[q + (size_t)min(c, q) * lda];
#pragma unroll
      for (int t = 0; t < B; ++t) {
        const T d = __shfl_sync(0xffffffffu, v[t], t), r1 = T(1) / d, l = v[t] * r1;
        if (q > t) ok = ok && tabs(d) >= alpha * tabs(v[t]);
        ok = ok && tabs(d) > T(0);
#pragma unroll
        for (int c = t + 1; c < B; ++c) v[c] -= __shfl_sync(0xffffffffu, l, c) * v[t];
        if (lane < B) Ld[t][lane] = l;
        if (lane == 0) {
          rinv[t] = r1;
          dv[t] = d;
        }
      }
    }
    __syncthreads();
    T x[B], lx[B];
    T *row = ab + B + min(tid, max(m - 1, 0));
    if (tid < m) {
#pragma unroll
      for (int c = 0; c < B; ++c) x[c] = row[(size_t)c * lda];
#pragma unroll
      for (int c = 0; c < B; ++c) {
#pragma unroll
        for (int t = 0; t < c; ++t) x[c] -= Ld[t][c] * x[t];
        lx[c] = x[c] * rinv[c];
        ok = ok && tabs(dv[c]) >= alpha * tabs(x[c]);
      }
    }
    if (!__syncthreads_and(ok)) break;
    if (tid < m) {
#pragma unroll
      for (int c = 0; c < B; ++c) {
        row[(size_t)c * lda] = x[c];
        Ls[c][tid] = lx[c];
      }
    }
    if (tid < B) {
      for (int t = 0; t < tid; ++t) ab[tid + (size_t)t * lda] = Ld[t][tid];
      D[b + tid] = dv[tid];
      E[b + tid] = T(0);
    }
    __syncthreads();
#pragma unroll 1
    for (int j = wi; j < m; j += nw) {
      T lj[B];
#pragma unroll
      for (int t = 0; t < B; ++t) lj[t] = Ls[t][j];
#pragma unroll 1
      for (int i = j + lane; i < m; i += 32) {
        T *e = ab + B + i;
        T y = e[(size_t)(B + j) * lda];
#pragma unroll
        for (int t = 0; t < B; ++t) y -= lj[t] * e[(size_t)t * lda];
        e[(size_t)(B + j) * lda] = y;
      }
    }
    __syncthreads();
    if (tid < m)
#pragma unroll
      for (int c = 0; c < B; ++c) row[(size_t)c * lda] = lx[c];
  }
  __syncthreads();
  return b;
}

// Largest diagonal block k_bk_global stages in shared memory (bytes).
constexpr size_t BKG_STAGE_MAX = 200 * 1024;

// D^-1 of a block as diagonal and 2x2 off-diagonal: entry m of both (D, E: the
// w diagonals and 2x2 sub-diagonals; 2x2 pivots by Cramer's rule, the
// arithmetic of blocked_2by2_solver, Sym_BLAS.cpp:492-529).
template <class T>
__device__ __forceinline__ void d_inverse(const T *D, const T *E, int w, int m, T &inv, T &off) {
  const bool first = m + 1 < w && E[m] != T(0), second = m > 0 && E[m - 1] != T(0);
  off = T(0);
  if (first || second) {
    const int k = second ? m - 1 : m;
    const T e = E[k], det = T(1) / (D[k] * D[k + 1] - e * e);
    inv = det * D[second ? k : k + 1];
    if (first) off = -e * det;
  } else {
    inv = T(1) / D[m];
  }
}

// Block-wide OR of a per-thread flag.
__device__ bool block_any(bool f) { return __syncthreads_or(f ? 1 : 0) != 0; }

// Rows of X (m x w, entry (r, j) at X[r * lr + j * lj], columns already in pivot
// order) times L11^-T, by nt threads (tid) that call together: column j is
// final, the later ones lose x_j L11(t, j), so that each entry receives its
// terms in increasing j, as in the substitution.  L11(t, j) at L[t * li + j * ld].
template <class T>
__device__ __forceinline__ void rows_solve(T *X, int m, int w, int lr, int lj, const T *L, int li, int ld, int tid,
                                           int nt) {
  // a lane keeps its row: R of them, the other index over nt / R
  int R = 32;
  while (nt % (2 * R) == 0 && R < m) R *= 2;  // nt need not be a power of two
  const int rr = tid & (R - 1), cq = tid / R, cs = nt / R;
#pragma unroll 1
  for (int j = 0; j + 1 < w; ++j) {
    for (int r = rr; r < m; r += R) {
      T *xr = X + r * lr;
      const T xj = xr[j * lj];
      int t = j + 1 + cq;
#pragma unroll 1
      for (; t + 3 * cs < w; t += 4 * cs) {
        T l[4], v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          l[q] = L[(t + q * cs) * li + j * ld];
          v[q] = xr[(t + q * cs) * lj];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) xr[(t + q * cs) * lj] = v[q] - xj * l[q];
      }
      for (; t < w; t += cs) xr[t * lj] -= xj * L[t * li + j * ld];
    }
    if (cs > 1) __syncthreads();
  }
  __syncthreads();
}

}  // namespace
}  // namespace nqg
