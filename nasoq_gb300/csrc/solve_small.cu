// The refined solve of a small FP64 plan as one launch: triangular solves, D^-1,
// residuals and the GMRES loop of gmres_refine (solve.cu), whose level kernels
// and dot products are hundreds of launches of a few microseconds each on a
// system of a few thousand columns (a QP's active-set iteration solves one such
// system per step; 74 tree levels at 576 variables and 284 general rows: 106
// level kernels per application, 6 us each).
//
// Forward / backward sweeps: reference H2LeveledBlockedLsolve / LTsolve
// (src/triangularSolve/Triangular_BCSC.cpp:378-446, 534-600); D: 1x1 and 2x2
// blocks (blocked_2by2_solver, src/common/Sym_BLAS.cpp:492-529); GMRES:
// pmgmres_ldlt_auto (src/gmres/mgmres.cpp:1015-1211).
//
// One cluster of eight CTAs does all of it; the vectors live in L2, a level of
// the tree ends with a cluster barrier.  What bounds it is latency: per level
// 5000 to 15000 cycles (dependent reads of 330 cycles at L2, 95 at L1; 380 cycles
// for the barrier alone, 1000 to 2000 after stores and reductions), and per 32
// columns of a wide block 2300 and, for what its columns take from the ones
// before, 512 per chunk.  FP64 itself (one warp instruction per SM quarter and 64
// cycles) is why one CTA was not enough.  The solve of 4820 columns in 10 levels:
// 1.98 ms with the level kernels, 1.79 on one SM, 0.99 on eight with
// substitutions, 0.83 with inverted 32 x 32 triangles; 916 columns in 83
// levels: 6.1, 2.65, 1.29 and 1.03 ms.
// Loads are issued eight at a time before they are used, and never under a
// condition; entries below a block are added with reductions at L2.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "plan.hpp"

namespace nqg {

namespace {

constexpr int SS_CTAS = 8;            // CTAs of the cluster
constexpr int SS_THREADS = 256, SS_WARPS = SS_THREADS / 32;
constexpr int SS_ALL = SS_CTAS * SS_THREADS;
constexpr int SS_MR = 16;             // Krylov steps per restart
constexpr int SS_LONG = 16;           // rows of a single column above which it takes a warp
constexpr int SS_WARP_BLOCK = 128;    // rows x columns of the largest block a warp takes ...
constexpr int SS_WARP_CROWD = 1024;   // ... and in a level with more large blocks than SS_CROWD
constexpr int SS_CROWD = 2 * SS_CTAS;
constexpr int SS_WIDE = 448;          // widest block (merged) ...
constexpr int64_t SS_PER_LEVEL = 1 << 14;  // ... its square per level kernel, where there are many
constexpr int SS_ROW = 16;            // entries of K's longest rows that take a thread
constexpr int SS_N_MAX = 32000;       // columns: the column table has to fit in shared memory
constexpr int64_t SS_ENTRIES_MAX = 1 << 24;  // factor entries: offsets are 32-bit
constexpr int SS_SMEM_MAX = 160 * 1024;
constexpr unsigned FULL = 0xffffffffu;

struct Args {
  int n, nlev, itr_max, mr, nlong, solve_first, wmax;
  double tol_abs, tol_rel;
  const int4 *rec;  // blocks in the order of the levels: c0, w, nr, first row
  const int *inv0;  // first 32-column chunk of the blocks that take a CTA
  const int4 *chunk;  // those chunks: the block's first column, chunk's first column in it, its columns
  double *inv;      // their inverted unit triangles, by columns and by rows
  int nchunk;
  const int *seg;   // thread / warp / CTA blocks of every level: 3 nlev + 1 starts
  const int *colp, *col2sup;
  const int *ls;
  const double *L, *D;
  const uint8_t *visible, *hidden;
  const int *iperm;
  const int *Rp, *Rj, *long_rows;
  const double *Rx;
  const double *rhs;
  double *out;
  double *b, *x, *V, *dinv;
  double *xs;    // the vector of the solves, in the order of the factor
  double *part;  // sums of the CTAs, two sets
  double *info;  // inner steps, last residual norm, applications of the factor
};

// Columns [c0, c0 + w) and their nr rows, the block's own columns first.
struct Block {
  int c0, w, nr;
  const int *rows;
};

struct Shared {
  double part[2][SS_WARPS], sum[2];
  double left[SS_WARPS][32], tri[SS_WARPS][32];
  double c[SS_MR + 1], s[SS_MR + 1], g[SS_MR + 1], y[SS_MR + 1], h[SS_MR + 1][SS_MR];
  double rho, rho_tol, scale;
  int go, again, parity;
};

__device__ __forceinline__ Block block_at(const Args &a, int q) {
  const int4 u = a.rec[q];
  return {u.x, u.y, u.z, a.ls + u.w};
}

// Entry (i, k) of a block is L[cp[c0 + k] + i]; cp < 0 marks a masked column,
// whose entries count as zero.  i < nr keeps the masked read inside L.
__device__ __forceinline__ double entry(const double *L, int c, int i) {
  const double l = L[max(c, 0) + i];
  return c < 0 ? 0.0 : l;
}

__device__ __forceinline__ int cta_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}
// Every thread of the cluster; what was written before is seen after it.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void push(double *xs, int r, double y) {
  if (y != 0.0) atomicAdd(xs + r, -y);
}

// f(l, row) over the rows below a single column, four loads ahead.
template <class F> __device__ __forceinline__ void below_single(const double *Lc, const Block &b, F &&f) {
#pragma unroll 1
  for (int r0 = 1; r0 < b.nr; r0 += 4) {
    double l[4];
    int rr[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = min(r0 + q, b.nr - 1);
      l[q] = Lc[r];
      rr[q] = b.rows[r];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (r0 + q < b.nr) f(l[q], rr[q]);
  }
}

// Unit lower triangle of columns [jb, jb + kb), kb <= 32, by one warp: lane i
// holds entry jb + i; c: cp of the block.
__device__ __forceinline__ double tri_fwd(const double *L, const int *c, int jb, int kb, double t) {
  const int lane = threadIdx.x & 31;
  const int i = jb + min(lane, kb - 1);
#pragma unroll 1
  for (int j0 = 0; j0 + 1 < kb; j0 += 8) {
    double l[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) l[q] = entry(L, c[jb + min(j0 + q, kb - 1)], i);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (j0 + q + 1 < kb) {
        const double xj = __shfl_sync(FULL, t, j0 + q);
        if (lane > j0 + q) t -= l[q] * xj;
      }
  }
  return t;
}
// The same with its transpose.
__device__ __forceinline__ double tri_bwd(const double *L, const int *c, int jb, int kb, double t) {
  const int lane = threadIdx.x & 31;
  const int cl = c[jb + min(lane, kb - 1)];
#pragma unroll 1
  for (int i0 = kb - 1; i0 > 0; i0 -= 8) {
    double l[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) l[q] = entry(L, cl, jb + max(i0 - q, 0));
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (i0 - q > 0) {
        const double xi = __shfl_sync(FULL, t, i0 - q);
        if (lane < i0 - q) t -= l[q] * xi;
      }
  }
  return t;
}

// Row i of columns [k0, k1) times v(k), eight loads ahead.
template <class F>
__device__ __forceinline__ double row_sum(const double *L, const int *c, int i, int k0, int k1, F &&v) {
  double y = 0.0;
#pragma unroll 1
  for (int k = k0; k < k1; k += 8) {
    double l[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) l[q] = entry(L, c[min(k + q, k1 - 1)], i);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (k + q < k1) y += l[q] * v(k + q);
  }
  return y;
}
// Sums of columns j .. j+7 (those below jend) against x over the rows below the
// block, by one warp; lane 4q returns column j+q's.  Lanes take rows; the
// reduction halves the columns with the lanes (9 additions for 8 columns: an
// FP64 addition holds the quarter's pipe for 64 cycles).
__device__ __forceinline__ double below_sums(const double *L, const int *c, const Block &b, int j, int jend,
                                             const double *xs) {
  const int lane = threadIdx.x & 31;
  double acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = 0.0;
#pragma unroll 1
  for (int r0 = b.w; r0 < b.nr; r0 += 32) {
    const int r = min(r0 + lane, b.nr - 1);
    double l[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) l[q] = entry(L, c[min(j + q, jend - 1)], r);
    double x = __ldcg(xs + b.rows[r]);
    if (r0 + lane >= b.nr) x = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (j + q < jend) acc[q] += l[q] * x;
  }
#pragma unroll
  for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < h; ++q) {
      const double mine = up ? acc[q + h] : acc[q], other = up ? acc[q] : acc[q + h];
      acc[q] = mine + __shfl_xor_sync(FULL, other, o);
    }
  }
  acc[0] += __shfl_xor_sync(FULL, acc[0], 2);
  acc[0] += __shfl_xor_sync(FULL, acc[0], 1);
  return acc[0];
}

// Brings a block's first entries and rows to L1, by n threads: what follows
// reads them in several rounds, of 330 cycles each at L2 and 95 here (a cluster
// barrier empties L1, so nothing can be fetched ahead of the level).
__device__ __forceinline__ void fetch(const double *L, const int *c, const Block &b, int t, int n) {
  constexpr int LINES = 512;
  const int c0 = c[0], c1 = c[b.w - 1];
  if (c0 >= 0 && c1 >= 0) {
    const int lines = min((c1 + b.nr - c0 + 15) / 16, LINES);
    for (int q = t; q < lines; q += n) asm volatile("prefetch.global.L1 [%0];" ::"l"(L + c0 + min(16 * q, c1 + b.nr - 1 - c0)));
  }
  for (int q = 32 * t; q < b.nr; q += 32 * n) asm volatile("prefetch.global.L1 [%0];" ::"l"(b.rows + q));
}

// A block of up to 32 columns by one warp.
__device__ __forceinline__ void fwd_warp(const double *L, const int *cp, const Block &b, double *xs) {
  const int lane = threadIdx.x & 31;
  const int *c = cp + b.c0;
  fetch(L, c, b, lane, 32);
  double t = lane < b.w ? __ldcg(xs + b.c0 + lane) : 0.0;
  if (b.w > 1) {
    t = tri_fwd(L, c, 0, b.w, t);
    if (lane < b.w) xs[b.c0 + lane] = t;
  }
#pragma unroll 1
  for (int r0 = b.w; r0 < b.nr; r0 += 32) {
    const int r = min(r0 + lane, b.nr - 1);
    const int rr = b.rows[r];
    const double y = row_sum(L, c, r, 0, b.w, [&](int k) { return __shfl_sync(FULL, t, k); });
    if (r0 + lane < b.nr) push(xs, rr, y);
  }
}
__device__ __forceinline__ void bwd_warp(const double *L, const int *cp, const Block &b, double *xs) {
  const int lane = threadIdx.x & 31;
  const int *c = cp + b.c0;
  fetch(L, c, b, lane, 32);
  double t = lane < b.w ? __ldcg(xs + b.c0 + lane) : 0.0;
  if (b.nr > b.w) {
#pragma unroll 1
    for (int j = 0; j < b.w; j += 8) {
      const double y = __shfl_sync(FULL, below_sums(L, c, b, j, b.w, xs), 4 * (lane & 7));
      if ((lane & ~7) == j) t -= y;
    }
  }
  if (b.w > 1) t = tri_bwd(L, c, 0, b.w, t);
  if (lane < b.w) xs[b.c0 + lane] = t;
}

// The four entries 4 wi .. 4 wi + 3 of the sum of the warps' vectors v[][32], one
// in each lane by lane % 4.
__device__ __forceinline__ double own_four(const double (*v)[32], int wi) {
  const int lane = threadIdx.x & 31;
  double t = v[lane >> 2][4 * wi + (lane & 3)];
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) t += __shfl_xor_sync(FULL, t, o);
  return t;
}

// Inverts the unit triangles of the 32-column chunks, one per CTA at a time: lane =
// row, a warp does the columns wi, wi + 8, ... in the order of elimination.
__device__ __noinline__ void invert_chunks(const Args &a, const int *cp) {
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
#pragma unroll 1
  for (int q = cta_rank(); q < a.nchunk; q += SS_CTAS) {
    const int4 u = a.chunk[q];
    const int *c = cp + u.x + u.y;
    const int kb = u.z, i = u.y + min(lane, kb - 1);
    double l[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const double v = entry(a.L, c[min(k, kb - 1)], i);
      l[k] = k < lane && lane < kb ? v : 0.0;
    }
    double x[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) x[v] = lane == wi + 8 * v ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < 31; ++k)
#pragma unroll
      for (int v = 0; v < 4; ++v)
        if (k >= 8 * v) {
          const double xk = __shfl_sync(FULL, x[v], k);
          x[v] -= l[k] * xk;
        }
    double *out = a.inv + (size_t)q * 2048;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int col = wi + 8 * v;
      out[col * 32 + lane] = x[v];
      out[1024 + lane * 32 + col] = x[v];
    }
  }
}

// A block by the CTA, 32 columns (a chunk) at a time.  Of every chunk a warp has
// four columns: it adds up what they contribute to the later chunks, and its
// part of the product with the chunk's inverted triangle (a substitution is a
// chain of 31 steps of about 110 cycles; by chunks 9000 cycles each, with the
// inverse and the sums spread over the warps 2300).  xb: the block's part of the vector,
// in shared memory; inv: the block's inverted triangles.
__device__ __noinline__ void fwd_cta(Shared &sh, const double *L, const int *cp, const double *inv, const Block b,
                                     double *xb, double *xs) {
  const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5;
  const int *c = cp + b.c0;
  fetch(L, c, b, tid, SS_THREADS);
  for (int i = tid; i < b.w; i += SS_THREADS) xb[i] = __ldcg(xs + b.c0 + i);
  double acc = 0.0, x = 0.0;
  __syncthreads();
#pragma unroll 1
  for (int jb = 0; jb < b.w; jb += 32, inv += 2048) {
    const int kb = min(32, b.w - jb), mine = 4 * wi + (lane & 3);
    double m[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = inv[(4 * wi + q) * 32 + lane];
    double t = mine < kb ? xb[jb + mine] : 0.0;
    if (jb > 0) {
      const int i = jb + min(lane, kb - 1);
#pragma unroll
      for (int q = 0; q < 4; ++q) acc += entry(L, c[jb - 32 + 4 * wi + q], i) * __shfl_sync(FULL, x, q);
      sh.left[wi][lane] = acc;
      __syncthreads();
      const double left = own_four(sh.left, wi);
      if (mine < kb) t -= left;
    }
    double y = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) y += m[q] * __shfl_sync(FULL, t, q);
    sh.tri[wi][lane] = y;
    acc = 0.0;
    if (jb + 32 < b.w) {  // the chunks before this one, for the next
      const int i = min(jb + 32 + lane, b.w - 1);
#pragma unroll 1
      for (int k = 4 * wi; k < jb; k += 64) {
        double l[8];
        const int k2 = min(k + 32, jb - 32 + 4 * wi);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          l[q] = entry(L, c[k + q], i);
          l[q + 4] = entry(L, c[k2 + q], i);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) acc += l[q] * xb[k + q];
        if (k + 32 < jb)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc += l[q + 4] * xb[k2 + q];
      }
    }
    __syncthreads();
    x = own_four(sh.tri, wi);
    if (lane < 4 && mine < kb) {
      xb[jb + mine] = x;
      xs[b.c0 + jb + mine] = x;
    }
    __syncwarp();
  }
  __syncthreads();
  // rows below: chunks of 32 rows, and of the columns where there are fewer
  const int rc = (b.nr - b.w + 31) / 32;
  const int split = rc == 0 ? 1 : max(1, min(SS_WARPS / rc, b.w / 8)), per = (b.w + split - 1) / split;
#pragma unroll 1
  for (int q = wi; q < rc * split; q += SS_WARPS) {
    const int r = b.w + 32 * (q / split) + lane, k0 = min(q % split * per, b.w), k1 = min(k0 + per, b.w);
    const int rr = b.rows[min(r, b.nr - 1)];
    const double y = row_sum(L, c, min(r, b.nr - 1), k0, k1, [&](int k) { return xb[k]; });
    if (r < b.nr) push(xs, rr, y);
  }
  __syncthreads();  // xb is free again
}
__device__ __noinline__ void bwd_cta(Shared &sh, const double *L, const int *cp, const double *inv, const Block b,
                                     double *xb, double *xs) {
  const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5;
  const int *c = cp + b.c0;
  fetch(L, c, b, tid, SS_THREADS);
  for (int i = tid; i < b.w; i += SS_THREADS) xb[i] = __ldcg(xs + b.c0 + i);
  __syncthreads();
  // What the rows below contribute to chunk j's columns (a lane each): a warp
  // has an eighth of the rows.
  const int per = (b.nr - b.w + SS_WARPS - 1) / SS_WARPS;
  const int ra = min(b.w + per * wi, b.nr), rb = min(ra + per, b.nr);
  auto below = [&](int j) {
    const int cl = c[min(j + lane, b.w - 1)];
    double y = 0.0;
#pragma unroll 1
    for (int r0 = ra; r0 < rb; r0 += 32) {
      const int n = min(32, rb - r0);
      const double xr = __ldcg(xs + b.rows[r0 + min(lane, n - 1)]);
#pragma unroll 1
      for (int k = 0; k < n; k += 8) {
        double l[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) l[q] = entry(L, cl, r0 + min(k + q, n - 1));
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (k + q < n) y += l[q] * __shfl_sync(FULL, xr, k + q);
      }
    }
    return y;
  };
  const int last = (b.w - 1) / 32 * 32;
  double acc = below(last), x = 0.0;
  inv += (size_t)(last / 32) * 2048 + 1024;
#pragma unroll 1
  for (int jb = last; jb >= 0; jb -= 32, inv -= 2048) {
    const int kb = min(32, b.w - jb), mine = 4 * wi + (lane & 3);
    double m[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = inv[(4 * wi + q) * 32 + lane];
    double t = mine < kb ? xb[jb + mine] : 0.0;
    if (jb < last) {
      const int cl = c[jb + lane];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = jb + 32 + 4 * wi + q;
        const double l = entry(L, cl, min(i, b.w - 1)), v = __shfl_sync(FULL, x, q);
        if (i < b.w) acc += l * v;
      }
    }
    if (jb < last || b.nr > b.w) {
      sh.left[wi][lane] = acc;
      __syncthreads();
      const double left = own_four(sh.left, wi);
      if (mine < kb) t -= left;
    }
    double y = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) y += m[q] * __shfl_sync(FULL, t, q);
    sh.tri[wi][lane] = y;
    acc = 0.0;
    if (jb > 0) {  // the rows below and the chunks after this one, for the next
      if (b.nr > b.w) acc = below(jb - 32);
      const int cl = c[jb - 32 + lane];
#pragma unroll 1
      for (int i = jb + 32 + 4 * wi; i < b.w; i += 64) {
        double l[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          l[q] = entry(L, cl, min(i + q, b.w - 1));
          l[q + 4] = entry(L, cl, min(i + 32 + q, b.w - 1));
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (i + q < b.w) acc += l[q] * xb[i + q];
        if (i + 32 < b.w)
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i + 32 + q < b.w) acc += l[q + 4] * xb[i + 32 + q];
      }
    }
    __syncthreads();
    x = own_four(sh.tri, wi);
    if (lane < 4 && mine < kb) {
      xb[jb + mine] = x;
      xs[b.c0 + jb + mine] = x;
    }
    __syncwarp();
  }
  __syncthreads();  // xb is free again
}

// xs <- (L D L^T)^-1 xs.  A level's blocks are independent of each other:
// short single columns take a thread each, small blocks a warp, the others a CTA.
__device__ __noinline__ void ldlt(const Args &a, Shared &sh, const int *cp, const int *seg, double *xb) {
  const int tid = threadIdx.x, rank = cta_rank();
  const int thread = (SS_THREADS - 1 - tid) * SS_CTAS + rank, warp = (tid >> 5) * SS_CTAS + rank;
  double *xs = a.xs;
#pragma unroll 1
  for (int l = 0; l < a.nlev; ++l) {
    const int *sg = seg + 3 * l;
    const int s0 = sg[0], s1 = sg[1], s2 = sg[2], s3 = sg[3];
#pragma unroll 1
    for (int q = s0 + thread; q < s1; q += SS_ALL) {
      const Block b = block_at(a, q);
      const int c = cp[b.c0];
      if (c < 0) continue;
      const double t = __ldcg(xs + b.c0);
      below_single(a.L + c, b, [&](double v, int r) { push(xs, r, v * t); });
    }
    __syncwarp();
#pragma unroll 1
    for (int q = s1 + warp; q < s2; q += SS_CTAS * SS_WARPS) fwd_warp(a.L, cp, block_at(a, q), xs);
#pragma unroll 1
    for (int q = s2 + rank; q < s3; q += SS_CTAS)
      fwd_cta(sh, a.L, cp, a.inv + (size_t)a.inv0[q] * 2048, block_at(a, q), xb, xs);
    cluster_sync();
  }
  for (int i = rank * SS_THREADS + tid; i < a.n; i += SS_ALL) {
    const double d = a.dinv[i], e = a.dinv[a.n + i];
    if (i > 0 && a.dinv[a.n + i - 1] != 0.0) continue;  // second of a 2x2 block
    const double x1 = __ldcg(xs + i);
    if (e == 0.0) {
      xs[i] = d * x1;
    } else {
      const double x2 = __ldcg(xs + i + 1);
      xs[i] = d * x1 + e * x2;
      xs[i + 1] = a.dinv[i + 1] * x2 + e * x1;
    }
  }
  cluster_sync();
#pragma unroll 1
  for (int l = a.nlev - 1; l >= 0; --l) {
    const int *sg = seg + 3 * l;
    const int s0 = sg[0], s1 = sg[1], s2 = sg[2], s3 = sg[3];
#pragma unroll 1
    for (int q = s0 + thread; q < s1; q += SS_ALL) {
      const Block b = block_at(a, q);
      const int c = cp[b.c0];
      if (c < 0) continue;
      double t = __ldcg(xs + b.c0);
      below_single(a.L + c, b, [&](double v, int r) { t -= v * __ldcg(xs + r); });
      xs[b.c0] = t;
    }
    __syncwarp();
#pragma unroll 1
    for (int q = s1 + warp; q < s2; q += SS_CTAS * SS_WARPS) bwd_warp(a.L, cp, block_at(a, q), xs);
#pragma unroll 1
    for (int q = s2 + rank; q < s3; q += SS_CTAS)
      bwd_cta(sh, a.L, cp, a.inv + (size_t)a.inv0[q] * 2048, block_at(a, q), xb, xs);
    cluster_sync();
  }
}

// put(i, (K v)_i) for every row of K: short rows a thread each, the others a warp each.
template <class F> __device__ __forceinline__ void spmv(const Args &a, const double *v, F &&put) {
  const int tid = threadIdx.x, lane = tid & 31;
#pragma unroll 1
  for (int i = cta_rank() * SS_THREADS + tid; i < a.n; i += SS_ALL) {
    const int q0 = a.Rp[i], q1 = a.Rp[i + 1];
    if (q1 - q0 > SS_ROW) continue;
    double acc = 0.0;
#pragma unroll 1
    for (int q = q0; q < q1; q += 4) {
      int jj[4];
      double k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        jj[u] = a.Rj[min(q + u, q1 - 1)];
        k[u] = a.Rx[min(q + u, q1 - 1)];
      }
      double x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = __ldcg(v + jj[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (q + u < q1) acc += k[u] * x[u];
    }
    put(i, acc);
  }
#pragma unroll 1
  for (int p = (tid >> 5) * SS_CTAS + cta_rank(); p < a.nlong; p += SS_CTAS * SS_WARPS) {
    const int i = a.long_rows[p];
    double acc = 0.0;
    for (int q = a.Rp[i] + lane; q < a.Rp[i + 1]; q += 32) acc += a.Rx[q] * __ldcg(v + a.Rj[q]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
    if (lane == 0) put(i, acc);
  }
}

// Sums of two values over the cluster, the same in every CTA; in sh.sum after
// the barrier it ends with.  The two sets of partial sums take turns: a CTA
// writes a set again only after a barrier that the others reach having read it.
__device__ __forceinline__ void sums(const Args &a, Shared &sh, double u, double v) {
  const int tid = threadIdx.x, lane = tid & 31;
  const bool up = lane & 16;
  double t = (up ? v : u) + __shfl_xor_sync(FULL, up ? u : v, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
  if ((lane & 15) == 0) sh.part[lane >> 4][tid >> 5] = t;
  __syncthreads();
  double *part = a.part + 2 * SS_CTAS * sh.parity;
  if (tid < 16) {
    t = sh.part[tid >> 3][tid & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffu, t, o);
    if ((tid & 7) == 0) part[(tid >> 3) * SS_CTAS + cta_rank()] = t;
  }
  cluster_sync();
  if (tid < 16) {
    t = __ldcg(part + tid);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffu, t, o);
    if ((tid & 7) == 0) sh.sum[tid >> 3] = t;
    if (tid == 0) sh.parity ^= 1;
  }
  __syncthreads();
}
static_assert(SS_WARPS == 8 && SS_CTAS == 8, "sums() adds eight partial sums with eight lanes");

// y <- y - h x, and the sums of (y . y, y . z)
__device__ __forceinline__ void axpy_dot(const Args &a, Shared &sh, double h, const double *x, double *y, const double *z) {
  double s0 = 0.0, s1 = 0.0;
#pragma unroll 1
  for (int i = cta_rank() * SS_THREADS + threadIdx.x; i < a.n; i += SS_ALL) {
    const double t = y[i] - h * x[i];
    y[i] = t;
    s0 += t * t;
    if (z) s1 += t * z[i];
  }
  sums(a, sh, s0, s1);
}

__global__ void __cluster_dims__(SS_CTAS, 1, 1) __launch_bounds__(SS_THREADS) k_solve_small(const Args a) {
  extern __shared__ double xb[];
  __shared__ Shared sh;
  const int tid = threadIdx.x, n = a.n, me = cta_rank() * SS_THREADS + tid;
  int *cp = reinterpret_cast<int *>(xb + a.wmax), *seg = cp + n;
  for (int i = tid; i < 3 * a.nlev + 1; i += SS_THREADS) seg[i] = a.seg[i];
  double *xs = a.xs;
  for (int i = tid; i < n; i += SS_THREADS) {
    const int c = a.colp[i];
    cp[i] = a.visible && !a.visible[a.col2sup[i]] ? -1 : c;
  }
  // D^-1, in the order of the factor; hidden columns keep their values
  for (int i = me; i < n; i += SS_ALL) {
    auto hid = [&](int k) { return a.hidden && a.hidden[k]; };
    const double e = a.D[n + i];
    if (hid(i)) {
      a.dinv[i] = 1.0;
      a.dinv[n + i] = 0.0;
    } else if (i > 0 && a.D[n + i - 1] != 0.0 && !hid(i - 1)) {
      a.dinv[n + i] = 0.0;  // second of a 2x2 block
    } else if (e == 0.0) {
      a.dinv[i] = 1.0 / a.D[i];
      a.dinv[n + i] = 0.0;
    } else {
      const double d1 = a.D[i], d2 = a.D[i + 1], inv = 1.0 / (d1 * d2 - e * e);
      a.dinv[i] = d2 * inv;
      a.dinv[i + 1] = d1 * inv;
      a.dinv[n + i] = -e * inv;
    }
  }
  for (int i = me; i < n; i += SS_ALL) {
    const double v = a.rhs[i];
    a.b[i] = v;
    a.x[i] = v;
    if (a.solve_first) xs[a.iperm[i]] = v;
  }
  if (tid == 0) {
    sh.rho = 0.0;
    sh.parity = 0;
  }
  __syncthreads();
  invert_chunks(a, cp);
  cluster_sync();
  if (a.solve_first) {
    ldlt(a, sh, cp, seg, xb);
    for (int i = me; i < n; i += SS_ALL) a.x[i] = __ldcg(xs + a.iperm[i]);
    cluster_sync();
  }
  int used = 0, applied = a.solve_first;
  constexpr double delta = 1.0e-03;
#pragma unroll 1
  for (int itr = 0; itr < (a.mr > 0 ? a.itr_max : 0); ++itr) {
    spmv(a, a.x, [&](int i, double v) { xs[a.iperm[i]] = a.b[i] - v; });
    cluster_sync();
    ldlt(a, sh, cp, seg, xb);
    ++applied;
    double s0 = 0.0;
    for (int i = me; i < n; i += SS_ALL) s0 += __ldcg(xs + i) * __ldcg(xs + i);
    sums(a, sh, s0, 0.0);
    if (tid == 0) {
      const double rho = sqrt(sh.sum[0]);
      sh.rho = rho;
      sh.go = !(rho < a.tol_abs);
      if (itr == 0) sh.rho_tol = rho * a.tol_rel;
      sh.g[0] = rho;
      sh.scale = 1.0 / rho;
    }
    __syncthreads();
    if (!sh.go) break;
    {
      const double sc = sh.scale;
      for (int i = me; i < n; i += SS_ALL) a.V[i] = __ldcg(xs + a.iperm[i]) * sc;
    }
    cluster_sync();
    int k = 0;
#pragma unroll 1
    for (;; ++k) {
      double *vk = a.V + (size_t)k * n, *v1 = vk + n;
      spmv(a, vk, [&](int i, double v) { xs[a.iperm[i]] = v; });
      cluster_sync();
      ldlt(a, sh, cp, seg, xb);
      ++applied;
      s0 = 0.0;
      double s1 = 0.0;
      for (int i = me; i < n; i += SS_ALL) {
        const double v = __ldcg(xs + a.iperm[i]);
        v1[i] = v;
        s0 += v * v;
        s1 += v * a.V[i];
      }
      sums(a, sh, s0, s1);
      double av = 0.0;
      if (tid == 0) av = sqrt(sh.sum[0]);
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
#pragma unroll 1
        for (int j = 0; j <= k; ++j) {
          const double h = sh.sum[1];
          if (tid == 0) sh.h[j][k] = pass ? sh.h[j][k] + h : h;
          axpy_dot(a, sh, h, a.V + (size_t)j * n, v1, j < k ? a.V + (size_t)(j + 1) * n : (pass ? nullptr : a.V));
        }
        if (pass) break;
        if (tid == 0) sh.again = av + delta * sqrt(sh.sum[0]) == av;
        __syncthreads();
        if (!sh.again) break;
      }
      if (tid == 0) {
        const double hn = sqrt(sh.sum[0]);
        sh.scale = hn != 0.0 ? 1.0 / hn : 1.0;
        double t = sh.h[0][k];
        for (int j = 0; j < k; ++j) {  // the rotations of the previous steps
          const double u = sh.h[j + 1][k];
          sh.h[j][k] = sh.c[j] * t - sh.s[j] * u;
          t = sh.s[j] * t + sh.c[j] * u;
        }
        const double mu = sqrt(t * t + hn * hn);
        if (mu == 0.0) {
          sh.go = -1;
        } else {
          const double c = t / mu, s = -hn / mu, g = sh.g[k];
          sh.c[k] = c;
          sh.s[k] = s;
          sh.h[k][k] = c * t - s * hn;
          sh.g[k] = c * g;
          sh.g[k + 1] = s * g;
          const double rho = fabs(s * g);
          sh.rho = rho;
          sh.go = !((rho <= sh.rho_tol && rho <= a.tol_abs) || k + 1 == a.mr);
        }
      }
      __syncthreads();
      if (sh.go < 0) break;
      ++used;
      if (!sh.go) break;
      const double sc = sh.scale;
      for (int i = me; i < n; i += SS_ALL) v1[i] *= sc;
      cluster_sync();
    }
    if (sh.go < 0 || sh.h[k][k] == 0.0) break;
    if (tid == 0)
      for (int i = k; i >= 0; --i) {
        double t = sh.g[i];
        for (int j = i + 1; j <= k; ++j) t -= sh.h[i][j] * sh.y[j];
        sh.y[i] = t / sh.h[i][i];
      }
    __syncthreads();
    for (int i = me; i < n; i += SS_ALL) {
      double t = a.x[i];
      for (int j = 0; j <= k; ++j) t += a.V[(size_t)j * n + i] * sh.y[j];
      a.x[i] = t;
    }
    cluster_sync();
    if (sh.rho <= sh.rho_tol && sh.rho <= a.tol_abs) break;
  }
  __syncthreads();
  for (int i = me; i < n; i += SS_ALL) a.out[i] = a.x[i];
  if (me == 0) {
    a.info[0] = used;
    a.info[1] = sh.rho;
    a.info[2] = applied;
  }
}

}  // namespace

// Blocks, levels and long rows of K; called once, when the plan is made.
int solve_small_setup(Plan &P, const std::vector<int> &Rp) {
  const Symbolic &S = P.sym;
  const int ns = (int)S.super.size() - 1;
  P.ss_ok = false;
  if (P.set.precision != NQG_FP64 || P.n < 1 || P.n > SS_N_MAX || ns < 1 || P.set.max_inner_iter > SS_MR) return NQG_OK;
  if (S.lpx[ns] > SS_ENTRIES_MAX) return NQG_OK;
  // A supernode whose rows below are exactly the next one's rows joins it: a
  // dense tail that the factorization keeps as a chain of narrow supernodes
  // (constraints stay columns of their own) is one block for the solves.
  std::vector<int> first(1, 0), blk(ns, 0);
  for (int s = 1; s < ns; ++s) {
    const int w = S.super[s] - S.super[s - 1];
    const int64_t p = S.lpi[s - 1] + w, e = S.lpi[s];
    if (e - p != S.lpi[s + 1] - S.lpi[s] || !std::equal(S.ls.begin() + p, S.ls.begin() + e, S.ls.begin() + e))
      first.push_back(s);
    blk[s] = (int)first.size() - 1;
  }
  const int nb = (int)first.size();
  first.push_back(ns);
  std::vector<int> level(nb, 0), colp(P.n);
  int nlev = 0;
  for (int b = 0; b < nb; ++b) {
    const int last = first[b + 1] - 1;
    const int64_t below = S.lpi[last] + S.super[last + 1] - S.super[last];
    nlev = std::max(nlev, level[b] + 1);
    if (below < S.lpi[last + 1]) {
      int &up = level[blk[S.col2sup[S.ls[below]]]];
      up = std::max(up, level[b] + 1);
    }
    for (int s = first[b]; s <= last; ++s) {
      const int o = S.super[s] - S.super[first[b]], nr = (int)(S.lpi[s + 1] - S.lpi[s]);
      for (int c = S.super[s]; c < S.super[s + 1]; ++c)
        colp[c] = (int)S.lpx[s] + (c - S.super[s]) * nr - o;
    }
  }
  std::vector<std::vector<int>> lists((size_t)3 * nlev);
  auto width = [&](int b) { return S.super[first[b + 1]] - S.super[first[b]]; };
  auto height = [&](int b) { return (int)(S.lpi[first[b] + 1] - S.lpi[first[b]]); };
  auto size = [&](int b) { return (int64_t)width(b) * height(b); };
  std::vector<int> large(nlev, 0);
  for (int b = 0; b < nb; ++b) large[level[b]] += size(b) > SS_WARP_BLOCK;
  P.ss_wmax = 0;
  for (int b = 0; b < nb; ++b) {
    const int64_t limit = large[level[b]] > SS_CROWD ? SS_WARP_CROWD : SS_WARP_BLOCK;
    const int c = width(b) == 1 && height(b) <= SS_LONG ? 0 : width(b) <= 32 && size(b) <= limit ? 1 : 2;
    lists[(size_t)3 * level[b] + c].push_back(b);
    if (c == 2) P.ss_wmax = std::max(P.ss_wmax, width(b));
  }
  // The level kernels and the block kernels stay the better ones where one
  // wide block is most of the work (they spread it over the chip; here its cost
  // grows with the square of the width, there with the levels).  A refined
  // solve, here and there: dense 256 columns 0.31 and 0.62 ms, 384 0.55 and 0.70,
  // 512 0.84 and 0.71; 16^3 Laplacian (widest block 277) 0.84 and 1.11, 20^3 (615)
  // 2.44 and 2.32, 160^2 (237) 2.28 and 2.38.  An active-set iteration of a QP with
  // 2064 columns in 115 levels 6.6 and 15.6 ms, 6522 in 368 levels 41 and 91.
  int launches = 0;
  for (size_t l = 0; l < P.levels.size(); ++l)
    launches += (P.level_off[l + 1] > P.level_off[l]) + (P.blk_fwd_off[l + 1] > P.blk_fwd_off[l]);
  if ((int64_t)P.ss_wmax * P.ss_wmax > std::max<int64_t>(SS_WIDE * SS_WIDE, SS_PER_LEVEL * launches)) return NQG_OK;
  std::vector<int> rec, seg(1, 0), rows, inv0, chunk;
  for (auto &list : lists) {
    // the largest first: they are dealt out in turn
    std::stable_sort(list.begin(), list.end(),
                     [&](int x, int y) { return size(x) > size(y); });
    for (int b : list) {
      const int r[4] = {S.super[first[b]], width(b), height(b), (int)S.lpi[first[b]]};
      rec.insert(rec.end(), r, r + 4);
      inv0.push_back((int)chunk.size() / 4);
      if ((&list - lists.data()) % 3 == 2)
        for (int j = 0; j < r[1]; j += 32) chunk.insert(chunk.end(), {r[0], j, std::min(32, r[1] - j), 0});
    }
    seg.push_back((int)rec.size() / 4);
  }
  P.ss_nlev = nlev;
  for (int i = 0; i < P.n; ++i)
    if (Rp[i + 1] - Rp[i] > SS_ROW) rows.push_back(i);
  P.ss_nchunk = (int)chunk.size() / 4;
  P.ss_smem = (size_t)P.ss_wmax * sizeof(double) + ((size_t)P.n + seg.size()) * sizeof(int);
  if (P.ss_smem > SS_SMEM_MAX) return NQG_OK;
  P.ss_nlong = (int)rows.size();
  rows.push_back(0);
  chunk.resize(chunk.size() + 4);
  NQG_CUDA(cudaMalloc(&P.d_ss_rec, rec.size() * sizeof(int)));
  NQG_CUDA(cudaMalloc(&P.d_ss_seg, seg.size() * sizeof(int)));
  NQG_CUDA(cudaMalloc(&P.d_ss_colp, colp.size() * sizeof(int)));
  NQG_CUDA(cudaMemcpy(P.d_ss_colp, colp.data(), colp.size() * sizeof(int), cudaMemcpyHostToDevice));
  NQG_CUDA(cudaMalloc(&P.d_ss_inv0, inv0.size() * sizeof(int)));
  NQG_CUDA(cudaMemcpy(P.d_ss_inv0, inv0.data(), inv0.size() * sizeof(int), cudaMemcpyHostToDevice));
  NQG_CUDA(cudaMalloc(&P.d_ss_chunk, chunk.size() * sizeof(int)));
  NQG_CUDA(cudaMemcpy(P.d_ss_chunk, chunk.data(), chunk.size() * sizeof(int), cudaMemcpyHostToDevice));
  NQG_CUDA(cudaMalloc(&P.d_ss_inv, std::max<size_t>(P.ss_nchunk, 1) * 2048 * sizeof(double)));
  NQG_CUDA(cudaMalloc(&P.d_ss_rows, rows.size() * sizeof(int)));
  NQG_CUDA(cudaMalloc(&P.d_ss_dinv, 2 * (size_t)P.n * sizeof(double)));
  NQG_CUDA(cudaMemcpy(P.d_ss_rec, rec.data(), rec.size() * sizeof(int), cudaMemcpyHostToDevice));
  NQG_CUDA(cudaMemcpy(P.d_ss_seg, seg.data(), seg.size() * sizeof(int), cudaMemcpyHostToDevice));
  NQG_CUDA(cudaMemcpy(P.d_ss_rows, rows.data(), rows.size() * sizeof(int), cudaMemcpyHostToDevice));
  P.ss_ok = true;
  return NQG_OK;
}

// d_x = refined solution of K x = d_rhs (solve_first), or the refinement of x = d_rhs.
int solve_small(Plan &P, const double *d_rhs, double *d_x, bool solve_first) {
  Args a{};
  a.n = P.n;
  a.nlev = P.ss_nlev;
  a.itr_max = P.set.req_ref_iter;
  a.mr = P.set.max_inner_iter;
  a.nlong = P.ss_nlong;
  a.solve_first = solve_first;
  a.tol_abs = P.set.tol_abs;
  a.tol_rel = P.set.tol_rel;
  a.rec = reinterpret_cast<const int4 *>(P.d_ss_rec);
  a.seg = P.d_ss_seg;
  a.ls = P.d_ls;
  a.colp = P.d_ss_colp;
  a.col2sup = P.d_col2sup;
  a.L = static_cast<const double *>(P.d_L);
  a.D = static_cast<const double *>(P.d_D);
  a.visible = P.masked ? P.d_visible : nullptr;
  a.hidden = P.masked ? P.d_hidden : nullptr;
  a.iperm = P.d_iperm;
  a.Rp = P.d_Rp;
  a.Rj = P.d_Rj;
  a.Rx = P.d_Rx;
  a.long_rows = P.d_ss_rows;
  a.rhs = d_rhs;
  a.out = d_x;
  a.b = P.d_bo;
  a.x = P.d_xo;
  a.V = P.d_V;
  a.dinv = P.d_ss_dinv;
  a.inv0 = P.d_ss_inv0;
  a.chunk = reinterpret_cast<const int4 *>(P.d_ss_chunk);
  a.nchunk = P.ss_nchunk;
  a.inv = P.d_ss_inv;
  a.wmax = P.ss_wmax;
  a.xs = P.d_r;
  a.part = P.d_scal + 64;
  a.info = P.d_scal;
  NQG_CUDA(cudaFuncSetAttribute(k_solve_small, cudaFuncAttributeMaxDynamicSharedMemorySize, SS_SMEM_MAX));
  cudaEvent_t e0 = P.prof_begin();
  k_solve_small<<<SS_CTAS, SS_THREADS, P.ss_smem, P.stream>>>(a);
  P.prof_end(NQG_K_SOLVE, e0, 0.0, 0.0);
  P.nlaunch++;
  NQG_CUDA(cudaGetLastError());
  double info[3];
  NQG_CUDA(cudaMemcpyAsync(info, P.d_scal, sizeof(info), cudaMemcpyDeviceToHost, P.stream));
  NQG_CUDA(cudaStreamSynchronize(P.stream));
  // factor values read by both sweeps of every application
  if (P.prof && !P.prof_pending.empty()) P.prof_pending.back().bytes = 2.0 * info[2] * P.sym.xsize * sizeof(double);
  P.tm.num_ref_iter = (int)info[0];
  P.tm.last_residual = info[1];
  return NQG_OK;
}

}  // namespace nqg
