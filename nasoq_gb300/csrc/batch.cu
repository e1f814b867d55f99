// Batched NASOQ: thousands of small QPs of uneven size, each solved to the
// end by one CTA of a persistent kernel -- the dual active-set iteration
// (reference Nasoq::numeric_QP, src/nasoq.cpp:478-610), its SoMod partial
// refactorizations (update_ldl_left_sn_02_v2, src/ldl/Serial_update_ldl.cpp:
// 18-277), masked supernodal solves and GMRES refinement all run on the
// device; the host only fills the work queue.
//
// Per problem, in the CTA's scratch slot (or, for the factor and its row
// lists, in shared memory when they fit the launch's staging space):
//  * the supernodal factor, in blocks laid out for the kernels that read them
//    (see "blocks" below), the composed ordering perm/iperm and the row lists,
//    renamed after Bunch-Kaufman pivoting as the reference's row_reordering
//    does (without re-sorting the renamed rows: every consumer maps them
//    through the target's row list);
//  * the active set as a per-constraint flag.  Hidden (inactive) constraint
//    columns are width-1 supernodes whose entries read as zero; the
//    reference's hidden-column tree edits (linear_solver_wrapper.cpp:770-907)
//    become a visibility flag per supernode plus, per supernode, a bit mask
//    of its active constraint-column descendants, and the supernodes to
//    refactor after an edit are those on the elimination-tree paths from the
//    edited column and its variables to the root;
//  * two copies of K's values in CSR order (factorization values with the
//    regularization, refinement values without it), edited in place;
//  * the KKT vectors in the original numbering; the triangular solves gather
//    them into shared memory in the factor's order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "batch.hpp"
#include "bk.cuh"

namespace nqg {

namespace {

// Up to 256 threads per CTA at 128 registers: 4 CTAs of 128 threads per SM.
//
// The kernel runs a whole solver, and its size is a cost of its own: with every
// phase inlined where it is used and loops unrolled by the compiler it was 2 MB
// of code, 16 times what an SM's instruction cache holds, and a tenth of all
// issue slots waited for instructions.  So a phase is one function
// (__noinline__), and loops are unrolled only where loads have to overlap
// (#pragma unroll with a count; unroll 1 elsewhere): 0.3 MB.
constexpr int BT_MAX_THREADS = 256;
constexpr int WF_WARPS = BATCH_WF_WARPS;  // warps of the level-parallel factorization
constexpr int MR_CAP = BATCH_MR_CAP;  // Krylov steps per restart held in shared memory

// Counters of nqg_batch_get_profile.
enum { PH_TOTAL, PH_INIT, PH_FACTOR, PH_PRECOND, PH_SPMV, PH_REFINE, PH_SELECT, PH_UPDATE, PH_SN, PH_ITER,
       PH_FWD_WIDE, PH_FWD_NARROW, PH_DIAG, PH_BWD, PH_GATHER, PH_INIT_FACTOR,
       PH_SN_ASSEMBLE, PH_SN_UPDATES, PH_SN_BK, PH_SN_ROWS, PH_SN_INVERSE, PH_SN_STORE, PH_RENAME, PH_N };
struct GmresSmall {
  double h[MR_CAP + 1][MR_CAP], cs[MR_CAP + 1], sn[MR_CAP + 1], g[MR_CAP + 1], y[MR_CAP + 1];
  double scal[4];
};

// An array in the CTA's dynamic shared memory, by its offset: what is read
// through it is known to be shared (a plain pointer kept in memory is not, and
// costs a generic access; a generic atomic is compiled for both spaces).
template <class T> struct Sh {
  unsigned off;
  __device__ __forceinline__ operator T *() const {
    extern __shared__ __align__(16) unsigned char dsm[];
    return reinterpret_cast<T *>(dsm + off);
  }
  __device__ __forceinline__ Sh at(int n) const { return {off + (unsigned)(n * (int)sizeof(T))}; }
};

// Patterns of more columns than shared memory has room for with both vectors
// of the solves keep the second one, the refactorization marks and the levels'
// items in global memory: a kernel of its own (batch_large.cu), since a pointer
// that may be either costs a generic access everywhere.  FP64 from 11900
// columns on (horizon 360 of the MPC families), to 15800; FP32 from 22000 to
// 23400.  64 problems of horizon 400 (FP64) 87.7 ms, of horizon 700 (FP32) 219.5
// (the kernel with one vector for the solves, which still held them: 332.7 and
// 973.5); horizon 300, both vectors shared, 55.6.
#ifdef NQG_BATCH_LARGE_UNIT
constexpr bool LARGE = true;
template <class T> using Spill = T *;
#else
constexpr bool LARGE = false;
template <class T> using Spill = Sh<T>;
#endif

// The problem that the CTA works on, at the start of its dynamic shared memory.
template <class T> struct Ctx {
  // pattern (read-only)
  int n, meq, mineq, N, base, ns, nlev, nnzR, cmask_ok;
  const int *__restrict__ super, *__restrict__ sparent, *__restrict__ col2sup, *__restrict__ lpi, *__restrict__ lpx;
  const int *__restrict__ lev;
  const int *__restrict__ Rp, *__restrict__ Rj, *__restrict__ Rq, *__restrict__ ent;
  const int *__restrict__ bt_ptr, *__restrict__ bt_var, *__restrict__ bt_q, *__restrict__ bt_rpos;
  const int *__restrict__ sn_con, *__restrict__ con_sn, *__restrict__ eq_ptr, *__restrict__ eq_var,
      *__restrict__ eq_q;
  const int4 *__restrict__ snrec;  // 2 per supernode: {c0, w, nrow, value offset}, {row-list offset, pairs}
  // per pair (2): {descendant's first column, width << 16 | rows, its rows inside the target, row-list offset of
  // the first of them}, {its value offset, its Y offset (width > 1), descendant, its index in the descendant's rows}
  const int4 *__restrict__ prec;
  const int *__restrict__ con_ptr, *__restrict__ con_tgt;
  // solves: the single columns that may hide or are long, by level, then up to BATCH_SN_LONG rows / longer (so_seg:
  // 2 nlev + 1 group starts); the others (so_e); the rows and columns of the wide supernodes (see ldlt_solve_smem)
  const int *__restrict__ so_sn, *__restrict__ so_seg;
  const int4 *__restrict__ so_rec, *__restrict__ so_e, *__restrict__ so_f, *__restrict__ so_b;
  const int2 *__restrict__ so_g;  // groups of 32 targets of the single columns
  const int *__restrict__ so_gj, *__restrict__ so_gs;  // their variables, their entries' columns
  const int *__restrict__ gidx;   // per row-list position of a single column: its entry in G, or -1
  int n1;  // length of so_sn
  // problem
  const double *__restrict__ kv, *__restrict__ q, *__restrict__ bq, *__restrict__ dq;
  const uint8_t *__restrict__ pert;
  double reg, reg32;
  // slot
  T *L, *D, *S, *G;  // G: the single columns' entries by target (see gather_singles)
  T *Di;  // D^-1 of the wide supernodes: diagonal, then the 2x2 blocks' off-diagonals (N each)
  int *ls, *perm, *iperm, *lperm, *alist, *mlist;
  int4 *vrec;  // so_rec of the visible single columns
  int *arow;   // rows of the active constraints
  uint8_t *piv;
  T *Fv;       // factorization values of K in CSR order
  double *Rv;  // refinement values
  unsigned long long *cmask;  // per supernode: active constraint-column descendants (bit = pair - pair_mid)
  double *rhs, *sol, *r, *w, *V, *tmp;
  T *Z;
  // shared memory
  Sh<int> map;
  Sh<T> xs;      // vectors of the solves, in the factor's order (xo shares the row map's memory where it is shared)
  Spill<T> xo;
  Sh<T> B, rowbuf, Dsm, Esm, Binv;
  Sh<int> lp;
  // per-warp scratch of the level-parallel factorization (WF_WARPS warps,
  // wstride values each): block wcap x rcap, wcap x wcap, D, E, D^-1; pivot orders
  Sh<T> wB;
  Sh<int> wlp;
  int wstride;
  int wcap, rcap;  // widest / tallest supernode a warp takes (<= 32)
  int wf;          // level-parallel factorization on
  Sh<uint8_t> vis;  // per supernode: visible (structural, or the column of an active constraint)
  Sh<uint8_t> act;  // per constraint: active
  Sh<int> vseg;     // starts of each level's two groups in vrec (2 nlev + 1), then the length of arow
  Spill<int4> lvl;     // per level (3): the pattern's items of the solves (see BPat)
  Spill<uint8_t> mark;  // per supernode: to be refactored
  int nmark;    // > 0: edits wait for a refactorization; during one, the length of mlist
  double red[32];
  int redi[32];
  int status;  // device status bits of this problem
  int prof;    // per-phase SM cycles of this CTA are counted in cyc
  unsigned long long cyc[PH_N];
  GmresSmall gs;
};
static_assert(sizeof(Ctx<double>) <= BATCH_CTX_BYTES && sizeof(Ctx<float>) <= BATCH_CTX_BYTES, "context size");
template <class T> __device__ __forceinline__ Ctx<T> &ctx() {
  extern __shared__ __align__(16) unsigned char dsm[];
  return *reinterpret_cast<Ctx<T> *>(dsm);
}

static_assert(PH_N <= BATCH_PROFILE_COUNTERS, "profile counters");
#define BQ_T0(c) const long long t0_ = (c).prof ? clock64() : 0
#define BQ_T1(c, ph) \
  if ((c).prof && threadIdx.x == 0) (c).cyc[ph] += (unsigned long long)(clock64() - t0_)

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ int warp_id() { return threadIdx.x >> 5; }
__device__ __forceinline__ int num_warps() { return blockDim.x >> 5; }

template <class T> __device__ __forceinline__ bool visible(const Ctx<T> &c, int s) { return c.vis[s] != 0; }

// Calls f(pair) for every descendant pair of s (pairs [pp, pe), constraint
// columns from pm) whose descendant is visible: the structural ones, then the
// active constraint columns (bit mask, or a scan when a supernode has more
// than 64 of them).
template <class T, class F>
__device__ __forceinline__ void for_visible_pairs(const Ctx<T> &c, int pp, int pm, int pe, int s, F &&f) {
#pragma unroll 1
  for (int pq = pp; pq < pm; ++pq) f(pq);
  if (c.cmask_ok) {
    unsigned long long m = c.cmask[s];
    while (m) {
      const int b = __ffsll((long long)m) - 1;
      m &= m - 1ull;
      f(pm + b);
    }
  } else {
#pragma unroll 1
    for (int pq = pm; pq < pe; ++pq)
      if (c.vis[c.prec[2 * pq + 1].z]) f(pq);
  }
}

// Block-wide sum in a fixed order (per-thread strided partials, then a tree):
// the same inputs give the same bits on every run.
__device__ double block_sum(double v, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane_id() == 0) red[warp_id()] = v;
  __syncthreads();
  if (warp_id() == 0) {
    v = lane_id() < num_warps() ? red[lane_id()] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane_id() == 0) red[0] = v;
  }
  __syncthreads();
  v = red[0];
  __syncthreads();
  return v;
}

__device__ int block_sum_int(int v, int *redi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane_id() == 0) redi[warp_id()] = v;
  __syncthreads();
  if (warp_id() == 0) {
    v = lane_id() < num_warps() ? redi[lane_id()] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane_id() == 0) redi[0] = v;
  }
  __syncthreads();
  v = redi[0];
  __syncthreads();
  return v;
}

// Block-wide selection: the largest (sel_max) or smallest value, the
// smallest index winning ties -- the outcome of the reference's ascending
// scans with strict comparisons.  idx < 0 marks "no candidate".
__device__ void block_select(double &v, int &idx, bool sel_max, double *red, int *redi) {
  auto better = [&](double ov, int oi, double cv, int ci) {
    if (oi < 0) return false;
    if (ci < 0) return true;
    if (ov == cv) return oi < ci;
    return sel_max ? ov > cv : ov < cv;
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double ov = __shfl_down_sync(0xffffffffu, v, o);
    int oi = __shfl_down_sync(0xffffffffu, idx, o);
    if (better(ov, oi, v, idx)) {
      v = ov;
      idx = oi;
    }
  }
  __syncthreads();
  if (lane_id() == 0) {
    red[warp_id()] = v;
    redi[warp_id()] = idx;
  }
  __syncthreads();
  if (warp_id() == 0) {
    v = lane_id() < num_warps() ? red[lane_id()] : 0.0;
    idx = lane_id() < num_warps() ? redi[lane_id()] : -1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      double ov = __shfl_down_sync(0xffffffffu, v, o);
      int oi = __shfl_down_sync(0xffffffffu, idx, o);
      if (better(ov, oi, v, idx)) {
        v = ov;
        idx = oi;
      }
    }
    if (lane_id() == 0) {
      red[0] = v;
      redi[0] = idx;
    }
  }
  __syncthreads();
  v = red[0];
  idx = redi[0];
  __syncthreads();
}


// ---- values ---------------------------------------------------------------
// Factorization value of lower-CSC entry vq: inactive constraint entries read
// as zero (the reference zeroes them in its ordered matrix), perturbed
// diagonals as the regularization (find_perturbation,
// linear_solver_wrapper.cpp:352-363).
//
// An FP32 factor also gets a floor reg32 on its diagonal: pivots as small as
// the 1e-9 regularization create element growth of ~1e9 under Bunch-Kaufman
// restricted to supernode diagonal blocks, beyond what FP32 carries; the
// factor is only the preconditioner of the FP64 refinement, whose matrix keeps
// the reference's values.  The floor is negative on the constraints' rows: the
// Schur complement there is -A H^-1 A^T, which a positive one makes singular
// wherever an eigenvalue of A H^-1 A^T comes near it, and the refinement then
// ran out of steps (1 in 8000 uneven MPC problems ended up to 1e-1 off, which
// ones depending on rounding; with the negative floor none of 121856).
template <class T> __device__ __forceinline__ double fact_val(const Ctx<T> &c, int vq) {
  const int e = c.ent[vq];
  double v = c.kv[vq];
  if (e >= 0) return c.act[e] ? v : 0.0;
  if (e <= -2) {
    if (c.pert[-2 - e]) v = c.reg;
    if (sizeof(T) == 4 && fabs(v) < c.reg32) v = v < 0.0 || -2 - e >= c.n ? -c.reg32 : c.reg32;
  }
  return v;
}
// Refinement value: perturbed diagonals read as zero (set_diags(0),
// linear_solver_wrapper.cpp:1359-1394).
template <class T> __device__ __forceinline__ double ref_val(const Ctx<T> &c, int vq) {
  const int e = c.ent[vq];
  double v = c.kv[vq];
  if (e >= 0) return c.act[e] ? v : 0.0;
  if (e <= -2 && c.pert[-2 - e]) return 0.0;
  return v;
}

// ---- blocks ------------------------------------------------------------------
// A supernode of one column keeps [1/d; L21] in c.L.  Those of at most 32 rows
// that never hide are stored 32 at a time, entry r of 32 neighbours (in the
// order the solves take them) side by side, values and row list alike
// (stride 32): a warp of the solves, a lane per supernode, reads them in whole
// lines.  A wider supernode keeps in c.S, by rows of w4 = s_ld(w) values:
//   R = [L11^-1; L21]   nrow rows, for the solves (their forward sums run along
//                       a row, 16 bytes a load; the backward ones across rows,
//                       a lane per column) and, from row w on, for the updates;
//   Y = L21 D           m = nrow - w rows: an update is L21 Y^T, without a
//                       pivot block in sight.
__host__ __device__ __forceinline__ int s_ld(int w) { return (w + 3) & ~3; }
// supernode record: rows, and the stride of its values and row list
__device__ __forceinline__ int sn_rows(const int4 &r0) { return r0.z & 0xffff; }
__device__ __forceinline__ int sn_stride(const int4 &r0) { return r0.z >> 16 ? 32 : 1; }

// Four consecutive values from a multiple of four values into a block.
[[maybe_unused]] __device__ __forceinline__ void load4(const float *p, float (&v)[4]) {
  const float4 f = *reinterpret_cast<const float4 *>(p);
  v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
}
[[maybe_unused]] __device__ __forceinline__ void load4(const double *p, double (&v)[4]) {
  const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
  v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}



// bk_block on blocks in dynamic shared memory, by their offsets.
template <class T>
__device__ __noinline__ bool bk_block_at(Sh<T> a, int lda, int w, Sh<T> D, Sh<T> E, Sh<int> perm, int wi, int nw) {
  return bk_block<T>((T *)a, lda, w, (T *)D, (T *)E, (int *)perm, &ctx<T>().status, wi, nw);
}

[[maybe_unused]] __device__ __forceinline__ bool finite_bits(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
[[maybe_unused]] __device__ __forceinline__ bool finite_bits(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }
template <class T> __device__ __forceinline__ void check_finite(Ctx<T> &c, T v) {
  if (!finite_bits(v)) atomicOr(&c.status, ST_NONFINITE);
}

// Updates of target s from its visible descendants: the staged target block
// B (nr x w, rows found by pos(row)) loses L_d[rows] Y_d[rows in s]^T of every
// one (single columns: Y = d L).  Entries of a pair go to lanes one each, so
// that all lanes work whatever the pair's shape; small pairs are dealt to the
// warps in turn, large ones shared by all of them (wi of nw warps call).
// Pairs of different warps may hit the same entry: the subtraction is atomic
// when nw > 1 (the summation order varies between runs, as in the
// reference's threaded factorization).
template <class T, class F>
__device__ __forceinline__ void sn_updates(Ctx<T> &c, int s, int c0, int w, int nr, int pp, int pm, int pe, T *B,
                                           int wi, int nw, F &&pos) {
  const int lane = lane_id();
  int t = 0;
  for_visible_pairs(c, pp, pm, pe, s, [&](int pq) {
    const int4 ra = c.prec[2 * pq], rb = c.prec[2 * pq + 1];
    const int wd = (int)((unsigned)ra.y >> 16), nc = ra.z, md = (ra.y & 0xffff) - rb.w;
    const int total = md * nc;
    int e0 = lane, step = 32;
    if (nw > 1) {
      if (total <= 128) {
        if (t++ % nw != wi) return;
      } else {
        e0 += 32 * wi;
        step *= nw;
      }
    }
    // wd 0, 1: a single column (stride 32, 1)
    const int st = wd == 0 ? 32 : 1, ld = s_ld(wd);
    const int *rd = c.ls + ra.w;  // descendant's rows from its first one inside s
    const T *Li = (wd < 2 ? c.L : c.S) + rb.x;  // its L21 from that row
    const T *Yj = c.S + rb.y;                   // its Y from that row (wd > 1)
    const T d1 = wd < 2 ? c.D[ra.x] : T(0);
#pragma unroll 1
    for (int eb = e0 - lane; eb < total; eb += step) {
      const int e = eb + lane;
      const int jj = e / md, i = e - jj * md;
      int ti = -1, tj = 0;
      if (e < total) {
        tj = rd[jj * st] - c0;
        ti = pos(rd[i * st]);
        if (ti < 0 || tj < 0 || tj >= w) {
          atomicOr(&c.status, ST_BOUNDS);
          ti = -1;
        }
      }
      if (e >= total || ti < tj) continue;  // lower triangle of the target only
      T acc = T(0);
      if (wd < 2) {
        acc = Li[i * st] * (d1 * Li[jj * st]);
      } else {
        const T *li = Li + i * ld, *yj = Yj + jj * ld;
#pragma unroll 2
        for (int k0 = 0; k0 < wd; k0 += 4) {
          T l[4], y[4];
          load4(li + k0, l);
          load4(yj + k0, y);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (k0 + q < wd) acc += l[q] * y[q];
        }
      }
      if (nw > 1) atomicAdd(&B[ti + tj * nr], -acc);
      else B[ti + tj * nr] -= acc;
    }
    if (nw == 1) __syncwarp();
  });
}

// ---- factorization of one single-column supernode (warp scope) ----------------
// The left-looking step of the reference (Serial_update_ldl.cpp:62-190) for a
// column of at most 32 rows, a lane per row: most supernodes of a KKT tree.
// Warp wi has 32 values of the row scratch and byte wi of every word of the row map.
template <class T> __device__ __noinline__ void factor_single(Ctx<T> &, int s, int wi) {
  Ctx<T> &c = ctx<T>();
  T *b = c.rowbuf + 32 * wi;
  const unsigned FULL = 0xffffffffu;
  const int lane = lane_id();
  if (c.prof && lane == 0) atomicAdd(&c.cyc[PH_SN], 1ull);
  const int4 r0 = c.snrec[2 * s], r1 = c.snrec[2 * s + 1];
  const int c0 = r0.x, nr = sn_rows(r0), ss = sn_stride(r0);
  const int *rows = c.ls + r1.x;
  uint8_t *map8 = Sh<uint8_t>{c.map.off};
  const int myrow = lane < nr ? rows[lane * ss] : -1;
  if (lane < nr) map8[4 * myrow + wi] = (uint8_t)lane;
  b[lane] = T(0);
  __syncwarp();
  // every lane calls; -1: not in the row list
  auto find = [&](int r) {
    const int p = r >= 0 ? map8[4 * r + wi] & 31 : 0;
    return __shfl_sync(FULL, myrow, p) == r && p < nr ? p : -1;
  };
  const int j = c.perm[c0], qb = c.Rp[j], qe = c.Rp[j + 1];
#pragma unroll 1
  for (int q0 = qb; q0 < qe; q0 += 32) {
    const int qq = q0 + lane;
    const int oi = qq < qe ? c.iperm[c.Rj[qq]] : -1;
    const T v = qq < qe ? c.Fv[qq] : T(0);
    const int p = find(oi);
    if (oi >= c0) {
      if (p < 0) atomicOr(&c.status, ST_BOUNDS);  // not in the row list: corrupted structure
      else b[p] = v;
    }
  }
  __syncwarp();
  for_visible_pairs(c, r1.y, r1.z, r1.w, s, [&](int pq) {
    const int4 ra = c.prec[2 * pq], rb = c.prec[2 * pq + 1];
    const int wd = (int)((unsigned)ra.y >> 16), md = (ra.y & 0xffff) - rb.w;
    const int st = wd == 0 ? 32 : 1, ld = s_ld(wd);
    const int *rd = c.ls + ra.w;
    const T *Li = (wd < 2 ? c.L : c.S) + rb.x, *y = c.S + rb.y;
#pragma unroll 1
    for (int i0 = 0; i0 < md; i0 += 32) {
      const int i = i0 + lane;
      const int p = find(i < md ? rd[i * st] : -1);
      if (i < md) {
        T acc = T(0);
        if (wd < 2) {
          acc = Li[i * st] * (c.D[ra.x] * Li[0]);
        } else {
#pragma unroll 1
          for (int k = 0; k < wd; ++k) acc += Li[i * ld + k] * y[k];
        }
        if (p < 0) atomicOr(&c.status, ST_BOUNDS);
        else b[p] -= acc;
      }
    }
    __syncwarp();
  });
  const T v = b[lane], d = __shfl_sync(FULL, v, 0);
  const T inv = T(1) / d;
  if (lane == 0 && !(tabs(d) > T(0))) atomicOr(&c.status, d == T(0) ? ST_ZERO_PIVOT : ST_NONFINITE);
  if (lane < nr) {
    const T l = lane ? v * inv : inv;
    check_finite(c, l);
    c.L[r0.w + lane * ss] = l;
    const int g = ss == 32 ? c.gidx[r1.x + lane * 32] : -1;
    if (g >= 0) c.G[g] = l;
  }
  if (lane == 0) {
    c.D[c0] = d;
    c.lperm[c0] = 0;
    c.piv[s] = 0;
  }
  __syncwarp();
}

// ---- factorization of one supernode -------------------------------------------
// Left-looking step of the reference (Serial_update_ldl.cpp:62-190): scatter
// the matrix columns, subtract every visible descendant's L D L^T restricted
// to the supernode, Bunch-Kaufman on the diagonal block, then the rows below
// permuted and solved with the unit L11^T.  The rows of the identity go along
// (their solutions are the columns of L11^-1).  The blocks stay in factored
// form: A11^-1 and L21 L11^-1 as such would make every solve a single product,
// but pivots as small as the 1e-9 regularization leave them with errors that
// the refinement then needs three times the steps for (measured).
//
// wi of nw warps call with the same scratch: the whole CTA (nw > 1, barriers)
// or one warp (nw = 1).  B: nr x w, I: w x w, dv: 2 w values (D^-1).
template <class T, bool CTA, class F>
__device__ __forceinline__ void sn_finish(Ctx<T> &c, int s, int c0, int w, int nr, const int4 &r0, T *B, T *I, T *D,
                                          T *E, int *lp, T *dv, bool pivoted, int tid, int nt, F &&lap) {
  auto sync = [&]() {
    if (CTA) __syncthreads();
    else __syncwarp();
  };
  const int m = nr - w;
  // a lane keeps its row: R of them, the other index over nt / R
  int R = 32;
  while (nt % (2 * R) == 0 && R < nr) R *= 2;  // nt need not be a power of two
  const int rr = tid & (R - 1), cq = tid / R, cs = nt / R;
  if (pivoted) {  // columns of the rows below into pivot order (cycles, in place)
#pragma unroll 1
    for (int r = w + tid; r < nr; r += nt) {
      T *br = B + r;
#pragma unroll 1
      for (int j0 = 0; j0 < w; ++j0) {
        int q = lp[j0], g = 0;
        while (q > j0 && g++ < w) q = lp[q];
        if (q != j0 || lp[j0] == j0) continue;  // the smallest index of a cycle turns it
        const T first = br[j0 * nr];
        int j = j0;
#pragma unroll 1
        for (g = 0; g < w; ++g) {
          const int src = lp[j];
          br[j * nr] = src == j0 ? first : br[src * nr];
          if (src == j0) break;
          j = src;
        }
      }
    }
  }
#pragma unroll 1
  for (int j = cq; j < w; j += cs)
#pragma unroll 1
    for (int r = rr; r < w; r += R) I[r + j * w] = r == j ? T(1) : T(0);
  if (tid < w) {
    T inv, off;
    d_inverse(D, E, w, tid, inv, off);
    dv[tid] = inv;
    dv[w + tid] = off;
  }
#pragma unroll 1
  for (int k = tid + nt; k < w; k += nt) {
    T inv, off;
    d_inverse(D, E, w, k, inv, off);
    dv[k] = inv;
    dv[w + k] = off;
  }
  sync();
  // V L11^T = [I; A21]: column j is final, the later ones lose x_j L11(t, j)
  // (each entry receives its terms in increasing j, as in the substitution)
#pragma unroll 1
  for (int j = 0; j + 1 < w; ++j) {
    const T *Lj = B + j * nr;
#pragma unroll 1
    for (int r = rr; r < nr; r += R) {
      if (r < w && r > j) continue;  // still zero
      T *vr = r < w ? I + r : B + r;
      const int ld = r < w ? w : nr;
      const T xj = vr[j * ld];
      int t = j + 1 + cq;
#pragma unroll 1
      for (; t + 3 * cs < w; t += 4 * cs) {
        const T l0 = Lj[t], l1 = Lj[t + cs], l2 = Lj[t + 2 * cs], l3 = Lj[t + 3 * cs];
        const T v0 = vr[t * ld], v1 = vr[(t + cs) * ld], v2 = vr[(t + 2 * cs) * ld], v3 = vr[(t + 3 * cs) * ld];
        vr[t * ld] = v0 - xj * l0;
        vr[(t + cs) * ld] = v1 - xj * l1;
        vr[(t + 2 * cs) * ld] = v2 - xj * l2;
        vr[(t + 3 * cs) * ld] = v3 - xj * l3;
      }
#pragma unroll 1
      for (; t < w; t += cs) vr[t * ld] -= xj * Lj[t];
    }
    if (CTA && cs > 1) __syncthreads();
    // a row's columns all belong to its lane otherwise
  }
  sync();
  lap(PH_SN_ROWS);
  // out: L11^-1 by rows (I(r, k) = L11^-1(k, r)), Y as it stands, L21 = Y D^-1
  const int w4 = s_ld(w);
  T *Rb = c.S + r0.w, *Yb = Rb + nr * w4;
#pragma unroll 1
  for (int e = tid; e < w * w4; e += nt) {
    const int i = e / w4, j = e - i * w4;
    const T v = j < w ? I[j + i * w] : T(0);
    check_finite(c, v);
    Rb[e] = v;
  }
#pragma unroll 1
  for (int e = tid; e < m * w4; e += nt) {
    const int r = w + e / w4, j = e % w4;
    T y = T(0), v = T(0);
    if (j < w) {
      y = B[r + j * nr];
      v = y * dv[j];
      if (dv[w + j] != T(0)) v += dv[w + j] * B[r + (j + 1) * nr];
      if (j > 0 && dv[w + j - 1] != T(0)) v += dv[w + j - 1] * B[r + (j - 1) * nr];
      check_finite(c, v);
    }
    Yb[e] = y;
    Rb[w * w4 + e] = v;
  }
#pragma unroll 1
  for (int k = tid; k < w; k += nt) {
    check_finite(c, dv[k]);
    c.D[c0 + k] = D[k];
    c.Di[c0 + k] = dv[k];
    c.Di[c.N + c0 + k] = dv[w + k];
    c.lperm[c0 + k] = lp[k];
  }
  if (tid == 0) c.piv[s] = pivoted ? 1 : 0;
  sync();
  lap(PH_SN_STORE);
}

// By the whole CTA.
template <class T> __device__ __noinline__ void factor_sn(Ctx<T> &, int s) {
  Ctx<T> &c = ctx<T>();
  const int tid = threadIdx.x, nt = blockDim.x;
  if (c.prof && tid == 0) c.cyc[PH_SN] += 1;
  const int4 r0 = c.snrec[2 * s], r1 = c.snrec[2 * s + 1];
  const int c0 = r0.x, w = r0.y, nr = sn_rows(r0);
  const int *rows = c.ls + r1.x;
  T *B = c.B;
  long long tq = c.prof ? clock64() : 0;
  auto lap = [&](int ph) {
    if (c.prof && tid == 0) {
      const long long now = clock64();
      c.cyc[ph] += (unsigned long long)(now - tq);
      tq = now;
    }
  };
#pragma unroll 1
  for (int p = tid; p < nr; p += nt) c.map[rows[p]] = p;
#pragma unroll 1
  for (int e = tid; e < nr * w; e += nt) B[e] = T(0);
  __syncthreads();
  // matrix columns (symmetric neighbours of the original column, ordered >=
  // the column): g threads per column, all columns at once
  const int g = w < nt ? nt / w : 1;
#pragma unroll 1
  for (int t = tid; t < w * g; t += nt) {
    const int m = t % w, k0 = t / w;
    const int col = c0 + m;
    const int j = c.perm[col];
#pragma unroll 1
    for (int qq = c.Rp[j] + k0; qq < c.Rp[j + 1]; qq += g) {
      const int oi = c.iperm[c.Rj[qq]];
      if (oi < col) continue;
      const int pos = c.map[oi];
      if (pos < 0 || pos >= nr || rows[pos] != oi) {  // not in the row list: corrupted structure
        atomicOr(&c.status, ST_BOUNDS);
        continue;
      }
      B[pos + m * nr] = c.Fv[qq];
    }
  }
  __syncthreads();
  lap(PH_SN_ASSEMBLE);
  sn_updates(c, s, c0, w, nr, r1.y, r1.z, r1.w, B, warp_id(), num_warps(), [&](int r) {
    const int p = c.map[r];
    return p >= 0 && p < nr && rows[p] == r ? p : -1;
  });
  __syncthreads();
  lap(PH_SN_UPDATES);
  if (w == 1) {  // a column of more than 32 rows
    const T d = B[0], inv = T(1) / d;
    if (tid == 0) {
      if (!(tabs(d) > T(0))) atomicOr(&c.status, d == T(0) ? ST_ZERO_PIVOT : ST_NONFINITE);
      c.D[c0] = d;
      c.lperm[c0] = 0;
      c.piv[s] = 0;
    }
#pragma unroll 1
    for (int r = tid; r < nr; r += nt) {
      const T l = r ? B[r] * inv : inv;
      check_finite(c, l);
      c.L[r0.w + r] = l;
    }
    __syncthreads();
    lap(PH_SN_STORE);
    return;
  }
  bool pivoted = false;
  if (w <= 64) pivoted = bk_block_at<T>(c.B, nr, w, c.Dsm, c.Esm, c.lp, warp_id(), num_warps());
  else bk_factor<T>(B, nr, w, c.Dsm, c.Esm, c.lp, &c.status, &pivoted);
  __syncthreads();
  lap(PH_SN_BK);
  sn_finish<T, true>(c, s, c0, w, nr, r0, B, c.Binv, c.Dsm, c.Esm, c.lp, c.rowbuf, pivoted, tid, nt, lap);
}

// By warp wi alone, in its own scratch: a supernode of at most wcap columns
// and rcap rows (both <= 32).
template <class T> __device__ __noinline__ void factor_sn_warp(Ctx<T> &, int s, int wi) {
  Ctx<T> &c = ctx<T>();
  const int lane = lane_id();
  if (c.prof && lane == 0) atomicAdd(&c.cyc[PH_SN], 1ull);
  const int4 r0 = c.snrec[2 * s], r1 = c.snrec[2 * s + 1];
  const int c0 = r0.x, w = r0.y, nr = sn_rows(r0);
  const int *rows = c.ls + r1.x;
  const Sh<T> sB = c.wB.at(wi * c.wstride), sD = sB.at(c.wcap * (c.rcap + c.wcap)), sE = sD.at(c.wcap);
  const Sh<int> slp = c.wlp.at(wi * c.wcap);
  T *B = sB, *I = B + c.wcap * c.rcap, *Dw = sD, *Ew = sE, *dv = Ew + c.wcap;
  int *lpw = slp;
  uint8_t *map8 = Sh<uint8_t>{c.map.off};
  const int myrow = lane < nr ? rows[lane] : -1;
  if (lane < nr) map8[4 * myrow + wi] = (uint8_t)lane;
#pragma unroll 1
  for (int e = lane; e < nr * w; e += 32) B[e] = T(0);
  __syncwarp();
  // matrix columns (entries of rows >= the column), one lane per entry
#pragma unroll 1
  for (int m = 0; m < w; ++m) {
    const int col = c0 + m, j = c.perm[col];
    const int qb = c.Rp[j], qe = c.Rp[j + 1];
#pragma unroll 1
    for (int qq = qb + lane; qq < qe; qq += 32) {
      const int oi = c.iperm[c.Rj[qq]];
      if (oi < col) continue;
      const int p = map8[4 * oi + wi];
      if (p >= nr || rows[p] != oi) atomicOr(&c.status, ST_BOUNDS);  // not in the row list: corrupted structure
      else B[p + m * nr] = c.Fv[qq];
    }
  }
  __syncwarp();
  sn_updates(c, s, c0, w, nr, r1.y, r1.z, r1.w, B, 0, 1, [&](int r) {
    const int p = map8[4 * r + wi];
    return p < nr && rows[p] == r ? p : -1;
  });
  const bool pivoted = bk_block_at<T>(sB, nr, w, sD, sE, slp, 0, 1);
  sn_finish<T, false>(c, s, c0, w, nr, r0, B, I, Dw, Ew, lpw, dv, pivoted, lane, 32, [](int) {});
}

// Factor the supernodes of mlist (ascending ids: children before parents,
// the reference's order of mod_indices), then fold the pivots into the row
// lists of the descendants (row_reordering, Sym_BLAS.cpp:327-490) and into
// the ordering (reorder_matrix, linear_solver_wrapper.cpp:1432-1460).
// Supernodes of one level of the tree are independent (each reads only
// descendants on lower levels and writes only itself), so a long list goes
// level by level: single columns a warp each, wider ones a warp each where
// there are enough of them to keep the warps busy (and the launch has the
// scratch), else one after another by the CTA.  A short list (the one or two
// paths to the root of an active-set step) runs through in order.
template <class T> __device__ __noinline__ void factor_marked(Ctx<T> &) {
  Ctx<T> &c = ctx<T>();
  const int m = c.nmark;
  const unsigned FULL = 0xffffffffu;
  const int wi = warp_id(), lane = lane_id(), nwf = min(num_warps(), WF_WARPS);
  // 0: a single column a warp takes, 1: a wide one that fits a warp, 2: the rest
  auto kind = [&](int s) {
    const int w = c.snrec[2 * s].y, nr = sn_rows(c.snrec[2 * s]);
    if (w == 1 && nr <= 32) return 0;
    return w > 1 && w <= c.wcap && nr <= c.rcap ? 1 : 2;
  };
  if (m > 2 * c.nlev) {
#pragma unroll 1
    for (int l = 0; l < c.nlev; ++l) {
      // every warp counts the level's supernodes the same way (uniform over the CTA)
      int n1 = 0, nw1 = 0, n2 = 0;
#pragma unroll 1
      for (int t0 = 0; t0 < m; t0 += 32) {
        const int s = t0 + lane < m ? c.mlist[t0 + lane] : -1;
        const int k = s >= 0 && c.lev[s] == l ? kind(s) : -1;
        n1 += __popc(__ballot_sync(FULL, k == 0));
        nw1 += __popc(__ballot_sync(FULL, k == 1));
        n2 += __popc(__ballot_sync(FULL, k == 2));
      }
      const bool warps = c.wf && nw1 >= 2;
      if (n1 + (warps ? nw1 : 0) > 0) {
        int seen = 0;
#pragma unroll 1
        for (int t0 = 0; t0 < m; t0 += 32) {
          const int s = t0 + lane < m ? c.mlist[t0 + lane] : -1;
          const int k = s >= 0 && c.lev[s] == l ? kind(s) : -1;
          unsigned bal = __ballot_sync(FULL, k == 0 || (k == 1 && warps));
          while (bal) {
            const int b = __ffs(bal) - 1;
            bal &= bal - 1u;
            const int sb_ = __shfl_sync(FULL, s, b), kb = __shfl_sync(FULL, k, b);
            if (seen++ % nwf == wi) {
              if (kb == 0) factor_single(c, sb_, wi);
              else factor_sn_warp(c, sb_, wi);
            }
          }
        }
        __syncthreads();
      }
      if (n2 + (warps ? 0 : nw1) > 0)
#pragma unroll 1
        for (int t = 0; t < m; ++t) {
          const int s = c.mlist[t];
          if (c.lev[s] != l) continue;
          const int k = kind(s);
          if (k == 2 || (k == 1 && !warps)) factor_sn(c, s);
        }
    }
  } else {
#pragma unroll 1
    for (int t = 0; t < m; ++t) {
      const int s = c.mlist[t];
      if (kind(s) == 0) {
        if (wi == 0) factor_single(c, s, 0);
        __syncthreads();
      } else {
        factor_sn(c, s);
      }
    }
  }
  BQ_T0(c);
  // renaming: rows of descendants that fall into a pivoted supernode
#pragma unroll 1
  for (int t = 0; t < m; ++t) {
    const int s = c.mlist[t];
    if (!c.piv[s]) continue;
    const int4 r0 = c.snrec[2 * s], r1 = c.snrec[2 * s + 1];
    const int c0 = r0.x, w = r0.y;
    // inverse of the local pivot order: old local position -> new position;
    // composed ordering: new position q holds the column that was at lperm[q]
    // (old values staged in the free row map)
#pragma unroll 1
    for (int q = threadIdx.x; q < w; q += blockDim.x) {
      const int o = c.lperm[c0 + q];
      c.lp[o] = q;
      c.map[q] = c.perm[c0 + o];
    }
    __syncthreads();
#pragma unroll 1
    for (int q = threadIdx.x; q < w; q += blockDim.x) {
      const int j = c.map[q];
      c.perm[c0 + q] = j;
      c.iperm[j] = c0 + q;
    }
#pragma unroll 1
    for (int pq = r1.y + threadIdx.x; pq < r1.w; pq += blockDim.x) {  // a pair per thread
      const int4 ra = c.prec[2 * pq];
      const int st = (unsigned)ra.y >> 16 ? 1 : 32;
      int *rd = c.ls + ra.w;
#pragma unroll 1
      for (int i = 0; i < ra.z; ++i) {
        const int o = rd[i * st] - c0;
        if (o >= 0 && o < w) rd[i * st] = c0 + c.lp[o];
        else atomicOr(&c.status, ST_BOUNDS);
      }
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int t = threadIdx.x; t < m; t += blockDim.x) c.mark[c.mlist[t]] = 0;
  __syncthreads();
  if (threadIdx.x == 0) c.nmark = 0;
  __syncthreads();
  BQ_T1(c, PH_RENAME);
}

// ---- triangular solves (factor order, vectors in shared memory) ----------------
// Forward (reference H2LeveledBlockedLsolve, Triangular_BCSC.cpp:378-446):
// t_s = L11^-1 x_s, then the rows below lose L21 t_s (pushes of supernodes of
// the same level may meet, so they are atomic, as in the reference's threaded
// solve, :435).  Backward (:534-600): v_s = D^-1 t_s - L21^T x(rows below),
// x_s = L11^-T v_s.  Two vectors, xs and xo, take turns, so that all rows
// (columns) of a level's supernodes can be formed at once: xs holds the
// accumulated right hand side, then v; xo holds t, then the solution.  Single
// columns need no t: theirs is x_s.
//
// What bounds them: latency (a chain of row index, factor entry and push per
// level, 16 warps on an SM that issue one instruction in 16 cycles each), the
// instructions of a step, the lines that a warp's loads touch, and in FP64
// operations (a multiply-add holds the FP64 pipe of its SM quarter for 64
// cycles whatever the number of lanes at work).  So
//  * the rows (columns) of all wide supernodes of a level form one list (so_f,
//    so_b, in the pattern), dealt to the threads with as many lanes to a row
//    as keep the CTA full;
//  * a step issues its first loads, which no other step writes, before the
//    barrier that it has to wait for, and no load stands under a condition:
//    places beyond the end read a valid entry with a zero factor (a branch per
//    term made every load wait for the one before: 230k cycles per
//    application of horizon-50 MPC, FP32, 4 CTAs per SM);
//  * where a level has many single columns, their targets gather (so_g: the
//    factor entries once more, by target) instead of the columns pushing: an
//    FP32 atomic of shared memory takes 88 cycles for every lane that meets
//    another on its entry, an FP64 one 140.
template <class T> __device__ __forceinline__ void push(const Ctx<T> &c, int rr, T y) {
  if (y != T(0)) atomicAdd(&c.xs[min((unsigned)rr, (unsigned)c.N - 1u)], -y);
}

// Four rows below of a single column (entry r0 on, stride st), zeros beyond the end.
template <class T> struct Single4 {
  T l[4];
  int rr[4];
  __device__ __forceinline__ void load(const Ctx<T> &c, const int4 &v, int r0, int st) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = min(r0 + q, v.y - 1);
      l[q] = c.L[v.z + r * st];
      rr[q] = c.ls[v.w + r * st];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (r0 + q >= v.y) l[q] = T(0);
  }
};
template <class T> __device__ __noinline__ void fwd_single(Ctx<T> &, const int4 v, int st) {
  Ctx<T> &c = ctx<T>();
  const T t = c.xs[v.x];
#pragma unroll 1
  for (int r0 = 1; r0 < v.y; r0 += 4) {
    Single4<T> b;
    b.load(c, v, r0, st);
#pragma unroll
    for (int q = 0; q < 4; ++q) push(c, b.rr[q], b.l[q] * t);
  }
}
// b: the first four rows, loaded
template <class T> __device__ __forceinline__ void bwd_single(Ctx<T> &c, const int4 &v, Single4<T> &b, T dinv, int st) {
  T acc = dinv * c.xs[v.x];
#pragma unroll 1
  for (int r0 = 1; r0 < v.y;) {
    T x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = c.xo[min((unsigned)b.rr[q], (unsigned)c.N - 1u)];
#pragma unroll
    for (int q = 0; q < 4; ++q) acc -= b.l[q] * x[q];
    r0 += 4;
    if (r0 < v.y) b.load(c, v, r0, st);
  }
  c.xo[v.x] = acc;
}
// Single columns of constraints and long ones: few are visible at a time.
template <class T> __device__ __noinline__ void fwd_listed(Ctx<T> &, int a, int m, int e) {
  Ctx<T> &c = ctx<T>();
#pragma unroll 1
  for (int q = a + threadIdx.x; q < m; q += blockDim.x) fwd_single(c, c.vrec[q], 1);
#pragma unroll 1
  for (int q = m + warp_id(); q < e; q += num_warps()) {
    const int4 v = c.vrec[q];
    const T t = c.xs[v.x];
#pragma unroll 4
    for (int r = 1 + lane_id(); r < v.y; r += 32) push(c, c.ls[v.w + r], c.L[v.z + r] * t);
  }
}
template <class T> __device__ __noinline__ void bwd_listed(Ctx<T> &, int a, int m, int e) {
  Ctx<T> &c = ctx<T>();
#pragma unroll 1
  for (int q = a + threadIdx.x; q < m; q += blockDim.x) {
    const int4 v = c.vrec[q];
    Single4<T> b;
    b.load(c, v, 1, 1);
    bwd_single(c, v, b, c.L[v.z], 1);
  }
#pragma unroll 1
  for (int q = m + warp_id(); q < e; q += num_warps()) {
    const int4 v = c.vrec[q];
    T acc = T(0);
#pragma unroll 4
    for (int r = 1 + lane_id(); r < v.y; r += 32)
      acc += c.L[v.z + r] * c.xo[min((unsigned)c.ls[v.w + r], (unsigned)c.N - 1u)];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane_id() == 0) c.xo[v.x] = c.L[v.z] * c.xs[v.x] - acc;
  }
}

// The targets of a level's single columns: x_j loses the sum of its entries
// times the columns' x.  g: first group of 32 targets, n of them;
// `alone`: no other thread pushes meanwhile.
template <class T> __device__ __noinline__ void gather_singles(Ctx<T> &, int g0, int n, bool alone) {
  Ctx<T> &c = ctx<T>();
#pragma unroll 1
  for (int g = g0 + warp_id(); g < g0 + n; g += num_warps()) {
    const int2 gr = c.so_g[g];  // first entry, entries per lane (a multiple of 4)
    const int j = c.so_gj[32 * g + lane_id()];  // variable, -1 beyond the end
    const int pos = c.iperm[max(j, 0)];
    T acc = T(0);
#pragma unroll 1
    for (int k = 0; k < gr.y; k += 4) {
      const int e = gr.x + 32 * k + lane_id();
      T l[4], x[4];
      int src[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        src[q] = c.so_gs[e + 32 * q];
        l[q] = c.G[e + 32 * q];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = c.xs[src[q]];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc += l[q] * x[q];
    }
    if (j >= 0) {
      if (alone) c.xs[pos] -= acc;
      else atomicAdd(&c.xs[pos], -acc);
    }
  }
}

// Sum over the G = 2^lg neighbouring lanes that share an item.
template <class T> __device__ __forceinline__ T lanes_sum(T v, int lg) {
#pragma unroll 1
  for (int o = 1 << lg >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of a block's row with x[0 ..] (zeros follow its terms up to a multiple
// of four): lane g of G takes every G-th group of four, from k0 = 4 g; p: its
// first two groups, loaded.
template <class T> struct RowTerms {
  T p[2][4];
  __device__ __forceinline__ void load(const T *row, int k0, int terms, int lg) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = k0 + (4 << lg) * h;
#pragma unroll
      for (int q = 0; q < 4; ++q) p[h][q] = T(0);
      if (k < terms) load4(row + k, p[h]);
    }
  }
  __device__ __forceinline__ T sum(const T *row, const T *x, int terms, int k0, int lg) {
    T acc = T(0);
    const int last = terms - 1;
#pragma unroll 1
    for (; k0 < terms;) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = k0 + (4 << lg) * h;
        if (h == 1 && k >= terms) break;
        T v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = x[min(k + q, last)];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc += p[h][q] * v[q];
      }
      k0 += 8 << lg;
      if (k0 < terms) load(row, k0, terms, lg);
    }
    return acc;
  }
};
// Sum down a block's column (stride ld, terms terms): lane g of G takes every
// G-th row from r0 = g; p: its first four, loaded (zeros beyond the end).
template <class T> struct ColTerms {
  T p[4];
  __device__ __forceinline__ void load(const T *col, int r0, int ld, int terms, int lg) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + (q << lg);
      p[q] = T(0);
      if (r < terms) p[q] = col[r * ld];
    }
  }
};

// xo <- (L D L^T)^-1 xs on the visible part, in the factor's order (xs is
// overwritten).  The caller's writes to xs and xo need no barrier before;
// one follows the last step.
template <class T> __device__ __noinline__ void ldlt_solve_smem(Ctx<T> &) {
  Ctx<T> &c = ctx<T>();
  const int tid = threadIdx.x, nt = blockDim.x, lane = lane_id();
  const T *const S = c.S;
  const int *const ls = c.ls;
  T *const xs = c.xs, *const xo = c.xo;
  const int nlev = c.nlev;
  const unsigned top = (unsigned)c.N - 1u;
  {
    BQ_T0(c);
#pragma unroll 1
    for (int l = 0; l < nlev; ++l) {
      const int a = c.vseg[2 * l], m = c.vseg[2 * l + 1], e = c.vseg[2 * l + 2];
      const int4 lf = c.lvl[3 * l], lb = c.lvl[3 * l + 1], lg_ = c.lvl[3 * l + 2];
      const int n1 = lf.y >> 5, lg1 = lf.y & 31, n2 = lf.w >> 5, lg2 = lf.w & 31, es = lb.z, en = lb.w;
      if (a == e && n1 == 0 && en == 0) continue;
      // t of the wide supernodes (an item: a row of L11^-1), then the single columns
      if (n1 > 0) {
        int t = tid, it = t >> lg1, k0 = 4 * (t & ((1 << lg1) - 1));
        int4 v = c.so_f[lf.x + min(it, n1 - 1)];  // {row in S, first column, terms, row-list position}
        RowTerms<T> rt;
        rt.load(S + v.x, k0, v.z, lg1);
        __syncthreads();
#pragma unroll 1
        for (; t - lane < n1 << lg1;) {
          const T y = lanes_sum(rt.sum(S + v.x, xs + v.y, v.z, k0, lg1), lg1);
          if (k0 == 0 && it < n1) xo[v.y + v.z - 1] = y;
          t += nt;
          if (t - lane >= n1 << lg1) break;
          it = t >> lg1;
          v = c.so_f[lf.x + min(it, n1 - 1)];
          rt.load(S + v.x, k0, v.z, lg1);
        }
      } else {
        __syncthreads();
      }
      if (lg_.y > 0) {
        gather_singles(c, lg_.x, lg_.y, a == e);
      } else {
#pragma unroll 1
        for (int q = tid; q < en; q += nt) fwd_single(c, c.so_e[es + q], 32);
      }
      if (a != e) fwd_listed(c, a, m, e);
      if (n1 > 0) {
        // pushes of the wide ones (an item: a row of L21)
        int t = tid, it = t >> lg2, k0 = 4 * (t & ((1 << lg2) - 1));
        int4 v = make_int4(0, 0, 0, 0);
        RowTerms<T> rt;
        int rr = 0;
        if (n2 > 0) {
          v = c.so_f[lf.z + min(it, n2 - 1)];
          rt.load(S + v.x, k0, v.z, lg2);
          rr = ls[v.w];
        }
        __syncthreads();
#pragma unroll 1
        for (; t - lane < n2 << lg2;) {
          const T y = lanes_sum(rt.sum(S + v.x, xo + v.y, v.z, k0, lg2), lg2);
          if (k0 == 0 && it < n2) push(c, rr, y);
          t += nt;
          if (t - lane >= n2 << lg2) break;
          it = t >> lg2;
          v = c.so_f[lf.z + min(it, n2 - 1)];
          rt.load(S + v.x, k0, v.z, lg2);
          rr = ls[v.w];
        }
      }
    }
    BQ_T1(c, PH_FWD_WIDE);
  }
  BQ_T0(c);
#pragma unroll 1
  for (int l = nlev - 1; l >= 0; --l) {
    const int a = c.vseg[2 * l], m = c.vseg[2 * l + 1], e = c.vseg[2 * l + 2];
    const int4 lb = c.lvl[3 * l + 1];
    const int n = lb.y >> 5, lg = lb.y & 31, es = lb.z, en = lb.w;
    if (a == e && n == 0 && en == 0) continue;
    const int g = tid & ((1 << lg) - 1), total = n << lg;
    // an item: a column {its first entry in L21, c0 << 16 | w, place in the block << 16 | rows below, row-list offset}
    int4 v0 = make_int4(0, 0, 0, 0);
    if (n > 0) {
      int t = tid, it = t >> lg;
      int4 v = c.so_b[lb.x + min(it, n - 1)];
      v0 = v;
      ColTerms<T> ct;
      int rr[4];
      T d, db, dbm;
      auto load = [&]() {
        const int ld = s_ld(v.y & 0xffff), mm = v.z & 0xffff, j = (int)((unsigned)v.z >> 16);
        const int cj = (int)((unsigned)v.y >> 16) + j;
        ct.load(S + v.x, g, ld, mm, lg);
#pragma unroll
        for (int q = 0; q < 4; ++q) rr[q] = ls[v.w + max(min(g + (q << lg), mm - 1), -1)];
        d = c.Di[cj];
        db = c.Di[c.N + cj];
        dbm = c.Di[c.N + cj - (j > 0 ? 1 : 0)];
        if (j == 0) dbm = T(0);
      };
      load();
      __syncthreads();
#pragma unroll 1
      for (; t - lane < total;) {
        const int ld = s_ld(v.y & 0xffff), mm = v.z & 0xffff, j = (int)((unsigned)v.z >> 16);
        const int cj = (int)((unsigned)v.y >> 16) + j;
        T y = T(0);
#pragma unroll 1
        for (int r0 = g; r0 < mm;) {
          T x[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) x[q] = xo[min((unsigned)rr[q], top)];
#pragma unroll
          for (int q = 0; q < 4; ++q) y += ct.p[q] * x[q];
          r0 += 4 << lg;
          if (r0 < mm) {
            ct.load(S + v.x, r0, ld, mm, lg);
#pragma unroll
            for (int q = 0; q < 4; ++q) rr[q] = ls[v.w + min(r0 + (q << lg), mm - 1)];
          }
        }
        y = lanes_sum(y, lg);
        const T u = d * xo[cj] + db * xo[cj + (db != T(0) ? 1 : 0)] + dbm * xo[cj - (dbm != T(0) ? 1 : 0)] - y;
        if (g == 0 && it < n) xs[cj] = u;
        t += nt;
        if (t - lane >= total) break;
        it = t >> lg;
        v = c.so_b[lb.x + min(it, n - 1)];
        load();
      }
    } else {
      __syncthreads();
    }
#pragma unroll 1
    for (int q = tid; q < en; q += nt) {
      const int4 v = c.so_e[es + q];
      Single4<T> b;
      b.load(c, v, 1, 32);
      bwd_single(c, v, b, c.L[v.z], 32);
    }
    if (a != e) bwd_listed(c, a, m, e);
    if (n > 0) {
      // x_j = v_j + sum over i > j of L11^-1(i, j) v_i: the rows j + 1 .. w of the column
      int t = tid, it = t >> lg;
      int4 v = v0;
      ColTerms<T> ct;
      int terms, ld, cj;
      const T *col;
      auto load = [&]() {
        const int w = v.y & 0xffff, j = (int)((unsigned)v.z >> 16);
        cj = (int)((unsigned)v.y >> 16) + j;
        ld = s_ld(w);
        terms = w - 1 - j;
        col = S + v.x - terms * ld;  // L21's first row is row w
        ct.load(col, g, ld, terms, lg);
      };
      load();
      __syncthreads();
#pragma unroll 1
      for (; t - lane < total;) {
        T y = T(0);
#pragma unroll 1
        for (int r0 = g; r0 < terms;) {
          T x[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) x[q] = xs[cj + min(1 + r0 + (q << lg), terms)];
#pragma unroll
          for (int q = 0; q < 4; ++q) y += ct.p[q] * x[q];
          r0 += 4 << lg;
          if (r0 < terms) ct.load(col, r0, ld, terms, lg);
        }
        y = lanes_sum(y, lg);
        if (g == 0 && it < n) xo[cj] = xs[cj] + y;
        t += nt;
        if (t - lane >= total) break;
        it = t >> lg;
        v = c.so_b[lb.x + min(it, n - 1)];
        load();
      }
    }
  }
  __syncthreads();
  BQ_T1(c, PH_BWD);
}

// The visible single columns' records, compacted from the pattern's order (by
// level, then short / long) after every change of the active set, where each
// level's two groups start, and the rows of the active constraints.  Each
// warp counts, then writes, its own stretch of the order.
template <class T> __device__ __noinline__ void build_vlist(Ctx<T> &) {
  Ctx<T> &c = ctx<T>();
  const int lane = lane_id(), wi = warp_id(), nw = num_warps(), ns = c.n1;
  const int per = ((ns + nw - 1) / nw + 31) / 32 * 32;
  const int t0 = min(wi * per, ns), t1 = min(t0 + per, ns);
  int cnt = 0;  // visible ones, and constraint columns among them (high half)
#pragma unroll 1
  for (int t = t0 + lane; t < t1; t += 32) {
    const int s = c.so_sn[t];
    if (c.vis[s]) cnt += c.sn_con[s] >= 0 ? 0x10001 : 1;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (lane == 0) c.redi[wi] = cnt;
  __syncthreads();
  int before = 0, total = 0;
#pragma unroll 1
  for (int k = 0; k < nw; ++k) {
    if (k < wi) before += c.redi[k];
    total += c.redi[k];
  }
  int pos = before & 0xffff, pcon = before >> 16;
  const unsigned below = (1u << lane) - 1u;
#pragma unroll 1
  for (int tb = t0; tb < t1; tb += 32) {
    const int t = tb + lane;
    const int s = t < t1 ? c.so_sn[t] : 0;
    const bool v = t < t1 && c.vis[s] != 0;
    const int k = v ? c.sn_con[s] : -1;
    const unsigned bal = __ballot_sync(0xffffffffu, v), bcon = __ballot_sync(0xffffffffu, k >= 0);
    const int p = pos + __popc(bal & below);
    if (t < t1) c.map[t] = p;  // records before position t (the row map is free here)
    if (v) c.vrec[p] = c.so_rec[t];
    if (k >= 0) c.arow[pcon + __popc(bcon & below)] = c.base + k;
    pos += __popc(bal);
    pcon += __popc(bcon);
  }
  __syncthreads();
#pragma unroll 1
  for (int k = threadIdx.x; k <= 2 * c.nlev; k += blockDim.x) {
    const int t = c.so_seg[k];
    c.vseg[k] = t < ns ? c.map[t] : total & 0xffff;
  }
  if (threadIdx.x == 0) c.vseg[2 * c.nlev + 1] = total >> 16;
  __syncthreads();
}

// Rows of K that take part: the structural ones, then the active
// constraints (c.arow, kept by build_vlist).  Everything below runs over
// them alone: the hidden rows of a small batch QP outnumber them (900 of
// 1650 at horizon 50), and FP64 operations are what the vectors cost.
template <class T> __device__ __forceinline__ int vis_rows(const Ctx<T> &c) { return c.base + c.vseg[2 * c.nlev + 1]; }
template <class T> __device__ __forceinline__ int vis_row(const Ctx<T> &c, int t) {
  return t < c.base ? t : c.arow[t - c.base];
}
// f(i) for every hidden row i
template <class T, class F> __device__ __forceinline__ void hidden_rows(const Ctx<T> &c, F &&f) {
#pragma unroll 1
  for (int k = threadIdx.x; k < c.mineq; k += blockDim.x)
    if (!c.act[k]) f(c.base + k);
}

// out(i, M^-1 v) over the visible rows (original numbering), v(i) the right
// hand side; the solve runs in shared memory.  Both permutations go through
// iperm, so that the global side is read and written in order.  Ends with a
// barrier.  Cycles per application of horizon-50 MPC with 4 CTAs on the SM,
// against one thread or warp per supernode walking its entries: FP32 458k ->
// 126k, FP64 969k -> 248k; 2048 cold QPs (FP32) 121 -> 46 ms, 1024 (FP64)
// 92 -> 32 ms.
template <class T, class VI, class VO> __device__ void precond(Ctx<T> &c, VI &&v, VO &&out) {
  BQ_T0(c);
  const long long tg0 = c.prof ? clock64() : 0;
  const int M = vis_rows(c);
#pragma unroll 4
  for (int t = threadIdx.x; t < M; t += blockDim.x) {
    const int i = vis_row(c, t);
    c.xs[c.iperm[i]] = T(v(i));
  }
  hidden_rows(c, [&](int i) { c.xo[c.iperm[i]] = T(0); });  // read by the products with hidden rows' zeros
  if (c.prof && threadIdx.x == 0) c.cyc[PH_GATHER] += (unsigned long long)(clock64() - tg0);
  ldlt_solve_smem(c);
  const long long tg1 = c.prof ? clock64() : 0;
#pragma unroll 4
  for (int t = threadIdx.x; t < M; t += blockDim.x) {
    const int i = vis_row(c, t);
    out(i, c.xo[c.iperm[i]]);
  }
  __syncthreads();
  if (c.prof && threadIdx.x == 0) c.cyc[PH_GATHER] += (unsigned long long)(clock64() - tg1);
  BQ_T1(c, PH_PRECOND);
}

// Row i of K x with the refinement values (original numbering).  Entries of
// hidden constraints are zeros and skipped by their bits: the columns there
// hold no value of this problem.
template <class T> __device__ __forceinline__ double spmv_row(const Ctx<T> &c, const double *x, int i) {
  double acc = 0.0;
  const int q1 = c.Rp[i + 1];
#pragma unroll 1
  for (int q0 = c.Rp[i]; q0 < q1; q0 += 4) {
    double v[4], u[4];
    int j[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int q = min(q0 + e, q1 - 1);
      v[e] = c.Rv[q];
      j[e] = c.Rj[q];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) u[e] = x[j[e]];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (q0 + e < q1 && __double_as_longlong(v[e]) << 1) acc += v[e] * u[e];
  }
  return acc;
}

// Block-wide sums of K values in a fixed order (the same inputs give the
// same bits on every run).  `par` alternates between two halves of red, so
// one barrier per call is enough; every thread adds the warps' sums itself.
template <int K> __device__ __forceinline__ void block_sums(double (&v)[K], double *red, int &par) {
  static_assert(K <= 2, "two halves of 16 doubles, up to 8 warps");
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < K; ++q) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
  double *h = red + 16 * par;
  par ^= 1;
  if (lane_id() == 0)
#pragma unroll
    for (int q = 0; q < K; ++q) h[q * 8 + warp_id()] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < K; ++q) {
    v[q] = h[q * 8];
#pragma unroll 1
    for (int t = 1; t < num_warps(); ++t) v[q] += h[q * 8 + t];
  }
}

// ---- refinement (reference pmgmres_ldlt_auto, src/gmres/mgmres.cpp:1015-1211)

// Solves K x = b (x holds the preconditioned solution on entry).  flexible:
// right-preconditioned FGMRES with stored directions Z (Saad 1993) -- the
// residual it minimises is the FP64 b - Kx itself; else the reference's
// left-preconditioned GMRES.  adaptive: stop once the residual estimate is
// below rtol * ||b||; else the reference's rule (rho <= tol_rel * rho0 and
// rho <= tol_abs).  Returns the Krylov steps taken.
//
// The vectors are a few hundred FP64 entries in L2: what they cost is FP64
// operations and block-wide sums.  So a pass forms all it can of the next
// step (residual and its norm, K z with its norm and first projection, each
// projection with the next one), vectors are scaled by a reciprocal (an FP64
// division takes nine multiply-adds) and only if a further step reads them.
// A row belongs to the same thread in every pass, so barriers stand only
// where a product with K or a solve crosses rows.
template <class T>
__device__ int refine(Ctx<T> &c, const double *b, double *x, int itr_max, int mr, bool flexible, bool adaptive,
                      double rtol, double tol_abs, double tol_rel) {
  if (itr_max <= 0 || mr <= 0) return 0;
  mr = min(mr, MR_CAP);
  GmresSmall &gs = c.gs;
  const int N = c.N, M = vis_rows(c), tid = threadIdx.x, nt = blockDim.x;
  const double delta = 1.0e-03;
  double *r = c.r, *V = c.V;
  double rho = 0.0, rho_tol = 0.0, stop_abs = tol_abs;
  int used = 0, par = 0;
  __syncthreads();  // red is free
  if (adaptive) {
    double s[1] = {0.0};
#pragma unroll 1
    for (int t = tid; t < M; t += nt) {
      const double v = b[vis_row(c, t)];
      s[0] += v * v;
    }
    block_sums<1>(s, c.red, par);
    stop_abs = rtol * sqrt(s[0]);
  }
#pragma unroll 1
  for (int itr = 0; itr < itr_max; ++itr) {
    double s1[1] = {0.0};
    {
      BQ_T0(c);
#pragma unroll 1
      for (int t = tid; t < M; t += nt) {
        const int i = vis_row(c, t);
        const double v = b[i] - spmv_row(c, x, i);
        r[i] = v;
        if (flexible) s1[0] += v * v;
      }
      BQ_T1(c, PH_SPMV);
    }
    if (!flexible) {
      __syncthreads();
      precond(c, [&](int i) { return r[i]; }, [&](int i, T v) {
        const double u = (double)v;
        r[i] = u;
        s1[0] += u * u;
      });
    }
    block_sums<1>(s1, c.red, par);
    rho = sqrt(s1[0]);
    if (adaptive ? rho <= stop_abs : rho < tol_abs) return used;
    if (itr == 0) rho_tol = rho * tol_rel;
    double scale = 1.0 / rho;  // of the newest basis vector, applied when a step reads it
#pragma unroll 1
    for (int t = tid; t < M; t += nt) {
      const int i = vis_row(c, t);
      V[i] = r[i] * scale;
    }
    if (tid == 0) {
      gs.g[0] = rho;
#pragma unroll 1
      for (int i = 1; i <= mr; ++i) gs.g[i] = 0.0;
    }
    int k_copy = 0;
    bool stop = false;
#pragma unroll 1
    for (int k = 0; k < mr; ++k) {
      k_copy = k;
      double *vk = V + (size_t)k * N, *vk1 = V + (size_t)(k + 1) * N;
      double s[2] = {0.0, 0.0};  // |K z|^2 and its product with V_0
      if (flexible) {
        T *zk = c.Z + (size_t)k * N;
        double *w = c.w;
        precond(c, [&](int i) { return vk[i]; }, [&](int i, T v) {
          zk[i] = v;
          w[i] = (double)v;  // widened for K z in FP64
        });
        BQ_T0(c);
#pragma unroll 1
        for (int t = tid; t < M; t += nt) {
          const int i = vis_row(c, t);
          const double v = spmv_row(c, w, i);
          vk1[i] = v;
          s[0] += v * v;
          s[1] += v * V[i];
        }
        BQ_T1(c, PH_SPMV);
      } else {
        __syncthreads();
        {
          BQ_T0(c);
#pragma unroll 1
          for (int t = tid; t < M; t += nt) {
            const int i = vis_row(c, t);
            vk1[i] = spmv_row(c, vk, i);
          }
          BQ_T1(c, PH_SPMV);
        }
        precond(c, [&](int i) { return vk1[i]; }, [&](int i, T v) {
          const double u = (double)v;
          vk1[i] = u;
          s[0] += u * u;
          s[1] += u * V[i];
        });
      }
      block_sums<2>(s, c.red, par);
      const double av = sqrt(s[0]);
      double hj = s[1], hk1 = 0.0;
#pragma unroll 1
      for (int j = 0; j <= k; ++j) {  // modified Gram-Schmidt, each pass forming the next product
        const double *vj = V + (size_t)j * N, *vn = V + (size_t)(j + 1) * N;
        if (tid == 0) gs.h[j][k] = hj;
        double p[1] = {0.0};
#pragma unroll 1
        for (int t = tid; t < M; t += nt) {
          const int i = vis_row(c, t);
          const double v = vk1[i] - hj * vj[i];
          vk1[i] = v;
          p[0] += j < k ? v * vn[i] : v * v;
        }
        block_sums<1>(p, c.red, par);
        hj = p[0];
      }
      hk1 = sqrt(hj);
      if ((av + delta * hk1) == av) {  // reorthogonalisation
#pragma unroll 1
        for (int j = 0; j <= k; ++j) {
          const double *vj = V + (size_t)j * N;
          double p[1] = {0.0};
#pragma unroll 1
          for (int t = tid; t < M; t += nt) {
            const int i = vis_row(c, t);
            p[0] += vk1[i] * vj[i];
          }
          block_sums<1>(p, c.red, par);
#pragma unroll 1
          for (int t = tid; t < M; t += nt) {
            const int i = vis_row(c, t);
            vk1[i] -= p[0] * vj[i];
          }
          if (tid == 0) gs.h[j][k] += p[0];
        }
        double p[1] = {0.0};
#pragma unroll 1
        for (int t = tid; t < M; t += nt) {
          const double v = vk1[vis_row(c, t)];
          p[0] += v * v;
        }
        block_sums<1>(p, c.red, par);
        hk1 = sqrt(p[0]);
      }
      if (tid == 0) {
        double hk = hk1;
#pragma unroll 1
        for (int j = 0; j < k; ++j) {  // previous Givens rotations
          const double g1 = gs.cs[j] * gs.h[j][k] - gs.sn[j] * gs.h[j + 1][k];
          const double g2 = gs.sn[j] * gs.h[j][k] + gs.cs[j] * gs.h[j + 1][k];
          gs.h[j][k] = g1;
          gs.h[j + 1][k] = g2;
        }
        const double h0 = gs.h[k][k], mu = sqrt(h0 * h0 + hk * hk);
        gs.scal[0] = mu;
        if (mu != 0.0) {
          const double im = 1.0 / mu, cs = h0 * im, sn = -hk * im;
          gs.cs[k] = cs;
          gs.sn[k] = sn;
          gs.h[k][k] = cs * h0 - sn * hk;
          const double g0 = gs.g[k], gk1 = gs.g[k + 1];
          gs.g[k] = cs * g0 - sn * gk1;
          gs.g[k + 1] = sn * g0 + cs * gk1;
        }
      }
      __syncthreads();
      if (gs.scal[0] == 0.0) return used;
      rho = fabs(gs.g[k + 1]);
      used++;
      stop = adaptive ? rho <= stop_abs : (rho <= rho_tol && rho <= tol_abs);
      if (stop) break;
      if (k + 1 < mr && hk1 != 0.0) {
        scale = 1.0 / hk1;
#pragma unroll 1
        for (int t = tid; t < M; t += nt) vk1[vis_row(c, t)] *= scale;
      }
    }
    const int k = k_copy;
    if (gs.h[k][k] == 0.0) return used;
    if (tid == 0) {
      gs.y[k] = gs.g[k] / gs.h[k][k];
#pragma unroll 1
      for (int i = k - 1; 0 <= i; i--) {
        double yi = gs.g[i];
#pragma unroll 1
        for (int j = i + 1; j < k + 1; j++) yi = yi - gs.h[i][j] * gs.y[j];
        gs.y[i] = yi / gs.h[i][i];
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int t = tid; t < M; t += nt) {
      const int i = vis_row(c, t);
      double acc = 0.0;
      if (flexible)
#pragma unroll 1
        for (int j = 0; j <= k; ++j) acc += (double)c.Z[(size_t)j * N + i] * gs.y[j];
      else
#pragma unroll 1
        for (int j = 0; j <= k; ++j) acc += V[(size_t)j * N + i] * gs.y[j];
      x[i] += acc;
    }
    __syncthreads();
    if (stop) break;
  }
  return used;
}

// x = M^-1 b, then refine; hidden rows of x are zero.  Returns the Krylov steps.
template <class T>
__device__ __noinline__ int solve_refined(Ctx<T> &, const double *b, double *x, int itr_max, int mr, bool flexible, bool adaptive,
                             double rtol, double tol_abs, double tol_rel) {
  Ctx<T> &c = ctx<T>();
  hidden_rows(c, [&](int i) { x[i] = 0.0; });
  precond(c, [&](int i) { return b[i]; }, [&](int i, T v) { x[i] = (double)v; });
  return refine(c, b, x, itr_max, mr, flexible, adaptive, rtol, tol_abs, tol_rel);
}

// ---- NASOQ on one problem ------------------------------------------------------
// Marks the supernodes on the elimination-tree path from supernode s to the
// root for the next refactorization (the reference marks the visible ones of
// its edited tree, which are a subset; refactoring an unchanged supernode
// reproduces it).  A marked supernode's path is marked, or being marked by
// another thread, already.
template <class T> __device__ void mark_path(Ctx<T> &c, int s) {
  while (s >= 0 && !c.mark[s]) {
    c.mark[s] = 1;
    s = c.sparent[s];
  }
}

// KKT edit of constraint k (reference edit_kkt -> add_del_matrix_qp,
// linear_solver_wrapper.cpp:1020-1137): the constraint's entries become
// visible / hidden in both value copies and in the descendant masks of its
// targets, and the paths of its column and of its variables are marked for
// the next partial refactorization.  One thread per constraint; several may
// edit different constraints at once.
template <class T> __device__ __noinline__ void edit_constraint(Ctx<T> &, int k, bool add) {
  Ctx<T> &c = ctx<T>();
  c.act[k] = add ? 1 : 0;
  c.vis[c.con_sn[k]] = add ? 1 : 0;
  c.nmark = 1;  // edits wait for a refactorization
#pragma unroll 1
  for (int e = c.bt_ptr[k]; e < c.bt_ptr[k + 1]; ++e) {
    const int qq = c.bt_rpos[e];
    const double v = add ? c.kv[c.bt_q[e]] : 0.0;
    c.Fv[qq] = T(v);
    c.Rv[qq] = v;
  }
  const int row = c.base + k;
#pragma unroll 1
  for (int qq = c.Rp[row]; qq < c.Rp[row + 1]; ++qq)
    if (c.Rj[qq] != row) {
      const double v = add ? c.kv[c.Rq[qq]] : 0.0;
      c.Fv[qq] = T(v);
      c.Rv[qq] = v;
    }
#pragma unroll 1
  for (int e = c.con_ptr[k]; e < c.con_ptr[k + 1]; ++e) {
    const int tg = c.con_tgt[2 * e], bit = c.con_tgt[2 * e + 1];
    if (bit < 64) {
      if (add) atomicOr(c.cmask + tg, 1ull << bit);
      else atomicAnd(c.cmask + tg, ~(1ull << bit));
    }
  }
  mark_path(c, c.con_sn[k]);
#pragma unroll 1
  for (int e = c.bt_ptr[k]; e < c.bt_ptr[k + 1]; ++e) mark_path(c, c.col2sup[c.iperm[c.bt_var[e]]]);
}

// Every visible supernode is to be factored.
template <class T> __device__ void mark_visible(Ctx<T> &c) {
#pragma unroll 1
  for (int s = threadIdx.x; s < c.ns; s += blockDim.x) c.mark[s] = c.vis[s];
  __syncthreads();
}

// mlist = the marked supernodes in ascending order (children before parents).
// Each warp counts, then writes, its own stretch.
template <class T> __device__ __noinline__ void collect_marked(Ctx<T> &) {
  Ctx<T> &c = ctx<T>();
  const int lane = lane_id(), wi = warp_id(), nw = num_warps(), ns = c.ns;
  const int per = ((ns + nw - 1) / nw + 31) / 32 * 32;
  const int t0 = min(wi * per, ns), t1 = min(t0 + per, ns);
  int cnt = 0;
#pragma unroll 1
  for (int t = t0 + lane; t < t1; t += 32) cnt += c.mark[t] ? 1 : 0;
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) c.redi[wi] = cnt;
  __syncthreads();
  int pos = 0, total = 0;
#pragma unroll 1
  for (int k = 0; k < nw; ++k) {
    if (k < wi) pos += c.redi[k];
    total += c.redi[k];
  }
#pragma unroll 1
  for (int tb = t0; tb < t1; tb += 32) {
    const int t = tb + lane;
    const bool v = t < t1 && c.mark[t] != 0;
    const unsigned bal = __ballot_sync(0xffffffffu, v);
    if (v) c.mlist[pos + __popc(bal & ((1u << lane) - 1u))] = t;
    pos += __popc(bal);
  }
  if (threadIdx.x == 0) c.nmark = total;
  __syncthreads();
}

// The marked supernodes factored again, and the solves' lists brought up to date.
template <class T> __device__ __noinline__ void refactor(Ctx<T> &) {
  Ctx<T> &c = ctx<T>();
  collect_marked(c);
  factor_marked(c);
  build_vlist(c);
}

// Slot state of a problem whose group shares one factorization: the factor,
// its pivoting state and both value copies of K with every inequality
// hidden, copied from the group's base slot; visibility likewise.
template <class T> __device__ __noinline__ void copy_base(Ctx<T> &, const unsigned char *bs, const BSlot &L, const BPat &pt) {
  Ctx<T> &c = ctx<T>();
  const int tid = threadIdx.x, nt = blockDim.x, N = c.N;
  const T *bL = reinterpret_cast<const T *>(bs + L.o_L);
  const T *bD = reinterpret_cast<const T *>(bs + L.o_D);
  const T *bS = reinterpret_cast<const T *>(bs + L.o_S);
  const T *bG = reinterpret_cast<const T *>(bs + L.o_G);
  const int *bls = reinterpret_cast<const int *>(bs + L.o_ls);
  const int *bperm = reinterpret_cast<const int *>(bs + L.o_perm);
  const int *biperm = reinterpret_cast<const int *>(bs + L.o_iperm);
  const int *blperm = reinterpret_cast<const int *>(bs + L.o_lperm);
  const T *bF = reinterpret_cast<const T *>(bs + L.o_Fv);
  const double *bR = reinterpret_cast<const double *>(bs + L.o_Rv);
  const unsigned long long *bmask = reinterpret_cast<const unsigned long long *>(bs + L.o_cmask);
#pragma unroll 4
  for (int i = tid; i < pt.lsize; i += nt) c.L[i] = bL[i];
#pragma unroll 4
  for (int i = tid; i < pt.sbsize; i += nt) c.S[i] = bS[i];
#pragma unroll 4
  for (int i = tid; i < pt.gsize; i += nt) c.G[i] = bG[i];
#pragma unroll 4
  for (int i = tid; i < pt.rsize; i += nt) c.ls[i] = bls[i];
#pragma unroll 4
  for (int i = tid; i < N; i += nt) {
#pragma unroll 1
    for (int k = 0; k < 3; ++k) c.D[k * N + i] = bD[k * N + i];
    c.perm[i] = bperm[i];
    c.iperm[i] = biperm[i];
    c.lperm[i] = blperm[i];
  }
#pragma unroll 4
  for (int i = tid; i < c.nnzR; i += nt) {
    c.Fv[i] = bF[i];
    c.Rv[i] = bR[i];
  }
#pragma unroll 4
  for (int s = tid; s < c.ns; s += nt) {
    c.piv[s] = bs[L.o_piv + s];
    c.cmask[s] = bmask[s];
    c.mark[s] = 0;
    c.vis[s] = c.sn_con[s] < 0 ? 1 : 0;
  }
  if (tid == 0) c.nmark = 0;
  __syncthreads();
}

// Visibility, descendant masks and both value copies of K from the active set.
template <class T> __device__ __noinline__ void load_state(Ctx<T> &) {
  Ctx<T> &c = ctx<T>();
#pragma unroll 1
  for (int s = threadIdx.x; s < c.ns; s += blockDim.x) {
    const int k = c.sn_con[s];
    c.vis[s] = (k < 0 || c.act[k]) ? 1 : 0;
    c.cmask[s] = 0ull;
  }
  __syncthreads();
#pragma unroll 1
  for (int k = threadIdx.x; k < c.mineq; k += blockDim.x)
    if (c.act[k])
#pragma unroll 1
      for (int e = c.con_ptr[k]; e < c.con_ptr[k + 1]; ++e) {
        const int bit = c.con_tgt[2 * e + 1];
        if (bit < 64) atomicOr(c.cmask + c.con_tgt[2 * e], 1ull << bit);
      }
#pragma unroll 1
  for (int qq = threadIdx.x; qq < c.nnzR; qq += blockDim.x) {
    const int vq = c.Rq[qq];
    c.Fv[qq] = T(fact_val(c, vq));
    c.Rv[qq] = ref_val(c, vq);
  }
  __syncthreads();
}

}  // namespace

template <class T, bool LARGE_PATTERNS>
__global__ void __launch_bounds__(BT_MAX_THREADS, 2) k_nasoq_batch(BArgs a) {
  static_assert(LARGE_PATTERNS == LARGE, "one of the two per translation unit");
  __shared__ int s_prob;
  __shared__ int s_int[8];
  __shared__ double s_dbl[8];
  Ctx<T> &c = ctx<T>();
  double *red = c.red;
  int *redi = c.redi;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid < PH_N) c.cyc[tid] = 0;
  // shared-memory carve-up (sizes from the largest pattern of the batch)
  unsigned sp = BATCH_CTX_BYTES;
  auto take = [&](size_t bytes) {
    const unsigned o = sp;
    sp += (unsigned)((bytes + 15) / 16 * 16);
    return o;
  };
  // the row map of a factorization, and xo of the solves
  const unsigned o_map = take((size_t)a.N_max * (LARGE ? sizeof(int) : sizeof(T)));
  const unsigned o_xs = take((size_t)a.N_max * sizeof(T));
  const unsigned o_rowbuf = take(batch_rowbuf(a) * sizeof(T));
  const unsigned o_D = take((size_t)a.w_max * sizeof(T)), o_E = take((size_t)a.w_max * sizeof(T));
  const unsigned o_lp = take((size_t)a.w_max * sizeof(int));
  const unsigned o_lvl = take(LARGE ? 0 : (size_t)3 * a.nlev_max * sizeof(int4));
  const unsigned o_vseg = take((size_t)(2 * a.nlev_max + 2) * sizeof(int));
  const unsigned o_vis = take((size_t)a.ns_max), o_mark = take(LARGE ? 0 : (size_t)a.ns_max), o_act = take((size_t)a.mi_max);
  // blocks of the factorization: the CTA's, or one set per warp in the same memory
  const int wcap = a.warp_factor ? min(a.w_max, 32) : 0, rcap = a.warp_factor ? min(a.nr_max, 32) : 0;
  const int wstride = wcap * (rcap + wcap + 4);
  const unsigned o_B = take(batch_block_bytes(a, sizeof(T)));
  unsigned char *stage = Sh<unsigned char>{sp};  // the factor and row lists of a problem that fits

  unsigned char *const own_slot = a.slots + (size_t)blockIdx.x * a.slot.bytes;
  const bool build_bases = a.mode == 1;
#pragma unroll 1
  for (;;) {
    if (tid == 0) {
      const int qi = atomicAdd(a.head, 1);
      if (build_bases) s_prob = qi < a.nbase ? qi : -1;  // a group
      else s_prob = qi < a.nprob ? a.order[qi] : -1;
      c.status = 0;
      c.nmark = 0;
    }
    __syncthreads();
    if (s_prob < 0) break;
    // mode 1: the group's shared factorization is built in its base slot,
    // for the group's representative problem
    const int grp = build_bases ? s_prob : -1;
    const int pi = build_bases ? a.base_rep[grp] : s_prob;
    unsigned char *const slot = build_bases ? a.bases + (size_t)grp * a.slot.bytes : own_slot;
    const BProb &P = a.probs[pi];
    const BPat &pt = a.pats[P.pat];
    if (tid == 0) {
      const int *ip = a.ipool;
      c.n = pt.n;
      c.meq = pt.meq;
      c.mineq = pt.mineq;
      c.N = pt.N;
      c.base = pt.base;
      c.ns = pt.ns;
      c.nlev = pt.nlev;
      c.nnzR = pt.nnzR;
      c.cmask_ok = pt.cmask_ok;
      c.super = ip + pt.o_super;
      c.sparent = ip + pt.o_sparent;
      c.col2sup = ip + pt.o_col2sup;
      c.lpi = ip + pt.o_lpi;
      c.lpx = ip + pt.o_lpx;
      c.lev = ip + pt.o_lev;
      c.Rp = ip + pt.o_Rp;
      c.Rj = ip + pt.o_Rj;
      c.Rq = ip + pt.o_Rq;
      c.ent = ip + pt.o_ent;
      c.bt_ptr = ip + pt.o_bt_ptr;
      c.bt_var = ip + pt.o_bt_var;
      c.bt_q = ip + pt.o_bt_q;
      c.bt_rpos = ip + pt.o_bt_rpos;
      c.sn_con = ip + pt.o_sn_con;
      c.con_sn = ip + pt.o_con_sn;
      c.eq_ptr = ip + pt.o_eq_ptr;
      c.eq_var = ip + pt.o_eq_var;
      c.eq_q = ip + pt.o_eq_q;
      c.snrec = reinterpret_cast<const int4 *>(ip + pt.o_snrec);
      c.prec = reinterpret_cast<const int4 *>(ip + pt.o_prec);
      c.con_ptr = ip + pt.o_con_ptr;
      c.con_tgt = ip + pt.o_con_tgt;
      c.so_sn = ip + pt.o_so_sn;
      c.so_seg = ip + pt.o_so_seg;
      c.so_rec = reinterpret_cast<const int4 *>(ip + pt.o_so_rec);
      c.so_e = reinterpret_cast<const int4 *>(ip + pt.o_so_e);
      c.so_f = reinterpret_cast<const int4 *>(ip + pt.o_so_f);
      c.so_b = reinterpret_cast<const int4 *>(ip + pt.o_so_b);
      c.so_g = reinterpret_cast<const int2 *>(ip + pt.o_so_g);
      c.so_gj = ip + pt.o_so_gj;
      c.so_gs = ip + pt.o_so_gs;
      c.gidx = ip + pt.o_gidx;
      c.G = reinterpret_cast<T *>(slot + a.slot.o_G);
      c.n1 = pt.n1;
      c.kv = a.dpool + P.o_kv;
      c.q = a.dpool + P.o_q;
      c.bq = a.dpool + P.o_b;
      c.dq = a.dpool + P.o_d;
      c.pert = reinterpret_cast<const uint8_t *>(a.dpool) + P.o_pert;
      c.reg = P.reg;
      c.reg32 = P.reg32;
      // the factor and the row lists live in shared memory when they fit
      const size_t lbytes = ((size_t)pt.lsize * sizeof(T) + 15) / 16 * 16, sbytes = (size_t)pt.sbsize * sizeof(T);
      if (!build_bases && lbytes + sbytes + (size_t)pt.rsize * sizeof(int) <= (size_t)a.stage_bytes) {
        c.S = reinterpret_cast<T *>(stage);
        c.L = reinterpret_cast<T *>(stage + sbytes);
        c.ls = reinterpret_cast<int *>(stage + sbytes + lbytes);
      } else {
        c.L = reinterpret_cast<T *>(slot + a.slot.o_L);
        c.S = reinterpret_cast<T *>(slot + a.slot.o_S);
        c.ls = reinterpret_cast<int *>(slot + a.slot.o_ls);
      }
      c.D = reinterpret_cast<T *>(slot + a.slot.o_D);
      c.Di = c.D + c.N;
      c.perm = reinterpret_cast<int *>(slot + a.slot.o_perm);
      c.iperm = reinterpret_cast<int *>(slot + a.slot.o_iperm);
      c.lperm = reinterpret_cast<int *>(slot + a.slot.o_lperm);
#ifdef NQG_BATCH_LARGE_UNIT
      c.mark = slot + a.slot.o_mark;
      c.lvl = reinterpret_cast<int4 *>(slot + a.slot.o_lvl);
      c.xo = reinterpret_cast<T *>(slot + a.slot.o_xo);
#else
      c.mark.off = o_mark;
      c.lvl.off = o_lvl;
      c.xo.off = o_map;
#endif
      c.piv = slot + a.slot.o_piv;
      c.alist = reinterpret_cast<int *>(slot + a.slot.o_alist);
      c.vrec = reinterpret_cast<int4 *>(slot + a.slot.o_vrec);
      c.arow = reinterpret_cast<int *>(slot + a.slot.o_arow);
      c.mlist = reinterpret_cast<int *>(slot + a.slot.o_mlist);
      c.Fv = reinterpret_cast<T *>(slot + a.slot.o_Fv);
      c.Rv = reinterpret_cast<double *>(slot + a.slot.o_Rv);
      c.cmask = reinterpret_cast<unsigned long long *>(slot + a.slot.o_cmask);
      c.rhs = reinterpret_cast<double *>(slot + a.slot.o_rhs);
      c.sol = reinterpret_cast<double *>(slot + a.slot.o_sol);
      c.r = reinterpret_cast<double *>(slot + a.slot.o_r);
      c.w = reinterpret_cast<double *>(slot + a.slot.o_w);
      c.V = reinterpret_cast<double *>(slot + a.slot.o_V);
      c.Z = reinterpret_cast<T *>(slot + a.slot.o_Z);
      c.tmp = reinterpret_cast<double *>(slot + a.slot.o_tmp);
      c.map.off = o_map;
      c.xs.off = o_xs;
      c.B.off = o_B;
      c.rowbuf.off = o_rowbuf;
      c.Dsm.off = o_D;
      c.Esm.off = o_E;
      c.Binv.off = o_B + (unsigned)(a.b_max * (int)sizeof(T));
      c.lp.off = o_lp;
      c.wB.off = o_B;
      c.wstride = wstride;
      c.wlp.off = o_B + (unsigned)(WF_WARPS * wstride * (int)sizeof(T));
      c.wcap = wcap;
      c.rcap = rcap;
      c.wf = a.warp_factor ? 1 : 0;
      c.vis.off = o_vis;
      c.act.off = o_act;
      c.vseg.off = o_vseg;
      c.prof = a.prof ? 1 : 0;
    }
    __syncthreads();
    const long long tp0 = clock64();
    const int *ip = a.ipool;
    double *xv = a.dout + P.o_x, *yv = a.dout + P.o_y, *zv = a.dout + P.o_z;
    int *as_out = a.iout + P.o_as;
    const int n = c.n, meq = c.meq, mineq = c.mineq, N = c.N;
    const bool flexible = sizeof(T) == 4 || a.refine == 1;
    const bool adaptive = a.refine == 1;
    int steps = 0, solves = 0, warm_dropped = 0;

    // ---- set-up: pattern state into the slot (a problem of a group starts
    // from the group's factorization instead, below)
    if (build_bases || P.base < 0) {
#pragma unroll 1
      for (int i = tid; i < N; i += nt) {
        const int p0 = ip[pt.o_perm0 + i];
        c.perm[i] = p0;
        c.iperm[p0] = i;
#pragma unroll 1
        for (int k = 0; k < 3; ++k) c.D[k * N + i] = T(0);
      }
#pragma unroll 1
      for (int i = tid; i < pt.rsize; i += nt) c.ls[i] = ip[pt.o_ls0 + i];
#pragma unroll 1
      for (int i = tid; i < pt.lsize; i += nt) c.L[i] = T(0);
#pragma unroll 1
      for (int i = tid; i < pt.sbsize; i += nt) c.S[i] = T(0);
#pragma unroll 1
      for (int i = tid; i < pt.gsize; i += nt) c.G[i] = T(0);
#pragma unroll 1
      for (int s = tid; s < c.ns; s += nt) {
        c.mark[s] = 0;
        c.piv[s] = 0;
      }
    }
#pragma unroll 1
    for (int k = tid; k < mineq; k += nt) c.act[k] = 0;
#pragma unroll 1
    for (int l = tid; l < 3 * c.nlev; l += nt) c.lvl[l] = reinterpret_cast<const int4 *>(ip + pt.o_lvl)[l];
    __syncthreads();
    if (build_bases) {  // every inequality hidden: the cold start's factorization
      load_state(c);
      mark_visible(c);
      refactor(c);
      continue;
    }
    const unsigned char *const bslot = P.base >= 0 ? a.bases + (size_t)P.base * a.slot.bytes : nullptr;
    int nact = 0;
    // warm start: proposed active set (constraints listed in as_out), then
    // the equality-constrained solution on it (below)
    const bool warm = P.ws_n >= 0;
    if (warm) {
#pragma unroll 1
      for (int t = tid; t < P.ws_n; t += nt) {
        const int k = as_out[t];
        if (k >= 0 && k < mineq) c.act[k] = 1;
      }
      __syncthreads();
    }
    // ---- initial factorization and solution (reference initialize_x,
    // src/nasoq.cpp:448-476): every visible supernode; rhs [-q; b; d on the
    // active rows]
    // Only visible supernodes are factored: a hidden one contributes zeros
    // and is skipped by the solves.  After the first warm round, dropped
    // constraints are hidden by the partial refactorization of their paths.
    bool cold = !warm, full = true;
#pragma unroll 1
    for (int round = 0; round < 5; ++round) {
      const long long tf0 = c.prof ? clock64() : 0;
      if (full && bslot) {
        // the group's cold factorization, then the active rows made visible
        // by partial refactorization of their paths
        copy_base(c, bslot, a.slot, pt);
#pragma unroll 1
        for (int k = tid; k < mineq; k += nt)
          if (c.act[k]) edit_constraint(c, k, true);
        __syncthreads();
        refactor(c);
      } else if (full) {
        load_state(c);
        mark_visible(c);
        refactor(c);
      } else {
        refactor(c);
      }
      if (c.prof && tid == 0) c.cyc[PH_INIT_FACTOR] += (unsigned long long)(clock64() - tf0);
#pragma unroll 1
      for (int i = tid; i < N; i += nt) {
        double v = 0.0;
        if (i < n) v = -c.q[i];
        else if (i < c.base) v = c.bq[i - n];
        else if (c.act[i - c.base]) v = c.dq[i - c.base];
        c.rhs[i] = v;
      }
      __syncthreads();
      solves++;
      steps += solve_refined(c, c.rhs, c.sol, P.outer, P.inner, flexible, adaptive, a.refine_tol, P.tol_abs, P.tol_rel);
      if (cold) break;
      // a proposed set that makes the KKT matrix singular (dependent
      // constraints): start cold instead
      int bad = 0;
#pragma unroll 1
      for (int i = tid; i < N; i += nt)
        if (!isfinite(c.sol[i])) bad++;
      bad = block_sum_int(bad, redi);
      if (bad > 0 || (c.status & (ST_ZERO_PIVOT | ST_NONFINITE))) {
#pragma unroll 1
        for (int k = tid; k < mineq; k += nt) c.act[k] = 0;
        __syncthreads();
        if (tid == 0) c.status = 0;
        cold = true;
        full = true;
        __syncthreads();
        continue;
      }
      // drop proposed constraints with negative multipliers, then solve again
      int ndrop = 0;
#pragma unroll 1
      for (int k = tid; k < mineq; k += nt)
        if (c.act[k] && c.sol[c.base + k] < 0.0) {
          edit_constraint(c, k, false);
          ndrop++;
        }
      ndrop = block_sum_int(ndrop, redi);
      warm_dropped += ndrop;
      if (ndrop == 0) break;
      full = false;
      if (round >= 2) {  // no consistent set after three rounds: cold start
#pragma unroll 1
        for (int k = tid; k < mineq; k += nt) c.act[k] = 0;
#pragma unroll 1
        for (int s = tid; s < c.ns; s += nt) c.mark[s] = 0;
        if (tid == 0) c.nmark = 0;
        cold = true;
        full = true;
        __syncthreads();
      }
    }
#pragma unroll 1
    for (int i = tid; i < n; i += nt) xv[i] = c.sol[i];
#pragma unroll 1
    for (int i = tid; i < meq; i += nt) yv[i] = c.sol[n + i];
#pragma unroll 1
    for (int k = tid; k < mineq; k += nt) zv[k] = c.act[k] ? c.sol[c.base + k] : 0.0;
    __syncthreads();
    if (tid == 0) {
#pragma unroll 1
      for (int k = 0; k < mineq; ++k)
        if (c.act[k]) c.alist[nact++] = k;
      s_int[0] = nact;
    }
    __syncthreads();
    nact = s_int[0];
    if (c.prof && tid == 0) c.cyc[PH_INIT] += (unsigned long long)(clock64() - tp0);

    // ---- the dual active-set iteration (reference numeric_QP)
    int num_iter = 0, converged = 0, nxt_active = -1, nxt_drop = -1, to_add = 1;
    int typ = 0;  // 0 solve, 1 update (partial refactorization first)
    const double DMAX = DBL_MAX;
#pragma unroll 1
    for (int pol = 0;; ++pol) {
#pragma unroll 1
    for (;;) {
      if (num_iter > P.max_iter_nas) {
        converged = 0;
        break;
      }
      if (to_add == 1) {
        BQ_T0(c);
        // primal_feasibility (src/nasoq.cpp:787-840): most violated row beyond eps_abs
        int viol = 0;
        double best = P.eps_abs;
        int bi = -1;
#pragma unroll 1
        for (int k = tid; k < mineq; k += nt) {
          double t = 0.0;
#pragma unroll 1
          for (int e = c.bt_ptr[k]; e < c.bt_ptr[k + 1]; ++e) t += c.kv[c.bt_q[e]] * xv[c.bt_var[e]];
          t -= c.dq[k];
          if (t > P.eps_abs) viol++;
          if (t > best) {
            best = t;
            bi = k;
          }
        }
        viol = block_sum_int(viol, redi);
        block_select(best, bi, true, red, redi);
        if (viol == 0) {
          converged = 1;
          break;
        }
        if (bi < 0) {
          converged = 0;
          break;
        }
        nxt_active = bi;
        // update_rhs (src/nasoq.cpp:880-889): the constraint's row as the rhs
#pragma unroll 1
        for (int i = tid; i < N; i += nt) c.rhs[i] = 0.0;
        __syncthreads();
#pragma unroll 1
        for (int e = c.bt_ptr[nxt_active] + tid; e < c.bt_ptr[nxt_active + 1]; e += nt)
          c.rhs[c.bt_var[e]] = c.kv[c.bt_q[e]];
        __syncthreads();
        BQ_T1(c, PH_SELECT);
      }
      // solve_kkt (src/nasoq.cpp:918-957)
      if (typ == 1) {
        BQ_T0(c);
        refactor(c);
        typ = 0;
        BQ_T1(c, PH_FACTOR);
      }
      {
        BQ_T0(c);
        solves++;
        steps += solve_refined(c, c.rhs, c.sol, P.outer, P.inner, flexible, adaptive, a.refine_tol, P.tol_abs, P.tol_rel);
        BQ_T1(c, PH_REFINE);
      }
      const long long tu0 = clock64();
      // step lengths (src/nasoq.cpp:852-878)
      double dual_step = DMAX;
      int drop = -1;
#pragma unroll 1
      for (int t = tid; t < nact; t += nt) {
        const int k = c.alist[t];
        const double lm = c.sol[c.base + k];
        if (lm > 0.0) {
          const double ratio = zv[k] / lm;
          if (drop < 0 || ratio < dual_step || (ratio == dual_step && k < drop)) {
            dual_step = ratio;
            drop = k;
          }
        }
      }
      block_select(dual_step, drop, false, red, redi);
      if (drop < 0) dual_step = DMAX;
      if (tid == 0) {
        double bdotx = 0.0, ddotb = 0.0;
#pragma unroll 1
        for (int e = c.bt_ptr[nxt_active]; e < c.bt_ptr[nxt_active + 1]; ++e) {
          bdotx += c.kv[c.bt_q[e]] * xv[c.bt_var[e]];
          ddotb += c.kv[c.bt_q[e]] * c.sol[c.bt_var[e]];
        }
        double prime_step = DMAX;
        if (!(ddotb < P.zero_thresh)) prime_step = -(c.dq[nxt_active] - bdotx) / ddotb;
        s_dbl[0] = prime_step;
      }
      __syncthreads();
      const double prime_step = s_dbl[0];
      if (drop >= 0) nxt_drop = drop;
      const double step = prime_step > dual_step ? dual_step : prime_step;
      if (step == DMAX) {
        converged = 0;
        break;
      }
      const bool dual_only = prime_step == DMAX && step == dual_step;
      // update_primal / update_dual (src/nasoq.cpp:612-632)
      if (!dual_only)
#pragma unroll 1
        for (int i = tid; i < n; i += nt) xv[i] = xv[i] - step * c.sol[i];
#pragma unroll 1
      for (int i = tid; i < meq; i += nt) yv[i] -= step * c.sol[n + i];
#pragma unroll 1
      for (int t = tid; t < nact; t += nt) {
        const int k = c.alist[t];
        zv[k] -= step * c.sol[c.base + k];
      }
      __syncthreads();
      if (tid == 0) {
        zv[nxt_active] = zv[nxt_active] + step;
        int add = -1, del = -1;
        if (dual_only) del = nxt_drop;
        else if (step == prime_step) add = nxt_active;
        else if (step == dual_step) del = nxt_drop;
        if (add >= 0) {
          const bool fresh = !c.act[add];
          edit_constraint(c, add, true);
          if (fresh && nact < mineq) c.alist[nact++] = add;
          s_int[1] = 1;
        } else if (del >= 0) {
          edit_constraint(c, del, false);
          int pos = -1;
#pragma unroll 1
          for (int t = 0; t < nact; ++t)
            if (c.alist[t] == del) pos = t;
          if (pos >= 0) {
#pragma unroll 1
            for (int t = pos; t + 1 < nact; ++t) c.alist[t] = c.alist[t + 1];
            nact--;
          }
          s_int[1] = 0;
        } else {
          s_int[1] = -1;
        }
        s_int[0] = nact;
      }
      __syncthreads();
      nact = s_int[0];
      if (s_int[1] >= 0) {
        to_add = s_int[1];
        typ = 1;
      }
      num_iter++;
      if (c.prof && tid == 0) {
        c.cyc[PH_UPDATE] += (unsigned long long)(clock64() - tu0);
        c.cyc[PH_ITER] += 1;
      }
    }
    // Polish (adaptive refinement only): the updates x -= step * descent
    // carry each solve's residual (1e-12 relative) through every iteration,
    // so the final point is recomputed as the equality-constrained solution
    // on the final active set (constraints whose multipliers come out
    // negative are dropped and the solve repeated); if the point then
    // violates a constraint, the active-set iteration continues from it (at
    // most twice).  The reference's fixed schedule runs to 1e-15 and needs
    // none of this.
    if (!adaptive || !converged || pol >= 2) break;
    // no iteration since the initial solution: it already is the solution on
    // the final active set (negative multipliers were dropped before), so
    // polishing would repeat the same solve
    if (pol == 0 && num_iter == 0) break;
    // the final solution is refined further than the loop's solves: after a
    // long trajectory its active set is settled, and its KKT norms decide the
    // status
    const double polish_tol = fmin(a.refine_tol, 1e-12);
    if (c.nmark > 0) {
      refactor(c);
    }
    typ = 0;
#pragma unroll 1
    for (int i = tid; i < N; i += nt) {
      double v = 0.0;
      if (i < n) v = -c.q[i];
      else if (i < c.base) v = c.bq[i - n];
      else if (c.act[i - c.base]) v = c.dq[i - c.base];
      c.rhs[i] = v;
    }
    __syncthreads();
    solves++;
    steps += solve_refined(c, c.rhs, c.sol, P.outer, P.inner, flexible, adaptive, polish_tol, P.tol_abs, P.tol_rel);
    // a negative multiplier: that constraint does not belong to the active
    // set of this point; drop it and solve again (at most three times)
#pragma unroll 1
    for (int rep = 0; rep < 3; ++rep) {
      if (tid == 0) {
        int nd = 0;
#pragma unroll 1
        for (int t = 0; t < nact;) {
          const int k = c.alist[t];
          if (c.sol[c.base + k] < 0.0) {
            edit_constraint(c, k, false);
#pragma unroll 1
            for (int u = t; u + 1 < nact; ++u) c.alist[u] = c.alist[u + 1];
            nact--;
            nd++;
          } else {
            ++t;
          }
        }
        s_int[0] = nact;
        s_int[2] = nd;
      }
      __syncthreads();
      nact = s_int[0];
      if (s_int[2] == 0) break;
      refactor(c);
#pragma unroll 1
      for (int i = c.base + tid; i < N; i += nt)
        if (!c.act[i - c.base]) c.rhs[i] = 0.0;
      __syncthreads();
      solves++;
      steps += solve_refined(c, c.rhs, c.sol, P.outer, P.inner, flexible, adaptive, polish_tol, P.tol_abs, P.tol_rel);
    }
#pragma unroll 1
    for (int k = tid; k < mineq; k += nt)
      if (!c.act[k]) zv[k] = 0.0;
#pragma unroll 1
    for (int i = tid; i < n; i += nt) xv[i] = c.sol[i];
#pragma unroll 1
    for (int i = tid; i < meq; i += nt) yv[i] = c.sol[n + i];
#pragma unroll 1
    for (int t = tid; t < nact; t += nt) {
      const int k = c.alist[t];
      zv[k] = c.sol[c.base + k];
    }
    __syncthreads();
    int viol = 0;
#pragma unroll 1
    for (int k = tid; k < mineq; k += nt) {
      double t = 0.0;
#pragma unroll 1
      for (int e = c.bt_ptr[k]; e < c.bt_ptr[k + 1]; ++e) t += c.kv[c.bt_q[e]] * xv[c.bt_var[e]];
      if (t - c.dq[k] > P.eps_abs) viol++;
    }
    viol = block_sum_int(viol, redi);
    if (viol == 0) break;
    converged = 0;
    to_add = 1;
    }

    // ---- results: objective and KKT norms (src/nasoq.cpp:712-728, 1013-1106)
    // Hx, Ax, Cx and H x + A^T y + C^T z from the original values
#pragma unroll 1
    for (int i = tid; i < N; i += nt) {
      double v = 0.0;
      if (i < n) v = xv[i];
      c.w[i] = v;
      double u = v;
      if (i >= n && i < c.base) u = yv[i - n];
      else if (i >= c.base) u = zv[i - c.base];
      c.tmp[i] = u;
    }
    __syncthreads();
    double quad = 0.0, lin = 0.0, lag = 0.0;
#pragma unroll 1
    for (int i = tid; i < n; i += nt) {
      double hx = 0.0, full = 0.0;
#pragma unroll 1
      for (int qq = c.Rp[i]; qq < c.Rp[i + 1]; ++qq) {
        const int j = c.Rj[qq];
        const double v = c.kv[c.Rq[qq]];
        if (j < n) hx += v * c.w[j];
        full += v * c.tmp[j];
      }
      quad += hx * xv[i];
      lin += c.q[i] * xv[i];
      lag = fmax(lag, fabs(full + c.q[i]));
    }
    double cons = 0.0, dual_obj = 0.0, nonneg = 0.0, comp = 0.0;
#pragma unroll 1
    for (int k = tid; k < mineq; k += nt) {
      double t = 0.0;
#pragma unroll 1
      for (int e = c.bt_ptr[k]; e < c.bt_ptr[k + 1]; ++e) t += c.kv[c.bt_q[e]] * xv[c.bt_var[e]];
      t -= c.dq[k];
      cons = fmax(cons, t < 0.0 ? 0.0 : t);
      dual_obj += t * zv[k];
      nonneg = fmax(nonneg, zv[k] > 0.0 ? 0.0 : fabs(zv[k]));
      comp = fmax(comp, fabs(zv[k] * t));
    }
#pragma unroll 1
    for (int r = tid; r < meq; r += nt) {
      double t = 0.0;
#pragma unroll 1
      for (int e = c.eq_ptr[r]; e < c.eq_ptr[r + 1]; ++e) t += c.kv[c.eq_q[e]] * xv[c.eq_var[e]];
      cons = fmax(cons, fabs(t - c.bq[r]));
    }
    // a non-finite solution (non-finite data, or a breakdown the loop could
    // not recover from) is never reported as converged
    int nonfin = 0;
#pragma unroll 1
    for (int i = tid; i < N; i += nt)
      if (!isfinite(c.tmp[i]) || !isfinite(c.w[i])) nonfin = 1;
    nonfin = block_sum_int(nonfin, redi);
    quad = block_sum(quad, red);
    lin = block_sum(lin, red);
    dual_obj = block_sum(dual_obj, red);
    double mx[4] = {lag, cons, nonneg, comp};
#pragma unroll 1
    for (int m = 0; m < 4; ++m) {
      double v = mx[m];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
      __syncthreads();
      if (lane_id() == 0) red[warp_id()] = v;
      __syncthreads();
      if (tid == 0) {
        double w = 0.0;
#pragma unroll 1
        for (int t = 0; t < num_warps(); ++t) w = fmax(w, red[t]);
        s_dbl[m] = w;
      }
      __syncthreads();
      mx[m] = s_dbl[m];
      __syncthreads();
    }
#pragma unroll 1
    for (int t = tid; t < mineq; t += nt) as_out[t] = t < nact ? c.alist[t] : -1;
    if (tid == 0) {
      BResult &R = a.res[pi];
      R.num_iter = num_iter;
      R.active_size = nact;
      R.flags = c.status | (nonfin ? ST_NONFINITE : 0);
      R.refine_steps = steps;
      R.solves = solves;
      R.warm_dropped = warm_dropped;
      R.primal_obj = 0.5 * quad + lin;
      R.dual_obj = dual_obj;
      R.objective = R.primal_obj + dual_obj;
      R.lag_res = mx[0];
      R.cons_sat_norm = mx[1];
      R.non_negativity_infn = mx[2];
      R.complementarity_infn = mx[3];
      int st;
      if (nonfin) st = 3;      // NotConverged
      else if (!converged) st = 0;  // check_solve_status: Infeasible when the loop did not converge
      else if (mx[0] <= P.eps_abs && mx[1] <= P.eps_abs && mx[2] <= P.eps_abs) st = 1;
      else if (mx[1] <= P.eps_abs) st = 2;
      else st = 3;
      R.status = st;
      if (c.prof) c.cyc[PH_TOTAL] += (unsigned long long)(clock64() - tp0);
    }
    __syncthreads();
  }
  if (a.prof && tid < PH_N) atomicAdd(a.prof + tid, c.cyc[tid]);
}

// batch_fp64.cu and batch_large.cu compile this file again with
// NQG_BATCH_FP64_UNIT / NQG_BATCH_LARGE_UNIT defined for their instantiations
// alone (they then build in parallel); the non-template kernels and host
// functions belong to this unit.
#if !defined(NQG_BATCH_FP64_UNIT) && !defined(NQG_BATCH_LARGE_UNIT)

// Warm-start sets from per-constraint scores (e.g. the logits of the active-set
// model): problem i proposes every constraint k with scores[i * ld + k] >
// threshold, in ascending order, except one parallel to a constraint it
// already proposed (same variables, proportional coefficients -- the two
// sides of a box): both active would make the KKT matrix singular.  A
// problem with no proposal keeps a cold start.  One warp per problem: lanes
// read 32 scores at a time (coalesced); the candidates of a chunk are taken
// in constraint order, each checked by all lanes at once against the
// constraints already proposed.
__global__ void k_ws_scores(int nprob, BProb *probs, const BPat *pats, const int *ipool, const double *dpool,
                            int *iout, const float *scores, int ld, float thr) {
  const int lane = threadIdx.x & 31;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= nprob) return;
  BProb &P = probs[i];
  const BPat &pt = pats[P.pat];
  const int *bt_ptr = ipool + pt.o_bt_ptr, *bt_var = ipool + pt.o_bt_var, *bt_q = ipool + pt.o_bt_q;
  const double *kv = dpool + P.o_kv;
  int *as = iout + P.o_as;
  const float *sc = scores + (size_t)i * ld;
  int cnt = 0;
  const int mi = min(pt.mineq, ld);
#pragma unroll 1
  for (int c0 = 0; c0 < mi; c0 += 32) {
    const int kk = c0 + lane;
    unsigned cand = __ballot_sync(0xffffffffu, kk < mi && sc[kk] > thr);
    while (cand) {
      const int k = c0 + __ffs(cand) - 1;
      cand &= cand - 1;
      const int ka = bt_ptr[k], kn = bt_ptr[k + 1] - ka;
      bool parallel = false;
#pragma unroll 1
      for (int t = lane; t < cnt; t += 32) {
        const int j = as[t], ja = bt_ptr[j], jn = bt_ptr[j + 1] - ja;
        if (jn != kn || kn == 0) continue;
        bool same = true;
        const double r = kv[bt_q[ka]] / kv[bt_q[ja]];
#pragma unroll 1
        for (int e = 0; e < kn && same; ++e)
          same = bt_var[ka + e] == bt_var[ja + e] &&
                 fabs(kv[bt_q[ka + e]] - r * kv[bt_q[ja + e]]) <= 1e-12 * fabs(kv[bt_q[ka + e]]);
        parallel = parallel || same;
      }
      if (!__any_sync(0xffffffffu, parallel)) {
        if (lane == 0) as[cnt] = k;
        ++cnt;
        __syncwarp();
      }
    }
  }
  if (lane == 0) P.ws_n = cnt > 0 ? cnt : -1;
}

// One block per problem: its q, b and d from the stacked staging buffer.
__global__ void k_scatter_vectors(int nprob, const BProb *probs, const BPat *pats, const int64_t *voff,
                                  const double *stage, double *dpool) {
  const int i = blockIdx.x;
  if (i >= nprob) return;
  const BProb &P = probs[i];
  const BPat &pt = pats[P.pat];
  const int64_t oq = voff[3 * i], ob = voff[3 * i + 1], od = voff[3 * i + 2];
  if (oq >= 0)
#pragma unroll 1
    for (int t = threadIdx.x; t < pt.n; t += blockDim.x) dpool[P.o_q + t] = stage[oq + t];
  if (ob >= 0)
#pragma unroll 1
    for (int t = threadIdx.x; t < pt.meq; t += blockDim.x) dpool[P.o_b + t] = stage[ob + t];
  if (od >= 0)
#pragma unroll 1
    for (int t = threadIdx.x; t < pt.mineq; t += blockDim.x) dpool[P.o_d + t] = stage[od + t];
}

int batch_scatter_vectors(int nprob, const BProb *probs, const BPat *pats, const int64_t *voff, const double *stage,
                          double *dpool, cudaStream_t st) {
  if (nprob <= 0) return NQG_OK;
  k_scatter_vectors<<<nprob, 128, 0, st>>>(nprob, probs, pats, voff, stage, dpool);
  return cudaGetLastError() == cudaSuccess ? NQG_OK : NQG_ERR_CUDA;
}

__global__ void k_ws_clear(int nprob, BProb *probs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nprob) probs[i].ws_n = -1;
}

int batch_ws_from_scores(int nprob, BProb *probs, const BPat *pats, const int *ipool, const double *dpool, int *iout,
                         const float *scores, int ld, float thr, cudaStream_t st) {
  k_ws_scores<<<(nprob + 7) / 8, 256, 0, st>>>(nprob, probs, pats, ipool, dpool, iout, scores, ld, thr);
  return cudaGetLastError() == cudaSuccess ? NQG_OK : NQG_ERR_CUDA;
}

int batch_ws_clear(int nprob, BProb *probs, cudaStream_t st) {
  k_ws_clear<<<(nprob + 127) / 128, 128, 0, st>>>(nprob, probs);
  return cudaGetLastError() == cudaSuccess ? NQG_OK : NQG_ERR_CUDA;
}

size_t batch_smem_bytes(const BArgs &a, size_t tsize) {
  auto up = [](size_t b) { return (b + 15) / 16 * 16; };
  return BATCH_CTX_BYTES + up((size_t)a.N_max * tsize) + up((size_t)a.N_max * (a.large ? sizeof(int) : tsize)) +
         up(batch_rowbuf(a) * tsize) + 2 * up((size_t)a.w_max * tsize) + up((size_t)a.w_max * sizeof(int)) +
         (a.large ? 0 : (size_t)a.nlev_max * 48 + up((size_t)a.ns_max)) + up((size_t)(2 * a.nlev_max + 2) * sizeof(int)) +
         up((size_t)a.ns_max) + up((size_t)a.mi_max) + batch_block_bytes(a, tsize) + (size_t)a.stage_bytes;
}

#endif

// Raises the kernel's dynamic shared-memory limit (outside any stream capture) and
// returns how many CTAs of `smem` bytes fit on an SM.  The limit belongs to the
// kernel, not to a batch: always the device's largest, so that a batch made later
// with less shared memory does not take it from an earlier one.
template <class T, bool LARGE_PATTERNS>
int batch_prepare(int threads, size_t smem_attr, size_t smem, int *blocks_per_sm) {
  const auto kernel = k_nasoq_batch<T, LARGE_PATTERNS>;
  int dev = 0, most = 0;
  cudaFuncAttributes fa;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, kernel) != cudaSuccess)
    return NQG_ERR_CUDA;
  most -= (int)fa.sharedSizeBytes;
  if (smem_attr > (size_t)most ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess)
    return NQG_ERR_CUDA;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, threads, smem) != cudaSuccess)
    return NQG_ERR_CUDA;
  return NQG_OK;
}

template <class T, bool LARGE_PATTERNS>
int launch_batch(const BArgs &a, int grid, int threads, size_t smem, cudaStream_t st) {
  k_nasoq_batch<T, LARGE_PATTERNS><<<grid, threads, smem, st>>>(a);
  return cudaGetLastError() == cudaSuccess ? NQG_OK : NQG_ERR_CUDA;
}

#define NQG_BATCH_INSTANCE(T)                                                           \
  template int launch_batch<T, LARGE>(const BArgs &, int, int, size_t, cudaStream_t); \
  template int batch_prepare<T, LARGE>(int, size_t, size_t, int *);
#if defined(NQG_BATCH_FP64_UNIT) || defined(NQG_BATCH_LARGE_UNIT)
NQG_BATCH_INSTANCE(double)
#endif
#if !defined(NQG_BATCH_FP64_UNIT)
NQG_BATCH_INSTANCE(float)
#endif

}  // namespace nqg
