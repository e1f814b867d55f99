// Active-set predictor for parametric QP families: a multilayer perceptron
// theta -> one logit per inequality constraint (positive: predicted active at
// the optimum), whose prediction seeds the batched NASOQ solve as a warm start
// (nqg_batch_warm_start_from_scores); the active-set iteration then corrects
// it and alone decides whether the final tolerance is met.  The reference has no
// learned component; its warm-start entry is Nasoq::set_warm_start
// (src/nasoq.cpp:413-436).
//
// Weights are kept as FP32 master copies (the optimizer's) and as BF16 copies
// that the forward and backward products read; activations and gradients are
// FP32 and every product accumulates in FP32.  Kernels (all hand-written):
//  * k_mlp_tc: C = A B^T on the fifth-generation tensor cores (see there):
//    X W^T (forward), dY W (input gradient) and dY^T X (weight gradient);
//    epilogues: bias + ReLU, ReLU mask of the layer below, plain store;
//  * k_sum_parts (weight gradient's parts), k_colsum (bias gradient), k_bce
//    (weighted sigmoid cross-entropy and its gradient), k_adam (Adam step,
//    BF16 refresh), k_gather (mini-batch rows).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <string>
#include <vector>

#include "../../include/nasoq_gb300.h"
#include "tcgen05.cuh"

namespace {

namespace t5 = nqg::t5;

enum { EPI_STORE = 0, EPI_BIAS_RELU = 1, EPI_BIAS = 2, EPI_RELU_MASK = 3 };

// One operand of a product, rows x K: entry (r, k) at p[r * ld + k], or at
// p[k * ld + r] when `across` (the rows run along memory).  FP32, or BF16 where
// bf is given (ld a multiple of 8, zeros behind K).  vec: FP32 rows may be read
// 16 bytes at a time.
struct Operand {
  const float *p;
  const __nv_bfloat16 *bf;
  int rows, ld;
  bool across, vec;
};

// C (M x N) = A B^T over K, 128 x NT tiles (64 or 128 columns), one CTA of 256
// threads each.
//
// FP32 values go through the BF16 tensor cores without losing bits: a value is
// the sum of three BF16 ones (its significand cut into three runs of eight
// bits), and the products of the parts are exact in the FP32 accumulator.  A
// product with BF16 weights takes three MMAs; one of two FP32 operands six
// (the parts' products down to 2^-16 of the leading one; the three left out
// are below 2^-24).  The threads split their share of A and B, eight entries of
// K at a time, into the swizzled K-major layout of tcgen05.cuh, 64 entries of
// K per stage, two stages: the next chunk's loads run while the tensor cores
// work.  Neighbouring threads take neighbouring memory: units of one row where
// the rows lie along it, rows where they lie across.
//
// The tensor cores cut a sum's low bits at every step (3e-8 of it each; a chain
// of 48 steps over 256 entries of K left 1.5e-6, five times what FP32
// multiply-adds do).  So the leading products take turns in NACC accumulators,
// the others, 2^-8 of them and less, have one of their own, and after SEG chunks
// the four are added to FP32 registers: at most 8 steps in a chain.
//
// The 64 x 64 CUDA-core tiles before reached 8.7 TFLOP/s (4096-row forward of
// the 32-256-256-900 model: 287 us).  What bounds it now is the splitting of A
// and the latency of a chunk (load, split, barrier, MMA: about 3 us), so a
// wide product takes 128 columns at a time (tile_columns).
//
// gridDim.z > 1: part z takes every gridDim.z-th chunk of K and stores to
// C + z * part (plain store).  If an MMA wait gives up (after wait_limit polls),
// the tile's entries are NaN and `timeout` (host memory) is set.
constexpr int MT = 128, KT = 64;      // rows of a tile, K entries per stage
constexpr int A_PART = MT * 128;     // bytes of one BF16 part of A in a stage

// Eight values as their three BF16 parts, one 16-byte unit each.
__device__ __forceinline__ void split8(const float *x, uint4 (&part)[3]) {
  uint32_t w[3][4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t h[2], m[2], l[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float v = x[2 * q + e];
      const uint32_t b = __float_as_uint(v);
      // a NaN may have its payload in the low bits alone, which would leave an infinity
      h[e] = (b & 0x7fffffffu) > 0x7f800000u ? 0x7fff0000u : b & 0xffff0000u;
      const float r = (b & 0x7f800000u) == 0x7f800000u ? 0.f : v - __uint_as_float(h[e]);  // exact; infinities and NaN stay in h
      m[e] = __float_as_uint(r) & 0xffff0000u;
      l[e] = __float_as_uint(r - __uint_as_float(m[e]));
    }
    w[0][q] = h[0] >> 16 | h[1];
    w[1][q] = m[0] >> 16 | m[1];
    w[2][q] = l[0] >> 16 | (l[1] & 0xffff0000u);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) part[q] = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
}

constexpr int TC_THREADS = 256;
constexpr int NACC = 3, SEG = 6;  // accumulators of the leading products, chunks until they are read

// The units (row, eight entries of K) of a rows x 64 operand tile that this
// thread moves: U of them, unit i of thread tid.
template <int ROWS> struct Units {
  static constexpr int U = ROWS * (KT / 8) / TC_THREADS;
  __device__ static __forceinline__ void at(bool across, int i, int &r, int &u) {
    const int tid = threadIdx.x;
    if (across) {
      r = tid % ROWS;
      u = (tid / ROWS) * U + i;
    } else {
      r = tid / 8 + (TC_THREADS / 8) * i;
      u = tid % 8;
    }
  }
};

// Entries k0 .. k0 + 8 of row r (0 outside the operand).
__device__ __forceinline__ void load_unit(const Operand &o, int r, int k0, int K, float *x) {
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] = 0.f;
  if (r >= o.rows) return;
  if (o.across) {
    const float *p = o.p + r + (size_t)k0 * o.ld;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k0 + k < K) x[k] = p[(size_t)k * o.ld];
  } else if (o.vec) {  // ld a multiple of 4: a group of four that begins inside the row ends inside it
    const float *p = o.p + (size_t)r * o.ld + k0;
#pragma unroll
    for (int k = 0; k < 8; k += 4)
      if (k0 + k < K) {
        const float4 f = *reinterpret_cast<const float4 *>(p + k);
        x[k] = f.x, x[k + 1] = f.y, x[k + 2] = f.z, x[k + 3] = f.w;
      }
  } else {
    const float *p = o.p + (size_t)r * o.ld + k0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k0 + k < K) x[k] = p[k];
  }
}

__host__ __device__ constexpr int tc_stage(int nb, int nt) { return 3 * A_PART + nb * nt * 128; }
__host__ __device__ constexpr int tc_smem(int nb, int nt) { return 2 * tc_stage(nb, nt) + 1024 + 64; }

// Entry (r, k) of an operand.
__device__ __forceinline__ float value(const Operand &o, int r, int k) {
  if (o.bf) return __bfloat162float(o.bf[(size_t)r * o.ld + k]);
  return o.across ? o.p[r + (size_t)k * o.ld] : o.p[(size_t)r * o.ld + k];
}
// Entry (m, n) of part z of nz of a product, by FP32 multiply-adds.  A result
// that is not a number is formed again by it: an infinity times a part of the
// other value that happens to be zero is no product of the values.
__device__ __noinline__ float plain_entry(const Operand &A, const Operand &B, int m, int n, int K, int z, int nz) {
  float s = 0.f;
#pragma unroll 1
  for (int k0 = z * KT; k0 < K; k0 += nz * KT)
#pragma unroll 4
    for (int k = k0; k < min(k0 + KT, K); ++k) s = fmaf(value(A, m, k), value(B, n, k), s);
  return s;
}

// NB: BF16 parts of B (1: BF16 operand, 3: FP32 one).
template <int NB, int NT>
__global__ void __launch_bounds__(TC_THREADS) k_mlp_tc(int M, int N, int K, Operand A, Operand B, float *C, int ldc, size_t part,
                                                int epi, const float *bias, const float *mask, int *timeout,
                                                long long wait_limit) {
  extern __shared__ __align__(16) unsigned char tc_raw[];
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int STAGE = tc_stage(NB, NT), B_PART = NT * 128;
  uint64_t *mbar = reinterpret_cast<uint64_t *>(base + 2 * STAGE);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(base + 2 * STAGE + 32);
  const int m0 = blockIdx.y * MT, n0 = blockIdx.x * NT;
  if (warp == 0) t5::tmem_alloc(t5::smem_u32(tslot), (NACC + 1) * NT);
  if (tid == 0) {
    s_fail = 0;
    t5::mbar_init(t5::smem_u32(&mbar[0]), 1);
    t5::mbar_init(t5::smem_u32(&mbar[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  t5::fence_before();
  __syncthreads();
  t5::fence_after();
  const uint32_t tmem = *tslot;
  constexpr uint32_t IDESC = t5::idesc_bf16(MT, NT);
  const int nchunk = (K + KT - 1) / KT;
  using UA = Units<MT>;
  using UB = Units<NT>;
  float xa[UA::U][8], xb[NB == 3 ? UB::U : 1][8];
  uint4 wb[NB == 1 ? UB::U : 1];
  auto load = [&](int ch) {
    int r, u;
#pragma unroll
    for (int i = 0; i < UA::U; ++i) {
      UA::at(A.across, i, r, u);
      load_unit(A, m0 + r, ch * KT + 8 * u, K, xa[i]);
    }
#pragma unroll
    for (int i = 0; i < UB::U; ++i) {
      UB::at(NB == 3 && B.across, i, r, u);
      const int k0 = ch * KT + 8 * u;
      if constexpr (NB == 3) load_unit(B, n0 + r, k0, K, xb[i]);
      else wb[i] = n0 + r < B.rows && k0 < K ? *reinterpret_cast<const uint4 *>(B.bf + (size_t)(n0 + r) * B.ld + k0)
                                             : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  uint32_t uses[2] = {0u, 0u};
  bool ok = true;
  int it = 0;
  // this thread's part of the result: accumulator row 32 (w % 4) + lane (warp w may read that quarter), every other
  // 32 columns
  float sum[NT / 64][32];
#pragma unroll
  for (int h = 0; h < NT / 64; ++h)
#pragma unroll
    for (int q = 0; q < 32; ++q) sum[h][q] = 0.f;
  // adds what the accumulators hold, once the MMAs have completed; every thread calls
  static_assert(KT / 16 >= NACC, "a chunk has written every accumulator");
  auto collect = [&]() {
    if (tid == 0)
      for (int s = 0; s < 2; ++s)
        if (uses[s] > 0 && !t5::mbar_wait(t5::smem_u32(&mbar[s]), (uses[s] - 1) & 1, wait_limit)) s_fail = 1;
    __syncthreads();
    t5::fence_after();
    if (s_fail) return false;
#pragma unroll
    for (int h = 0; h < NT / 64; ++h)
#pragma unroll 1
      for (int g = NACC; g >= 0; --g) {
        uint32_t v[32];
        t5::tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * NT + 64 * h + 32 * (warp >> 2)), v);
#pragma unroll
        for (int q = 0; q < 32; ++q) sum[h][q] += __uint_as_float(v[q]);
      }
    t5::fence_before();
    __syncthreads();  // the accumulators may be written again
    t5::fence_after();
    return true;
  };
  if ((int)blockIdx.z < nchunk) load(blockIdx.z);
  for (int ch = blockIdx.z; ch < nchunk; ch += gridDim.z, ++it) {
    const int s = it & 1;
    unsigned char *stg = base + s * STAGE;
    if (uses[s] > 0) {  // the MMAs that last read this stage must have completed
      if (tid == 0 && !t5::mbar_wait(t5::smem_u32(&mbar[s]), (uses[s] - 1) & 1, wait_limit)) s_fail = 1;
      __syncthreads();
      if (s_fail) {
        ok = false;
        break;
      }
    }
    unsigned char *stb = stg + 3 * A_PART;
    int r, u;
#pragma unroll
    for (int i = 0; i < UA::U; ++i) {
      UA::at(A.across, i, r, u);
      const int off = r * 128 + ((u ^ (r & 7)) << 4);
      uint4 p[3];
      split8(xa[i], p);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4 *>(stg + q * A_PART + off) = p[q];
    }
#pragma unroll
    for (int i = 0; i < UB::U; ++i) {
      UB::at(NB == 3 && B.across, i, r, u);
      const int off = r * 128 + ((u ^ (r & 7)) << 4);
      if constexpr (NB == 3) {
        uint4 p[3];
        split8(xb[i], p);
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4 *>(stb + q * B_PART + off) = p[q];
      } else {
        *reinterpret_cast<uint4 *>(stb + off) = wb[i];
      }
    }
    t5::fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      t5::fence_after();
      const uint32_t a = t5::smem_u32(stg), b = a + 3 * A_PART;
      const int step0 = (it % SEG) * (KT / 16);
#pragma unroll
      for (int ks = 0; ks < KT / 16; ++ks) {
        // the smaller products first
#pragma unroll
        for (int o = 2; o >= 0; --o)
#pragma unroll
          for (int ib = 0; ib <= o; ++ib) {
            const int ia = o - ib;
            if (ib >= NB) continue;
            const int g = o > 0 ? NACC : (step0 + ks) % NACC;
            const uint32_t acc = o == 0 ? step0 + ks >= NACC : (step0 + ks > 0 || o < 2 || ib > 0);
            t5::mma_bf16(tmem + g * NT, t5::desc_sw128(a + ia * A_PART + 32 * ks), t5::desc_sw128(b + ib * B_PART + 32 * ks),
                         IDESC, acc);
          }
      }
      t5::mma_commit(t5::smem_u32(&mbar[s]));
    }
    ++uses[s];
    const bool more = ch + (int)gridDim.z < nchunk;
    if (more) load(ch + gridDim.z);
    if (it % SEG == SEG - 1 || !more)
      if (!collect()) {
        ok = false;
        break;
      }
  }
  if (!ok) {  // a wait gave up: give the MMAs in flight their time (bounded) before the memory they use goes
    if (tid == 0)
      for (int s = 0; s < 2; ++s)
        if (uses[s] > 0) t5::mbar_wait(t5::smem_u32(&mbar[s]), (uses[s] - 1) & 1);
    __syncthreads();
  }
  if (tid == 0) {
    for (int s = 0; s < 2; ++s)
      asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(t5::smem_u32(&mbar[s])) : "memory");
    if (!ok) *(volatile int *)timeout = 1;
  }
  // accumulator rows through shared memory (the stages are free), so that
  // global rows are written in whole lines
  float *out = reinterpret_cast<float *>(base);
  constexpr int LDO = NT + 1;
  bool nan = false;
  if (ok) {
    const int row = (warp & 3) * 32 + lane;
#pragma unroll
    for (int h = 0; h < NT / 64; ++h)
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        out[row * LDO + 64 * h + 32 * (warp >> 2) + q] = sum[h][q];
        nan |= sum[h][q] != sum[h][q];
      }
  }
  // a loop of its own: as a call in the epilogue's it cost 8 us of 65 (4096-row forward)
  if (__syncthreads_or(nan)) {
#pragma unroll 1
    for (int e = tid; e < MT * NT; e += TC_THREADS) {
      const int m = m0 + e / NT, n = n0 + e % NT;
      float &v = out[(e / NT) * LDO + e % NT];
      if (m < M && n < N && v != v) v = plain_entry(A, B, m, n, K, blockIdx.z, gridDim.z);
    }
    __syncthreads();
  }
  float *Cz = C + blockIdx.z * part;
  if (!ok) {
    for (int e = tid; e < MT * NT; e += TC_THREADS)
      if (m0 + e / NT < M && n0 + e % NT < N) Cz[(size_t)(m0 + e / NT) * ldc + n0 + e % NT] = __int_as_float(0x7fffffff);
  } else {
#pragma unroll 4
    for (int r = warp * 16; r < warp * 16 + 16; ++r) {
      const int m = m0 + r;
      if (m >= M) break;
#pragma unroll
      for (int h = 0; h < NT; h += 32) {
        const int n = n0 + h + lane;
        if (n >= N) continue;
        float v = out[r * LDO + h + lane];
        if (epi == EPI_BIAS_RELU) v = fmaxf(v + bias[n], 0.f);
        else if (epi == EPI_BIAS) v = v + bias[n];
        else if (epi == EPI_RELU_MASK) v = mask[(size_t)m * ldc + n] > 0.f ? v : 0.f;
        Cz[(size_t)m * ldc + n] = v;
      }
    }
  }
  t5::fence_before();
  __syncthreads();
  if (warp == 0) t5::tmem_dealloc(tmem, (NACC + 1) * NT);
}

// out = the sum of `parts` arrays of n values, `part` apart, in order; 0 where
// the mask (if given) is not positive.
__global__ void k_sum_parts(long n, int parts, size_t part, const float *src, const float *mask, float *out) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    float s = src[i];
    for (int q = 1; q < parts; ++q) s += src[q * part + i];
    out[i] = !mask || mask[i] > 0.f ? s : 0.f;
  }
}

// Column sums of Y (M x N): 32 columns per block, 32 groups of rows each
// summed by one thread per column, then the groups in order (one thread per
// column over all rows before: 1024 rows x 900 columns 94 us).
__global__ void __launch_bounds__(1024) k_colsum(int M, int N, const float *Y, float *out) {
  __shared__ float part[32][33];
  const int n = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (n < N) {
#pragma unroll 4
    for (int m = threadIdx.y; m < M; m += 32) s += Y[(long)m * N + n];
  }
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && n < N) {
    s = part[0][threadIdx.x];
    for (int q = 1; q < 32; ++q) s += part[q][threadIdx.x];
    out[n] = s;
  }
}

// Weighted sigmoid cross-entropy, mean over the batch rows:
//   l = -(pw y log s(z) + (1 - y) log(1 - s(z))),  dl/dz = s(z) (pw y + 1 - y) - pw y
// (computed with log1p(exp(-|z|)) for stability); grad = dl/dz / M.
// One wave of blocks: the FP64 sums of a block (an FP64 addition holds its pipe
// for 64 cycles) cost as much as hundreds of its entries.
__global__ void k_bce(long total, int M, const float *Z, const float *Y, float pw, float *grad, double *loss) {
  double part = 0.0;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const float z = Z[e], y = Y[e];
    const float t = expf(-fabsf(z)), lp = log1pf(t);
    const float sp_neg = fmaxf(-z, 0.f) + lp;  // -log s(z)
    const float sp_pos = fmaxf(z, 0.f) + lp;   // -log(1 - s(z))
    part += (double)(pw * y * sp_neg + (1.f - y) * sp_pos);
    const float s = (z < 0.f ? t : 1.f) / (1.f + t);
    grad[e] = (s * (pw * y + 1.f - y) - pw * y) / (float)M;
  }
  __shared__ double red[256];
  red[threadIdx.x] = part;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, red[0] / M);
}

// BF16 copies of a layer's weights (out x in): by rows and across, rows padded
// to a multiple of 8 entries (the padding stays zero).
__host__ __device__ inline int pad8(int n) { return (n + 7) & ~7; }
__device__ __forceinline__ void store_bf16(__nv_bfloat16 *wb, __nv_bfloat16 *wt, long i, int out, int in, float w) {
  const int o = (int)(i / in), k = (int)(i - (long)o * in);
  const __nv_bfloat16 v = __float2bfloat16(w);
  wb[(size_t)o * pad8(in) + k] = v;
  wt[(size_t)k * pad8(out) + o] = v;
}

__global__ void k_adam(long n, float *w, __nv_bfloat16 *wb, __nv_bfloat16 *wt, int out, int in, const float *g, float *m,
                       float *v, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (wb) store_bf16(wb, wt, i, out, in, wi);
  }
}

__global__ void k_to_bf16(long n, const float *w, __nv_bfloat16 *wb, __nv_bfloat16 *wt, int out, int in) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    store_bf16(wb, wt, i, out, in, w[i]);
}

__global__ void k_gather(int rows, int cols, const int *idx, const float *src, float *dst) {
  const long total = (long)rows * cols;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long r = e / cols, c = e % cols;
    dst[e] = src[(long)idx[r] * cols + c];
  }
}

inline int blocks_for(long n) { return (int)std::max<long>(1, std::min<long>((n + 255) / 256, 4096)); }

}  // namespace

struct nqg_mlp {
  std::vector<int> sizes;  // sizes[0] inputs, ..., sizes[L] outputs
  int L = 0;
  std::vector<float *> W, b, gW, gb, mW, vW, mb, vb;
  std::vector<__nv_bfloat16 *> Wb, Wt;  // out x in, in x out
  std::vector<float *> act;  // act[0]: input rows, act[l]: output of layer l (act[L]: logits)
  std::vector<float *> dact;
  int cap = 0;               // rows the activation buffers hold
  float *d_X = nullptr, *d_Y = nullptr;  // training set (device)
  int n_train = 0;
  float *d_lab = nullptr;    // labels of the current mini-batch
  int *d_idx = nullptr;
  double *d_loss = nullptr;
  float *d_parts = nullptr;  // parts of a gradient's product (see k_parts)
  // host memory, set by kernels whose MMA wait gave up: on the model's own stream, on a caller's
  int *timeout = nullptr;
  long long wait_limit = t5::WAIT_LIMIT;
  long step = 0;
  cudaStream_t stream = nullptr, own_stream = nullptr;  // where launches go; the model's own
  std::string err;
};

namespace {

#define MQ(call)                                                         \
  do {                                                                   \
    cudaError_t e_ = (call);                                             \
    if (e_ != cudaSuccess) {                                             \
      m->err = std::string(#call) + ": " + cudaGetErrorString(e_);       \
      return NQG_ERR_CUDA;                                               \
    }                                                                    \
  } while (0)

constexpr int PARTS_MAX = 8;
constexpr int SM_COUNT = 152;

// Parts of K of a gradient's product: its tiles alone (32 at 900 x 256 weights
// or 1024 x 256 inputs) leave the chip idle, so K is split until they fill it,
// two chunks to a part at least.  A part of its own costs one more launch (the
// sum), so the forward pass, four chunks deep at most in the usual models, is
// not split.
int k_parts(int M, int N, int K) {
  const int tiles = ((M + MT - 1) / MT) * ((N + 63) / 64), chunks = (K + KT - 1) / KT;
  return std::max(1, std::min({PARTS_MAX, chunks / 2, SM_COUNT / tiles}));
}

int ensure_rows(nqg_mlp *m, int rows) {
  if (rows <= m->cap) return NQG_OK;
  for (auto *p : m->act) cudaFree(p);
  for (auto *p : m->dact) cudaFree(p);
  cudaFree(m->d_lab);
  cudaFree(m->d_idx);
  m->act.assign(m->L + 1, nullptr);
  m->dact.assign(m->L + 1, nullptr);
  for (int l = 0; l <= m->L; ++l) {
    MQ(cudaMalloc(&m->act[l], (size_t)rows * m->sizes[l] * sizeof(float)));
    MQ(cudaMalloc(&m->dact[l], (size_t)rows * m->sizes[l] * sizeof(float)));
  }
  MQ(cudaMalloc(&m->d_lab, (size_t)rows * m->sizes[m->L] * sizeof(float)));
  MQ(cudaMalloc(&m->d_idx, (size_t)rows * sizeof(int)));
  m->cap = rows;
  return NQG_OK;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// entry (r, k) of an FP32 operand at p[r * ld + k] / p[k * ld + r]
Operand along(const float *p, int rows, int ld) { return {p, nullptr, rows, ld, false, ld % 4 == 0 && aligned16(p)}; }
Operand across(const float *p, int rows, int ld) { return {p, nullptr, rows, ld, true, false}; }
Operand weights(const __nv_bfloat16 *p, int rows, int K) { return {nullptr, p, rows, pad8(K), false, true}; }

// Columns of a tile: 128 where 64 would take more than a wave of CTAs (every
// tile splits the same rows of A again).
int tile_columns(int M, int N) { return (long)((M + MT - 1) / MT) * ((N + 63) / 64) > SM_COUNT && N > 64 ? 128 : 64; }

// Shared-memory limits of the kernels below, for the device that a model is
// made on (they belong to a device, not to the process).
template <int NB, int NT> cudaError_t allow_smem() {
  return cudaFuncSetAttribute(k_mlp_tc<NB, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem(NB, NT));
}
cudaError_t allow_smem_all() {
  for (cudaError_t e : {allow_smem<1, 64>(), allow_smem<1, 128>(), allow_smem<3, 64>()})
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

template <int NB, int NT>
void launch_tc(nqg_mlp *m, int M, int N, int K, const Operand &A, const Operand &B, float *C, int ldc, int epi,
               const float *bias, const float *mask, int parts) {
  const dim3 grid((N + NT - 1) / NT, (M + MT - 1) / MT, parts);
  int *const report = m->timeout + (m->stream == m->own_stream ? 0 : 1);
  k_mlp_tc<NB, NT><<<grid, TC_THREADS, tc_smem(NB, NT), m->stream>>>(M, N, K, A, B, C, ldc, (size_t)M * N, epi, bias, mask,
                                                                     report, m->wait_limit);
}

// B FP32 (NB 3) or BF16 (NB 1).
template <int NB>
void gemm(nqg_mlp *m, int M, int N, int K, const Operand &A, const Operand &B, float *C, int ldc, int epi,
          const float *bias, const float *mask, int parts = 1) {
  if (NB == 1 && tile_columns(M, N) == 128) launch_tc<1, 128>(m, M, N, K, A, B, C, ldc, epi, bias, mask, parts);
  else launch_tc<NB, 64>(m, M, N, K, A, B, C, ldc, epi, bias, mask, parts);
}

// Forward over rows given in x; act[1 ..] receive the hidden layers, `logits`
// the last one.
void forward(nqg_mlp *m, int rows, const float *x, float *logits) {
  for (int l = 0; l < m->L; ++l) {
    const int in = m->sizes[l], out = m->sizes[l + 1];
    const bool last = l + 1 == m->L;
    // act[l+1][r, o] = sum_i act[l][r, i] W[o, i]  (+ b, ReLU below the last layer)
    gemm<1>(m, rows, out, in, along(l ? m->act[l] : x, rows, in), weights(m->Wb[l], out, in),
            last ? logits : m->act[l + 1], out, last ? EPI_BIAS : EPI_BIAS_RELU, m->b[l], nullptr);
  }
}
void forward(nqg_mlp *m, int rows) { forward(m, rows, m->act[0], m->act[m->L]); }

// Backward from dact[L] (dloss/dlogits); fills gW, gb.
void backward(nqg_mlp *m, int rows) {
  for (int l = m->L - 1; l >= 0; --l) {
    const int in = m->sizes[l], out = m->sizes[l + 1];
    // gW[o, i] = sum_r dact[l+1][r, o] act[l][r, i]
    const int pw = k_parts(out, in, rows);
    gemm<3>(m, out, in, rows, across(m->dact[l + 1], out, out), across(m->act[l], in, in), pw > 1 ? m->d_parts : m->gW[l],
            in, EPI_STORE, nullptr, nullptr, pw);
    if (pw > 1) {
      const long nw = (long)in * out;
      k_sum_parts<<<blocks_for(nw), 256, 0, m->stream>>>(nw, pw, (size_t)nw, m->d_parts, nullptr, m->gW[l]);
    }
    k_colsum<<<(out + 31) / 32, dim3(32, 32), 0, m->stream>>>(rows, out, m->dact[l + 1], m->gb[l]);
    if (l > 0) {  // dact[l][r, i] = sum_o dact[l+1][r, o] W[o, i], masked by the ReLU of layer l
      const int px = k_parts(rows, in, out);
      gemm<1>(m, rows, in, out, along(m->dact[l + 1], rows, out), weights(m->Wt[l], in, out),
              px > 1 ? m->d_parts : m->dact[l], in, px > 1 ? EPI_STORE : EPI_RELU_MASK, nullptr, m->act[l], px);
      if (px > 1) {
        const long nx = (long)rows * in;
        k_sum_parts<<<blocks_for(nx), 256, 0, m->stream>>>(nx, px, (size_t)nx, m->d_parts, m->act[l], m->dact[l]);
      }
    }
  }
}

// `which`: 0 the model's own stream, 1 callers' streams.
int mma_status(nqg_mlp *m, int which = 0) {
  volatile int *t = m->timeout + which;
  if (!*t) return NQG_OK;
  *t = 0;
  m->err = "a tensor-core wait timed out";
  return NQG_ERR_TIMEOUT;
}

}  // namespace

extern "C" int nqg_mlp_create(int nsizes, const int *sizes, unsigned long long seed, nqg_mlp **out) {
  if (!out || nsizes < 2 || !sizes) return NQG_ERR_ARG;
  for (int l = 0; l < nsizes; ++l)
    if (sizes[l] <= 0) return NQG_ERR_ARG;
  if (allow_smem_all() != cudaSuccess) return NQG_ERR_CUDA;
  auto *m = new nqg_mlp;
  m->sizes.assign(sizes, sizes + nsizes);
  m->L = nsizes - 1;
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete m;
    return NQG_ERR_CUDA;
  }
  m->own_stream = m->stream;
  std::mt19937_64 rng(seed);
  for (int l = 0; l < m->L; ++l) {
    const int in = sizes[l], o = sizes[l + 1];
    const long nw = (long)in * o;
    // He initialisation for the ReLU layers
    std::normal_distribution<float> nd(0.f, std::sqrt(2.f / in));
    std::vector<float> w(nw), z(std::max<long>(nw, o), 0.f);
    for (auto &v : w) v = nd(rng);
    float *p;
    for (auto *vec : {&m->W, &m->gW, &m->mW, &m->vW}) {
      if (cudaMalloc(&p, nw * sizeof(float)) != cudaSuccess) return NQG_ERR_CUDA;
      vec->push_back(p);
    }
    for (auto *vec : {&m->b, &m->gb, &m->mb, &m->vb}) {
      if (cudaMalloc(&p, o * sizeof(float)) != cudaSuccess) return NQG_ERR_CUDA;
      vec->push_back(p);
    }
    for (auto [vec, n] : {std::make_pair(&m->Wb, (size_t)o * pad8(in)), std::make_pair(&m->Wt, (size_t)in * pad8(o))}) {
      __nv_bfloat16 *pb;
      if (cudaMalloc(&pb, n * sizeof(__nv_bfloat16)) != cudaSuccess) return NQG_ERR_CUDA;
      vec->push_back(pb);
      if (cudaMemsetAsync(pb, 0, n * sizeof(__nv_bfloat16), m->stream) != cudaSuccess) return NQG_ERR_CUDA;
    }
    cudaMemcpy(m->W[l], w.data(), nw * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(m->b[l], z.data(), o * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(m->mW[l], z.data(), nw * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(m->vW[l], z.data(), nw * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(m->mb[l], z.data(), o * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(m->vb[l], z.data(), o * sizeof(float), cudaMemcpyHostToDevice);
    k_to_bf16<<<blocks_for(nw), 256, 0, m->stream>>>(nw, m->W[l], m->Wb[l], m->Wt[l], o, in);
  }
  if (cudaMalloc(&m->d_loss, sizeof(double)) != cudaSuccess) return NQG_ERR_CUDA;
  // parts > 1 only while parts x tiles <= SM_COUNT
  if (cudaMalloc(&m->d_parts, (size_t)SM_COUNT * MT * 64 * sizeof(float)) != cudaSuccess) return NQG_ERR_CUDA;
  if (cudaHostAlloc(&m->timeout, 2 * sizeof(int), cudaHostAllocDefault) != cudaSuccess) return NQG_ERR_CUDA;
  m->timeout[0] = m->timeout[1] = 0;
  if (cudaStreamSynchronize(m->stream) != cudaSuccess) return NQG_ERR_CUDA;
  *out = m;
  return NQG_OK;
}

extern "C" int nqg_mlp_num_params(const nqg_mlp *m, long *n_weights, long *n_biases) {
  if (!m) return NQG_ERR_ARG;
  long nw = 0, nb = 0;
  for (int l = 0; l < m->L; ++l) {
    nw += (long)m->sizes[l] * m->sizes[l + 1];
    nb += m->sizes[l + 1];
  }
  if (n_weights) *n_weights = nw;
  if (n_biases) *n_biases = nb;
  return NQG_OK;
}

// Host copies of every layer's FP32 master weights (row-major out x in,
// layer after layer) and biases; set also refreshes the BF16 copies and
// restarts the optimizer.
extern "C" int nqg_mlp_set_weights(nqg_mlp *m, const float *w_all, const float *b_all) {
  if (!m || !w_all || !b_all) return NQG_ERR_ARG;
  long ow = 0, ob = 0;
  for (int l = 0; l < m->L; ++l) {
    const long nw = (long)m->sizes[l] * m->sizes[l + 1];
    const int o = m->sizes[l + 1];
    MQ(cudaMemcpy(m->W[l], w_all + ow, nw * sizeof(float), cudaMemcpyHostToDevice));
    MQ(cudaMemcpy(m->b[l], b_all + ob, o * sizeof(float), cudaMemcpyHostToDevice));
    MQ(cudaMemset(m->mW[l], 0, nw * sizeof(float)));
    MQ(cudaMemset(m->vW[l], 0, nw * sizeof(float)));
    MQ(cudaMemset(m->mb[l], 0, o * sizeof(float)));
    MQ(cudaMemset(m->vb[l], 0, o * sizeof(float)));
    k_to_bf16<<<blocks_for(nw), 256, 0, m->stream>>>(nw, m->W[l], m->Wb[l], m->Wt[l], o, m->sizes[l]);
    ow += nw;
    ob += o;
  }
  m->step = 0;
  MQ(cudaStreamSynchronize(m->stream));
  return NQG_OK;
}

extern "C" int nqg_mlp_get_weights(nqg_mlp *m, float *w_all, float *b_all) {
  if (!m) return NQG_ERR_ARG;
  long ow = 0, ob = 0;
  MQ(cudaStreamSynchronize(m->stream));
  for (int l = 0; l < m->L; ++l) {
    const long nw = (long)m->sizes[l] * m->sizes[l + 1];
    const int o = m->sizes[l + 1];
    if (w_all) MQ(cudaMemcpy(w_all + ow, m->W[l], nw * sizeof(float), cudaMemcpyDeviceToHost));
    if (b_all) MQ(cudaMemcpy(b_all + ob, m->b[l], o * sizeof(float), cudaMemcpyDeviceToHost));
    ow += nw;
    ob += o;
  }
  return NQG_OK;
}

// Logits of `rows` inputs (device pointers, row-major), on `stream` (NULL:
// the model's own stream, synchronised before returning).
extern "C" int nqg_mlp_forward_device(nqg_mlp *m, int rows, const float *d_x, float *d_logits, void *stream) {
  if (!m || rows <= 0 || !d_x || !d_logits) return NQG_ERR_ARG;
  int rc = ensure_rows(m, rows);
  if (rc) return rc;
  cudaStream_t st = stream ? (cudaStream_t)stream : m->stream;
  cudaStream_t keep = m->stream;
  m->stream = st;
  forward(m, rows, d_x, d_logits);
  const cudaError_t launched = cudaGetLastError();
  m->stream = keep;
  MQ(launched);
  if (stream) return NQG_OK;
  MQ(cudaStreamSynchronize(st));
  return mma_status(m);
}

extern "C" int nqg_mlp_set_wait_limit(nqg_mlp *m, long long polls) {
  if (!m) return NQG_ERR_ARG;
  m->wait_limit = polls == 0 ? t5::WAIT_LIMIT : std::clamp(polls, 0ll, t5::WAIT_LIMIT);
  return NQG_OK;
}

// What forwards on callers' streams have reported since the last call.
extern "C" int nqg_mlp_stream_status(nqg_mlp *m) { return m ? mma_status(m, 1) : NQG_ERR_ARG; }

// Host-buffer variant of nqg_mlp_forward_device.
extern "C" int nqg_mlp_forward(nqg_mlp *m, int rows, const float *x, float *logits) {
  if (!m || rows <= 0 || !x || !logits) return NQG_ERR_ARG;
  int rc = ensure_rows(m, rows);
  if (rc) return rc;
  MQ(cudaMemcpyAsync(m->act[0], x, (size_t)rows * m->sizes[0] * sizeof(float), cudaMemcpyHostToDevice, m->stream));
  forward(m, rows);
  MQ(cudaMemcpyAsync(logits, m->act[m->L], (size_t)rows * m->sizes[m->L] * sizeof(float), cudaMemcpyDeviceToHost,
                     m->stream));
  MQ(cudaStreamSynchronize(m->stream));
  return mma_status(m);
}

// Loss and gradients of one batch (host buffers): loss = mean over rows of
// the weighted cross-entropy summed over outputs; gradients copied to the
// host (layer after layer, as in nqg_mlp_get_weights) when the pointers are
// non-null.  No optimizer step.
extern "C" int nqg_mlp_loss_grad(nqg_mlp *m, int rows, const float *x, const float *y, float pos_weight,
                                 double *loss, float *gw_all, float *gb_all) {
  if (!m || rows <= 0 || !x || !y) return NQG_ERR_ARG;
  int rc = ensure_rows(m, rows);
  if (rc) return rc;
  const int out = m->sizes[m->L];
  MQ(cudaMemcpyAsync(m->act[0], x, (size_t)rows * m->sizes[0] * sizeof(float), cudaMemcpyHostToDevice, m->stream));
  MQ(cudaMemsetAsync(m->d_loss, 0, sizeof(double), m->stream));
  forward(m, rows);  // runs while the labels are staged
  MQ(cudaMemcpyAsync(m->d_lab, y, (size_t)rows * out * sizeof(float), cudaMemcpyHostToDevice, m->stream));
  const long tot = (long)rows * out;
  k_bce<<<std::min(blocks_for(tot), 2 * SM_COUNT), 256, 0, m->stream>>>(tot, rows, m->act[m->L], m->d_lab, pos_weight, m->dact[m->L],
                                                 m->d_loss);
  backward(m, rows);
  double h = 0.0;
  MQ(cudaMemcpyAsync(&h, m->d_loss, sizeof(double), cudaMemcpyDeviceToHost, m->stream));
  MQ(cudaStreamSynchronize(m->stream));
  if (const int rc = mma_status(m)) return rc;
  if (loss) *loss = h;
  long ow = 0, ob = 0;
  for (int l = 0; l < m->L; ++l) {
    const long nw = (long)m->sizes[l] * m->sizes[l + 1];
    const int o = m->sizes[l + 1];
    if (gw_all) MQ(cudaMemcpy(gw_all + ow, m->gW[l], nw * sizeof(float), cudaMemcpyDeviceToHost));
    if (gb_all) MQ(cudaMemcpy(gb_all + ob, m->gb[l], o * sizeof(float), cudaMemcpyDeviceToHost));
    ow += nw;
    ob += o;
  }
  return NQG_OK;
}

// Training set (host buffers, row-major): n rows of inputs and of 0/1 labels.
extern "C" int nqg_mlp_set_data(nqg_mlp *m, int n, const float *x, const float *y) {
  if (!m || n <= 0 || !x || !y) return NQG_ERR_ARG;
  cudaFree(m->d_X);
  cudaFree(m->d_Y);
  MQ(cudaMalloc(&m->d_X, (size_t)n * m->sizes[0] * sizeof(float)));
  MQ(cudaMalloc(&m->d_Y, (size_t)n * m->sizes[m->L] * sizeof(float)));
  MQ(cudaMemcpy(m->d_X, x, (size_t)n * m->sizes[0] * sizeof(float), cudaMemcpyHostToDevice));
  MQ(cudaMemcpy(m->d_Y, y, (size_t)n * m->sizes[m->L] * sizeof(float), cudaMemcpyHostToDevice));
  m->n_train = n;
  return NQG_OK;
}

// Adam (beta1 0.9, beta2 0.999, eps 1e-8) over shuffled mini-batches of the
// training set; epoch_loss (nullable, `epochs` entries) receives the mean
// mini-batch loss of each epoch.
extern "C" int nqg_mlp_train(nqg_mlp *m, int epochs, int batch, float lr, float pos_weight, unsigned long long seed,
                             double *epoch_loss) {
  if (!m || epochs <= 0 || batch <= 0 || m->n_train <= 0) return NQG_ERR_ARG;
  batch = std::min(batch, m->n_train);
  int rc = ensure_rows(m, batch);
  if (rc) return rc;
  const int in = m->sizes[0], out = m->sizes[m->L];
  std::mt19937_64 rng(seed);
  std::vector<int> perm(m->n_train);
  for (int i = 0; i < m->n_train; ++i) perm[i] = i;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int ep = 0; ep < epochs; ++ep) {
    std::shuffle(perm.begin(), perm.end(), rng);
    MQ(cudaMemsetAsync(m->d_loss, 0, sizeof(double), m->stream));
    int nb = 0;
    for (int s0 = 0; s0 + batch <= m->n_train; s0 += batch, ++nb) {
      MQ(cudaMemcpyAsync(m->d_idx, perm.data() + s0, batch * sizeof(int), cudaMemcpyHostToDevice, m->stream));
      k_gather<<<blocks_for((long)batch * in), 256, 0, m->stream>>>(batch, in, m->d_idx, m->d_X, m->act[0]);
      k_gather<<<blocks_for((long)batch * out), 256, 0, m->stream>>>(batch, out, m->d_idx, m->d_Y, m->d_lab);
      forward(m, batch);
      const long tot = (long)batch * out;
      k_bce<<<std::min(blocks_for(tot), 2 * SM_COUNT), 256, 0, m->stream>>>(tot, batch, m->act[m->L], m->d_lab, pos_weight, m->dact[m->L],
                                                     m->d_loss);
      backward(m, batch);
      m->step++;
      const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
      for (int l = 0; l < m->L; ++l) {
        const long nw = (long)m->sizes[l] * m->sizes[l + 1];
        const int o = m->sizes[l + 1];
        k_adam<<<blocks_for(nw), 256, 0, m->stream>>>(nw, m->W[l], m->Wb[l], m->Wt[l], o, m->sizes[l], m->gW[l], m->mW[l],
                                                        m->vW[l], lr, b1, b2, eps, c1, c2);
        k_adam<<<blocks_for(o), 256, 0, m->stream>>>(o, m->b[l], nullptr, nullptr, o, 1, m->gb[l], m->mb[l], m->vb[l], lr,
                                                       b1, b2, eps, c1, c2);
      }
      // the host index buffer of the next batch must not change before the copy ran
      MQ(cudaStreamSynchronize(m->stream));
    }
    double h = 0.0;
    MQ(cudaMemcpyAsync(&h, m->d_loss, sizeof(double), cudaMemcpyDeviceToHost, m->stream));
    MQ(cudaStreamSynchronize(m->stream));
    if (epoch_loss) epoch_loss[ep] = nb ? h / nb : 0.0;
  }
  MQ(cudaGetLastError());
  return mma_status(m);
}

extern "C" const char *nqg_mlp_last_error(const nqg_mlp *m) { return m ? m->err.c_str() : ""; }

extern "C" int nqg_mlp_destroy(nqg_mlp *m) {
  if (!m) return NQG_ERR_ARG;
  cudaStreamSynchronize(m->stream);
  for (auto *vec : {&m->W, &m->b, &m->gW, &m->gb, &m->mW, &m->vW, &m->mb, &m->vb, &m->act, &m->dact})
    for (float *p : *vec) cudaFree(p);
  for (auto *vec : {&m->Wb, &m->Wt})
    for (auto *p : *vec) cudaFree(p);
  cudaFree(m->d_X);
  cudaFree(m->d_Y);
  cudaFree(m->d_lab);
  cudaFree(m->d_idx);
  cudaFree(m->d_loss);
  cudaFree(m->d_parts);
  if (m->timeout) cudaFreeHost(m->timeout);
  cudaStreamDestroy(m->stream);
  delete m;
  return NQG_OK;
}
