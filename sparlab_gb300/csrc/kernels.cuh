// Device kernels of the AMG-PCG solve: deterministic reductions, CSR
// operator applications with fused smoother epilogues, the Galerkin numeric
// products over node-level patterns, and the PCG vector updates.
//
// Determinism: every reduction has a fixed shape (grid, block, tree), every
// output entry is written by one thread that sums its terms in a fixed order,
// and no value path uses atomics, so results are bitwise reproducible run to
// run.  The setup products sum in exactly the order of the reference's
// multiply/multiply_numeric (src/fem/Multigrid.cpp:121-225) with rounded
// (unfused) multiply-adds, so their FP64 values equal the CPU oracle's.
#pragma once

#include "common.h"

#include <type_traits>

#include <cuda_runtime.h>

namespace simp {

// Scalar column indices of a CSR from its node pattern (defined in amg.cu).
__global__ void k_expand_columns(i32 n, const i32* __restrict__ node_of, NodeView p,
                                 const i32* __restrict__ col_first, const i32* __restrict__ rowptr,
                                 i32* __restrict__ col);

constexpr int kRedBlocks = 1024;   // fixed reduction grid
constexpr int kRedThreads = 256;

// Kernels below have internal linkage: every translation unit instantiates
// the ones it launches.
namespace {
// ---------------------------------------------------------------------------
// exact-order arithmetic (no contraction into FMA)
// ---------------------------------------------------------------------------
__device__ __forceinline__ double xmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double xadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float xmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float xadd(float a, float b) { return __fadd_rn(a, b); }

// Double-float arithmetic (a value is an unevaluated sum hi + lo of two
// floats, about 48 significant bits): Knuth's TwoSum and Dekker's product
// with a fused multiply-add for the exact product error.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// (sh, sl) += (ah + al)(bh + bl), dropping al * bl
__device__ __forceinline__ void df_fma(float ah, float al, float bh, float bl, float& sh, float& sl) {
  const float p = __fmul_rn(ah, bh);
  float pe = __fmaf_rn(ah, bh, -p);
  pe = __fmaf_rn(ah, bl, __fmaf_rn(al, bh, pe));
  float t, e;
  two_sum(sh, p, t, e);
  sh = t;
  sl = __fadd_rn(sl, __fadd_rn(e, pe));
}

// hi = fl32(v), lo = fl32(v - hi), both rounded to nearest even.  Where
// both halves are normal floats (v's exponent field in [949, 1149]: |v| in
// [2^-74, 2^127)), from v's bits with integer operations -- GB300 runs FP64
// conversions and arithmetic at 1/64 of its FP32 rate -- and otherwise by
// FP64 conversion.  The 53-bit significand M splits into its top 24 bits K
// and low 29 bits R; K rounds to nearest even on R (a carry out of K moves
// into the float exponent field), and v - hi is the remainder r = R or
// R - 2^29 in units of 2^(e - 1075), which one int -> float conversion
// rounds to 24 bits and a power of two scales exactly.
__device__ __forceinline__ void df_split(double v, float& hi, float& lo) {
  const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
  const int e = static_cast<int>((u >> 52) & 0x7FFull);
  if (e >= 949 && e <= 1149) {
    const unsigned long long m = (u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    unsigned k = static_cast<unsigned>(m >> 29);
    const int rr = static_cast<int>(m & 0x1FFFFFFFull);
    int r = rr;
    if (rr > 0x10000000 || (rr == 0x10000000 && (k & 1u))) {
      k += 1u;
      r = rr - 0x20000000;
    }
    const bool neg = (u >> 63) != 0;
    const unsigned bits = (static_cast<unsigned>(neg) << 31) | ((static_cast<unsigned>(e - 896) << 23) + (k - 0x800000u));
    hi = __uint_as_float(bits);
    lo = __int2float_rn(neg ? -r : r) * __uint_as_float(static_cast<unsigned>(e - 948) << 23);
    return;
  }
  hi = __double2float_rn(v);
  lo = __double2float_rn(v - static_cast<double>(hi));
}

// hi = float(v) and the interleaved (hi, lo) pairs of the double-float operator
__global__ void k_split_values_pairs(i64 n, const double* __restrict__ v, float* __restrict__ hi,
                                     float2* __restrict__ pair) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    float h, l;
    df_split(v[i], h, l);
    hi[i] = h;
    pair[i] = make_float2(h, l);
  }
}

__global__ void k_split_pairs(i64 n, const double* __restrict__ v, float2* __restrict__ out) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    float h, l;
    df_split(v[i], h, l);
    out[i] = make_float2(h, l);
  }
}

template <class T>
__device__ __forceinline__ double todbl(T v) { return static_cast<double>(v); }

// Block-wide sum of one double per thread (fixed tree), valid in thread 0.
template <int BS>
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double warp_part[BS / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) warp_part[w] = v;
  __syncthreads();
  double s = 0.0;
  if (w == 0) {
    s = l < BS / 32 ? warp_part[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  __syncthreads();
  return s;
}

// First statement of every kernel that chain_launch launches, as
// `if (!chain_start()) return;` (always true: the branch keeps the compiler
// from moving loads that it takes for invariant above the wait).  All threads
// wait here until the previous kernel of the stream has completed and its
// writes are visible; then the next kernel may be scheduled, which waits in
// turn, so completion stays in stream order.  A grid of more than two blocks an
// SM lets the next one in only as its blocks end: earlier, the next grid's
// blocks would fill the slots that happen to be free and the SMs would have
// unequal shares of it (46800 rows, FP64, 731 blocks after 731: a CG iteration
// of 227 us against 181 without any overlap).
constexpr unsigned kChainBlocks = 2 * kSms;
__device__ __forceinline__ bool chain_start() {
  unsigned lane;
  asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, %%laneid;" : "=r"(lane)::"memory");
  if (gridDim.x * gridDim.y * gridDim.z <= kChainBlocks) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  return lane < 32u;
}

// Sum over the grid of one double per block (valid in thread 0): every block
// stores its partial and takes a ticket, and the last one adds the partials in
// order, so the value does not depend on which block that is.  True in that
// block's thread 0, with the total; the ticket is back at zero for the next
// launch.  `also` runs in all threads of that block.
template <class Last>
__device__ __forceinline__ bool grid_sum(double block, double* __restrict__ part, unsigned* __restrict__ ticket,
                                         double& total, Last also) {
  __shared__ int last;
  if (threadIdx.x == 0) {
    part[blockIdx.x] = block;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double s = 0.0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += 256) s += __ldcg(part + i);
  s = block_sum<256>(s);
  also();
  if (threadIdx.x != 0) return false;
  *ticket = 0u;
  total = s;
  return true;
}

__device__ __forceinline__ bool grid_sum(double block, double* __restrict__ part, unsigned* __restrict__ ticket,
                                         double& total) {
  return grid_sum(block, part, ticket, total, [] {});
}

// Sums of K values of every thread over the grid, in one launch and in the
// order in which grid_sum would add each of them: the
// lanes of a warp halve the set of values that they still hold at each step
// (K = 7 costs 9 additions where 7 separate sums cost 35; the FP64 pipe takes
// 16 clocks for each), every block stores its K partials, and a warp of the
// last block adds up a row of partials and stores the total in page-locked
// memory that the host polls.  Blocks of 256 threads; part holds K * gridDim.x.
template <int D>  // K = 2^D - 1 values and a zero
__device__ __forceinline__ void grid_sums_to_host(double (&s)[1 << D], double* __restrict__ part,
                                                  unsigned* __restrict__ ticket, SumPost* host, unsigned seq) {
  constexpr int P = 1 << D, K = P - 1;
  static_assert(K <= SumPost::kValues, "");
  __shared__ double warp_part[P][9];
  __shared__ int last;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int step = 0; step < D; ++step) {
    const int half = P >> (step + 1), off = 16 >> step;
    const bool up = (l & off) != 0;
#pragma unroll
    for (int i = 0; i < P / 2; ++i) {
      if (i >= half) continue;
      const double give = up ? s[i] : s[i + half], keep = up ? s[i + half] : s[i];
      s[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
#pragma unroll
  for (int off = 16 >> D; off > 0; off >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
  if ((l & ((32 >> D) - 1)) == 0) warp_part[l >> (5 - D)][w] = s[0];
  auto of_warps = [](const double* v) { return ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7])); };
  __syncthreads();
  const unsigned nb = gridDim.x;
  if (threadIdx.x < K) {
    part[threadIdx.x * nb + blockIdx.x] = of_warps(warp_part[threadIdx.x]);
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == nb - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int k = w; k < K; k += 8) {
    double v[8] = {};
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (q * 32u >= nb) continue;
      double t = 0.0;
      for (unsigned i = q * 32u + l; i < nb; i += 256) t += __ldcg(part + k * nb + i);
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      v[q] = t;
    }
    if (l == 0) {
      host->v[k] = of_warps(v);
      __threadfence_system();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *ticket = 0u;
    *reinterpret_cast<volatile unsigned*>(&host->seq) = seq;
  }
}

// ---------------------------------------------------------------------------
// elementwise
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_fill(T* __restrict__ x, T v, i64 n) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) x[i] = v;
}

template <class A, class B>
__global__ void k_convert(const A* __restrict__ a, B* __restrict__ b, i64 n) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
    b[i] = static_cast<B>(a[i]);
}

// three unknowns a node: node order (3 I + k) to component planes (k nodes + I) and back
template <class A, class B>
__global__ void k_to_planes(const A* __restrict__ a, B* __restrict__ b, i64 nodes) {
  if (!chain_start()) return;
  for (i64 I = blockIdx.x * (i64)blockDim.x + threadIdx.x; I < nodes; I += (i64)gridDim.x * blockDim.x)
#pragma unroll
    for (int k = 0; k < 3; ++k) b[k * nodes + I] = static_cast<B>(a[3 * I + k]);
}

template <class A, class B>
__global__ void k_from_planes(const A* __restrict__ a, B* __restrict__ b, i64 nodes) {
  if (!chain_start()) return;
  for (i64 I = blockIdx.x * (i64)blockDim.x + threadIdx.x; I < nodes; I += (i64)gridDim.x * blockDim.x)
#pragma unroll
    for (int k = 0; k < 3; ++k) b[3 * I + k] = static_cast<B>(a[k * nodes + I]);
}

// ---------------------------------------------------------------------------
// PCG scalars and vector updates (FP64 CG scalars in device memory).  Each
// reduction is one launch (grid_sum); a CG iteration is the V-cycle and five
// launches: r^T z with beta, the direction, the operator, p^T q with alpha, the
// update.  z is read where the V-cycle left it (its level-0 iterate, FP32 in
// mixed precision) and the update writes the next V-cycle's right-hand side,
// so no pass converts or copies between them.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void post_to_host(const PcgScalars* sc, PcgPost* host) {
  host->rr = sc->rr;
  host->pq = sc->pq;
  host->status = sc->status;
  __threadfence_system();
  *reinterpret_cast<volatile unsigned*>(&host->seq) = sc->seq;
}

// Place of unknown i in a vector in component planes of `nodes` nodes, three
// unknowns a node.
__device__ __forceinline__ i32 plane_of(i32 i, i32 nodes) { return i % 3 * nodes + i / 3; }

// out[0] = a^T b, to the host
__global__ void __launch_bounds__(kRedThreads) k_dot(const double* __restrict__ a, const double* __restrict__ b, i64 n,
                                                     double* __restrict__ part, PcgScalars* sc, PcgPost* host,
                                                     unsigned seq) {
  double s = 0.0;
  for (i64 i = blockIdx.x * (i64)kRedThreads + threadIdx.x; i < n; i += (i64)gridDim.x * kRedThreads) s += a[i] * b[i];
  double total;
  if (grid_sum(block_sum<kRedThreads>(s), part, &sc->ticket, total)) {
    sc->rr = total;
    sc->seq = seq;
    post_to_host(sc, host);
  }
}

// ||r||^2 to the host, the V-cycle's FP32 right-hand side (planes > 0: in
// component planes), and the scalars of a new CG run
__global__ void __launch_bounds__(kRedThreads) k_pcg_begin(const double* __restrict__ r, i32 n, float* __restrict__ b32,
                                                           i32 planes, double* __restrict__ part, PcgScalars* sc,
                                                           PcgPost* host, unsigned seq) {
  if (!chain_start()) return;
  double s = 0.0;
  for (i32 i = blockIdx.x * kRedThreads + threadIdx.x; i < n; i += gridDim.x * kRedThreads) {
    const double ri = r[i];
    s += ri * ri;
    if (b32) b32[planes > 0 ? plane_of(i, planes) : i] = static_cast<float>(ri);
  }
  double total;
  if (grid_sum(block_sum<kRedThreads>(s), part, &sc->ticket, total)) {
    sc->rr = total;
    sc->rz = 0.0;
    sc->status = 0;
    sc->fresh = 1;
    sc->seq = seq;
    post_to_host(sc, host);
  }
}

// r^T z; beta = r^T z / the last one (0 for the first direction)
template <class TZ>
__global__ void __launch_bounds__(kRedThreads) k_pcg_rz(const double* __restrict__ r, const TZ* __restrict__ z, i32 n,
                                                        i32 planes, double* __restrict__ part, PcgScalars* sc) {
  if (!chain_start()) return;
  double s = 0.0;
  for (i32 i = blockIdx.x * kRedThreads + threadIdx.x; i < n; i += gridDim.x * kRedThreads)
    s += r[i] * static_cast<double>(z[planes > 0 ? plane_of(i, planes) : i]);
  double total;
  if (grid_sum(block_sum<kRedThreads>(s), part, &sc->ticket, total)) {
    sc->beta = sc->fresh ? 0.0 : total / sc->rz;
    sc->rz = total;
    sc->fresh = 0;
  }
}

// p = z + beta p (p = z where a run starts); with ps, also its double-float
// split (the operator's input in mixed precision); with p32, its FP32 copy
// (the input of the matrix-free CG operator).  U values a thread, all loads
// before the first use: one a thread is 17 waves of blocks that wait for one
// load each at 5.4 M values (192x96x96's design pass 65.45 -> 64.83 ms).
template <class TZ, int U>
__global__ void __launch_bounds__(256) k_pcg_direction(double* __restrict__ p, const TZ* __restrict__ z, i32 n,
                                                       i32 planes, const PcgScalars* __restrict__ sc,
                                                       float2* __restrict__ ps, float* __restrict__ p32) {
  if (!chain_start()) return;
  const double beta = sc->beta;
  const i64 first = blockIdx.x * static_cast<i64>(256 * U) + threadIdx.x;
  double v[U], old[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const i64 at = first + u * 256;
    v[u] = old[u] = 0.0;
    if (at >= n) continue;
    const i32 i = static_cast<i32>(at);
    v[u] = static_cast<double>(z[planes > 0 ? plane_of(i, planes) : i]);
    if (beta != 0.0) old[u] = p[i];
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const i64 i = first + u * 256;
    if (i >= n) continue;
    if (beta != 0.0) v[u] += beta * old[u];
    p[i] = v[u];
    if (ps) {
      float h, l;
      df_split(v[u], h, l);
      ps[i] = make_float2(h, l);
    }
    if (p32) p32[i] = __double2float_rn(v[u]);
  }
}

// p^T q and alpha
__global__ void __launch_bounds__(kRedThreads) k_pcg_pq(const double* __restrict__ p, const double* __restrict__ q,
                                                        i32 n, double* __restrict__ part, PcgScalars* sc) {
  if (!chain_start()) return;
  double s = 0.0;
  for (i32 i = blockIdx.x * kRedThreads + threadIdx.x; i < n; i += gridDim.x * kRedThreads) s += p[i] * q[i];
  double total;
  if (grid_sum(block_sum<kRedThreads>(s), part, &sc->ticket, total)) {
    sc->pq = total;
    if (!(total > 0.0) || !isfinite(total)) {
      sc->status = 2;
      sc->alpha = 0.0;
    } else {
      sc->alpha = sc->rz / total;
    }
  }
}

// x += alpha p ; r -= alpha q ; ||r||^2 to the host ; r's FP32 copy as the next
// V-cycle's right-hand side
__global__ void __launch_bounds__(kRedThreads) k_pcg_update(double* __restrict__ x, double* __restrict__ r,
                                                            const double* __restrict__ p,
                                                            const double* __restrict__ q, i32 n,
                                                            float* __restrict__ b32, i32 planes,
                                                            double* __restrict__ part, PcgScalars* sc, PcgPost* host) {
  if (!chain_start()) return;
  const double alpha = sc->alpha;
  double s = 0.0;
  for (i32 i = blockIdx.x * kRedThreads + threadIdx.x; i < n; i += gridDim.x * kRedThreads) {
    x[i] += alpha * p[i];
    const double ri = r[i] - alpha * q[i];
    r[i] = ri;
    if (b32) b32[planes > 0 ? plane_of(i, planes) : i] = static_cast<float>(ri);
    s += ri * ri;
  }
  double total;
  if (grid_sum(block_sum<kRedThreads>(s), part, &sc->ticket, total)) {
    sc->rr = total;
    sc->seq += 1u;
    post_to_host(sc, host);
  }
}

// ---------------------------------------------------------------------------
// Chebyshev smoothing (Saad, Alg. 12.1 in D^-1 A; src/fem/Multigrid.cpp:
// 783-855): the operator steps live with the operator kernels (nbspmv.cuh,
// mfree.cuh); the zero-guess start needs no operator.
// ---------------------------------------------------------------------------
// zero guess: d = dinv b / theta ; x = d
template <class TX>
__global__ void k_cheb_zero(i64 n, const TX* __restrict__ b, const TX* __restrict__ dinv,
                            TX* __restrict__ d, TX* __restrict__ x, const TX* __restrict__ inv_theta) {
  if (!chain_start()) return;
  const TX it = *inv_theta;
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    const TX di = dinv[i] * b[i] * it;
    d[i] = di;
    x[i] = di;
  }
}

// x += d
template <class TX>
__global__ void k_add_to(i64 n, const TX* __restrict__ d, TX* __restrict__ x) {
  if (!chain_start()) return;
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) x[i] += d[i];
}

// ---------------------------------------------------------------------------
// Lanczos on S A S, S = D^-1/2 (src/fem/Multigrid.cpp:288-327), two launches a
// step instead of eight: the operator's rows with the step's vector update and
// the partial sums of alpha_j in their epilogue (k_lz_rows, or a matrix-free
// product and k_lz_post), then k_lz_norm; the last block of each adds the
// partials in order.  The vector of a step stays unnormalised: u = beta_{j-1}
// v_j is in w and t = s u is the operator's input, scaled in the rows'
// epilogue, so no pass divides by beta (the first u is the start vector, of
// unit norm, with beta_0 = 1).  FP32 vectors (the mixed-precision reuse setups)
// take FP32 arithmetic with FP64 scalars, and a row's products are added up in
// FP64: GB300 runs FP64 at 1/64 of the FP32 rate, so a block of rows leaves its
// products in shared memory and one warp adds them, 7 FP64 additions a block
// where sums in every warp take 32.
// ---------------------------------------------------------------------------
// Device scalars of a level's Lanczos run (alpha_j and beta_j follow the host's
// order in an array of their own).
struct LzScalars {
  double inv;       // 1 / beta of the last step (1 before the first) ...
  double inv_low;   // ... and what rounding cut off it
  double last;      // that beta
  int stop;         // breakdown: the later steps change nothing
  int bad;          // first non-positive diagonal entry, or kLzGood
  unsigned ticket;  // grid_sum's
  int pad;
};
constexpr int kLzGood = 0x7fffffff;

// Sum in FP64 of the block's row values, which lane 0 of each VS group holds
// (256 threads; valid in thread 0).
template <int VS, class T>
__device__ __forceinline__ double rows_block_sum(T v) {
  constexpr int kRows = 256 / VS;
  __shared__ T row_value[kRows];
  if (threadIdx.x % VS == 0) row_value[threadIdx.x / VS] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = threadIdx.x; k < kRows; k += 32) s += static_cast<double>(row_value[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;
}

// x / beta.  FP64 multiplies by 1 / beta in two parts, which rounds once, as the
// division would; FP32 by the rounded 1 / beta.
struct LzScale {
  double inv, low;
  __device__ __forceinline__ LzScale(const LzScalars& sc) : inv(sc.inv), low(sc.inv_low) {}
  __device__ __forceinline__ float operator()(float x) const { return x * static_cast<float>(inv); }
  __device__ __forceinline__ double operator()(double x) const { return fma(x, inv, x * low); }
};

// u_j and v_{j-1} of row i become w = S A v_j - beta_{j-1} v_{j-1} and v_j, from
// y = (A t)_i; returns w_i v_i.
template <class T>
__device__ __forceinline__ T lz_row(T y, i64 i, const T* __restrict__ s, T* __restrict__ w, T* __restrict__ v,
                                    const LzScale& over_beta, T beta) {
  const T vn = over_beta(w[i]);
  const T wn = over_beta(y) * s[i] - beta * v[i];
  w[i] = wn;
  v[i] = vn;
  return wn * vn;
}

// matrix-free operators: y = A t is a vector
template <class T>
__global__ void __launch_bounds__(kRedThreads) k_lz_post(const T* __restrict__ y, const T* __restrict__ s,
                                                         T* __restrict__ w, T* __restrict__ v, i64 n,
                                                         double* __restrict__ alpha, double* __restrict__ part,
                                                         LzScalars* __restrict__ sc) {
  if (!chain_start()) return;
  if (sc->stop) return;
  const LzScale over_beta(*sc);
  const T beta = static_cast<T>(sc->last);
  T c = T(0);
  for (i64 i = blockIdx.x * (i64)kRedThreads + threadIdx.x; i < n; i += (i64)gridDim.x * kRedThreads)
    c += lz_row(y[i], i, s, w, v, over_beta, beta);
  double total;
  if (grid_sum(block_sum<kRedThreads>(static_cast<double>(c)), part, &sc->ticket, total)) *alpha = total;
}

// w -= alpha_j v, t = s w, beta_j = ||w|| and the reference's breakdown test
// (beta_j <= 1e-12 |alpha_j|); ab = alpha_j, beta_j
template <class T>
__global__ void __launch_bounds__(kRedThreads) k_lz_norm(const T* __restrict__ s, T* __restrict__ w,
                                                         const T* __restrict__ v, T* __restrict__ t, i64 n,
                                                         double* __restrict__ ab, double* __restrict__ part,
                                                         LzScalars* __restrict__ sc) {
  if (!chain_start()) return;
  if (sc->stop) return;
  const T a = static_cast<T>(ab[0]);
  T c = T(0);
  for (i64 i = blockIdx.x * (i64)kRedThreads + threadIdx.x; i < n; i += (i64)gridDim.x * kRedThreads) {
    const T wi = w[i] - a * v[i];
    w[i] = wi;
    t[i] = s[i] * wi;
    c += wi * wi;
  }
  double total;
  if (grid_sum(block_sum<kRedThreads>(static_cast<double>(c)), part, &sc->ticket, total)) {
    const double b = sqrt(total);
    ab[1] = b;
    if (!(b > 1.0e-12 * fabs(ab[0]))) sc->stop = 1;
    const double inv = 1.0 / b;
    sc->last = b;
    sc->inv = inv;
    sc->inv_low = fma(-inv, b, 1.0) * inv;
  }
}

// The scalars before a level's first kernel.
__global__ void k_lz_reset(LzScalars* sc) {
  sc->inv = 1.0;
  sc->inv_low = 0.0;
  sc->last = 1.0;
  sc->stop = 0;
  sc->bad = kLzGood;
  sc->ticket = 0;
}

// Inverse diagonal of a level (1 / a_ii; the first entry that is not positive
// is recorded) and the Lanczos start: s = sqrt(1 / a_ii), w = start, t = s w,
// v = 0.  planes > 0: dinv32, s, w, t and v in component planes of that many
// nodes (three unknowns a node).
template <class T>
__global__ void k_level_start(i32 n, const i32* __restrict__ node_of, const i32* __restrict__ first,
                              const i32* __restrict__ self_slot, NodeView a, const i32* __restrict__ rowptr,
                              const T* __restrict__ val, const double* __restrict__ start, double* __restrict__ dinv,
                              float* __restrict__ dinv32, T* __restrict__ s, T* __restrict__ w, T* __restrict__ t,
                              T* __restrict__ v, i64 planes, LzScalars* __restrict__ sc) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    const i32 I = node_of[i];
    const i32 li = static_cast<i32>(i) - first[I];
    const double d = static_cast<double>(val[rowptr[i] + a.off[self_slot[I]] + li]);
    double inv = 0.0;
    if (!(d > 0.0)) atomicMin(&sc->bad, static_cast<int>(i));
    else inv = 1.0 / d;
    dinv[i] = inv;
    const i64 o = planes > 0 ? (i % 3) * planes + i / 3 : i;
    if (dinv32) dinv32[o] = static_cast<float>(inv);
    const T si = static_cast<T>(sqrt(inv)), wi = static_cast<T>(start[i]);
    s[o] = si;
    w[o] = wi;
    t[o] = si * wi;
    v[o] = T(0);
  }
}

// Chebyshev coefficients and the prolongator's damping into device memory.
struct ChebValues {
  double v[64];
  double omega;
  int count;
};
__global__ void k_set_cheb(const __grid_constant__ ChebValues c, double* __restrict__ c64, float* __restrict__ c32,
                           float* __restrict__ omega) {
  const int k = threadIdx.x;
  if (k < c.count) {
    c64[k] = c.v[k];
    c32[k] = static_cast<float>(c.v[k]);
  }
  if (k == 0) *omega = static_cast<float>(c.omega);
}

// ---------------------------------------------------------------------------
// Setup numerics over node-level patterns
// ---------------------------------------------------------------------------
// Block sums of squares per node-level slot (strength of connection,
// src/fem/Multigrid.cpp:460-513): rows of the row node in order, then the
// slot's columns in order.
__global__ void k_block_sumsq(i32 nnodes, const i32* __restrict__ first, NodeView a,
                              const i32* __restrict__ col_first, const i32* __restrict__ rowptr,
                              const double* __restrict__ val, double* __restrict__ acc) {
  for (i64 I = blockIdx.x * (i64)blockDim.x + threadIdx.x; I < nnodes; I += (i64)gridDim.x * blockDim.x) {
    for (i32 t = a.ptr[I]; t < a.ptr[I + 1]; ++t) {
      const i32 J = a.nbr[t];
      const i32 sz = col_first[J + 1] - col_first[J];
      double s = 0.0;
      for (i32 i = first[I]; i < first[I + 1]; ++i) {
        const double* v = val + rowptr[i] + a.off[t];
        for (i32 k = 0; k < sz; ++k) s = xadd(s, xmul(v[k], v[k]));
      }
      acc[t] = s;
    }
  }
}

// P = (I - omega D^-1 A) P-hat over P's node pattern
// (src/fem/Multigrid.cpp:671-716).  One TPR-lane group per fine row.
template <int TPR, class T>
__global__ void __launch_bounds__(256) k_prolongator(
    i32 n, const i32* __restrict__ node_of, const i32* __restrict__ first,
    const i32* __restrict__ first1, const i32* __restrict__ agg, NodeView a,
    const i32* __restrict__ arow, const T* __restrict__ aval, NodeView p,
    const i32* __restrict__ prow, T* __restrict__ pval, const i32* __restrict__ phat_ptr,
    const T* __restrict__ phat, const double* __restrict__ dinv, double omega) {
  const i64 t0 = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  const i32 i = static_cast<i32>(t0 / TPR);
  const int lane = static_cast<int>(t0 % TPR);
  if (i >= n) return;
  const i32 I = node_of[i];
  const T scale = static_cast<T>(omega * dinv[i]);
  const i32 aI = agg[I];
  for (i32 s = p.ptr[I] + lane; s < p.ptr[I + 1]; s += TPR) {
    const i32 g = p.nbr[s];
    const i32 rg = first1[g + 1] - first1[g];
    T acc[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    for (i32 t = a.ptr[I]; t < a.ptr[I + 1]; ++t) {
      const i32 J = a.nbr[t];
      if (agg[J] != g) continue;
      const i32 sJ = first[J + 1] - first[J];
      const T* av = aval + arow[i] + a.off[t];
      for (i32 kb = 0; kb < sJ; ++kb) {
        const T v = av[kb];
        const T* ph = phat + phat_ptr[first[J] + kb];
#pragma unroll
        for (int j = 0; j < 6; ++j)
          if (j < rg) acc[j] = xadd(acc[j], xmul(v, ph[j]));
      }
    }
    T* out = pval + prow[i] + p.off[s];
    const T* own = phat + phat_ptr[i];
#pragma unroll
    for (int j = 0; j < 6; ++j)
      if (j < rg) {
        T v = xmul(acc[j], -scale);
        if (aI == g) v = xadd(v, own[j]);
        out[j] = v;
      }
  }
}

// R = P^T refill: R(c, (I, ka)) = P((I, ka), c)
template <int TPR, class T>
__global__ void __launch_bounds__(256) k_restriction(
    i32 nc, const i32* __restrict__ node_of1, const i32* __restrict__ first1,
    const i32* __restrict__ first, NodeView r, const i32* __restrict__ rrow, T* __restrict__ rval,
    const i32* __restrict__ r_to_p, NodeView p, const i32* __restrict__ prow,
    const T* __restrict__ pval) {
  const i64 t0 = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  const i32 c = static_cast<i32>(t0 / TPR);
  const int lane = static_cast<int>(t0 % TPR);
  if (c >= nc) return;
  const i32 g = node_of1[c];
  const i32 lc = c - first1[g];
  for (i32 t = r.ptr[g] + lane; t < r.ptr[g + 1]; t += TPR) {
    const i32 I = r.nbr[t];
    const i32 u = r_to_p[t];
    T* out = rval + rrow[c] + r.off[t];
    for (i32 ka = 0; ka < first[I + 1] - first[I]; ++ka) out[ka] = pval[prow[first[I] + ka] + p.off[u] + lc];
  }
}

// AP = A P over AP's node pattern (multiply_numeric order).
template <int TPR, class T>
__global__ void __launch_bounds__(256) k_product_ap(
    i32 n, const i32* __restrict__ node_of, const i32* __restrict__ first,
    const i32* __restrict__ first1, NodeView a, const i32* __restrict__ arow,
    const T* __restrict__ aval, NodeView p, const i32* __restrict__ prow,
    const T* __restrict__ pval, NodeView ap, const i32* __restrict__ aprow, T* __restrict__ apval) {
  const i64 t0 = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  const i32 i = static_cast<i32>(t0 / TPR);
  const int lane = static_cast<int>(t0 % TPR);
  if (i >= n) return;
  const i32 I = node_of[i];
  for (i32 s = ap.ptr[I] + lane; s < ap.ptr[I + 1]; s += TPR) {
    const i32 h = ap.nbr[s];
    const i32 rh = first1[h + 1] - first1[h];
    T acc[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    for (i32 t = a.ptr[I]; t < a.ptr[I + 1]; ++t) {
      const i32 J = a.nbr[t];
      i32 u = p.ptr[J];
      const i32 ue = p.ptr[J + 1];
      while (u < ue && p.nbr[u] < h) ++u;
      if (u == ue || p.nbr[u] != h) continue;
      const i32 sJ = first[J + 1] - first[J];
      const T* av = aval + arow[i] + a.off[t];
      for (i32 kb = 0; kb < sJ; ++kb) {
        const T v = av[kb];
        const T* pv = pval + prow[first[J] + kb] + p.off[u];
#pragma unroll
        for (int j = 0; j < 6; ++j)
          if (j < rh) acc[j] = xadd(acc[j], xmul(v, pv[j]));
      }
    }
    T* out = apval + aprow[i] + ap.off[s];
#pragma unroll
    for (int j = 0; j < 6; ++j)
      if (j < rh) out[j] = acc[j];
  }
}

// RAW = R (AP) over the coarse node pattern (multiply_numeric order).
template <int TPR, class T>
__global__ void __launch_bounds__(256) k_product_rap(
    i32 nc, const i32* __restrict__ node_of1, const i32* __restrict__ first1,
    const i32* __restrict__ first, NodeView r, const i32* __restrict__ rrow,
    const T* __restrict__ rval, NodeView ap, const i32* __restrict__ aprow,
    const T* __restrict__ apval, NodeView c, const i32* __restrict__ crow, T* __restrict__ cval) {
  const i64 t0 = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  const i32 row = static_cast<i32>(t0 / TPR);
  const int lane = static_cast<int>(t0 % TPR);
  if (row >= nc) return;
  const i32 g = node_of1[row];
  for (i32 s = c.ptr[g] + lane; s < c.ptr[g + 1]; s += TPR) {
    const i32 h = c.nbr[s];
    const i32 rh = first1[h + 1] - first1[h];
    T acc[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    for (i32 t = r.ptr[g]; t < r.ptr[g + 1]; ++t) {
      const i32 I = r.nbr[t];
      i32 u = ap.ptr[I];
      const i32 ue = ap.ptr[I + 1];
      while (u < ue && ap.nbr[u] < h) ++u;
      if (u == ue || ap.nbr[u] != h) continue;
      const i32 sI = first[I + 1] - first[I];
      const T* rv = rval + rrow[row] + r.off[t];
      for (i32 ka = 0; ka < sI; ++ka) {
        const T v = rv[ka];
        const T* apv = apval + aprow[first[I] + ka] + ap.off[u];
#pragma unroll
        for (int j = 0; j < 6; ++j)
          if (j < rh) acc[j] = xadd(acc[j], xmul(v, apv[j]));
      }
    }
    T* out = cval + crow[row] + c.off[s];
#pragma unroll
    for (int j = 0; j < 6; ++j)
      if (j < rh) out[j] = acc[j];
  }
}

// A_c = (RAW + RAW^T) / 2 on the (structurally symmetric) coarse pattern: a
// warp a row, a lane a slot (a thread a row was a serial walk of strided reads:
// 0.95 -> 0.34 ms for 26136 nodes of six unknowns, 94 -> 10 us for 127).
template <class T, class TO>
__global__ void k_symmetrize(i32 nc, const i32* __restrict__ node_of1, const i32* __restrict__ first1,
                             NodeView c, const i32* __restrict__ crow, const i32* __restrict__ tslot,
                             const T* __restrict__ raw, TO* __restrict__ out, double* __restrict__ out64) {
  const int lane = threadIdx.x & 31;
  for (i64 row = (blockIdx.x * (i64)blockDim.x + threadIdx.x) >> 5; row < nc;
       row += ((i64)gridDim.x * blockDim.x) >> 5) {
    const i32 g = node_of1[row];
    const i32 lc = static_cast<i32>(row) - first1[g];
    for (i32 s = c.ptr[g] + lane; s < c.ptr[g + 1]; s += 32) {
      const i32 h = c.nbr[s];
      const i32 st = tslot[s];
      const i32 base = crow[row] + c.off[s];
      for (i32 j = 0; j < first1[h + 1] - first1[h]; ++j) {
        const T a = raw[base + j];
        const T b = raw[crow[first1[h] + j] + c.off[st] + lc];
        const T v = xmul(T(0.5), xadd(a, b));
        out[base + j] = static_cast<TO>(v);
        if (out64) out64[base + j] = static_cast<double>(v);
      }
    }
  }
}

}  // namespace
}  // namespace simp
