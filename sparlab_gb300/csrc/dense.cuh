// Coarsest-level direct solve in FP64 (src/fem/Multigrid.cpp:749-781, 859-865).
// The reference factors the dense coarse operator (LDL^T) and runs two
// triangular sweeps per V-cycle.  Here the SPD coarse operator is inverted
// once per setup by a blocked symmetric sweep (Gauss-Jordan elimination
// without pivoting, which is stable for SPD matrices because every pivot is a
// Schur complement's diagonal), and a V-cycle's coarse solve is one GEMV.
//
// Sweeping pivot block k of a symmetric M (P = M_kk^-1, U = M_{:,k}, V = U P):
//   M_ij <- M_ij - V_i U_j^T   (i, j outside k)
//   M_ik <- V_i,  M_kj <- V_j^T,  M_kk <- -P
// After all blocks M = -A^-1.  Only the lower triangle is stored and updated
// (GB300's FP64 rate makes the halved update worth the bookkeeping).  The
// scalar pivots met inside the pivot blocks are the squared Cholesky pivots
// (the D of A = L D L^T), recorded for the singularity check.
// Row-major n x n storage.
//
// The same sweep inverts the indefinite shifted pencil K - sigma G of the
// buckling spectral transformation (SIGNED pivots: any nonzero finite pivot
// is taken).  Its pivots are then the D of A = L D L^T in the natural order,
// so by Sylvester's law of inertia the count of negative pivots is the count
// of negative eigenvalues whenever no leading minor vanishes -- the number
// src/fem/Buckling.cpp:190-201 reads off its sparse LDL^T.
#pragma once

#include "common.h"
#include "kernels.cuh"

#include <algorithm>

namespace simp {
namespace {

constexpr int kNB = 32;         // pivot block width
constexpr int kSweepRows = 4;   // rows of U and V per block of k_sweep_panel, one a warp
constexpr int kTileRows = 16;   // rows of an update tile (kNB columns)

// What a sweep costs: n^2 / 2 x 32 FMA a pivot block at GB300's two FP64 FMA a
// clock and SM (22 us at n = 864), and the serial chain through a pivot block,
// 32 dependent divides.  A pivot block therefore takes two launches: the panel
// (U and V = U P), and the update, whose first block updates the NEXT pivot
// block's tile ahead of everything else and sweeps it while the other blocks
// work through the triangle, so that the chain runs beside the update instead
// of before it (a 32 x 16 x 8 Hex8 design pass in FP64: 9.04 -> 6.73 ms a
// pass with the same bits; before, every panel block repeated the chain, 40 us
// a pivot block, ahead of a 38 us update).

// Sweeps the kb x kb block in s (identity outside) into its negative inverse
// -P, and writes P, the pivots and the status.  Warp w keeps rows 4w .. 4w + 3
// in registers, lane = column; the warp that owns the next pivot row updates
// that row first and publishes it with its divide, so a pivot costs one
// barrier and one divide instead of two barriers around shared-memory sweeps.
template <bool SIGNED>
__device__ void sweep_pivot_block(const double (*s)[kNB + 1], int kb, double* __restrict__ pout,
                                  double* __restrict__ piv, int* __restrict__ status) {
  __shared__ double urow[2][kNB], trow[2][kNB], pj[2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double a[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) a[q] = s[4 * warp + q][lane];
  auto publish = [&](int j, double x) {
    const double d = __shfl_sync(0xffffffffu, x, j);
    const bool ok = (SIGNED ? d != 0.0 : d > 0.0) && isfinite(d);
    const double p = ok ? 1.0 / d : 1.0;
    urow[j & 1][lane] = x;
    trow[j & 1][lane] = p * x;
    if (lane == 0) {
      pj[j & 1] = p;
      piv[j] = d;
      if (!ok) *status = 1;
    }
  };
  if (warp == 0) publish(0, a[0]);
  __syncthreads();
  for (int jw = 0; 4 * jw < kb; ++jw) {
#pragma unroll
    for (int jq = 0; jq < 4; ++jq) {
      const int j = 4 * jw + jq;
      if (j >= kb) break;
      const double* ur = urow[j & 1];
      const double* tr = trow[j & 1];
      const double tc = tr[lane], p = pj[j & 1];
      auto update = [&](int q) {
        const int r = 4 * warp + q;
        if (r == j) a[q] = lane == j ? -p : tc;
        else a[q] = lane == j ? tr[r] : fma(-ur[r], tc, a[q]);
      };
      constexpr int nq_of[4] = {1, 2, 3, 0};
      const int nq = nq_of[jq];
      update(nq);
      if (warp == (jq == 3 ? jw + 1 : jw) && j + 1 < kb) publish(j + 1, a[nq]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q != nq) update(q);
      __syncthreads();
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) pout[(4 * warp + q) * kNB + lane] = -a[q];
}

// P and the pivots of the first pivot block (one block of 256 threads).
template <bool SIGNED>
__global__ void __launch_bounds__(256) k_sweep_first(const double* __restrict__ m, int n, int kb,
                                                     double* __restrict__ pout, double* __restrict__ piv,
                                                     int* __restrict__ status) {
  if (!chain_start()) return;
  __shared__ double s[kNB][kNB + 1];
  for (int e = threadIdx.x; e < kNB * kNB; e += blockDim.x) {
    const int r = e / kNB, c = e % kNB;
    s[r][c] = r < kb && c < kb ? m[(size_t)max(r, c) * n + min(r, c)] : r == c ? 1.0 : 0.0;
  }
  __syncthreads();
  sweep_pivot_block<SIGNED>(s, kb, pout, piv, status);
}

// U_i = M[i, k0:k0+kb] and V_i = U_i P for the rows i outside the pivot block,
// one row a warp (n / 4 blocks, so that the FP64 pipes of all SMs share them).
__global__ void __launch_bounds__(32 * kSweepRows) k_sweep_panel(const double* __restrict__ m, int n, int k0, int kb,
                                                                 const double* __restrict__ p,
                                                                 double* __restrict__ u, double* __restrict__ v) {
  if (!chain_start()) return;
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * kSweepRows + (threadIdx.x >> 5);
  if (i >= n || (i >= k0 && i < k0 + kb)) return;
  double pc[kNB];
#pragma unroll
  for (int d = 0; d < kNB; ++d) pc[d] = p[d * kNB + lane];
  double ui = 0.0;
  if (lane < kb) ui = i >= k0 + kb ? m[(size_t)i * n + k0 + lane] : m[(size_t)(k0 + lane) * n + i];
  double acc = 0.0;
#pragma unroll
  for (int d = 0; d < kNB; ++d) acc = fma(__shfl_sync(0xffffffffu, ui, d), pc[d], acc);
  if (lane < kb) {
    u[(size_t)i * kNB + lane] = ui;
    v[(size_t)i * kNB + lane] = acc;
  }
}

// The update of pivot block k0 over the lower triangle, 16 x 32 per block (a
// 32-row tile leaves the last SM's third tile as the tail at n = 864: 26 us of
// FP64 pipe against 21), a grid of nt x (2 nt + 1) blocks; those above the
// diagonal return at once.  Reads only U, V, P and its own tile.  Row 0 of the
// grid is the block that prepares the next pivot block (see above): the lower
// half of its 32 x 32 tile, mirrored, swept in place into pnext.
template <bool SIGNED>
__global__ void __launch_bounds__(256) k_sweep_update(double* __restrict__ m, int n, int k0, int kb,
                                                      const double* __restrict__ u,
                                                      const double* __restrict__ v,
                                                      const double* __restrict__ p, double* __restrict__ pnext,
                                                      double* __restrict__ piv, int* __restrict__ status) {
  if (!chain_start()) return;
  const int kt = k0 / kNB;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  __shared__ double vs[kNB][kNB + 1];
  __shared__ double us[kNB][kNB + 1];
  __shared__ double s[kNB][kNB + 1];
  if (blockIdx.y == 0) {
    const int k1 = k0 + kNB, kb1 = min(kNB, n - k1);
    if (blockIdx.x != 0 || kb1 <= 0) return;
    for (int q = ty; q < kNB; q += 8) {
      vs[q][tx] = q < kb1 ? v[(size_t)(k1 + q) * kNB + tx] : 0.0;
      us[q][tx] = q < kb1 ? u[(size_t)(k1 + q) * kNB + tx] : 0.0;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kNB * (kNB + 1) / 2; e += 256) {
      int r = static_cast<int>((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
      if ((r + 1) * (r + 2) / 2 <= e) ++r;
      if (r * (r + 1) / 2 > e) --r;
      const int c = e - r * (r + 1) / 2;
      double x = r == c ? 1.0 : 0.0;
      if (r < kb1) {
        x = m[(size_t)(k1 + r) * n + k1 + c];
        double acc = 0.0;
#pragma unroll
        for (int d = 0; d < kNB; ++d) acc = fma(vs[r][d], us[c][d], acc);
        x -= acc;
      }
      s[r][c] = x;
      s[c][r] = x;
    }
    __syncthreads();
    sweep_pivot_block<SIGNED>(s, kb1, pnext, piv + k1, status);
    return;
  }
  const int half = (blockIdx.y - 1) & 1, ti = (blockIdx.y - 1) >> 1, tj = blockIdx.x;
  if (tj > ti || (ti == kt + 1 && tj == ti)) return;  // the next pivot block's tile is overwritten unread
  const int r0 = ti * kNB + half * kTileRows, c0 = tj * kNB;
  if (ti == kt && tj == kt) {
    for (int q = half * kTileRows + ty; q < (half + 1) * kTileRows; q += 8)
      if (q < kb && tx < kb) m[(size_t)(k0 + q) * n + k0 + tx] = -p[q * kNB + tx];
    return;
  }
  if (ti == kt) {  // M_kj <- V_j^T for the columns j of tile J
    for (int q = ty; q < kNB; q += 8) {
      const int j = c0 + q;
      vs[q][tx] = (j < n && tx < kb) ? v[(size_t)j * kNB + tx] : 0.0;
    }
    __syncthreads();
    for (int q = half * kTileRows + ty; q < min(kb, (half + 1) * kTileRows); q += 8)
      if (c0 + tx < n) m[(size_t)(k0 + q) * n + c0 + tx] = vs[tx][q];
    return;
  }
  if (tj == kt) {  // M_ik <- V_i for the rows i of tile I
    for (int q = ty; q < kTileRows; q += 8) {
      const int i = r0 + q;
      if (i < n && tx < kb) m[(size_t)i * n + k0 + tx] = v[(size_t)i * kNB + tx];
    }
    return;
  }
  const int j = c0 + tx;
  double old[kTileRows / 8];
#pragma unroll
  for (int qq = 0; qq < kTileRows / 8; ++qq) {
    const int i = r0 + ty + 8 * qq;
    old[qq] = i < n && j <= i ? m[(size_t)i * n + j] : 0.0;
  }
  for (int q = ty; q < kNB; q += 8) {
    const int i = r0 + q, jj = c0 + q;
    if (q < kTileRows) vs[q][tx] = (i < n && tx < kb) ? v[(size_t)i * kNB + tx] : 0.0;
    us[q][tx] = (jj < n && tx < kb) ? u[(size_t)jj * kNB + tx] : 0.0;
  }
  __syncthreads();
  double acc[kTileRows / 8] = {};
#pragma unroll
  for (int d = 0; d < kNB; ++d) {
    const double uj = us[tx][d];
#pragma unroll
    for (int qq = 0; qq < kTileRows / 8; ++qq) acc[qq] = fma(vs[ty + 8 * qq][d], uj, acc[qq]);
  }
#pragma unroll
  for (int qq = 0; qq < kTileRows / 8; ++qq) {
    const int i = r0 + ty + 8 * qq;
    if (i < n && j <= i) m[(size_t)i * n + j] = old[qq] - acc[qq];
  }
}

// Doubles of the panel workspace of dense_sweep: U, V and two P.
inline size_t sweep_panel_size(int n) { return 2 * static_cast<size_t>(n) * kNB + 2 * kNB * kNB; }

// M (lower triangle) -> -A^-1 with its n scalar pivots; *status, zeroed by the
// caller, becomes 1 on a pivot that is not positive and finite (SIGNED: zero
// or not finite).
template <bool SIGNED>
void dense_sweep(double* m, int n, double* panel, double* piv, int* status, cudaStream_t stream) {
  double* u = panel;
  double* v = u + static_cast<size_t>(n) * kNB;
  double* p[2] = {v + static_cast<size_t>(n) * kNB, v + static_cast<size_t>(n) * kNB + kNB * kNB};
  const int nt = (n + kNB - 1) / kNB;
  chain_launch(k_sweep_first<SIGNED>, 1, 256, 0, stream, m, n, std::min(kNB, n), p[0], piv, status);
  SIMP_CHECK_LAUNCH();
  for (int k0 = 0; k0 < n; k0 += kNB) {
    const int kb = std::min(kNB, n - k0), b = (k0 / kNB) & 1;
    chain_launch(k_sweep_panel, (n + kSweepRows - 1) / kSweepRows, 32 * kSweepRows, 0, stream, m, n, k0, kb, p[b], u, v);
    SIMP_CHECK_LAUNCH();
    chain_launch(k_sweep_update<SIGNED>, dim3(nt, 2 * nt + 1), 256, 0, stream, m, n, k0, kb, u, v, p[b], p[b ^ 1], piv, status);
    SIMP_CHECK_LAUNCH();
  }
}

// F = -M mirrored from the lower triangle to full storage: one 32 x 32 tile
// (I, J), J <= I, per block, written to (I, J) and (J, I).
__global__ void __launch_bounds__(256) k_sweep_finish(const double* __restrict__ m, double* __restrict__ f,
                                                      int n) {
  if (!chain_start()) return;
  const int ti = blockIdx.y, tj = blockIdx.x;
  if (tj > ti) return;
  const int r0 = ti * kNB, c0 = tj * kNB;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  __shared__ double t[kNB][kNB + 1];
  for (int q = ty; q < kNB; q += 8) {
    const int i = r0 + q, j = c0 + tx;
    t[q][tx] = (i < n && j < n && (ti != tj || j <= i)) ? -m[(size_t)i * n + j] : 0.0;
  }
  __syncthreads();
  for (int q = ty; q < kNB; q += 8) {
    const int i = r0 + q, j = c0 + tx;
    if (i < n && j < n) f[(size_t)i * n + j] = ti != tj || tx <= q ? t[q][tx] : t[tx][q];
    if (ti != tj) {
      const int i2 = c0 + q, j2 = r0 + tx;
      if (i2 < n && j2 < n) f[(size_t)i2 * n + j2] = t[tx][q];
    }
  }
}

// y = M x for row-major M, one warp per row.
template <class TX, class TY>
__global__ void __launch_bounds__(256) k_gemv(const double* __restrict__ m, int n, const TX* __restrict__ x,
                                              TY* __restrict__ y) {
  if (!chain_start()) return;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n) return;
  const double* row = m + (size_t)warp * n;
  double s = 0.0;
  for (int c = lane; c < n; c += 32) s += row[c] * static_cast<double>(x[c]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) y[warp] = static_cast<TY>(s);
}

// one warp a row
__global__ void k_dense_from_csr(int n, const i32* __restrict__ ptr, const i32* __restrict__ col,
                                 const double* __restrict__ val, double* __restrict__ a) {
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += (gridDim.x * blockDim.x) >> 5)
    for (i32 k = ptr[r] + (threadIdx.x & 31); k < ptr[r + 1]; k += 32) a[(size_t)r * n + col[k]] = val[k];
}

// a = K - s G densely, K and G on the same CSR pattern (a zeroed before).
__global__ void k_dense_shifted(int n, const i32* __restrict__ ptr, const i32* __restrict__ col,
                                const double* __restrict__ kval, const double* __restrict__ gval, double s,
                                double* __restrict__ a) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    for (i32 k = ptr[r]; k < ptr[r + 1]; ++k) a[(size_t)r * n + col[k]] = kval[k] - s * gval[k];
}

// Z = F Y for a row-major n x n F and column-major n x q Y, Z: one 32 x 32
// tile (rows i0.., columns c0..) per block of 256 threads, the inner index
// staged 32 at a time; every output sums its terms in ascending inner order.
__global__ void __launch_bounds__(256) k_dense_gemm_cols(const double* __restrict__ f, int n, int q,
                                                         const double* __restrict__ y, double* __restrict__ z) {
  __shared__ double fs[kNB][kNB + 1];  // fs[i][k] = F[i0 + i][k0 + k]
  __shared__ double ys[kNB][kNB + 1];  // ys[c][k] = Y[k0 + k][c0 + c]
  const int i0 = blockIdx.x * kNB, c0 = blockIdx.y * kNB;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double acc[kNB / 8] = {};
  for (int k0 = 0; k0 < n; k0 += kNB) {
    for (int q2 = ty; q2 < kNB; q2 += 8) {
      const int i = i0 + q2, k = k0 + tx, c = c0 + q2;
      fs[q2][tx] = (i < n && k < n) ? f[(size_t)i * n + k] : 0.0;
      ys[q2][tx] = (c < q && k < n) ? y[(size_t)c * n + k] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int qq = 0; qq < kNB / 8; ++qq) {
      const int c = ty + 8 * qq;
      double a = acc[qq];
#pragma unroll 8
      for (int k = 0; k < kNB; ++k) a = fma(fs[tx][k], ys[c][k], a);
      acc[qq] = a;
    }
    __syncthreads();
  }
#pragma unroll
  for (int qq = 0; qq < kNB / 8; ++qq) {
    const int i = i0 + tx, c = c0 + ty + 8 * qq;
    if (i < n && c < q) z[(size_t)c * n + i] = acc[qq];
  }
}

}  // namespace
}  // namespace simp
