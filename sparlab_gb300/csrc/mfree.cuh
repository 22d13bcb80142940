// Matrix-free level-0 operator of a structured Q4 / Hex8 grid (FP32).
//
// y_I = sum over the cells e around node I of s_e sum_J K_e^0(I, J) x_J, with
// one thread per free node gathering its (at most 8) cells: every output is
// written once, no atomics, and the result does not depend on the launch
// shape.  The 8 (4) cells around a node are visited in a fixed order, so all
// threads of a warp read the same K_e^0 rows at the same time (a broadcast
// from shared memory).  Used where every node is either fully free or fully
// clamped (the free DOFs of node I are 3I', 3I'+1, 3I'+2 for its free index
// I'); the assembled operator is used otherwise.
#pragma once

#include "kernels.cuh"

namespace simp {
namespace {

struct MfView {
  i32 nx, ny, nz;      // cells (nz = 1 in 2-D)
  i32 nnx, nny;        // nodes per axis in x, y
  const i32* nindex;   // grid node -> free node or -1
  const float* scale;  // s_e
};

// ---------------------------------------------------------------------------
// 2-D operator: one thread per grid node (32 x 4 nodes a block), K_e^0 a
// kernel parameter indexed by compile-time constants.  Every index, then every
// value and scale of the 3 x 3 neighbourhood is loaded before the first
// product: two load latencies a thread, which bound the kernel at the sizes of
// 2-D problems (against a loop over cells and corners with a division-decoded
// node index, 11.6 us a Chebyshev step at 120x40 cells, a SIMP iteration went
// from 4.85 to 4.27 ms there and from 10.6 to 9.4 ms at 600x200 with three load
// cases; the products and their order are the same).  Modes as in k_mf3_tile:
// 0 y = A x, 1 y = b - A x, 3 Chebyshev step, 4 Chebyshev first step.
// ---------------------------------------------------------------------------
struct KeQ4 {
  float k[8 * 8];  // K_e^0, row-major
};

template <int MODE>
__global__ void __launch_bounds__(128) k_mf2(MfView m, const float* __restrict__ x, float* __restrict__ y,
                                             const float* b, float* r, float* __restrict__ dn, float* xs,
                                             const float* __restrict__ dinv, const float* __restrict__ coef, int add_d,
                                             const __grid_constant__ KeQ4 ke) {
  if (!chain_start()) return;
  const i32 across = (m.nnx + 31) / 32;  // blocks of a row of blocks
  const i32 ix = blockIdx.x % across * 32 + (threadIdx.x & 31), iy = blockIdx.x / across * 4 + (threadIdx.x >> 5);
  if (ix >= m.nnx || iy >= m.nny) return;
  i32 J[3][3];
  float s[2][2];
#pragma unroll
  for (int v = 0; v < 3; ++v)
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const i32 jx = ix + u - 1, jy = iy + v - 1;
      J[v][u] = jx >= 0 && jx < m.nnx && jy >= 0 && jy < m.nny ? m.nindex[static_cast<i64>(jy) * m.nnx + jx] : -1;
    }
#pragma unroll
  for (int v = 0; v < 2; ++v)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const i32 cx = ix + u - 1, cy = iy + v - 1;
      s[v][u] = cx >= 0 && cx < m.nx && cy >= 0 && cy < m.ny ? m.scale[static_cast<i64>(cy) * m.nx + cx] : 0.0f;
    }
  const i32 I = J[1][1];
  if (I < 0) return;
  float2 xv[3][3];
#pragma unroll
  for (int v = 0; v < 3; ++v)
#pragma unroll
    for (int u = 0; u < 3; ++u)
      xv[v][u] = J[v][u] >= 0 ? reinterpret_cast<const float2*>(x)[J[v][u]] : make_float2(0.0f, 0.0f);
  // the epilogue's operands are in flight during the products
  const i64 row = 2 * static_cast<i64>(I);
  float bi[2] = {}, di[2] = {}, xi[2] = {}, c0 = 0.0f, c1 = 0.0f;
  if (MODE != 0) {
    bi[0] = b[row];
    bi[1] = b[row + 1];
  }
  if (MODE == 3 || MODE == 4) {
    di[0] = dinv[row];
    di[1] = dinv[row + 1];
    c0 = coef[0];
  }
  if (MODE == 3) {
    c1 = coef[1];
    xi[0] = xs[row];
    xi[1] = xs[row + 1];
  }
  float out[2] = {0.0f, 0.0f};
#pragma unroll
  for (int v = 0; v < 2; ++v)
#pragma unroll
    for (int u = 0; u < 2; ++u) {  // cell (ix + u - 1, iy + v - 1); this node is its corner (1 - u, 1 - v)
      const int ox = 1 - u, oy = 1 - v, a = oy ? 3 - ox : ox;
      float acc[2] = {0.0f, 0.0f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int bx = c == 1 || c == 2, by = c >= 2;
        const float2 t = xv[v + by][u + bx];
#pragma unroll
        for (int k = 0; k < 2; ++k)
          acc[k] = fmaf(ke.k[(2 * a + k) * 8 + 2 * c + 1], t.y, fmaf(ke.k[(2 * a + k) * 8 + 2 * c], t.x, acc[k]));
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) out[k] = fmaf(s[v][u], acc[k], out[k]);
    }
  const float self[2] = {xv[1][1].x, xv[1][1].y};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (MODE == 0) {
      y[row + k] = out[k];
    } else if (MODE == 1) {
      y[row + k] = bi[k] - out[k];
    } else {
      const float ri = bi[k] - out[k];
      r[row + k] = ri;
      if (MODE == 4) {
        dn[row + k] = di[k] * ri * c0;
      } else {
        const float dv = c0 * self[k] + c1 * di[k] * ri;
        dn[row + k] = dv;
        xs[row + k] = (add_d ? xi[k] + self[k] : xi[k]) + dv;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Tiled 3-D variant: a block of 32 x 4 x 2 threads owns a 32 x 4 x (2 kNZ)
// tile of grid nodes (kNZ node layers per thread; two layers per thread
// measured slower at 192 x 96 x 96, 109 against 105 us); the tile's node
// values plus a one-node halo (one shared array per component) and the
// scales of the cells that touch it are staged in shared memory once (see
// MfHalo for the node values' layouts).  Each thread sums
// the 64 (cell, corner) 3 x 3 block products with K_e^0 taken from the kernel
// parameter (a __grid_constant__ struct indexed by compile-time constants,
// so its entries are constant-bank operands of the FMAs rather than loads).
// Modes: 0 y = A x, 1 y = b - A x, 3 Chebyshev step, 4 Chebyshev first step
// (same epilogues as the other operator kernels); and the pieces of the
// smoothed-prolongator transfers P = (I - w D^-1 A) P^ applied without P:
// 5 x_s += t - w D^-1 A t (t = P^ x_c, the input), 6 y = b - A x with
// dn = D^-1 y, 7 y = b - w A x (x = D^-1 r, b = r: the vector P^T maps to
// the coarse right-hand side); 8 y64 = A x in FP64 storage (the FP32 product
// as the CG operator of the matrix-free variant).
// ---------------------------------------------------------------------------
constexpr int kTX = 32, kTY = 4, kTZ = 2;  // threads per block axis (the default tile)
constexpr int kNZ = 1;                      // node layers per thread
// Tile shapes the launch-shape tuner chooses among (TX x TY x TZ threads,
// one node each), each with both halo layouts (variant v: shape v % 5, the
// float4 layout for v >= 5): every variant sums each node's cells and
// corners in the same order, so all give the same values bit for bit.
constexpr int kMfTiles = 10;
constexpr int kMfTileShape[5][3] = {{32, 4, 2}, {32, 8, 1}, {32, 2, 4}, {64, 2, 2}, {32, 4, 1}};

struct KeF32 {
  float k[24 * 24];  // K_e^0, row-major
};

struct MfArgs {
  const float* x;     // input (d for the Chebyshev step)
  float* y;           // mode 0/1: output
  const float* b;     // mode 1/4: right-hand side; mode 3: r_in
  float* r;           // mode 3/4: residual out
  float* dn;          // mode 3: new direction; mode 4: d out
  float* xs;          // mode 3: smoothed iterate (updated)
  const float* dinv;  // mode 3/4/5/6
  const float* coef;  // mode 3: (c1, c2); mode 4: 1 / theta; mode 5/7: w (device memory)
  int add_d;
  double* y64;        // mode 8: output
  i32 nodes;          // free nodes (stride of the component planes)
};

// Unknown (node I, component k) of a level-0 vector: node by node, or (SOA)
// in component planes, as a plane's base (the same for every thread) and a
// 32-bit byte offset shared by all vectors and planes.
template <bool SOA, class T>
__device__ __forceinline__ T* mf_place(const MfArgs& a, T* v, i32 I, int k) {
  if constexpr (SOA)
    return reinterpret_cast<T*>(reinterpret_cast<uintptr_t>(v + static_cast<i64>(k) * a.nodes) +
                                static_cast<uint32_t>(I) * static_cast<uint32_t>(sizeof(T)));
  else
    return v + 3 * static_cast<i64>(I) + k;
}

// The epilogue of a node's product o = (A x)_I (3 components) in each mode,
// in two parts: the node's operand loads (mf_node_load: right-hand side,
// inverse diagonal, smoothed iterate, as the mode reads them) and the
// arithmetic and stores (mf_node_store), so a kernel can issue the loads
// early.  self = the input x at node I itself (mode 3: the direction d,
// mode 5: t); c0, c1 = coef[0], coef[1] of the modes that read them.
struct MfNodeIn {
  float b[3], dinv[3], xs[3];
};

template <int MODE, bool SOA = false>
__device__ __forceinline__ void mf_node_load(const MfArgs& a, i32 I, MfNodeIn& in) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    auto at = [&](auto* v) -> auto& { return *mf_place<SOA>(a, v, I, k); };
    if (MODE == 1 || MODE == 3 || MODE == 4 || MODE == 6 || MODE == 7) in.b[k] = at(a.b);
    if (MODE == 3 || MODE == 4 || MODE == 5 || MODE == 6) in.dinv[k] = at(a.dinv);
    if (MODE == 3 || MODE == 5) in.xs[k] = at(a.xs);
  }
}

template <int MODE, bool SOA = false>
__device__ __forceinline__ void mf_node_store(const MfArgs& a, i32 I, const float (&o)[3], const float (&self)[3],
                                              const MfNodeIn& in, float c0, float c1) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    auto at = [&](auto* v) -> auto& { return *mf_place<SOA>(a, v, I, k); };
    if (MODE == 0) {
      at(a.y) = o[k];
    } else if (MODE == 1) {
      at(a.y) = in.b[k] - o[k];
    } else if (MODE == 3) {
      const float ri = in.b[k] - o[k];
      at(a.r) = ri;
      const float dv = self[k];
      const float di = c0 * dv + c1 * in.dinv[k] * ri;
      at(a.dn) = di;
      float xi = in.xs[k];
      if (a.add_d) xi = xi + dv;
      at(a.xs) = xi + di;
    } else if (MODE == 4) {
      const float ri = in.b[k] - o[k];
      at(a.r) = ri;
      at(a.dn) = in.dinv[k] * ri * c0;
    } else if (MODE == 5) {
      at(a.xs) = in.xs[k] + (self[k] - c0 * (in.dinv[k] * o[k]));
    } else if (MODE == 6) {
      const float ri = in.b[k] - o[k];
      at(a.y) = ri;
      at(a.dn) = in.dinv[k] * ri;
    } else if (MODE == 8) {
      a.y64[3 * static_cast<i64>(I) + k] = static_cast<double>(o[k]);
    } else {
      at(a.y) = in.b[k] - c0 * o[k];
    }
  }
}

// coef[0], coef[1] of the modes that read them (device scalars)
template <int MODE>
__device__ __forceinline__ void mf_coefs(const MfArgs& a, float& c0, float& c1) {
  c0 = c1 = 0.0f;
  if (MODE == 3) {
    c0 = a.coef[0];
    c1 = a.coef[1];
  } else if (MODE == 4 || MODE == 5 || MODE == 7) {
    c0 = a.coef[0];
  }
}

template <int MODE>
__device__ __forceinline__ void mf_node_out(const MfArgs& a, i32 I, const float (&o)[3], const float (&self)[3]) {
  MfNodeIn in;
  mf_node_load<MODE>(a, I, in);
  float c0, c1;
  mf_coefs<MODE>(a, c0, c1);
  mf_node_store<MODE>(a, I, o, self, in, c0, c1);
}

// Node values of a tile in shared memory: one array per component (V4
// false: three 4-byte loads per corner, fewer registers) or (x, y, z,
// unused) per node (V4 true: one 16-byte load per corner).  The tuner picks;
// the arithmetic is the same.
template <bool V4, int NZ, int TY, int TX>
struct MfHalo;
template <int NZ, int TY, int TX>
struct MfHalo<false, NZ, TY, TX> {
  float v[3][NZ + 2][TY + 2][TX + 2];
  __device__ __forceinline__ void put(int z, int y, int x, float a, float b, float c) {
    v[0][z][y][x] = a;
    v[1][z][y][x] = b;
    v[2][z][y][x] = c;
  }
  __device__ __forceinline__ void get(int z, int y, int x, float (&o)[3]) const {
    o[0] = v[0][z][y][x];
    o[1] = v[1][z][y][x];
    o[2] = v[2][z][y][x];
  }
};
template <int NZ, int TY, int TX>
struct MfHalo<true, NZ, TY, TX> {
  float4 v[NZ + 2][TY + 2][TX + 2];
  __device__ __forceinline__ void put(int z, int y, int x, float a, float b, float c) {
    v[z][y][x] = make_float4(a, b, c, 0.0f);
  }
  __device__ __forceinline__ void get(int z, int y, int x, float (&o)[3]) const {
    const float4 t = v[z][y][x];
    o[0] = t.x;
    o[1] = t.y;
    o[2] = t.z;
  }
};

template <int MODE, int TX = kTX, int TY = kTY, int TZ = kTZ, bool V4 = false>
__global__ void __launch_bounds__(TX* TY* TZ) k_mf3_tile(MfView m, MfArgs a, const __grid_constant__ KeF32 ke) {
  if (!chain_start()) return;
  constexpr int NZ = TZ * kNZ;  // node layers of the tile
  __shared__ MfHalo<V4, NZ, TY, TX> xh;
  __shared__ float sc[NZ + 1][TY + 1][TX + 1];
  const int tid = threadIdx.x;
  const i32 x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = blockIdx.z * NZ;
  const i32 nnz = m.nz + 1;
  // node values of the tile and its halo (zero outside the grid / clamped):
  // every thread first loads the free-node indices of all its halo entries,
  // then their values, so the loads of one thread are independent
  constexpr int kHalo = (NZ + 2) * (TY + 2) * (TX + 2);
  constexpr int kPer = (kHalo + TX * TY * TZ - 1) / (TX * TY * TZ);
  i32 hj[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int e = tid + q * TX * TY * TZ;
    const int hx = e % (TX + 2), hy = (e / (TX + 2)) % (TY + 2), hz = e / ((TX + 2) * (TY + 2));
    const i32 gx = x0 - 1 + hx, gy = y0 - 1 + hy, gz = z0 - 1 + hz;
    hj[q] = -1;
    if (e < kHalo && gx >= 0 && gx < m.nnx && gy >= 0 && gy < m.nny && gz >= 0 && gz < nnz)
      hj[q] = m.nindex[(static_cast<i64>(gz) * m.nny + gy) * m.nnx + gx];
  }
  float hv[kPer][3];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    hv[q][0] = hv[q][1] = hv[q][2] = 0.0f;
    if (hj[q] >= 0) {
      const float* p = a.x + static_cast<i64>(hj[q]) * 3;
      hv[q][0] = p[0];
      hv[q][1] = p[1];
      hv[q][2] = p[2];
    }
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int e = tid + q * TX * TY * TZ;
    if (e < kHalo) {
      const int hx = e % (TX + 2), hy = (e / (TX + 2)) % (TY + 2), hz = e / ((TX + 2) * (TY + 2));
      xh.put(hz, hy, hx, hv[q][0], hv[q][1], hv[q][2]);
    }
  }
  // cell scales (zero outside the grid)
  for (int e = tid; e < (NZ + 1) * (TY + 1) * (TX + 1); e += TX * TY * TZ) {
    const int cx = e % (TX + 1), cy = (e / (TX + 1)) % (TY + 1), cz = e / ((TX + 1) * (TY + 1));
    const i32 gx = x0 - 1 + cx, gy = y0 - 1 + cy, gz = z0 - 1 + cz;
    float s = 0.0f;
    if (gx >= 0 && gx < m.nx && gy >= 0 && gy < m.ny && gz >= 0 && gz < m.nz)
      s = m.scale[(static_cast<i64>(gz) * m.ny + gy) * m.nx + gx];
    sc[cz][cy][cx] = s;
  }
  __syncthreads();
  const int tx = tid % TX, ty = (tid / TX) % TY, tz = tid / (TX * TY);
  const i32 gx = x0 + tx, gy = y0 + ty;
  if (gx >= m.nnx || gy >= m.nny) return;
  // kNZ consecutive node layers per thread: their neighbourhoods share
  // layers, so each shared value is loaded once per thread
#pragma unroll
  for (int q = 0; q < kNZ; ++q) {
    const int lz = tz * kNZ + q;  // node layer in the tile
    const i32 gz = z0 + lz;
    if (gz >= nnz) break;
    const i32 I = m.nindex[(static_cast<i64>(gz) * m.nny + gy) * m.nnx + gx];
    if (I < 0) continue;
    float out0 = 0.0f, out1 = 0.0f, out2 = 0.0f;
#pragma unroll
    for (int dz = -1; dz <= 0; ++dz)
#pragma unroll
      for (int dy = -1; dy <= 0; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 0; ++dx) {
          const float s = sc[lz + dz + 1][ty + dy + 1][tx + dx + 1];
          const int ox = -dx, oy = -dy, oz = -dz;
          const int aI = 4 * oz + (oy ? 3 - ox : ox);
          float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const int bx = (b == 1 || b == 2 || b == 5 || b == 6) ? 1 : 0;
            const int by = (b == 2 || b == 3 || b == 6 || b == 7) ? 1 : 0;
            const int bz = b >= 4 ? 1 : 0;
            float xb[3];
            xh.get(lz + dz + 1 + bz, ty + dy + 1 + by, tx + dx + 1 + bx, xb);
#pragma unroll
            for (int kb = 0; kb < 3; ++kb) {
              const float xv = xb[kb];
              a0 = fmaf(ke.k[(3 * aI + 0) * 24 + 3 * b + kb], xv, a0);
              a1 = fmaf(ke.k[(3 * aI + 1) * 24 + 3 * b + kb], xv, a1);
              a2 = fmaf(ke.k[(3 * aI + 2) * 24 + 3 * b + kb], xv, a2);
            }
          }
          out0 = fmaf(s, a0, out0);
          out1 = fmaf(s, a1, out1);
          out2 = fmaf(s, a2, out2);
        }
    const float o[3] = {out0, out1, out2};
    float self[3];
    xh.get(lz + 1, ty + 1, tx + 1, self);
    mf_node_out<MODE>(a, I, o, self);
  }
}

// FP64 variant of the tiled operator (same tile, halo and cell order): y =
// A x (MODE 0) or y = b - A x (MODE 1) with FP64 values, scales and K_e^0.
// It gives the matrix-free CG operator's true residuals, whose accuracy the
// FP32 products inside CG lack; FP64-pipe bound (576 multiply-adds per
// node), so it runs only at the restarts.
struct KeF64 {
  double k[24 * 24];
};

template <int MODE>
__global__ void __launch_bounds__(kTX* kTY* kTZ) k_mf3_tile64(MfView m, const double* __restrict__ scale,
                                                              const double* __restrict__ x, double* __restrict__ y,
                                                              const double* __restrict__ b,
                                                              const __grid_constant__ KeF64 ke) {
  if (!chain_start()) return;
  constexpr int NZ = kTZ * kNZ;
  __shared__ double xh[3][NZ + 2][kTY + 2][kTX + 2];
  __shared__ double sc[NZ + 1][kTY + 1][kTX + 1];
  const int tid = threadIdx.x;
  const i32 x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY, z0 = blockIdx.z * NZ;
  const i32 nnz = m.nz + 1;
  constexpr int kHalo = (NZ + 2) * (kTY + 2) * (kTX + 2);
  for (int e = tid; e < kHalo; e += kTX * kTY * kTZ) {
    const int hx = e % (kTX + 2), hy = (e / (kTX + 2)) % (kTY + 2), hz = e / ((kTX + 2) * (kTY + 2));
    const i32 gx = x0 - 1 + hx, gy = y0 - 1 + hy, gz = z0 - 1 + hz;
    i32 j = -1;
    if (gx >= 0 && gx < m.nnx && gy >= 0 && gy < m.nny && gz >= 0 && gz < nnz)
      j = m.nindex[(static_cast<i64>(gz) * m.nny + gy) * m.nnx + gx];
    double v0 = 0.0, v1 = 0.0, v2 = 0.0;
    if (j >= 0) {
      const double* p = x + static_cast<i64>(j) * 3;
      v0 = p[0];
      v1 = p[1];
      v2 = p[2];
    }
    xh[0][hz][hy][hx] = v0;
    xh[1][hz][hy][hx] = v1;
    xh[2][hz][hy][hx] = v2;
  }
  for (int e = tid; e < (NZ + 1) * (kTY + 1) * (kTX + 1); e += kTX * kTY * kTZ) {
    const int cx = e % (kTX + 1), cy = (e / (kTX + 1)) % (kTY + 1), cz = e / ((kTX + 1) * (kTY + 1));
    const i32 gx = x0 - 1 + cx, gy = y0 - 1 + cy, gz = z0 - 1 + cz;
    double s = 0.0;
    if (gx >= 0 && gx < m.nx && gy >= 0 && gy < m.ny && gz >= 0 && gz < m.nz)
      s = scale[(static_cast<i64>(gz) * m.ny + gy) * m.nx + gx];
    sc[cz][cy][cx] = s;
  }
  __syncthreads();
  const int tx = tid % kTX, ty = (tid / kTX) % kTY, tz = tid / (kTX * kTY);
  const i32 gx = x0 + tx, gy = y0 + ty, gz = z0 + tz;
  if (gx >= m.nnx || gy >= m.nny || gz >= nnz) return;
  const i32 I = m.nindex[(static_cast<i64>(gz) * m.nny + gy) * m.nnx + gx];
  if (I < 0) return;
  double out0 = 0.0, out1 = 0.0, out2 = 0.0;
#pragma unroll
  for (int dz = -1; dz <= 0; ++dz)
#pragma unroll
    for (int dy = -1; dy <= 0; ++dy)
#pragma unroll
      for (int dx = -1; dx <= 0; ++dx) {
        const double s = sc[tz + dz + 1][ty + dy + 1][tx + dx + 1];
        const int ox = -dx, oy = -dy, oz = -dz;
        const int aI = 4 * oz + (oy ? 3 - ox : ox);
        double a0 = 0.0, a1 = 0.0, a2 = 0.0;
#pragma unroll
        for (int bb = 0; bb < 8; ++bb) {
          const int bx = (bb == 1 || bb == 2 || bb == 5 || bb == 6) ? 1 : 0;
          const int by = (bb == 2 || bb == 3 || bb == 6 || bb == 7) ? 1 : 0;
          const int bz = bb >= 4 ? 1 : 0;
#pragma unroll
          for (int kb = 0; kb < 3; ++kb) {
            const double xv = xh[kb][tz + dz + 1 + bz][ty + dy + 1 + by][tx + dx + 1 + bx];
            a0 = fma(ke.k[(3 * aI + 0) * 24 + 3 * bb + kb], xv, a0);
            a1 = fma(ke.k[(3 * aI + 1) * 24 + 3 * bb + kb], xv, a1);
            a2 = fma(ke.k[(3 * aI + 2) * 24 + 3 * bb + kb], xv, a2);
          }
        }
        out0 = fma(s, a0, out0);
        out1 = fma(s, a1, out1);
        out2 = fma(s, a2, out2);
      }
  const double o[3] = {out0, out1, out2};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const i64 row = static_cast<i64>(I) * 3 + k;
    if (MODE == 0) y[row] = o[k];
    else y[row] = b[row] - o[k];
  }
}

// The tentative prolongator P^ of level 0 (3 unknowns per node, B1 per
// aggregate; SOA: t in component planes; aggregate g owns coarse unknowns g B1 .. g B1 + B1 - 1; the row
// of fine unknown i is phat[phat_ptr[i] ...], B1 values, empty for a node in
// no aggregate).  t = P^ x_c, one thread per fine unknown.
template <int B1, bool SOA>
__global__ void __launch_bounds__(256) k_phat_prolong(i32 n, const i32* __restrict__ agg,
                                                      const i32* __restrict__ phat_ptr,
                                                      const float* __restrict__ phat, const float* __restrict__ xc,
                                                      float* __restrict__ t) {
  if (!chain_start()) return;
  const i32 i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const i32 g = agg[i / 3];
  float s = 0.0f;
  if (g >= 0) {
    const float* ph = phat + phat_ptr[i];
    const float* xg = xc + static_cast<i64>(g) * B1;
#pragma unroll
    for (int j = 0; j < B1; ++j) s = fmaf(ph[j], xg[j], s);
  }
  t[SOA ? static_cast<i64>(i % 3) * (n / 3) + i / 3 : i] = s;
}

// b_c = P^T t: one warp per aggregate; lane q takes the aggregate's member
// unknowns q, q + 32, ... (members ascending, 3 unknowns each) into B1 partial
// sums, reduced across the warp in a fixed butterfly order.
template <int B1, bool SOA>
__global__ void __launch_bounds__(256) k_phat_restrict(i32 naggs, i64 nodes, const i32* __restrict__ mptr,
                                                       const i32* __restrict__ members,
                                                       const i32* __restrict__ phat_ptr,
                                                       const float* __restrict__ phat, const float* __restrict__ t,
                                                       float* __restrict__ bc) {
  if (!chain_start()) return;
  const i32 g = static_cast<i32>((blockIdx.x * static_cast<i64>(blockDim.x) + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (g >= naggs) return;
  const i32 q0 = mptr[g], cnt = 3 * (mptr[g + 1] - q0);
  float acc[B1];
#pragma unroll
  for (int j = 0; j < B1; ++j) acc[j] = 0.0f;
  for (i32 q = lane; q < cnt; q += 32) {
    const i32 i = 3 * members[q0 + q / 3] + q % 3;
    const float ti = t[SOA ? (i % 3) * nodes + i / 3 : i];
    const float* ph = phat + phat_ptr[i];
#pragma unroll
    for (int j = 0; j < B1; ++j) acc[j] = fmaf(ph[j], ti, acc[j]);
  }
#pragma unroll
  for (int j = 0; j < B1; ++j)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  if (lane < B1) {
    float v = acc[0];
#pragma unroll
    for (int j = 1; j < B1; ++j)
      if (lane == j) v = acc[j];
    bc[static_cast<i64>(g) * B1 + lane] = v;
  }
}

}  // namespace
}  // namespace simp
