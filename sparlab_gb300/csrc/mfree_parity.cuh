// Matrix-free level-0 operator of a structured Hex8 grid in the cell's
// parity basis.
//
// A box cell's K_e^0 is unchanged by the mirror reflections of the cell.  In
// the basis of sums and differences of its corner values along each axis
// (T = H x H x H per component, H = [[1, 1], [-1, 1]]), K_e^0 = T^T K^ T where
// K^ = T K_e^0 T^T / 64 couples only modes of the same mirror parities: eight
// 3 x 3 blocks, one mode of each component in each, of which the rigid
// translations and the split of shear and hourglass modes leave 45 entries.
// A cell's product is then 45 multiply-adds instead of 576, and the sums and
// differences along x and y belong to the node layers, so neighbouring cells
// share them: about 190 FP32 operations a cell where the direct product
// takes 576 (k_mf3_tile, kept for small grids and for element matrices
// without the symmetry).  The differences of close values come first, so
// smooth fields lose fewer digits than in the direct sums.
//
// A block owns 31 x TY node columns and marches `chunk` node layers along z,
// one warp per row of cells: lane i holds the node column x0 - 1 + i and the
// cell column to its right.  Along x neighbours exchange by shuffles (lane 31
// loads its right neighbour), along y through shared memory, along z in
// registers.  One barrier per layer: before it a warp stores its row's x
// sums and differences of layer L, and the upper halves of the cell rows'
// results for node layer L - 2 stored at the end of the last step; after it
// node layer L - 2 is finished and the cells between layers L - 1 and L are
// computed.  Every value is summed in the same order whatever TY and
// `chunk`, so all launch shapes give the same bits.
//
// The arithmetic is FP32 (the V-cycle's operator, with k_mf3_tile's epilogues)
// or double-float (the CG operator: (hi, lo) float pairs in, FP64 output and
// right-hand side).
//
// Bound by instruction issue: 965 instructions a node, most of them node
// indices and their tests, addresses, shuffles and exchanges beside the
// arithmetic (FP32 at 120x64x64: 56 % of the issue slots, 0.2 of the load/store
// wavefronts, the rest barrier and load latency at 18 warps an SM).  Measured,
// us a launch, before -> after: y = A x double-float 700 -> 193 at 192x96x96
// (the assembled rows read 3.8 GB, this 0.1 GB) and 97 -> 39 at 96x48x48; FP32
// Chebyshev step 87 -> 60 and 16.9 -> 14.8, the other modes 79-86 -> 43-52 and
// 15-16.9 -> 12.8.  Errors against FP64 fall too:
// double-float 8.6e-15 -> 3.6e-15 (2-norm, random x) and 1.7e-12 -> 3.3e-13
// (smooth x), FP32 7.2e-8 -> 6.8e-8 and 1.1e-5 -> 8.5e-6.
#pragma once

#include "mfree.cuh"

namespace simp {
namespace {

constexpr int kParCols = 31;    // node columns a warp row owns
constexpr int kParRows = 8;     // node rows a block owns (FP32)
constexpr int kParRowsDf = 4;   // (double-float)

struct KePar32 {
  float k[8][3][3];  // K^ blocks: label l holds the modes (l ^ 1, x), (l ^ 2, y), (l ^ 4, z)
};
struct KeParDf {
  float2 k[8][3][3];  // (hi, lo)
};

// Entries of block l that can be nonzero.  Labels 1, 2, 4 hold a rigid
// translation (zero row and column of component log2 l); in labels 3, 5, 6 the
// xyz hourglass mode of component log2(7 - l) stands alone.
__host__ __device__ constexpr int par_alone(int l) {
  return l == 1 || l == 6 ? 0 : l == 2 || l == 5 ? 1 : l == 4 || l == 3 ? 2 : -1;
}
__host__ __device__ constexpr bool par_rigid(int l, int k) {
  return (l == 1 || l == 2 || l == 4) && par_alone(l) == k;
}
__host__ __device__ constexpr bool par_couples(int l, int r, int c) {
  if (par_rigid(l, r) || par_rigid(l, c)) return false;
  return r == c || (par_alone(l) != r && par_alone(l) != c);
}

// FP32 arithmetic.
struct ParF32 {
  using V = float;
  using Ke = KePar32;
  using X2 = float2;
  static __device__ __forceinline__ V zero() { return 0.0f; }
  // rounded operations, so that no launch shape's compilation contracts them differently
  static __device__ __forceinline__ V add(V a, V b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ V renorm(V a) { return a; }
  static __device__ __forceinline__ V mul(float k, V a) { return __fmul_rn(k, a); }
  static __device__ __forceinline__ V mad(float k, V a, V t) { return fmaf(k, a, t); }
  // s a + s b and s a - s b
  static __device__ __forceinline__ void scaled(V s, V a, V b, V& sum, V& diff) {
    const float sb = __fmul_rn(s, b);
    sum = fmaf(s, a, sb);
    diff = fmaf(s, a, -sb);
  }
  static __device__ __forceinline__ void scaled(V s, V b, V& sum, V& diff) {  // a = 0
    sum = __fmul_rn(s, b);
    diff = -sum;
  }
  static __device__ __forceinline__ V down(V a) { return __shfl_down_sync(0xffffffffu, a, 1); }
  static __device__ __forceinline__ V up(V a) { return __shfl_up_sync(0xffffffffu, a, 1); }
  static __device__ __forceinline__ X2 pack(V a, V b) { return make_float2(a, b); }
  static __device__ __forceinline__ void unpack(X2 v, V& a, V& b) {
    a = v.x;
    b = v.y;
  }
};

// Double-float arithmetic: sums keep (hi, lo) with lo possibly a few ulps of
// hi; renorm makes |lo| <= ulp(hi) / 2 again before a product, whose lo * lo
// term is dropped (after a cancellation that leaves |hi| < |lo|, both below
// 2^-22 of the summands, renorm rounds to a float: 2^-46 of the summands).
struct ParDf {
  struct V {
    float h, l;
  };
  using Ke = KeParDf;
  using X2 = float4;
  static __device__ __forceinline__ V zero() { return {0.0f, 0.0f}; }
  static __device__ __forceinline__ V add(V a, V b) {
    float s, e;
    two_sum(a.h, b.h, s, e);
    return {s, __fadd_rn(e, __fadd_rn(a.l, b.l))};
  }
  static __device__ __forceinline__ V sub(V a, V b) { return add(a, {-b.h, -b.l}); }
  static __device__ __forceinline__ V renorm(V a) {
    const float s = __fadd_rn(a.h, a.l);
    return {s, __fsub_rn(a.l, __fsub_rn(s, a.h))};
  }
  static __device__ __forceinline__ V mul(float2 k, V a) {
    const float p = __fmul_rn(k.x, a.h);
    float e = __fmaf_rn(k.x, a.h, -p);
    e = __fmaf_rn(k.x, a.l, __fmaf_rn(k.y, a.h, e));
    return {p, e};
  }
  static __device__ __forceinline__ V mad(float2 k, V a, V t) { return add(t, mul(k, a)); }
  static __device__ __forceinline__ void scaled(V s, V a, V b, V& sum, V& diff) {
    const V sa = mul(make_float2(s.h, s.l), a), sb = mul(make_float2(s.h, s.l), b);
    sum = add(sa, sb);
    diff = sub(sa, sb);
  }
  static __device__ __forceinline__ void scaled(V s, V b, V& sum, V& diff) {
    sum = mul(make_float2(s.h, s.l), b);
    diff = {-sum.h, -sum.l};
  }
  static __device__ __forceinline__ V down(V a) {
    return {__shfl_down_sync(0xffffffffu, a.h, 1), __shfl_down_sync(0xffffffffu, a.l, 1)};
  }
  static __device__ __forceinline__ V up(V a) {
    return {__shfl_up_sync(0xffffffffu, a.h, 1), __shfl_up_sync(0xffffffffu, a.l, 1)};
  }
  static __device__ __forceinline__ X2 pack(V a, V b) { return make_float4(a.h, a.l, b.h, b.l); }
  static __device__ __forceinline__ void unpack(X2 v, V& a, V& b) {
    a = {v.x, v.y};
    b = {v.z, v.w};
  }
};

// row r of block l times v
template <class AR>
__device__ __forceinline__ typename AR::V par_row(const typename AR::Ke& ke, int l, int r,
                                                  const typename AR::V (&v)[3]) {
  typename AR::V t = AR::zero();
  bool first = true;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (!par_couples(l, r, c)) continue;
    t = first ? AR::mul(ke.k[l][r][c], v[c]) : AR::mad(ke.k[l][r][c], v[c], t);
    first = false;
  }
  return AR::renorm(t);
}

struct MfArgs64 {
  const float2* x;      // input, (hi, lo) pairs
  double* y;            // output
  const double* b;      // mode 1: right-hand side
  const float2* scale;  // s_e, (hi, lo)
};

// Arithmetic and arguments of a kernel: FP32 with the epilogues of mfree.cuh
// (MfArgs), or double-float on FP64 vectors (modes 0 y = A x, 1 y = b - A x).
template <class AR>
struct ParIo;

// FP32 vectors in component planes (unknown (node I, component k) at
// k nodes + I): a warp's loads and stores are contiguous, where the
// node-by-node order takes three times the load/store cycles, which then
// bound the kernel (85 against 51 us for the Chebyshev step at 192x96x96).
template <>
struct ParIo<ParF32> {
  using Args = MfArgs;
  struct In {
    MfNodeIn n;
    float self[3];
  };
  using Raw = float;  // a value as stored
  static __device__ __forceinline__ float value(Raw r) { return r; }
  static __device__ __forceinline__ Raw scale(const MfView& m, const Args&, i32 c) { return m.scale[c]; }
  static __device__ __forceinline__ Raw input(const Args& a, i32 I, int k) { return *mf_place<true>(a, a.x, I, k); }
  template <int MODE>
  static __device__ __forceinline__ void fetch(const Args& a, i32 I, In& in) {
    mf_node_load<MODE, true>(a, I, in.n);
    if (MODE == 3 || MODE == 5)  // the input at the node itself, loaded two layers ago
#pragma unroll
      for (int k = 0; k < 3; ++k) in.self[k] = input(a, I, k);
  }
  template <int MODE>
  static __device__ __forceinline__ void store(const Args& a, i32 I, const float (&o)[3], const In& in, float c0,
                                               float c1) {
    mf_node_store<MODE, true>(a, I, o, in.self, in.n, c0, c1);
  }
  template <int MODE>
  static __device__ __forceinline__ void coefs(const Args& a, float& c0, float& c1) {
    mf_coefs<MODE>(a, c0, c1);
  }
};

template <>
struct ParIo<ParDf> {
  using Args = MfArgs64;
  struct In {
    double b[3];
  };
  using Raw = float2;
  static __device__ __forceinline__ ParDf::V value(Raw r) { return {r.x, r.y}; }
  static __device__ __forceinline__ Raw scale(const MfView&, const Args& a, i32 c) { return a.scale[c]; }
  static __device__ __forceinline__ Raw input(const Args& a, i32 I, int k) { return a.x[3 * I + k]; }
  template <int MODE>
  static __device__ __forceinline__ void fetch(const Args& a, i32 I, In& in) {
    if (MODE == 1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) in.b[k] = a.b[static_cast<i64>(I) * 3 + k];
    }
  }
  template <int MODE>
  static __device__ __forceinline__ void store(const Args& a, i32 I, const ParDf::V (&o)[3], const In& in, float,
                                               float) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double v = static_cast<double>(o[k].h) + static_cast<double>(o[k].l);
      a.y[static_cast<i64>(I) * 3 + k] = MODE == 1 ? in.b[k] - v : v;
    }
  }
  template <int MODE>
  static __device__ __forceinline__ void coefs(const Args&, float&, float&) {}
};

// Two resident blocks bound the registers (FP32, 10 warps: 96; double-float, 6
// warps: 168); three spill (192x96x96: double-float 422 against 319 us).  They
// are full, so nothing that a layer can form again is kept across layers: with
// the coefficients and the sizes of node and cell planes kept, modes 3 and 5
// spill 8 bytes (192x96x96 design pass 62.4 against 61.0 ms).
template <int MODE, class AR, int TY>
__global__ void __launch_bounds__(32 * (TY + 2), 2) k_mf3_par(MfView m, typename ParIo<AR>::Args a,
                                                            const __grid_constant__ typename AR::Ke ke, int chunk) {
  if (!chain_start()) return;
  using V = typename AR::V;
  using X2 = typename AR::X2;
  using Io = ParIo<AR>;
  using Raw = typename Io::Raw;
  // per component (sum, difference) along x of a node row; upper halves of a
  // cell row's result
  __shared__ X2 fwd[2][TY + 2][3][32];
  __shared__ X2 bwd[2][TY][3][32];
  const int lane = threadIdx.x & 31, j = threadIdx.x >> 5;
  const i32 gx = static_cast<i32>(blockIdx.x) * kParCols - 1 + lane;
  const i32 gy = static_cast<i32>(blockIdx.y) * TY - 1 + j;
  const i32 nnz = m.nz + 1;
  const i32 z0 = static_cast<i32>(blockIdx.z) * chunk, z1 = min(z0 + chunk, nnz);
  const bool row_in = gy >= 0 && gy < m.nny;
  const bool node_in = row_in && gx >= 0 && gx < m.nnx;
  const bool edge_in = row_in && lane == 31 && gx + 1 < m.nnx;  // the right neighbour of lane 31
  const bool cell_in = gx >= 0 && gx < m.nx && gy >= 0 && gy < m.ny;
  const bool owns = node_in && lane >= 1 && j >= 1 && j <= TY;

  // free-node index of this thread's column (and lane 31's neighbour) in layer L
  // (32-bit indices: the unknowns are counted in 32 bits)
  auto index_of = [&](i32 L, i32& I, i32& E) {
    I = E = -1;
    if (L >= 0 && L < nnz) {
      if (node_in) I = m.nindex[(L * m.nny + gy) * m.nnx + gx];
      if (edge_in) E = m.nindex[(L * m.nny + gy) * m.nnx + gx + 1];
    }
  };
  auto values_of = [&](i32 I, Raw (&u)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) u[k] = I >= 0 ? Io::input(a, I, k) : Raw{};
  };

  i32 In, En;          // indices of the layer whose values are in flight
  Raw un[3], ue[3];    // its values
  index_of(z0 - 1, In, En);
  values_of(In, un);
  values_of(En, ue);
  i32 I2, E2;          // indices of the layer after it
  index_of(z0, I2, E2);
  Raw sn = Raw{};     // scale of the next cell (between the layers L - 1 and L)
  i32 Ia = -1, Ib = -1;           // free indices of this column in layers L - 1 and L - 2
  V P[4][3], C[4][3], low[2][3];  // layer L - 1's xy modes; upper halves of the cell below; lower rows' part of L - 2
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int q = 0; q < 4; ++q) P[q][k] = C[q][k] = AR::zero();
    low[0][k] = low[1][k] = AR::zero();
  }

  for (i32 L = z0 - 1; L <= z1 + 1; ++L) {
    const int buf = L & 1;
    V s[3], d[3];
    const i32 I = In;
    if (L <= z1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const V u = Io::value(un[k]);
        V right = AR::down(u);
        if (lane == 31) right = Io::value(ue[k]);
        s[k] = AR::add(u, right);
        d[k] = AR::sub(right, u);
        fwd[buf][j][k][lane] = AR::pack(s[k], d[k]);
      }
      if (L < z1) {  // the next layer's values and the indices after it
        In = I2;
        values_of(I2, un);
        values_of(E2, ue);
        index_of(L + 2, I2, E2);
      }
    }
    const V sc = Io::value(sn);  // scale of cell layer L - 1
    if (L < z1) sn = cell_in && L >= 0 && L < m.nz ? Io::scale(m, a, (L * m.ny + gy) * m.nx + gx) : Raw{};
    const bool out = owns && L - 2 >= z0 && Ib >= 0;
    typename Io::In in;
    if (out) Io::template fetch<MODE>(a, Ib, in);
    __syncthreads();
    if (j <= TY) {
      if (j >= 1 && L - 2 >= z0) {  // finish node layer L - 2
        V o[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          V hs, hd;
          AR::unpack(bwd[buf][j - 1][k][lane], hs, hd);
          const V as = AR::add(hs, low[0][k]), ad = AR::add(hd, low[1][k]);
          o[k] = AR::add(AR::up(AR::add(as, ad)), AR::sub(as, ad));
        }
        if (out) {
          float c0 = 0.0f, c1 = 0.0f;
          Io::template coefs<MODE>(a, c0, c1);
          Io::template store<MODE>(a, Ib, o, in, c0, c1);
        }
      }
      if (L <= z1) {
        // xy modes of layer L: bit 0 difference along x, bit 1 along y
        V s2[3], d2[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) AR::unpack(fwd[buf][j + 1][k][lane], s2[k], d2[k]);
        auto mode_of = [&](int q, int k) {
          return q == 0 ? AR::add(s[k], s2[k]) : q == 1 ? AR::add(d[k], d2[k])
               : q == 2 ? AR::sub(s2[k], s[k]) : AR::sub(d2[k], d[k]);
        };
        // the cells between layers L - 1 and L, two labels (l, l + 4) at a
        // time: they hold both z parities of three xy modes.  At L = z0 - 1
        // there is no layer below: only P is set.
        V Q[4][3];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          V v[2][3];  // by z parity of the mode
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int q = (l ^ (1 << k)) & 3;
            const V n = mode_of(q, k);
            v[0][k] = q == 0 ? AR::zero() : AR::renorm(AR::add(P[q][k], n));  // q = 0: a rigid translation
            v[1][k] = AR::renorm(AR::sub(n, P[q][k]));
            P[q][k] = n;
          }
          // label l: components x and y at z parity 0, z at 1; label l + 4 the others
          const V va[3] = {v[0][0], v[0][1], v[1][2]}, vb[3] = {v[1][0], v[1][1], v[0][2]};
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int q = (l ^ (1 << k)) & 3;
            const int l0 = k < 2 ? l : l + 4, l1 = k < 2 ? l + 4 : l;
            V top, bottom;
            const V w1 = par_row<AR>(ke, l1, k, k < 2 ? vb : va);
            if (par_rigid(l0, k)) AR::scaled(sc, w1, top, bottom);
            else AR::scaled(sc, par_row<AR>(ke, l0, k, k < 2 ? va : vb), w1, top, bottom);
            Q[q][k] = AR::add(C[q][k], bottom);
            C[q][k] = top;
          }
        }
        // node layer L - 1: upper halves of the cell below, lower of this one
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          low[0][k] = AR::sub(Q[0][k], Q[2][k]);
          low[1][k] = AR::sub(Q[1][k], Q[3][k]);
          if (j < TY) bwd[buf ^ 1][j][k][lane] = AR::pack(AR::add(Q[0][k], Q[2][k]), AR::add(Q[1][k], Q[3][k]));
        }
      }
    }
    Ib = Ia;
    Ia = L <= z1 ? I : -1;
  }
}

}  // namespace

// K^ of a Hex8 element matrix (row-major 24 x 24); false when an entry that
// par_couples rules out exceeds 1e-14 of the largest (an element without the
// box cell's symmetry).
inline bool parity_blocks(const double* ke, double (&k)[8][3][3]) {
  static const int cx[8] = {0, 1, 1, 0, 0, 1, 1, 0}, cy[8] = {0, 0, 1, 1, 0, 0, 1, 1}, cz[8] = {0, 0, 0, 0, 1, 1, 1, 1};
  auto t = [&](int mode, int corner) {
    double v = 1.0;
    if ((mode & 1) && !cx[corner]) v = -v;
    if ((mode & 2) && !cy[corner]) v = -v;
    if ((mode & 4) && !cz[corner]) v = -v;
    return v;
  };
  double largest = 0.0, stray = 0.0;
  for (int m = 0; m < 8; ++m)
    for (int a = 0; a < 3; ++a)
      for (int n = 0; n < 8; ++n)
        for (int b = 0; b < 3; ++b) {
          double sum = 0.0;
          for (int p = 0; p < 8; ++p)
            for (int q = 0; q < 8; ++q) sum += t(m, p) * ke[(3 * p + a) * 24 + 3 * q + b] * t(n, q);
          sum /= 64.0;
          const double v = sum < 0.0 ? -sum : sum;
          const int l = m ^ (1 << a);
          if (!(v <= largest)) largest = v;
          if (l == (n ^ (1 << b)) && par_couples(l, a, b)) k[l][a][b] = sum;
          else if (!(v <= stray)) stray = v;
        }
  return largest > 0.0 && stray <= 1e-14 * largest;
}

}  // namespace simp
