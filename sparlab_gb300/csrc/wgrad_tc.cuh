// Weight and bias gradients of the surrogate's 3 x 3 x 3 convolutions on the
// fifth-generation tensor cores:
//   dW_t[co][ci] = sum_v dY[v][co] X[v + o_t][ci],  db[co] = sum_v dY[v][co].
//
// For one z offset dz a CTA walks tiles of 32 x 4 x 1 nodes v and holds the
// nine taps (dy, dx) of up to 32 input channels as FP32 accumulators in
// tensor memory: D (co x (dy, dx, ci)) += dY^T X with the nodes as the
// contraction.  Both operands are channels-last, so with the nodes as K they
// are "MN-major": 8 channels of a node are 16 contiguous bytes, and the plain
// (no-swizzle) canonical layout wants the 16-byte pieces of 8 consecutive
// nodes contiguous -- planes of one 8-channel group each, nodes 16 bytes
// apart, which cp.async writes directly.  A y offset is then a shift of the
// start address by a row of 32 nodes; the x offsets are three copies of the
// tile, side by side along N, so one instruction covers three taps (N = 48
// or 96 instead of 16 or 32: the A operand is read from shared memory once
// for the three).  dY is the A operand with M = 128: rows beyond its channels
// read whatever follows it in the block's shared memory and end in
// accumulator rows nobody reads.  The bias gradient is one more instruction
// per step against a constant tile of ones.
//
// The tensor core adds into its FP32 accumulator with truncation (about 0.4 x
// 2^-24 of the sum per instruction, always towards zero), so a long sum
// drifts: 3.6e-5 of the gradient over 193x97x97 nodes.  An accumulator
// therefore takes a run of up to eight instructions (a tile's 128 nodes) and is
// then added to FP32 registers, rounded to nearest, by the warps that own its
// rows; a ring of four accumulator sets keeps the tensor core busy meanwhile.
// Small grids, whose gradients have fewer terms to average over, take shorter
// runs (2 up to 2^13 nodes, 4 up to 2^15).
//
// Warps: 0, 4, 8 (and 1, 5, 9) add the accumulators (rows 32 (w % 4) .., a
// third of the columns each), 6 issues the instructions, the others load.
// Splits: blockIdx.y = (segment of <= 32 input channels, dz), blockIdx.x one
// of G walkers of the tiles; k_wgrad_tc_sum adds the G partials in order.
//
// Measured at 97x49x49 nodes, 16 -> 16 channels: 1,270 us on the CUDA cores
// (FP32 multiply-adds from shared memory, two loads each), 80 us with runs of
// four here (one issuing warp of uniform control: 162 us when a single
// divergent thread issued, about 70 cycles an instruction); bound by the
// loads' latency and the runs' barriers (0.25 us a run).  Error of the
// gradient against FP64: 3.8e-7 -> 1.5e-7 there, 7.9e-8 -> 4.6e-8 at 37x7x5.
#pragma once

#include "common.h"
#include "tc.cuh"

namespace simp {
namespace wg {

constexpr int kThreads = 384;
constexpr int kLoaders = 160;  // threads of the loading warps
constexpr int kSets = 4;       // accumulator sets in tensor memory
constexpr int kStages = 3;
constexpr int kTX = 32, kTY = 4, kNodes = kTX * kTY;
constexpr int kRowsX = kTY + 2;
// plane strides: 16 bytes a node, and 16 more so that the planes of a node's
// channel groups fall in different banks
constexpr int kPlaneY = kNodes * 16 + 16;
constexpr int kPlaneX = kTX * kRowsX * 16 + 16;
constexpr int kMaxSeg = 4;

struct Segment {
  const __nv_bfloat16* x;  // first channel of the segment at node 0
  int pitch;               // channels per node of its tensor
  int c;                   // channels (16 or 32)
  int ci0;                 // its first input channel of the convolution
};

struct Args {
  int nx, ny, nz;
  Segment seg[kMaxSeg];
  const __nv_bfloat16* dy;
  int cdy;  // 16, 32 or 64
  float* part;
  int* status;
  int run;  // instructions an accumulator takes before it is added (2, 4 or 8)
};

__host__ __device__ constexpr int stage_bytes(int cdy, int c) { return cdy / 8 * kPlaneY + 3 * (c / 8) * kPlaneX; }
// every stage, the window of 16 planes that M = 128 reads past the last
// stage's start, the ones tile and the barriers
__host__ __device__ constexpr int smem_bytes(int cdy, int c) {
  return kStages * stage_bytes(cdy, c) + 16 * kPlaneY + 256 + 128;
}
// floats of one walker's partial: co rows of (dy, dx, ci) and 16 bias columns
__host__ __device__ constexpr int part_cols(int c) { return 9 * c + 16; }

// MN-major operand in the plain layout: (mn, k) at (mn % 8) * 2 + (mn / 8) *
// sbo + (k % 8) * 16 + (k / 8) * lbo bytes.  cp16 copies one 16-byte piece,
// zeros outside the grid.
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool in) {
  const int bytes = in ? 16 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Arrives on a barrier (one thread).
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// A walker's rows of one (segment, dz): the adding warps' part.
template <int C>
__device__ __forceinline__ void add_sets(const Args& p, uint32_t tmem, int parts, bool bias, uint64_t* set_full,
                                         uint64_t* set_free, float* out) {
  constexpr int kWide = 3 * C + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int quad = warp & 3, third = warp >> 2;  // the x offset third - 1
  const uint32_t rows = static_cast<uint32_t>(quad * 32) << 16;
  float acc[3][C], ab = 0.0f;
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int k = 0; k < C; ++k) acc[d][k] = 0.0f;
  int unit = 0;
  bool ok = true;
  for (int n = 0; n < parts && ok; ++n) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int set = unit % kSets;
      ok = ok && tc::mbar_wait(&set_full[set], (unit / kSets) & 1, p.status);
      __syncwarp();
      tc::fence_after_sync();
      float v[C / 16][16], w[16];
#pragma unroll
      for (int h = 0; h < C / 16; ++h) tc::tmem_ld16(tmem + rows + set * kWide + third * C + h * 16, v[h]);
      if (bias && d == 1 && third == 0) tc::tmem_ld16(tmem + rows + set * kWide + 3 * C, w);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&set_free[set]);
#pragma unroll
      for (int k = 0; k < C; ++k) acc[d][k] += v[k / 16][k % 16];
      if (bias && d == 1 && third == 0) ab += w[0];
      ++unit;
    }
  }
  const int co = quad * 32 + lane;
  if (co < p.cdy) {
    float* o = out + static_cast<i64>(co) * part_cols(C);
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int k = 0; k < C; k += 4)
        *reinterpret_cast<float4*>(o + (d * 3 + third) * C + k) =
            make_float4(acc[d][k], acc[d][k + 1], acc[d][k + 2], acc[d][k + 3]);
    if (third == 0) o[9 * C] = ab;
  }
}

__global__ void __launch_bounds__(kThreads, 1) k_wgrad_tc(const Args p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int segi = blockIdx.y / 3, dz = static_cast<int>(blockIdx.y % 3) - 1;
  const Segment sg = p.seg[segi];
  const int py = p.cdy / 8, px = sg.c / 8;
  const int stage = stage_bytes(p.cdy, sg.c);
  uint8_t* tail = smem + kStages * stage + 16 * kPlaneY;
  uint64_t* full = reinterpret_cast<uint64_t*>(tail + 128);  // a stage is loaded
  uint64_t* empty = full + kStages;                          // its instructions are done
  uint64_t* set_full = empty + kStages;                      // an accumulator set is complete
  uint64_t* set_free = set_full + kSets;                     // it has been added
  uint32_t* tslot = reinterpret_cast<uint32_t*>(set_free + kSets);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform for the compiler
  const int wide = 3 * sg.c + 16;  // columns of a set
  const uint32_t ncols = kSets * wide <= 256 ? 256u : 512u;
  const int adders = p.cdy > 32 ? 6 : 3;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&full[s], kLoaders / 32);
      tc::mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < kSets; ++s) {
      tc::mbar_init(&set_full[s], 1);
      tc::mbar_init(&set_free[s], static_cast<uint32_t>(adders));
    }
    tc::fence_mbar_init();
  }
  // one 8 x 8 core matrix of ones: every core of the bias tile points at it
  if (tid < 64) reinterpret_cast<__nv_bfloat16*>(tail)[tid] = __float2bfloat16_rn(1.0f);
  tc::fence_proxy_async_smem();
  if (warp == 0) tc::tmem_alloc(tslot, ncols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  const bool bias = segi == 0 && dz == 0;
  const int parts = kNodes / 16 / p.run;  // accumulator runs of a tile

  const int tx = (p.nx + kTX - 1) / kTX, ty = (p.ny + kTY - 1) / kTY;
  const int tiles = tx * ty * p.nz, first = static_cast<int>(blockIdx.x), step = static_cast<int>(gridDim.x);
  const int mine = tiles > first ? (tiles - first + step - 1) / step : 0;

  if (warp == 6) {
    // the whole warp runs the loop, so that descriptors stay in uniform
    // registers; one elected lane issues
    const bool leader = tc::elect_one();
    const uint64_t bones = tc::smem_desc_plain(tc::smem_u32(tail), 0, 0);
    // BF16 operands, both MN-major (bits 15 and 16)
    const uint32_t id = tc::idesc_bf16(128, 3 * sg.c) | (1u << 15) | (1u << 16);
    const uint32_t idb = tc::idesc_bf16(128, 16) | (1u << 15) | (1u << 16);
    int unit = 0;
    bool ok = true;
    for (int n = 0; n < mine && ok; ++n) {
      const int s = n % kStages;
      ok = tc::mbar_wait(&full[s], (n / kStages) & 1, p.status);
      tc::fence_after_sync();
      // descriptors of the stage's first nodes: a later start adds its bytes / 16
      const uint32_t base = tc::smem_u32(smem + s * stage);
      const uint64_t a0 = tc::smem_desc_plain(base, 128, kPlaneY);
      const uint64_t b0 = tc::smem_desc_plain(base + py * kPlaneY, 128, kPlaneX);
      for (int part = 0; part < parts && ok; ++part)
        for (int dy = 0; dy < 3 && ok; ++dy) {
          const int set = unit % kSets;
          if (unit >= kSets) {
            ok = tc::mbar_wait(&set_free[set], (unit / kSets - 1) & 1, p.status);
            tc::fence_after_sync();
          }
          const uint32_t d = tmem + set * wide;
          const uint64_t a = a0 + part * p.run * 16, b = b0 + part * p.run * 16 + dy * kTX;
          if (leader) {
#pragma unroll
            for (int k = 0; k < 8; ++k)  // 16 nodes each
              if (k < p.run) tc::mma_bf16(d, a + k * 16, b + k * 16, id, k != 0);
            if (bias && dy == 1)
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (k < p.run) tc::mma_bf16(d + 3 * sg.c, a + k * 16, bones, idb, k != 0);
            tc::mma_commit(&set_full[set]);
          }
          __syncwarp();
          ++unit;
        }
      if (leader) tc::mma_commit(&empty[s]);
      __syncwarp();
    }
    __syncwarp();
  } else if ((warp & 3) < 2) {
    float* out = p.part + (static_cast<i64>(blockIdx.y) * gridDim.x + blockIdx.x) * p.cdy * part_cols(32);
    if ((warp & 3) * 32 < p.cdy) {
      if (sg.c == 32) add_sets<32>(p, tmem, mine * parts, bias, set_full, set_free, out);
      else add_sets<16>(p, tmem, mine * parts, bias, set_full, set_free, out);
    }
  } else {
    const int lt = (warp < 4 ? warp - 2 : warp == 7 ? 2 : warp - 7) * 32 + lane;  // warps 2, 3, 7, 10, 11
    const int ly = 31 - __clz(py), lx = 31 - __clz(px);
    bool ok = true;
    for (int n = 0; n <= mine && ok; ++n) {
      if (n < mine) {
        const int s = n % kStages;
        if (n >= kStages) ok = tc::mbar_wait(&empty[s], (n / kStages - 1) & 1, p.status);
        const int t = first + n * step;
        const int x0 = t % tx * kTX, y0 = t / tx % ty * kTY, z = t / (tx * ty), zz = z + dz;
        const uint32_t base = tc::smem_u32(smem + s * stage), xb = base + py * kPlaneY;
        // a thread keeps one channel group; 16-byte pieces of consecutive
        // groups and nodes are consecutive in memory
        {
          const int pl = lt & (py - 1);
          const uint32_t dst = base + pl * kPlaneY;
          const __nv_bfloat16* src = p.dy + pl * 8;
          for (int v = lt >> ly; v < kNodes; v += kLoaders >> ly) {
            const int x = x0 + (v & (kTX - 1)), y = y0 + v / kTX;
            const bool in = x < p.nx && y < p.ny;
            const i64 node = in ? (static_cast<i64>(z) * p.ny + y) * p.nx + x : 0;
            cp16(dst + v * 16, src + (node << (ly + 3)), in);
          }
        }
        {
          const int pl = lt & (px - 1);
          const uint32_t dst = xb + pl * kPlaneX;
          const __nv_bfloat16* src = sg.x + pl * 8;
          const bool layer = zz >= 0 && zz < p.nz;
          for (int v = lt >> lx; v < kTX * kRowsX; v += kLoaders >> lx) {
            const int x = x0 + (v & (kTX - 1)) - 1, y = y0 + v / kTX - 1;
            const bool row = layer && y >= 0 && y < p.ny;
            const i64 node = row ? (static_cast<i64>(zz) * p.ny + y) * p.nx : 0;
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
              const bool in = row && x + dx >= 0 && x + dx < p.nx;
              cp16(dst + dx * px * kPlaneX + v * 16, src + (node + (in ? x + dx : 0)) * sg.pitch, in);
            }
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (n >= 1) {  // tile n - 1 has landed: visible to the tensor core
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        tc::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[(n - 1) % kStages]);
      }
    }
  }
  __syncwarp();
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, ncols);
  }
}

// gw[t][co][ci] += sum_g part, gb[co] += sum_g part: the walkers in order
__global__ void __launch_bounds__(256) k_wgrad_tc_sum(const Args p, int walkers, int cout, int cin, int nseg,
                                                      float* __restrict__ gw, float* __restrict__ gb) {
  const int total = 27 * cout * cin + cout;
  const i64 one = static_cast<i64>(p.cdy) * part_cols(32);  // floats of a walker's slot
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    const bool weight = e < 27 * cout * cin;
    int group = 1, at;
    if (weight) {
      const int ci = e % cin, co = e / cin % cout, t = e / (cin * cout);
      int s = 0;
      while (s + 1 < nseg && ci >= p.seg[s + 1].ci0) ++s;
      const int c = p.seg[s].c;
      group = s * 3 + t / 9;
      at = co * part_cols(c) + (t / 3 % 3 * 3 + t % 3) * c + ci - p.seg[s].ci0;
    } else {
      const int c = p.seg[0].c;
      at = (e - 27 * cout * cin) * part_cols(c) + 9 * c;
    }
    const float* q = p.part + static_cast<i64>(group) * walkers * one + at;
    // the partials' sum keeps its rounding errors (Knuth's TwoSum)
    float s = 0.0f, err = 0.0f;
    for (int g = 0; g < walkers; ++g) {
      const float v = q[g * one], t = __fadd_rn(s, v), b = __fsub_rn(t, s);
      err = __fadd_rn(err, __fadd_rn(__fsub_rn(s, __fsub_rn(t, b)), __fsub_rn(v, b)));
      s = t;
    }
    s += err;
    if (weight) gw[e] += s;
    else gb[e - 27 * cout * cin] += s;
  }
}

}  // namespace wg
}  // namespace simp
