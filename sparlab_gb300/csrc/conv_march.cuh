// 3 x 3 x 3 convolutions of the displacement surrogate whose weights fit in
// shared memory: a CTA owns 32 x 4 nodes in x and y and marches along z.
//
// conv_tc.cuh loads every input tile 27 times (once per tap) and issues one
// product per tap; with 16 or 32 output columns the A operand's shared-memory
// reads (4 KB an instruction) and the loads bound it.  Here an input layer is
// loaded once per x offset by TMA (32 x 6 nodes, K-major rows of a node's
// channels in the swizzle that spans them): a y offset is a shift of the
// operand's start address by 32 rows, a whole number of swizzle atoms.  One
// product per (y, x) tap serves the three output layers around the input
// layer: N = 3 n columns, with the accumulators of the chunk's layers side by
// side in tensor memory and the weights resident in the plain layout.  The
// layers run in the order in which each output meets its taps t = 0 .. 26 (z
// ascending, with flip descending), so every output sums the same products in
// the same order as in conv_tc.cuh and gets the same bits.
//
// Warps 0-3 finish output layers (bias, ReLU, store) while later layers are
// multiplied, warp 4 issues the products, warp 5 the loads.
//
// Measured at 193x97x97 nodes against conv_tc.cuh: 16 -> 16 channels 269 ->
// 59 us, 32 + 16 -> 16 552 -> 147 us; a chunk's start (weights, tensor memory,
// the first layers: 2 to 4 us) and about 40 cycles a product bound it.
#pragma once

#include "common.h"
#include "conv_tc.cuh"
#include "wgrad_tc.cuh"

namespace simp {
namespace conv {

constexpr int kMarchThreads = 192;
constexpr int kMarchRows = kTileY + 2;
constexpr int kMarchNodes = kTileX * kMarchRows;  // nodes of a loaded layer
constexpr int kMarchMaxStages = 4;
constexpr int kMarchMaxSteps = 40;  // input layers of a chunk

struct MarchArgs {
  ConvArgs c;
  const __nv_bfloat16* w;  // [27][n][K]
  int chunk;               // output layers of a CTA
  int stages;
};

__host__ __device__ constexpr int march_weight_bytes(int n, int k) { return 27 * n * k * 2; }
__host__ __device__ constexpr int march_stage_bytes(int k) { return 3 * k * 2 * kMarchNodes; }
__host__ __device__ constexpr int march_smem(int n, int k, int stages) {
  return 1024 + stages * march_stage_bytes(k) + march_weight_bytes(n, k) + (2 * kMarchMaxStages + kMarchMaxSteps) * 8 + 16;
}

// Start of tap u's operand in a loaded layer of c channels, in 16 bytes: the
// copy of its x offset, the row of its y offset.
template <bool FLIP>
__host__ __device__ constexpr int march_tap(int u, int c) {
  return ((FLIP ? 2 - u % 3 : u % 3) * kMarchNodes + (FLIP ? 2 - u / 3 : u / 3) * kTileX) * c / 8;
}

// C0, C1: channels of the input segments (C1 = 0: one segment).
template <int C0, int C1, bool FLIP>
__global__ void __launch_bounds__(kMarchThreads) k_conv_march(const __grid_constant__ CUtensorMap map0,
                                                              const __grid_constant__ CUtensorMap map1,
                                                              const __grid_constant__ MarchArgs m) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const ConvArgs& p = m.c;
  constexpr int K = C0 + C1, kc = K / 8;
  const int n = p.n;
  const int stage = march_stage_bytes(K);
  uint8_t* weights = smem + m.stages * stage;
  uint64_t* full = reinterpret_cast<uint64_t*>(weights + march_weight_bytes(n, K));
  uint64_t* empty = full + kMarchMaxStages;
  uint64_t* layer = empty + kMarchMaxStages;  // one per input layer: its products are done
  uint32_t* tslot = reinterpret_cast<uint32_t*>(layer + kMarchMaxSteps);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int x0 = blockIdx.x * kTileX, y0 = blockIdx.y * kTileY;
  const int z0 = blockIdx.z * m.chunk, z1 = min(z0 + m.chunk, p.nz), layers = z1 - z0, steps = layers + 2;
  const uint32_t ncols = tmem_cols(m.chunk * n);
  // step i reads input layer z0 - 1 + i (flip: z1 - i) and adds to the
  // output layers i - 2, i - 1, i of the marching order, with the taps
  // 9 a + u, a = 2, 1, 0
  auto load = [&](int i) {  // one thread; layers outside the grid read zero
    const int s = i % m.stages, z = FLIP ? z1 - i : z0 - 1 + i;
    uint8_t* dst = smem + s * stage;
    tc::mbar_arrive_expect_tx(&full[s], static_cast<uint32_t>(stage));
    for (int dx = 0; dx < 3; ++dx) {
      tc::tma_load_4d(dst + dx * C0 * 2 * kMarchNodes, &map0, 0, x0 + dx - 1, y0 - 1, z, &full[s]);
      if (C1) tc::tma_load_4d(dst + (3 * C0 + dx * C1) * 2 * kMarchNodes, &map1, 0, x0 + dx - 1, y0 - 1, z, &full[s]);
    }
  };
  if (warp == 5 && lane == 0) {
    tc::prefetch_map(&map0);
    if (C1) tc::prefetch_map(&map1);
    for (int s = 0; s < m.stages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < steps; ++s) tc::mbar_init(&layer[s], 1);
    tc::fence_mbar_init();
    for (int i = 0; i < min(m.stages, steps); ++i) load(i);
  }
  __syncwarp();
  if (warp == 0) tc::tmem_alloc(tslot, ncols);
  // weights: tap u of the layer at [u][k chunk][row], rows (a = 2, 1, 0; column)
  const uint32_t wb = tc::smem_u32(weights);
  for (int q = warp; q < 9 * kc; q += kMarchThreads / 32) {
    const int ch = q % kc, u = q / kc;
    for (int r = lane; r < 3 * n; r += 32) {
      const int third = r >= 2 * n ? 2 : r >= n ? 1 : 0;
      const i64 row = static_cast<i64>(9 * (2 - third) + u) * n + (r - third * n);
      wg::cp16(wb + (q * 3 * n + r) * 16, m.w + row * K + ch * 8, true);
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  tc::fence_proxy_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;

  if (warp == 5) {
    if (lane == 0) {
      for (int i = m.stages; i < steps; ++i) {
        if (!tc::mbar_wait(&empty[i % m.stages], (i / m.stages - 1) & 1, p.status)) break;
        load(i);
      }
    }
  } else if (warp == 4) {
    const bool leader = tc::elect_one();
    // The taps' operand offsets are constants of the channel counts and the
    // products are unrolled: address arithmetic between them cost 150 to 350
    // cycles a tap, ten times a product.
    const uint64_t b0 = tc::smem_desc_plain(wb, 3 * n * 16, 128);
    const uint64_t a0 = tc::smem_desc(tc::smem_u32(smem), C0 * 2);
    const uint64_t a1 = tc::smem_desc(tc::smem_u32(smem) + 3 * C0 * 2 * kMarchNodes, C1 ? C1 * 2 : 32);
    const int bk = 2 * 3 * n;  // two k chunks of the weights, in 16 bytes
    int s = 0, phase = 0;
    bool ok = true;
    for (int i = 0; i < steps && ok; ++i) {
      ok = tc::mbar_wait(&full[s], phase, p.status);
      if (!ok) break;
      tc::fence_after_sync();
      // output layers [lo, hi] of the marching order, weight rows from a = 2's
      const int lo = max(i - 2, 0), hi = min(i, layers - 1);
      const uint32_t d = tmem + lo * n, before = static_cast<uint32_t>(hi - lo) * n;
      const uint32_t id = tc::idesc_bf16(128, (hi - lo + 1) * n);
      const uint64_t as0 = a0 + s * (stage >> 4), as1 = a1 + s * (stage >> 4);
      uint64_t b = b0 + (lo - (i - 2)) * n;  // past the rows of layers before the chunk
      if (leader) {
        if (hi == i) {  // output layer i starts here: its columns are overwritten
          if (before) tc::mma_bf16(d, as0 + march_tap<FLIP>(0, C0), b, tc::idesc_bf16(128, before), 1u);
          tc::mma_bf16(d + before, as0 + march_tap<FLIP>(0, C0), b + before, tc::idesc_bf16(128, n), 0u);
        } else {
          tc::mma_bf16(d, as0 + march_tap<FLIP>(0, C0), b, id, 1u);
        }
        b += bk;
#pragma unroll
        for (int u = 0; u < 9; ++u) {
#pragma unroll
          for (int k = u == 0 ? 1 : 0; k < C0 / 16; ++k) {
            tc::mma_bf16(d, as0 + march_tap<FLIP>(u, C0) + 2 * k, b, id, 1u);
            b += bk;
          }
#pragma unroll
          for (int k = 0; k < C1 / 16; ++k) {
            tc::mma_bf16(d, as1 + march_tap<FLIP>(u, C1) + 2 * k, b, id, 1u);
            b += bk;
          }
        }
        tc::mma_commit(&empty[s]);
        tc::mma_commit(&layer[i]);
      }
      __syncwarp();
      if (++s == m.stages) {
        s = 0;
        phase ^= 1;
      }
    }
  } else {
    // output node of this thread: row 32 warp + lane of the 32 x 4 tile
    const int gx = x0 + lane, gy = y0 + warp;
    const bool in = gx < p.nx && gy < p.ny;
    bool ok = true;
    for (int q = 0; q < layers; ++q) {
      ok = ok && tc::mbar_wait(&layer[q + 2], 0, p.status);
      __syncwarp();
      tc::fence_after_sync();
      const int gz = FLIP ? z1 - 1 - q : z0 + q;
      const long long node = (static_cast<long long>(gz) * p.ny + gy) * p.nx + gx;
      for (int col = 0; col < n; col += 16) {
        float v[16];
        tc::tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(q * n + col), v);
        if (in && ok) conv_store(p, node, col, v);
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

}  // namespace conv
}  // namespace simp
