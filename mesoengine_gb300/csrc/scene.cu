// scene.cu -- device-resident brick-map scenes: build from the seeded terrain
// generator or from a dense grid, the dense/chunk generators of the meshing
// workloads, and sphere edits with a device brick allocator.
//
// The reference keeps chunks as host vectors of blocks in ring-buffer pools
// with importance eviction (Runtimes/Voxel/Chunk/ChunkPool.h:83-181,
// :446-622) and regenerates them from a sin-hash SDF on host threads
// (Runtimes/Helper/GeneratorHelper.h:120-150).  Here a scene is three device
// arrays: a pointer grid (one uint32 per 8^3 brick, all-ones = empty, the
// reference's INT_MAX-sentinel idea, Runtimes/Voxel/Block/Block.h:16-18), a
// pool of 64-byte occupancy masks (word z, bit x+8y; the FVolume 8^3 bitmask of
// Runtimes/Voxel/VoxelStructure.h:30-39) and a pool of 1 KiB uint16 material
// bricks.  Bricks are numbered in pointer-grid order by an exclusive scan, so
// a build is deterministic.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <set>
#include <vector>

#include "meso_internal.h"

namespace meso {
namespace {

using namespace ::meso::dev;

constexpr uint32_t kFull = 0xFFFFFFFFu;

struct TerrainDev {
  int32_t nx, ny, nz;
  uint32_t seed, height_period;
  int32_t height_octaves;
  float height_base, height_amp;
  uint32_t cave_period;
  float cave_threshold;
};

TerrainDev to_dev(const meso_terrain& t) {
  TerrainDev d;
  d.nx = t.nx;
  d.ny = t.ny;
  d.nz = t.nz;
  d.seed = t.seed;
  d.height_period = t.height_period;
  d.height_octaves = t.height_octaves;
  d.height_base = t.height_base;
  d.height_amp = t.height_amp;
  d.cave_period = t.cave_period;
  d.cave_threshold = t.cave_threshold;
  return d;
}

__device__ __forceinline__ uint16_t terrain_voxel(const TerrainDev& T, float h, uint32_t x, uint32_t y, uint32_t z) {
  if (!(__uint2float_rn(z) < h)) return 0;
  const float c = vnoise3(x, y, z, T.cave_period, T.seed + 100u);
  if (c > T.cave_threshold) return 0;
  const int depth = (int)floorf(h) - (int)z;
  return (uint16_t)(1 + ((depth >> 2) & 63));
}

__global__ void heights_kernel(TerrainDev T, float* heights) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= (uint64_t)T.nx * T.ny) return;
  const uint32_t x = (uint32_t)(i % T.nx), y = (uint32_t)(i / T.nx);
  const float f = fbm2(x, y, T.height_period, T.height_octaves, T.seed);
  heights[i] = __fadd_rn(T.height_base, __fmul_rn(T.height_amp, f));
}

__global__ void column_max_kernel(TerrainDev T, const float* heights, float* hmax) {
  const int bx = T.nx / 8, by = T.ny / 8;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= bx * by) return;
  const int X = (i % bx) * 8, Y = (i / bx) * 8;
  float m = -__builtin_huge_valf();
  for (int ly = 0; ly < 8; ly++)
    for (int lx = 0; lx < 8; lx++) m = fmaxf(m, heights[(size_t)(Y + ly) * T.nx + X + lx]);
  hmax[i] = m;
}

// The non-empty 2x2x2-voxel blocks of a brick (bit x + 4y + 16z) from its
// occupancy as 16 words of 32 voxels (word k: z = k/2, rows y = 4(k mod 2) ..
// +3 of 8 bits each).
__device__ __forceinline__ uint64_t sub_mask(const uint32_t (&w)[16]) {
  uint64_t m = 0;
#pragma unroll
  for (int z = 0; z < 4; z++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint32_t v = w[4 * z + h] | w[4 * z + 2 + h];  // both layers
      v |= v >> 8;                                   // both rows: bytes 0 and 2
      v |= v >> 1;                                   // both columns: even bits
      v &= 0x00550055u;
      v = (v | v >> 1) & 0x00330033u;
      v = (v | v >> 2) & 0x000F000Fu;
      m |= (uint64_t)((v | v >> 12) & 0xFFu) << (16 * z + 8 * h);
    }
  return m;
}

// Of the 8 squares of 2x2 voxels in 4 rows of 8 bits each: how many hold voxels and
// are not solid, and 16 bits higher how many are not solid.
__device__ __forceinline__ uint32_t square_counts(uint32_t rows) {
  uint32_t some = rows | rows >> 8, solid = rows & rows >> 8;
  some = (some | some >> 1) & 0x00550055u;
  solid = solid & solid >> 1 & 0x00550055u;
  return (uint32_t)__popc(some & ~solid) | (8u - (uint32_t)__popc(solid)) << 16;
}

// One warp per brick; lane covers voxels lane + 32k (x = i&7, y = (i>>3)&7, z = i>>6).
template <bool kFill>
__global__ void terrain_brick_kernel(TerrainDev T, const float* heights, const float* hmax, uint8_t* flags,
                                     const uint32_t* ptr, uint64_t* occ, uint16_t* mat) {
  const int bx = T.nx / 8, by = T.ny / 8, bz = T.nz / 8;
  const uint64_t nb = (uint64_t)bx * by * bz;
  const int lane = threadIdx.x & 31;
  const uint64_t wstride = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t b = blockIdx.x * (uint64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); b < nb; b += wstride) {
    const int X = (int)(b % bx), Y = (int)((b / bx) % by), Z = (int)(b / ((uint64_t)bx * by));
    if (kFill) {
      if (!flags[b]) continue;
    } else {
      if (!((float)(Z * 8) < hmax[(size_t)Y * bx + X])) {
        if (lane == 0) flags[b] = 0;
        continue;
      }
    }
    const uint32_t slot = kFill ? ptr[b] : 0u;
    bool any = false;
    for (int k = 0; k < 16; k++) {
      const int i = lane + 32 * k;
      const uint32_t x = X * 8 + (i & 7), y = Y * 8 + ((i >> 3) & 7), z = Z * 8 + (i >> 6);
      const float h = heights[(size_t)y * T.nx + x];
      const uint16_t m = terrain_voxel(T, h, x, y, z);
      if (kFill) {
        mat[(size_t)slot * 512 + i] = m;
        // voxel i = lane + 32k is bit (i mod 32) of 32-bit word k of the
        // brick's occupancy (word z of 64 bits = 32-bit words 2z, 2z+1)
        const uint32_t bits = __ballot_sync(kFull, m != 0);
        if (lane == 0) reinterpret_cast<uint32_t*>(occ + (size_t)slot * 8)[k] = bits;
      } else {
        any |= m != 0;
      }
    }
    if (!kFill) {
      const bool f = __any_sync(kFull, any);
      if (lane == 0) flags[b] = f ? 1 : 0;
    }
  }
}

// ---------------------------------------------------------------- scan
constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr int kScanTile = kScanThreads * kScanPer;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0u;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, s, o);
      if (lane >= o) s += y;
    }
    warp_sums[lane] = s;  // inclusive
  }
  __syncthreads();
  const uint32_t before = warp ? warp_sums[warp - 1] : 0u;
  total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before + x - v;
}

// flags (uint8) -> out (exclusive prefix within tile), tile sums.
__global__ void scan_tiles_kernel(const uint8_t* flags, uint64_t n, uint32_t* out, uint32_t* tile_sums) {
  __shared__ uint32_t ws[32];
  const uint64_t base = blockIdx.x * (uint64_t)kScanTile + threadIdx.x * (uint64_t)kScanPer;
  uint32_t v[kScanPer], s = 0;
  for (int k = 0; k < kScanPer; k++) {
    v[k] = (base + k < n) ? flags[base + k] : 0u;
    s += v[k];
  }
  uint32_t total;
  uint32_t ex = block_exclusive_scan(s, ws, total);
  for (int k = 0; k < kScanPer; k++) {
    if (base + k < n) out[base + k] = ex;
    ex += v[k];
  }
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// single block: exclusive scan of tile sums in place; grand total to *total.
__global__ void scan_sums_kernel(uint32_t* sums, uint32_t n, uint32_t* total) {
  __shared__ uint32_t ws[32];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < n; base += kScanThreads) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < n ? sums[i] : 0u;
    uint32_t t;
    const uint32_t ex = block_exclusive_scan(v, ws, t);
    if (i < n) sums[i] = carry + ex;
    carry += t;
  }
  if (threadIdx.x == 0) *total = carry;
}

// ptr[b] = flags[b] ? tile offset + local : EMPTY
__global__ void scan_finish_kernel(const uint8_t* flags, uint64_t n, const uint32_t* tile_sums, uint32_t* ptr) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  ptr[i] = flags[i] ? ptr[i] + tile_sums[i / kScanTile] : MESO_EMPTY_BRICK;
}

// Numbers bricks flagged nonzero in pointer-grid order.  Returns the count.
meso_status number_bricks(meso_ctx* ctx, const uint8_t* d_flags, uint64_t nb, uint32_t* d_ptr, cudaStream_t st,
                          uint64_t* count) {
  const uint64_t tiles = (nb + kScanTile - 1) / kScanTile;
  if (tiles > 0xFFFFFFFFull) return fail(MESO_ERR_INVALID_ARG, "scene too large");
  uint32_t* d_sums = nullptr;
  MESO_CUDA_TRY(dev_malloc_async(ctx, &d_sums, sizeof(uint32_t) * (tiles + 1), st));
  scan_tiles_kernel<<<(unsigned)tiles, kScanThreads, 0, st>>>(d_flags, nb, d_ptr, d_sums);
  scan_sums_kernel<<<1, kScanThreads, 0, st>>>(d_sums, (uint32_t)tiles, d_sums + tiles);
  scan_finish_kernel<<<(unsigned)((nb + 255) / 256), 256, 0, st>>>(d_flags, nb, d_sums, d_ptr);
  ctx->launches.fetch_add(3);
  uint32_t h_total = 0;
  MESO_CUDA_TRY(cudaMemcpyAsync(&h_total, d_sums + tiles, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  MESO_CUDA_TRY(cudaFreeAsync(d_sums, st));
  MESO_CUDA_TRY(cudaStreamSynchronize(st));
  MESO_CUDA_TRY(cudaGetLastError());
  *count = h_total;
  return MESO_OK;
}

// Numbers the set bits of n words in order: base[i] = set bits before word i,
// *total = all of them.  One block; a thread takes 8 words of a tile, and the next
// tile's words are on their way while this one is scanned.  (Three launches over
// a byte per brick and a copy of the pointers took a build 14 us longer: 512^3
// uint16 195 us and now 181, 256^3 89 and 72.  Of a uint8 build's kernels this one is 8
// of 88 us at 512^3, 40 of 635 at 1024^3, 299 of 5,050 at 2048^3; those three took 11,
// 21 and 114 there, of 312, 2,507 and 18,945.)
// It also adds up the sampled square_counts: total[1] and [2].
__global__ void __launch_bounds__(kScanThreads) scan_words_kernel(const uint32_t* words, uint64_t n, uint32_t* base,
                                                                  uint32_t* total, const uint32_t* squares,
                                                                  uint32_t n_squares) {
  __shared__ uint32_t ws[32];
  __shared__ uint32_t sums[2];
  if (threadIdx.x < 2) sums[threadIdx.x] = 0;
  uint32_t mixed = 0, open = 0;
  for (uint32_t i = threadIdx.x; i < n_squares; i += kScanThreads) {
    const uint32_t q = squares[i];
    mixed += q & 0xFFFFu;
    open += q >> 16;
  }
  constexpr int kPer = 8;
  uint32_t carry = 0, v[kPer];
  auto load = [&](uint64_t i0) {
#pragma unroll
    for (int k = 0; k < kPer; k++) v[k] = i0 + k < n ? words[i0 + k] : 0u;
  };
  load((uint64_t)threadIdx.x * kPer);
  for (uint64_t t = 0; t < n; t += (uint64_t)kScanThreads * kPer) {
    const uint64_t i0 = t + (uint64_t)threadIdx.x * kPer;
    uint32_t c[kPer], s = 0, all;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
      c[k] = s;
      s += __popc(v[k]);
    }
    load(i0 + (uint64_t)kScanThreads * kPer);
    const uint32_t ex = carry + block_exclusive_scan(s, ws, all);
#pragma unroll
    for (int k = 0; k < kPer; k++)
      if (i0 + k < n) base[i0 + k] = ex + c[k];
    carry += all;
  }
  __syncthreads();  // (sums are clear, with no tile too)
  mixed = __reduce_add_sync(kFull, mixed);
  open = __reduce_add_sync(kFull, open);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sums[0], mixed);
    atomicAdd(&sums[1], open);
  }
  __syncthreads();
  if (threadIdx.x < 3) total[threadIdx.x] = threadIdx.x ? sums[threadIdx.x - 1] : carry;
}

// ---------------------------------------------------------- dense -> bricks
// T: uint16_t or uint8_t materials of a dense grid (x fastest).
//
// Both passes are bound by HBM: the grid is read once to see which bricks hold
// anything, the occupied bricks again to be copied.  A CTA of 8 warps takes 32
// bricks that follow one another in the pointer grid; lane = brick, warp = z
// layer, so the 8 voxel rows of a lane are 16-byte (uint8: 8-byte) loads that
// are all in flight together, and a warp's loads cover whole lines along x.
// 512^3 uint16 (268 MB, 62 % of its bricks occupied): flags 112 us with a warp
// per brick reading 2 bytes per lane, 41 us now; fill 204 us and 70 us (6.5 and
// 4.9 TB/s of the bytes each has to move).  What the first pass read last is
// still in L2 when the second begins, so that one goes backwards and lets its
// output stream past: a build of 512x512x256 uint16 142 -> 132 us, of 512^3 uint8
// 157 -> 152; of 512^3 uint16, twice the L2, 194 and 193.
constexpr int kDenseBricks = 32, kDenseThreads = 256;

// The 8 voxels of a brick row as 8 uint16.  kWide: the grid's base is aligned
// to the load (its rows are, as nx is a multiple of 32); else element by
// element.
// kKeep: read again soon.
template <typename T, bool kWide, bool kKeep = false>
__device__ __forceinline__ uint4 load_row8(const T* src) {
  if constexpr (kWide && sizeof(T) == 2) {
    return kKeep ? __ldcg(reinterpret_cast<const uint4*>(src)) : __ldcs(reinterpret_cast<const uint4*>(src));
  } else if constexpr (kWide) {
    const uint2 v = kKeep ? __ldcg(reinterpret_cast<const uint2*>(src)) : __ldcs(reinterpret_cast<const uint2*>(src));
    return make_uint4(__byte_perm(v.x, 0, 0x4140), __byte_perm(v.x, 0, 0x4342), __byte_perm(v.y, 0, 0x4140),
                      __byte_perm(v.y, 0, 0x4342));
  } else {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = (uint32_t)src[2 * k] | (uint32_t)src[2 * k + 1] << 16;
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// Bit x set iff uint16 x of the row is not zero.
__device__ __forceinline__ uint32_t row8_bits(const uint4& v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t b = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) b |= ((w[k] & 0xFFFFu) != 0 ? 1u : 0u) << (2 * k) | (w[k] > 0xFFFFu ? 2u : 0u) << (2 * k);
  return b;
}

// First voxel of layer z of brick b.
template <typename T>
__device__ __forceinline__ const T* brick_layer(const T* grid, int nx, int ny, uint64_t b, int z) {
  const uint32_t bx = (uint32_t)nx / 8u, by = (uint32_t)ny / 8u;
  const uint32_t X = (uint32_t)(b % bx), YZ = (uint32_t)(b / bx), Y = YZ % by, Z = YZ / by;
  return grid + ((size_t)X * 8 + (size_t)nx * ((size_t)Y * 8 + (size_t)ny * ((size_t)Z * 8 + (size_t)z)));
}

template <typename T, bool kWide>
__global__ void __launch_bounds__(kDenseThreads) dense_flag_kernel(const T* grid, int nx, int ny, uint64_t nb,
                                                                   uint32_t* occupied, uint32_t* squares, uint32_t step) {
  __shared__ uint32_t any[kDenseThreads / 32], counts[kDenseThreads / 32];
  const int lane = threadIdx.x & 31, z = threadIdx.x >> 5;
  const uint64_t b = (uint64_t)blockIdx.x * kDenseBricks + lane;
  const bool sample = blockIdx.x % step == 0;  // of the squares, every step-th block's
  uint32_t acc = 0, q = 0;
  if (b < nb) {
    const T* src = brick_layer(grid, nx, ny, b, z);
    uint4 v[8];
#pragma unroll
    for (int y = 0; y < 8; y++) v[y] = load_row8<T, kWide, true>(src + (size_t)nx * y);
#pragma unroll
    for (int y = 0; y < 8; y++) acc |= v[y].x | v[y].y | v[y].z | v[y].w;
    if (sample) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t rows = 0;
#pragma unroll
        for (int y = 0; y < 4; y++) rows |= row8_bits(v[4 * h + y]) << (8 * y);
        q += square_counts(rows);
      }
    }
  }
  const uint32_t bits = __ballot_sync(kFull, acc != 0);
  if (sample) q = __reduce_add_sync(kFull, q);
  if (lane == 0) {
    any[z] = bits;
    counts[z] = q;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t m = 0, n = 0;
#pragma unroll
    for (int k = 0; k < kDenseThreads / 32; k++) {
      m |= any[k];
      n += counts[k];
    }
    occupied[blockIdx.x] = m;
    if (sample) squares[blockIdx.x / step] = n;
  }
}

// The layers go through shared memory (rows padded by 16 bytes against bank
// conflicts), so that a warp writes the 128 contiguous bytes of 4 bricks'
// layers per store and a brick's 8 occupancy words leave together.
template <typename T, bool kWide>
__global__ void __launch_bounds__(kDenseThreads) dense_fill_kernel(const T* grid, int nx, int ny, uint64_t nb,
                                                                   const uint32_t* occupied, const uint32_t* base,
                                                                   uint32_t* ptr, uint64_t* occ, uint16_t* mat,
                                                                   uint64_t* sub) {
  __shared__ uint4 rows[kDenseThreads / 32][8][kDenseBricks + 1];
  __shared__ uint64_t words[kDenseBricks][9];
  __shared__ uint32_t slots[kDenseBricks];
  const int lane = threadIdx.x & 31, z = threadIdx.x >> 5;
  const uint32_t group = gridDim.x - 1u - blockIdx.x, m = occupied[group];
  const uint64_t b = (uint64_t)group * kDenseBricks + lane;
  const uint32_t slot = (m >> lane) & 1u ? base[group] + __popc(m & ((1u << lane) - 1u)) : MESO_EMPTY_BRICK;
  if (z == 0) {
    slots[lane] = slot;
    if (b < nb) ptr[b] = slot;
  }
  uint64_t word = 0;
  if (slot != MESO_EMPTY_BRICK) {
    const T* src = brick_layer(grid, nx, ny, b, z);
    uint4 v[8];
#pragma unroll
    for (int y = 0; y < 8; y++) v[y] = load_row8<T, kWide>(src + (size_t)nx * y);
#pragma unroll
    for (int y = 0; y < 8; y++) {
      word |= (uint64_t)row8_bits(v[y]) << (8 * y);
      rows[z][y][lane] = v[y];
    }
  }
  words[lane][z] = word;
  __syncthreads();
  // store k of a warp: layer z of bricks 4k .. 4k+3, 8 lanes (rows) each
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int brick = 4 * k + (lane >> 3);
    const uint32_t s = slots[brick];
    if (s != MESO_EMPTY_BRICK)
      __stcs(reinterpret_cast<uint4*>(mat) + (size_t)s * 64 + z * 8 + (lane & 7), rows[z][lane & 7][brick]);
  }
  if (z == 0 && slot != MESO_EMPTY_BRICK) {
    uint32_t w[16];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      w[2 * k] = (uint32_t)words[lane][k];
      w[2 * k + 1] = (uint32_t)(words[lane][k] >> 32);
    }
    sub[slot] = sub_mask(w);
  }
  const int brick = threadIdx.x >> 3;
  const uint32_t s = slots[brick];
  if (s != MESO_EMPTY_BRICK) occ[(size_t)s * 8 + (threadIdx.x & 7)] = words[brick][threadIdx.x & 7];
}

// ------------------------------------------------------------- generators
__global__ void dense_u8_kernel(int nx, int ny, int nz, uint32_t seed, uint8_t* out) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= (uint64_t)nx * ny * nz) return;
  const uint32_t x = (uint32_t)(i % nx), y = (uint32_t)((i / nx) % ny), z = (uint32_t)(i / ((uint64_t)nx * ny));
  const float n0 = vnoise3(x, y, z, 64, seed);
  float n1 = vnoise3(x, y, z, 32, seed + 1);
  float n2 = vnoise3(x, y, z, 16, seed + 2);
  float s = n0;
  n1 = __fmul_rn(n1, 0.5f);
  s = __fadd_rn(s, n1);
  n2 = __fmul_rn(n2, 0.25f);
  s = __fadd_rn(s, n2);
  s = __fdiv_rn(s, 1.75f);
  uint8_t m = 0;
  if (s > 0.5f) m = (uint8_t)(1 + (int)floorf(__fmul_rn(s, 15.0f)));
  out[i] = m;
}

// One CTA (1024 threads) per standalone chunk: keys = 17-bit quantised value
// noise (period 8) over (32767 - index), the k-th largest key found by a
// 4-pass radix select, solid iff key >= it; material 1 + hash mod m.
__global__ void __launch_bounds__(1024) chunks_u16_kernel(uint32_t seed0, const uint32_t* targets, uint16_t* out,
                                                          uint32_t* solid_count) {
  extern __shared__ uint32_t keys[];  // 32768
  __shared__ uint32_t hist[256];
  __shared__ uint32_t s_prefix, s_k;
  const uint32_t c = blockIdx.x, seed = seed0 + c;
  const uint32_t k = targets[c];
  for (uint32_t i = threadIdx.x; i < 32768u; i += blockDim.x) {
    const float n = vnoise3(i & 31u, (i >> 5) & 31u, i >> 10, 8, seed);
    uint32_t q = (uint32_t)floorf(__fmul_rn(n, 131072.0f));
    if (q > 131071u) q = 131071u;
    keys[i] = (q << 15) | (32767u - i);
  }
  uint32_t prefix = 0, pmask = 0, kk = k;
  for (int shift = 24; shift >= 0 && k > 0; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < 32768u; i += blockDim.x) {
      const uint32_t key = keys[i];
      if ((key & pmask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t cum = 0;
      for (int d = 255; d >= 0; d--) {
        if (cum + hist[d] >= kk) {
          prefix |= (uint32_t)d << shift;
          kk -= cum;
          break;
        }
        cum += hist[d];
      }
      s_prefix = prefix;
      s_k = kk;
    }
    __syncthreads();
    prefix = s_prefix;
    kk = s_k;
    pmask |= 255u << shift;
  }
  const uint32_t m = 1u + pcg3d(seed, 0x77u, 0x3u) % 64u;
  uint16_t* dst = out + (size_t)c * 32768u;
  for (uint32_t i = threadIdx.x; i < 32768u; i += blockDim.x) {
    const bool solid = k > 0 && keys[i] >= prefix;
    dst[i] = solid ? (uint16_t)(1u + pcg3d(i, seed, 0x9E37u) % m) : (uint16_t)0;
  }
  if (threadIdx.x == 0 && solid_count) solid_count[c] = k;
}

// ------------------------------------------------------------------ edits
struct EditParams {
  const meso_sphere_edit* spheres;
  uint32_t n_spheres;
  const uint32_t* bricks;  // touched linear brick indices
  uint32_t n_bricks;
  int32_t bx, by;
  uint32_t* ptr;
  uint64_t* occ;
  uint16_t* mat;
  uint64_t* sub;
  uint16_t* temp;          // 512 per touched brick
  uint8_t* state;          // per touched brick: bit0 present, bit1 nonempty
  uint32_t* free_stack;
  int32_t* alloc;          // [0] bump, [1] top
  uint32_t capacity;
  uint32_t* err;
};

__global__ void edit_compute_kernel(EditParams P) {
  const int lane = threadIdx.x & 31;
  const uint32_t wi = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wi >= P.n_bricks) return;
  const uint32_t b = P.bricks[wi];
  const int X = (int)(b % P.bx) * 8, Y = (int)((b / P.bx) % P.by) * 8, Z = (int)(b / ((uint32_t)P.bx * P.by)) * 8;
  const uint32_t slot = P.ptr[b];
  const bool present = slot != MESO_EMPTY_BRICK;
  uint16_t v[16];
  for (int k = 0; k < 16; k++) v[k] = present ? P.mat[(size_t)slot * 512 + lane + 32 * k] : (uint16_t)0;
  for (uint32_t s = 0; s < P.n_spheres; s++) {
    const meso_sphere_edit e = P.spheres[s];
    const int r = e.radius;
    if (e.center[0] + r < X || e.center[0] - r > X + 7 || e.center[1] + r < Y || e.center[1] - r > Y + 7 ||
        e.center[2] + r < Z || e.center[2] - r > Z + 7)
      continue;
    const int r2 = r * r;
    for (int k = 0; k < 16; k++) {
      const int i = lane + 32 * k;
      const int dx = X + (i & 7) - e.center[0], dy = Y + ((i >> 3) & 7) - e.center[1], dz = Z + (i >> 6) - e.center[2];
      if (dx * dx + dy * dy + dz * dz <= r2) v[k] = e.material;
    }
  }
  bool any = false;
  for (int k = 0; k < 16; k++) any |= v[k] != 0;
  const bool nonempty = __any_sync(kFull, any);
  if (present && nonempty) {
    uint32_t w[16];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      P.mat[(size_t)slot * 512 + lane + 32 * k] = v[k];
      w[k] = __ballot_sync(kFull, v[k] != 0);
      if (lane == 0) reinterpret_cast<uint32_t*>(P.occ + (size_t)slot * 8)[k] = w[k];
    }
    if (lane == 0) P.sub[slot] = sub_mask(w);
  } else if (present && !nonempty) {
    if (lane == 0) {
      P.ptr[b] = MESO_EMPTY_BRICK;
      const int t = atomicAdd(&P.alloc[1], 1);
      P.free_stack[t] = slot;
    }
  } else if (!present && nonempty) {
    for (int k = 0; k < 16; k++) P.temp[(size_t)wi * 512 + lane + 32 * k] = v[k];
  }
  if (lane == 0) P.state[wi] = (uint8_t)((present ? 1 : 0) | (nonempty ? 2 : 0));
}

__global__ void edit_alloc_kernel(EditParams P) {
  const int lane = threadIdx.x & 31;
  const uint32_t wi = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wi >= P.n_bricks) return;
  if (P.state[wi] != 2) return;  // absent and now nonempty
  uint32_t slot = 0;
  int ok = 1;
  if (lane == 0) {
    const int t = atomicSub(&P.alloc[1], 1) - 1;
    if (t >= 0) {
      slot = P.free_stack[t];
    } else {
      const int nb = atomicAdd(&P.alloc[0], 1);
      if ((uint32_t)nb >= P.capacity) {
        ok = 0;
        atomicOr(P.err, ERR_POOL_FULL);
      } else {
        slot = (uint32_t)nb;
      }
    }
  }
  ok = __shfl_sync(kFull, ok, 0);
  slot = __shfl_sync(kFull, slot, 0);
  if (!ok) return;
  const uint32_t b = P.bricks[wi];
  uint32_t w[16];
#pragma unroll
  for (int k = 0; k < 16; k++) {
    const uint16_t m = P.temp[(size_t)wi * 512 + lane + 32 * k];
    P.mat[(size_t)slot * 512 + lane + 32 * k] = m;
    w[k] = __ballot_sync(kFull, m != 0);
    if (lane == 0) reinterpret_cast<uint32_t*>(P.occ + (size_t)slot * 8)[k] = w[k];
  }
  if (lane == 0) {
    P.ptr[b] = slot;
    P.sub[slot] = sub_mask(w);
  }
}

// Solid voxels of the live bricks: popcount of each linked brick's 8
// occupancy words, summed per warp and added to *count.
__global__ void count_solid_kernel(const uint32_t* ptr, uint64_t nb, const uint64_t* occ,
                                   unsigned long long* count) {
  uint32_t acc = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b < nb; b += stride) {
    const uint32_t p = ptr[b];
    if (p == MESO_EMPTY_BRICK) continue;
    const uint4* w = reinterpret_cast<const uint4*>(occ + (size_t)p * 8);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint4 v = w[k];
      acc += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
    }
  }
  const uint32_t tot = __reduce_add_sync(kFull, acc);
  if ((threadIdx.x & 31) == 0 && tot) atomicAdd(count, (unsigned long long)tot);
}

unsigned grid_for(uint64_t warps, int threads = 256) {
  const uint64_t per = threads / 32;
  uint64_t b = (warps + per - 1) / per;
  if (b > 1048576) b = 1048576;
  return (unsigned)(b ? b : 1);
}

}  // namespace

// One warp per macro cell (4x4x4 bricks): the mask of its occupied bricks
// (bit x + 4y + 16z), and a byte that says whether there are any.  Its first
// threads also do what must lie between the kernels before and behind it: of a
// whole rebuild, reset the bounds and clear the word before the block masks; of an
// edit (cells given), bring the pool's counters back into their range where
// allocations overran it.
__global__ void macro_kernel(const uint32_t* ptr, int bx, int by, uint8_t* macro, uint64_t* mask, int32_t* bounds,
                             uint64_t* sub, int32_t* alloc, uint32_t capacity, const uint32_t* cells, uint64_t n) {
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (blockIdx.x == 0) {
    if (!cells) {
      if (threadIdx.x < 8) bounds[threadIdx.x] = INT32_MIN / 2;  // nothing occupied
      if (threadIdx.x == 8) sub[-1] = 0;
    } else if (threadIdx.x == 0) {
      if (alloc[1] < 0) alloc[1] = 0;
      if ((uint32_t)alloc[0] > capacity) alloc[0] = (int32_t)capacity;
    }
  }
  if (w >= n) return;
  const uint32_t m = cells ? cells[w] : (uint32_t)w;
  const int mx = bx >> 2, my = by >> 2;
  const int cx = (int)(m % (uint32_t)mx), cy = (int)((m / (uint32_t)mx) % (uint32_t)my), cz = (int)(m / ((uint32_t)mx * my));
  const int x = cx * 4 + (lane & 3), y = cy * 4 + ((lane >> 2) & 3), z = cz * 4 + (lane >> 4);
  const uint64_t i = (uint64_t)x + (uint64_t)bx * ((uint64_t)y + (uint64_t)by * z);
  const uint32_t lo = __ballot_sync(0xFFFFFFFFu, ptr[i] != MESO_EMPTY_BRICK);
  const uint32_t hi = __ballot_sync(0xFFFFFFFFu, ptr[i + 2ull * bx * by] != MESO_EMPTY_BRICK);
  if (lane == 0) {
    macro[m] = (lo | hi) != 0 ? 1 : 0;
    mask[m] = (uint64_t)hi << 32 | lo;
  }
}

// Level bytes: per brick log2 of the edge, in voxels, of the largest aligned
// cube of empty space that it is part of and that lies in the grid (9: 64^3
// bricks .. 3: the brick), 0 if it is occupied; and the bounds of the occupied
// cells, widened where a 64^3-brick cell holds some outside them (looked at
// before, so that few send an atomic).
//
// The bricks of one 64^3-brick cell depend on nothing outside it, so an edit
// recomputes those of the cells it touches (list), a build all of them: 32
// blocks each, a thread per 4x4x4-brick cell.  Every block reads the cell's
// 16^3 occupancy bytes (4 KB, of which the 32 share the fetches) and derives the
// coarser levels itself.  (With the 16^3- and 64^3-brick cells' maps from two
// launches in between, and two more for what macro_kernel's first threads do, a
// 512^3 build took 202 us and now 194, 16 sphere edits with remesh and frame 318
// and now 308.)
constexpr int kLevelThreads = 128;

__global__ void __launch_bounds__(kLevelThreads)
    level_kernel(const uint64_t* mask, const uint8_t* macro, int bx, int by, int bz, uint8_t* level, int32_t* bounds,
                 const uint32_t* list) {
  // two rows of 16 4x4x4-brick cells a word (y = 2i and 2i + 1), bit x, outside of the grid set
  __shared__ uint32_t rows[16 * 8];
  __shared__ uint32_t set2[2];  // 16^3-brick cells that are not empty or reach past the grid, bit x + 4y + 16z
  const int mx = bx / 4, my = by / 4, mz = bz / 4;
  const uint32_t m3x = (uint32_t)(bx + 63) / 64, m3y = (uint32_t)(by + 63) / 64;
  const uint32_t r = list ? list[blockIdx.x >> 5] : blockIdx.x >> 5;
  const int ox = (int)(r % m3x) * 16, oy = (int)((r / m3x) % m3y) * 16, oz = (int)(r / (m3x * m3y)) * 16;
  const int t = (int)threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll 8
  for (int k = 0; k < 32; k++) {  // warp: layers 4 warp .. 4 warp + 3
    const int x = ox + (lane & 15), y = oy + 2 * (k & 7) + (lane >> 4), z = oz + 4 * warp + (k >> 3);
    const bool in = x < mx && y < my && z < mz;
    const uint32_t w = __ballot_sync(0xFFFFFFFFu, !in || macro[(size_t)x + (size_t)mx * ((size_t)y + (size_t)my * (size_t)z)] != 0);
    if (lane == 0) rows[32 * warp + k] = w;
  }
  __syncthreads();
  if (t < 64) {
    uint32_t any = 0;  // child (t & 3, t >> 2 & 3, t >> 4): 4 layers of 2 words
#pragma unroll
    for (int k = 0; k < 8; k++) any |= rows[32 * (t >> 4) + 8 * (k >> 1) + 2 * ((t >> 2) & 3) + (k & 1)];
    any |= any >> 16;
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, (any >> (4 * (t & 3))) & 15u);
    if (lane == 0) set2[warp] = b;
  } else if (warp == 2 && (blockIdx.x & 31u) == 0) {
    uint32_t xs = 0, ys = 0, zs = 0;
    const uint32_t inx = mx - ox < 16 ? (1u << (mx - ox)) - 1u : 0xFFFFu;
    for (int k = lane; k < 128; k += 32) {
      const int y = 2 * (k & 7), z = k >> 3;
      const uint32_t a = oz + z < mz && oy + y < my ? rows[k] & inx : 0u;
      const uint32_t b = oz + z < mz && oy + y + 1 < my ? (rows[k] >> 16) & inx : 0u;
      xs |= a | b;
      ys |= (uint32_t)(a != 0) << y | (uint32_t)(b != 0) << (y + 1);
      zs |= (uint32_t)((a | b) != 0) << z;
    }
    xs = __reduce_or_sync(0xFFFFFFFFu, xs);
    ys = __reduce_or_sync(0xFFFFFFFFu, ys);
    zs = __reduce_or_sync(0xFFFFFFFFu, zs);
    if (xs && lane < 6) {
      const int a = lane % 3;
      const uint32_t s = a == 0 ? xs : (a == 1 ? ys : zs);
      const int c = a == 0 ? ox : (a == 1 ? oy : oz);
      const int v = lane < 3 ? -32 * (c + __ffs((int)s) - 1) : 32 * (c + 31 - __clz((int)s)) + 31;
      int32_t* b = bounds + (lane < 3 ? a : 4 + a);
      if (v > *static_cast<volatile int32_t*>(b)) atomicMax(b, v);
    }
  }
  __syncthreads();
  const int k12 = (int)(blockIdx.x & 31u) * kLevelThreads + t;  // the thread's cell of the 16^3
  const int lx = k12 & 15, ly = (k12 >> 4) & 15, lz = k12 >> 8;
  const int cx = ox + lx, cy = oy + ly, cz = oz + lz;
  if (cx >= mx || cy >= my || cz >= mz) return;
  const uint64_t bricks = mask[(size_t)cx + (size_t)mx * ((size_t)cy + (size_t)my * (size_t)cz)];
  uint32_t l;
  if (bricks) l = 0;
  else if ((set2[0] | set2[1]) == 0) l = 9;
  else {
    const uint32_t half = set2[lz >> 3] >> ((lx >> 2 & 2) + 4 * (ly >> 2 & 2));  // the aligned 2x2x2 children's
    const uint32_t* w = rows + 8 * (lz & ~1) + (ly >> 1);                        // the aligned 2x2x2 cells'
    if ((half & 0x330033u) == 0) l = 8;
    else if (!((set2[lz >> 3] >> ((lx >> 2) + 4 * (ly >> 2) + 16 * (lz >> 2 & 1))) & 1u)) l = 7;
    else if ((((w[0] | w[8]) >> (lx & ~1)) & 0x30003u) == 0) l = 6;
    else l = 5;
  }
  // 16 rows of 4 bricks, a byte each
  uint32_t* dst = reinterpret_cast<uint32_t*>(level) + (size_t)cx + (size_t)mx * ((size_t)cy * 4 + (size_t)by * ((size_t)cz * 4));
#pragma unroll
  for (int k = 0; k < 16; k++) {
    uint32_t v = l * 0x01010101u;
    if (bricks) {
      const int y = k & 3, z = k >> 2;
#pragma unroll
      for (int x = 0; x < 4; x++) {
        const bool set = (bricks >> (x + 4 * y + 16 * z)) & 1ull;
        const bool block = (bricks >> ((x & 2) + 4 * (y & 2) + 16 * (z & 2))) & 0x330033ull;
        v |= (set ? 0u : (block ? 3u : 4u)) << (8 * x);
      }
    }
    dst[(size_t)mx * ((size_t)(k & 3) + (size_t)by * (size_t)(k >> 2))] = v;
  }
}

// d_sub of `slots` consecutive pool slots, one thread each; their square_counts are
// added to counts[0] and [1].
__global__ void sub_kernel(const uint64_t* occ, uint64_t slots, uint64_t* sub, unsigned long long* counts) {
  const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(occ + p * 8);
  uint32_t w[16];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint4 v = p < slots ? src[k] : make_uint4(0, 0, 0, 0);
    w[4 * k] = v.x;
    w[4 * k + 1] = v.y;
    w[4 * k + 2] = v.z;
    w[4 * k + 3] = v.w;
  }
  uint32_t q = 0;
  if (p < slots) {
    sub[p] = sub_mask(w);
#pragma unroll
    for (int k = 0; k < 16; k++) q += square_counts(w[k]);
  }
  q = __reduce_add_sync(kFull, q);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(counts, (unsigned long long)(q & 0xFFFFu));
    atomicAdd(counts + 1, (unsigned long long)(q >> 16));
  }
}

// ---------------------------------------------------------------- scene API

// Keeps the scene pool's release threshold at the live scenes' bytes plus
// kScenePoolKeep: what is free beyond that goes back to the device at the next
// synchronisation.  Returns the threshold.
static uint64_t scene_pool_account(meso_ctx* ctx, int64_t delta) {
  constexpr uint64_t kScenePoolKeep = 1ull << 30;
  std::lock_guard<std::mutex> lk(ctx->scene_pool_mu);
  ctx->scene_pool_live += (uint64_t)delta;
  uint64_t keep = ctx->scene_pool_live + kScenePoolKeep;
  cudaMemPoolSetAttribute(ctx->scene_pool, cudaMemPoolAttrReleaseThreshold, &keep);
  return keep;
}

bool scene_pool_give_back(meso_ctx* ctx) {
  uint64_t used = 0, held = 0;
  if (cudaMemPoolGetAttribute(ctx->scene_pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess ||
      cudaMemPoolGetAttribute(ctx->scene_pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess || held <= used)
    return false;
  cudaGetLastError();  // of the allocation that is tried again
  cudaStreamSynchronize(ctx->stream);
  return cudaMemPoolTrimTo(ctx->scene_pool, 0) == cudaSuccess;
}

meso_status scene_alloc(meso_ctx* ctx, int32_t nx, int32_t ny, int32_t nz, uint64_t capacity, meso_scene** out) {
  meso_scene* s = new meso_scene();
  s->nx = nx;
  s->ny = ny;
  s->nz = nz;
  s->bx = nx / 8;
  s->by = ny / 8;
  s->bz = nz / 8;
  s->capacity = capacity;
  const uint64_t nb = n_bricks_of(s), nm = std::max<uint64_t>(n_macro_of(s), 1), nslot = std::max<uint64_t>(capacity, 1);
  const uint64_t ptr_bytes = nb * 4, map_bytes = 32 + nm * (8 + 64 + 1), occ_bytes = nslot * 64, mat_bytes = nslot * 1024,
                 small_bytes = 8 + nslot * 12 + 16;
  const uint64_t bytes = ptr_bytes + map_bytes + occ_bytes + mat_bytes + small_bytes;
  if (ctx->budget_bytes && ctx->scene_bytes.load() + bytes > ctx->budget_bytes) {
    delete s;
    return fail(MESO_ERR_OVER_BUDGET, "scene exceeds the HBM budget");
  }
  // One allocation for the cell maps and one for the pool's small arrays.  All
  // come from the context's scene pool, which keeps up to kScenePoolKeep of
  // freed memory: a scene made in place of another reuses its memory instead
  // of mapping it afresh, which was most of such a build (512^3 uint16 grid:
  // create 360 us and destroy 230 us with cudaMalloc and cudaFree, 200 and 4 us
  // now).  The pool is the scenes' own: in the default pool they would count
  // against what that keeps of the per-call temporaries.
  const cudaStream_t st = ctx->stream;
  auto take = [&](auto** p, uint64_t n) {
    cudaError_t err = cudaMallocFromPoolAsync(reinterpret_cast<void**>(p), n, ctx->scene_pool, st);
    if (err == cudaErrorMemoryAllocation && scene_pool_give_back(ctx))
      err = cudaMallocFromPoolAsync(reinterpret_cast<void**>(p), n, ctx->scene_pool, st);
    if (err == cudaSuccess) s->pool_bytes += n;
    return err;
  };
  uint8_t* maps = nullptr;
  uint8_t* small = nullptr;
  cudaError_t e = take(&s->d_ptr, ptr_bytes);
  if (e == cudaSuccess) e = take(&maps, map_bytes);
  if (e == cudaSuccess) {
    s->d_bounds = reinterpret_cast<int32_t*>(maps);  // all written whole by rebuild_macro
    s->d_mask = reinterpret_cast<uint64_t*>(maps + 32);
    s->d_level = maps + 32 + nm * 8;
    s->d_macro = s->d_level + nm * 64;
  }
  if (e == cudaSuccess) e = take(&s->d_occ, occ_bytes);
  if (e == cudaSuccess) e = take(&s->d_mat, mat_bytes);
  if (e == cudaSuccess) e = take(&small, small_bytes);
  if (e == cudaSuccess) {
    s->d_sub = reinterpret_cast<uint64_t*>(small) + 1;
    s->d_alloc = reinterpret_cast<int64_t*>(s->d_sub + nslot);
    s->d_free = reinterpret_cast<uint32_t*>(s->d_alloc + 2);
  }
  scene_pool_account(ctx, (int64_t)s->pool_bytes);
  if (e != cudaSuccess) {
    scene_release(ctx, s);
    cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? MESO_ERR_OOM : MESO_ERR_CUDA,
                std::string("scene allocation failed: ") + cudaGetErrorString(e));
  }
  s->bytes = bytes;
  ctx->scene_bytes.fetch_add(bytes);
  *out = s;
  return MESO_OK;
}

void scene_release(meso_ctx* ctx, meso_scene* s) {
  if (!s) return;
  cudaFreeAsync(s->d_ptr, ctx->stream);   // cudaFreeAsync(nullptr) is a no-op
  cudaFreeAsync(s->d_bounds, ctx->stream);  // the base of the cell maps
  cudaFreeAsync(s->d_occ, ctx->stream);
  cudaFreeAsync(s->d_mat, ctx->stream);
  if (s->d_sub) cudaFreeAsync(s->d_sub - 1, ctx->stream);  // the base of the pool's small arrays
  const uint64_t keep = scene_pool_account(ctx, -(int64_t)s->pool_bytes);
  // what the pool then holds beyond the threshold goes back now, not at some
  // later synchronisation: the caller's next allocation may need it
  uint64_t held = 0;
  if (cudaMemPoolGetAttribute(ctx->scene_pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess && held > keep) {
    cudaStreamSynchronize(ctx->stream);
    cudaMemPoolTrimTo(ctx->scene_pool, keep);
  }
  if (s->bytes) ctx->scene_bytes.fetch_sub(s->bytes);
  delete s;
}

meso_status rebuild_macro(meso_ctx* ctx, meso_scene* s, const uint32_t* d_cells, uint32_t n, cudaStream_t st,
                          const uint32_t* d_cells3, uint32_t n3) {
  const uint64_t cells = d_cells ? n : n_macro_of(s), cells3 = d_cells3 ? n3 : n_macro3_of(s);
  if (cells == 0) return MESO_OK;
  macro_kernel<<<(unsigned)((cells * 32 + 255) / 256), 256, 0, st>>>(s->d_ptr, s->bx, s->by, s->d_macro, s->d_mask, s->d_bounds,
                                                                     s->d_sub, reinterpret_cast<int32_t*>(s->d_alloc),
                                                                     (uint32_t)s->capacity, d_cells, cells);
  level_kernel<<<(unsigned)(cells3 * 32), kLevelThreads, 0, st>>>(s->d_mask, s->d_macro, s->bx, s->by, s->bz, s->d_level,
                                                                  s->d_bounds, d_cells3);
  ctx->launches.fetch_add(2);
  MESO_CUDA_TRY(cudaGetLastError());
  return MESO_OK;
}

// Of the squares of 2x2 voxels of z layers (all, or a sample) that are not solid
// (`open`), `mixed` hold voxels.  A scene is rough if that is more than an eighth.
// Its rays then walk step by step: so few regions are empty that leaving them one by
// one costs more than the steps.  256^3 voxels, 1280x720 from outside, by region and
// by steps: 2 % solid at random (0.08 of the squares) 225 and 249 us, 3 % (0.12) 185
// and 182, 4 % (0.15) 158 and 146, 10 % (0.34) 87 and 69, 25 % (0.68) 48 and 35.
// Terrains, caves, foliage and the generator's noise lie below 0.06.
static void set_rough(meso_scene* s, uint64_t mixed, uint64_t open) { s->rough = 8 * mixed > open; }

meso_status rebuild_sub(meso_ctx* ctx, meso_scene* s, uint64_t slots, cudaStream_t st) {
  if (slots == 0) return MESO_OK;
  unsigned long long* d = nullptr;
  unsigned long long counts[2] = {0, 0};
  MESO_CUDA_TRY(dev_malloc_async(ctx, &d, sizeof(counts), st));
  cudaError_t e = cudaMemsetAsync(d, 0, sizeof(counts), st);
  if (e == cudaSuccess) {
    sub_kernel<<<(unsigned)((slots + 127) / 128), 128, 0, st>>>(s->d_occ, slots, s->d_sub, d);
    ctx->launches.fetch_add(1);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(counts, d, sizeof(counts), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(d, st);
  const cudaError_t e2 = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) return cuda_fail(e, "scene block masks");
  set_rough(s, counts[0], counts[1] + (n_bricks_of(s) - slots) * 128);
  return MESO_OK;
}

static meso_status finish_pools(meso_ctx* ctx, meso_scene* s, uint64_t count, cudaStream_t st) {
  MESO_TRY(rebuild_macro(ctx, s, nullptr, 0, st));
  int32_t init[4] = {(int32_t)count, 0, 0, 0};
  MESO_CUDA_TRY(cudaMemcpyAsync(s->d_alloc, init, 16, cudaMemcpyHostToDevice, st));
  MESO_CUDA_TRY(cudaStreamSynchronize(st));
  s->live_bricks_host = count;
  (void)ctx;
  return MESO_OK;
}

// A scene object for `count` bricks and `spare` more, its arrays not yet written.
static meso_status alloc_sized(meso_ctx* ctx, int32_t nx, int32_t ny, int32_t nz, uint64_t count, uint64_t spare,
                               meso_scene** out) {
  const uint64_t cap = count + spare;
  if (cap >= 0xFFFFFFFFull) return fail(MESO_ERR_INVALID_ARG, "brick pool too large");
  return scene_alloc(ctx, nx, ny, nz, cap, out);
}

meso_status scene_create_terrain(meso_ctx* ctx, const meso_terrain* t, uint64_t spare, meso_scene** out) {
  if (!t || !out) return fail(MESO_ERR_INVALID_ARG, "terrain: null argument");
  if (t->nx <= 0 || t->ny <= 0 || t->nz <= 0 || t->nx % 32 || t->ny % 32 || t->nz % 32 || t->nx > 8192 ||
      t->ny > 8192 || t->nz > 8192)
    return fail(MESO_ERR_INVALID_ARG, "terrain: dims must be positive multiples of 32 (<= 8192)");
  if (t->height_period == 0 || t->cave_period == 0 || t->height_octaves < 1 || t->height_octaves > 16)
    return fail(MESO_ERR_INVALID_ARG, "terrain: bad noise parameters");
  cudaStream_t st = ctx->stream;
  const TerrainDev T = to_dev(*t);
  const uint64_t ncol = (uint64_t)t->nx * t->ny;
  const int bx = t->nx / 8, by = t->ny / 8, bz = t->nz / 8;
  const uint64_t nb = (uint64_t)bx * by * bz;
  float* d_h = nullptr;
  float* d_hmax = nullptr;
  uint8_t* d_flags = nullptr;
  uint32_t* d_ptr_tmp = nullptr;
  cudaError_t ae = dev_malloc_async(ctx, &d_h, ncol * 4, st);
  if (ae == cudaSuccess) ae = dev_malloc_async(ctx, &d_hmax, (uint64_t)bx * by * 4, st);
  if (ae == cudaSuccess) ae = dev_malloc_async(ctx, &d_flags, nb, st);
  if (ae == cudaSuccess) ae = dev_malloc_async(ctx, &d_ptr_tmp, nb * 4, st);
  if (ae != cudaSuccess) {
    cudaFreeAsync(d_h, st);  // cudaFreeAsync(nullptr) is a no-op
    cudaFreeAsync(d_hmax, st);
    cudaFreeAsync(d_flags, st);
    cudaStreamSynchronize(st);
    return cuda_fail(ae, "terrain build: scratch allocation");
  }
  heights_kernel<<<(unsigned)((ncol + 255) / 256), 256, 0, st>>>(T, d_h);
  column_max_kernel<<<(bx * by + 255) / 256, 256, 0, st>>>(T, d_h, d_hmax);
  terrain_brick_kernel<false><<<grid_for(nb), 256, 0, st>>>(T, d_h, d_hmax, d_flags, nullptr, nullptr, nullptr);
  ctx->launches.fetch_add(3);
  uint64_t count = 0;
  meso_status rc = number_bricks(ctx, d_flags, nb, d_ptr_tmp, st, &count);
  meso_scene* s = nullptr;
  if (rc == MESO_OK) rc = alloc_sized(ctx, t->nx, t->ny, t->nz, count, spare, &s);
  if (rc == MESO_OK) {
    cudaMemcpyAsync(s->d_ptr, d_ptr_tmp, nb * 4, cudaMemcpyDeviceToDevice, st);
    terrain_brick_kernel<true><<<grid_for(nb), 256, 0, st>>>(T, d_h, d_hmax, d_flags, s->d_ptr, s->d_occ, s->d_mat);
    ctx->launches.fetch_add(1);
    rc = rebuild_sub(ctx, s, count, st);
    if (rc == MESO_OK) rc = finish_pools(ctx, s, count, st);
  }
  cudaFreeAsync(d_h, st);
  cudaFreeAsync(d_hmax, st);
  cudaFreeAsync(d_flags, st);
  cudaFreeAsync(d_ptr_tmp, st);
  cudaError_t e = cudaStreamSynchronize(st);
  if (rc == MESO_OK && e != cudaSuccess) rc = cuda_fail(e, "terrain build");
  if (rc != MESO_OK) {
    scene_release(ctx, s);
    return rc;
  }
  *out = s;
  return MESO_OK;
}

// Brick map of a dense grid already in device memory (T = uint8_t or
// uint16_t; a uint8 material m becomes the uint16 material m).
template <typename T>
static meso_status build_from_device_grid(meso_ctx* ctx, const T* d_grid, int32_t nx, int32_t ny, int32_t nz,
                                          uint64_t spare, cudaStream_t st, meso_scene** out) {
  const uint64_t nb = (uint64_t)nx * ny * nz / 512;
  const unsigned blocks = (unsigned)((nb + kDenseBricks - 1) / kDenseBricks);
  // a word per block: which of its bricks hold anything; their first slots, and the
  // count of bricks and of the sampled squares; the samples, about 1024
  const uint32_t step = blocks / 1024u | 1u, n_squares = (blocks + step - 1) / step;
  uint32_t* d_occupied = nullptr;
  const cudaError_t ae = dev_malloc_async(ctx, &d_occupied, 8 * (size_t)blocks + 12 + 4 * (size_t)n_squares, st);
  if (ae != cudaSuccess) {
    cudaStreamSynchronize(st);
    return cuda_fail(ae, "dense scene: scratch allocation");
  }
  uint32_t* const d_base = d_occupied + blocks;
  uint32_t* const d_total = d_base + blocks;
  uint32_t* const d_squares = d_total + 3;
  const bool wide = (reinterpret_cast<uintptr_t>(d_grid) & (8 * sizeof(T) - 1)) == 0;
  if (wide) dense_flag_kernel<T, true><<<blocks, kDenseThreads, 0, st>>>(d_grid, nx, ny, nb, d_occupied, d_squares, step);
  else dense_flag_kernel<T, false><<<blocks, kDenseThreads, 0, st>>>(d_grid, nx, ny, nb, d_occupied, d_squares, step);
  scan_words_kernel<<<1, kScanThreads, 0, st>>>(d_occupied, blocks, d_base, d_total, d_squares, n_squares);
  ctx->launches.fetch_add(2);
  uint32_t totals[3] = {0, 0, 0};
  cudaError_t e = cudaMemcpyAsync(totals, d_total, sizeof(totals), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  meso_status rc = e == cudaSuccess ? MESO_OK : cuda_fail(e, "dense scene build");
  const uint32_t count = totals[0];
  meso_scene* s = nullptr;
  if (rc == MESO_OK) rc = alloc_sized(ctx, nx, ny, nz, count, spare, &s);
  if (rc == MESO_OK) {
    if (wide)
      dense_fill_kernel<T, true><<<blocks, kDenseThreads, 0, st>>>(d_grid, nx, ny, nb, d_occupied, d_base, s->d_ptr, s->d_occ,
                                                                     s->d_mat, s->d_sub);
    else
      dense_fill_kernel<T, false><<<blocks, kDenseThreads, 0, st>>>(d_grid, nx, ny, nb, d_occupied, d_base, s->d_ptr, s->d_occ,
                                                                      s->d_mat, s->d_sub);
    ctx->launches.fetch_add(1);
    set_rough(s, totals[1], totals[2]);
    rc = finish_pools(ctx, s, count, st);
  }
  cudaFreeAsync(d_occupied, st);
  e = cudaStreamSynchronize(st);
  if (rc == MESO_OK && e != cudaSuccess) rc = cuda_fail(e, "dense scene build");
  if (rc != MESO_OK) {
    scene_release(ctx, s);
    return rc;
  }
  *out = s;
  return MESO_OK;
}

static meso_status check_grid_dims(int32_t nx, int32_t ny, int32_t nz) {
  if (nx <= 0 || ny <= 0 || nz <= 0 || nx % 32 || ny % 32 || nz % 32 || nx > 8192 || ny > 8192 || nz > 8192)
    return fail(MESO_ERR_INVALID_ARG, "dense scene: dims must be positive multiples of 32 (<= 8192)");
  return MESO_OK;
}

meso_status scene_create_dense(meso_ctx* ctx, const uint16_t* h_grid, int32_t nx, int32_t ny, int32_t nz,
                               uint64_t spare, meso_scene** out) {
  if (!h_grid || !out) return fail(MESO_ERR_INVALID_ARG, "dense scene: null argument");
  MESO_TRY(check_grid_dims(nx, ny, nz));
  cudaStream_t st = ctx->stream;
  const uint64_t nvox = (uint64_t)nx * ny * nz;
  uint16_t* d_grid = nullptr;
  cudaError_t ae = dev_malloc_async(ctx, &d_grid, nvox * 2, st);
  if (ae == cudaSuccess) ae = cudaMemcpyAsync(d_grid, h_grid, nvox * 2, cudaMemcpyHostToDevice, st);
  if (ae != cudaSuccess) {
    cudaFreeAsync(d_grid, st);
    cudaStreamSynchronize(st);
    return cuda_fail(ae, "dense scene: upload");
  }
  const meso_status rc = build_from_device_grid<uint16_t>(ctx, d_grid, nx, ny, nz, spare, st, out);
  cudaFreeAsync(d_grid, st);
  cudaStreamSynchronize(st);
  return rc;
}

meso_status scene_create_grid(meso_ctx* ctx, int32_t kind, const void* d_grid, int32_t nx, int32_t ny, int32_t nz,
                              uint64_t spare, meso_scene** out) {
  if (!d_grid || !out) return fail(MESO_ERR_INVALID_ARG, "grid scene: null argument");
  MESO_TRY(check_grid_dims(nx, ny, nz));
  if (kind == MESO_SRC_GRID_U8)
    return build_from_device_grid<uint8_t>(ctx, static_cast<const uint8_t*>(d_grid), nx, ny, nz, spare, ctx->stream,
                                           out);
  if (kind == MESO_SRC_GRID_U16)
    return build_from_device_grid<uint16_t>(ctx, static_cast<const uint16_t*>(d_grid), nx, ny, nz, spare,
                                            ctx->stream, out);
  return fail(MESO_ERR_INVALID_ARG, "grid scene: kind must be MESO_SRC_GRID_U8 or MESO_SRC_GRID_U16");
}

meso_status scene_count_solid(meso_ctx* ctx, const meso_scene* s, uint64_t* n_solid) {
  if (!s || !n_solid) return fail(MESO_ERR_INVALID_ARG, "scene_count_solid: null argument");
  cudaStream_t st = ctx->stream;
  unsigned long long* d = nullptr;
  MESO_CUDA_TRY(dev_malloc_async(ctx, &d, 8, st));
  cudaError_t e = cudaMemsetAsync(d, 0, 8, st);
  const uint64_t nb = n_bricks_of(s);
  if (e == cudaSuccess) {
    count_solid_kernel<<<(unsigned)std::min<uint64_t>((nb + 255) / 256, (uint64_t)ctx->sm_count * 16), 256, 0, st>>>(
        s->d_ptr, nb, s->d_occ, d);
    ctx->launches.fetch_add(1);
    e = cudaGetLastError();
  }
  unsigned long long h = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, 8, cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(d, st);
  const cudaError_t e2 = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = e2;
  if (e != cudaSuccess) return cuda_fail(e, "scene_count_solid");
  *n_solid = h;
  return MESO_OK;
}

meso_status generate_dense_u8(meso_ctx* ctx, int32_t nx, int32_t ny, int32_t nz, uint32_t seed, uint8_t* d_out,
                              cudaStream_t st) {
  if (!d_out || nx <= 0 || ny <= 0 || nz <= 0) return fail(MESO_ERR_INVALID_ARG, "generate_dense_u8: bad argument");
  const uint64_t n = (uint64_t)nx * ny * nz;
  dense_u8_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nx, ny, nz, seed, d_out);
  ctx->launches.fetch_add(1);
  MESO_CUDA_TRY(cudaGetLastError());
  return MESO_OK;
}

uint32_t chunk_solid_target(uint32_t seed) {
  // round(32768 * p), p = exp(U(ln 0.001, ln 0.9)), U from the chunk seed
  auto pcg = [](uint32_t x, uint32_t y, uint32_t z) {
    x = x * 1664525u + 1013904223u;
    y = y * 1664525u + 1013904223u;
    z = z * 1664525u + 1013904223u;
    x += y * z;
    y += z * x;
    z += x * y;
    x ^= x >> 16;
    y ^= y >> 16;
    z ^= z >> 16;
    x += y * z;
    y += z * x;
    z += x * y;
    return z;
  };
  const double u = (double)(pcg(seed, 0xA5A5u, 0x1234u) >> 8) / 16777216.0;
  const double lo = std::log(0.001), hi = std::log(0.9);
  const double p = std::exp(lo + (hi - lo) * u);
  return (uint32_t)std::floor(32768.0 * p + 0.5);
}

meso_status generate_chunks_u16(meso_ctx* ctx, uint32_t n, uint32_t seed0, uint16_t* d_out, uint32_t* d_solid,
                                cudaStream_t st) {
  if (!d_out || n == 0) return fail(MESO_ERR_INVALID_ARG, "generate_chunks_u16: bad argument");
  std::vector<uint32_t> targets(n);
  for (uint32_t i = 0; i < n; i++) targets[i] = chunk_solid_target(seed0 + i);
  uint32_t* d_t = nullptr;
  MESO_CUDA_TRY(dev_malloc_async(ctx, &d_t, 4ull * n, st));
  MESO_CUDA_TRY(cudaMemcpyAsync(d_t, targets.data(), 4ull * n, cudaMemcpyHostToDevice, st));
  static bool attr = false;
  if (!attr) {
    MESO_CUDA_TRY(cudaFuncSetAttribute(chunks_u16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 131072));
    attr = true;
  }
  chunks_u16_kernel<<<n, 1024, 131072, st>>>(seed0, d_t, d_out, d_solid);
  ctx->launches.fetch_add(1);
  MESO_CUDA_TRY(cudaFreeAsync(d_t, st));
  MESO_CUDA_TRY(cudaStreamSynchronize(st));
  MESO_CUDA_TRY(cudaGetLastError());
  return MESO_OK;
}

// Host side of an edit: touched bricks (sorted unique) and dirty chunks.
// Cells (bricks or chunks, edge `shift` bits of voxels) that the boxes
// [lo, hi] of the spheres touch, as sorted unique linear indices of a grid
// of G cells.  Small sets are collected and sorted; when the boxes cover a
// sizeable part of the grid, a bitmap over the grid is marked and scanned
// instead, so the cost stays bounded by the grid size.
// The cells (2^shift voxels on a side, grid G) that the boxes [lo, hi]
// overlap, unique; sorted unless `any_order` (then sorted only when two boxes
// share a cell: boxes that share none enumerate disjoint cells, and the
// sort is the costly part for a few thousand cells).
static void touched_cells(const int64_t (*lo)[3], const int64_t (*hi)[3], uint32_t n, int shift, const int64_t G[3],
                          std::vector<uint32_t>& out, bool any_order = false) {
  out.clear();
  uint64_t volume = 0;
  for (uint32_t i = 0; i < n; i++) {
    if (lo[i][0] > hi[i][0] || lo[i][1] > hi[i][1] || lo[i][2] > hi[i][2]) continue;
    uint64_t v = 1;
    for (int a = 0; a < 3; a++) v *= (uint64_t)((hi[i][a] >> shift) - (lo[i][a] >> shift) + 1);
    volume += v;
  }
  const uint64_t total = (uint64_t)(G[0] * G[1] * G[2]);
  const bool bitmap = volume > total / 64;
  std::vector<uint64_t> bits;
  if (bitmap) bits.assign((size_t)((total + 63) / 64), 0);
  else out.reserve((size_t)volume);
  for (uint32_t i = 0; i < n; i++) {
    if (lo[i][0] > hi[i][0] || lo[i][1] > hi[i][1] || lo[i][2] > hi[i][2]) continue;
    for (int64_t z = lo[i][2] >> shift; z <= hi[i][2] >> shift; z++)
      for (int64_t y = lo[i][1] >> shift; y <= hi[i][1] >> shift; y++)
        for (int64_t x = lo[i][0] >> shift; x <= hi[i][0] >> shift; x++) {
          const uint64_t k = (uint64_t)(x + G[0] * (y + G[1] * z));
          if (bitmap) bits[k >> 6] |= 1ull << (k & 63);
          else out.push_back((uint32_t)k);
        }
  }
  if (bitmap) {
    for (size_t w = 0; w < bits.size(); w++)
      for (uint64_t m = bits[w]; m; m &= m - 1) out.push_back((uint32_t)(w * 64 + (uint64_t)__builtin_ctzll(m)));
  } else {
    bool shared = !any_order;
    for (uint32_t i = 0; i < n && !shared; i++) {
      if (lo[i][0] > hi[i][0] || lo[i][1] > hi[i][1] || lo[i][2] > hi[i][2]) continue;
      for (uint32_t j = i + 1; j < n && !shared; j++) {
        if (lo[j][0] > hi[j][0] || lo[j][1] > hi[j][1] || lo[j][2] > hi[j][2]) continue;
        bool all = true;
        for (int a = 0; a < 3; a++)
          all = all && std::max(lo[i][a] >> shift, lo[j][a] >> shift) <= std::min(hi[i][a] >> shift, hi[j][a] >> shift);
        shared = all;
      }
    }
    if (shared) {
      std::sort(out.begin(), out.end());
      out.erase(std::unique(out.begin(), out.end()), out.end());
    }
  }
}

// The bricks a set of sphere edits may change (the voxel boxes of the
// spheres) and the chunks to remesh (the boxes grown by one voxel, whose
// faces may change), both sorted by linear index.
// The bricks and chunks the spheres' boxes touch, and the cells of 4^3 and
// 64^3 bricks holding those bricks (all unique; all but the bricks sorted).  A cell holds a
// touched brick iff the box overlaps it, so the cells come from the boxes
// directly, at the cells' own granularity.
static void edit_sets(const meso_scene* s, const meso_sphere_edit* sp, uint32_t n, std::vector<uint32_t>& bricks,
                      std::vector<uint32_t>& chunks, std::vector<uint32_t> (&cells)[2]) {
  const int64_t N[3] = {s->nx, s->ny, s->nz};
  std::vector<int64_t> box((size_t)n * 12);
  auto lo = reinterpret_cast<int64_t (*)[3]>(box.data());
  auto hi = lo + n;
  auto clo = hi + n;
  auto chi = clo + n;
  for (uint32_t i = 0; i < n; i++)
    for (int a = 0; a < 3; a++) {
      lo[i][a] = std::max<int64_t>((int64_t)sp[i].center[a] - sp[i].radius, 0);
      hi[i][a] = std::min<int64_t>((int64_t)sp[i].center[a] + sp[i].radius, N[a] - 1);
      clo[i][a] = std::max<int64_t>((int64_t)sp[i].center[a] - sp[i].radius - 1, 0);
      chi[i][a] = std::min<int64_t>((int64_t)sp[i].center[a] + sp[i].radius + 1, N[a] - 1);
    }
  const int64_t B[3] = {s->bx, s->by, s->bz}, C[3] = {s->nx / 32, s->ny / 32, s->nz / 32};
  touched_cells(lo, hi, n, 3, B, bricks, /*any_order=*/true);  // the edit kernels take them in any order
  touched_cells(clo, chi, n, 5, C, chunks);
  const int64_t M[3] = {s->bx / 4, s->by / 4, s->bz / 4}, M3[3] = {(s->bx + 63) / 64, (s->by + 63) / 64, (s->bz + 63) / 64};
  touched_cells(lo, hi, n, 5, M, cells[0]);
  touched_cells(lo, hi, n, 9, M3, cells[1]);
}

meso_status edit_spheres(meso_ctx* ctx, meso_scene* s, const meso_sphere_edit* h_sp, uint32_t n, uint32_t* h_dirty,
                         uint32_t dirty_cap, uint32_t* n_dirty, cudaStream_t st) {
  if (!s || (n && !h_sp)) return fail(MESO_ERR_INVALID_ARG, "edit: null argument");
  for (uint32_t i = 0; i < n; i++)
    if (h_sp[i].radius < 0 || h_sp[i].radius > 4096) return fail(MESO_ERR_INVALID_ARG, "edit: radius out of range");
  std::vector<uint32_t> bricks, chunks, cells[2];
  edit_sets(s, h_sp, n, bricks, chunks, cells);
  if (n_dirty) *n_dirty = (uint32_t)chunks.size();
  if (h_dirty) std::copy(chunks.begin(), chunks.begin() + std::min<size_t>(chunks.size(), dirty_cap), h_dirty);
  if (bricks.empty()) return chunks.size() > dirty_cap && h_dirty ? fail(MESO_ERR_OVERFLOW, "edit: dirty list overflow") : MESO_OK;
  const size_t nb = bricks.size();
  // only the maps of the cells holding touched bricks are recomputed
  // device scratch: [spheres | bricks | cells | cells3] uploaded in one copy,
  // then the per-brick temporaries
  const size_t nc = cells[0].size(), nc3 = cells[1].size();
  const size_t up = n * sizeof(meso_sphere_edit) + 4 * (nb + nc + nc3);
  const size_t up16 = (up + 15) & ~size_t(15);
  std::vector<uint8_t> h(up);
  std::memcpy(h.data(), h_sp, n * sizeof(meso_sphere_edit));
  size_t o = n * sizeof(meso_sphere_edit);
  std::memcpy(h.data() + o, bricks.data(), nb * 4);
  o += nb * 4;
  for (int l = 0; l < 2; l++) {
    std::memcpy(h.data() + o, cells[l].data(), cells[l].size() * 4);
    o += cells[l].size() * 4;
  }
  const size_t bytes = up16 + nb * 1024 + nb + 16;
  uint8_t* d = nullptr;
  MESO_CUDA_TRY(dev_malloc_async(ctx, &d, bytes, st));
  meso_sphere_edit* d_sp = reinterpret_cast<meso_sphere_edit*>(d);
  uint32_t* d_b = reinterpret_cast<uint32_t*>(d + n * sizeof(meso_sphere_edit));
  uint32_t* d_cells = d_b + nb;
  uint32_t* d_cells3 = d_cells + nc;
  uint16_t* d_temp = reinterpret_cast<uint16_t*>(d + up16);
  uint8_t* d_state = reinterpret_cast<uint8_t*>(d_temp) + nb * 1024;
  const cudaError_t ce = cudaMemcpyAsync(d, h.data(), up, cudaMemcpyHostToDevice, st);
  if (ce != cudaSuccess) {
    cudaFreeAsync(d, st);
    return cuda_fail(ce, "edit: upload");
  }
  EditParams P;
  P.spheres = d_sp;
  P.n_spheres = n;
  P.bricks = d_b;
  P.n_bricks = (uint32_t)nb;
  P.bx = s->bx;
  P.by = s->by;
  P.ptr = s->d_ptr;
  P.occ = s->d_occ;
  P.mat = s->d_mat;
  P.sub = s->d_sub;
  P.temp = d_temp;
  P.state = d_state;
  P.free_stack = s->d_free;
  P.alloc = reinterpret_cast<int32_t*>(s->d_alloc);
  P.capacity = (uint32_t)s->capacity;
  P.err = ctx->d_scratch + 1;
  const unsigned blocks = (unsigned)((nb + 7) / 8);
  edit_compute_kernel<<<blocks, 256, 0, st>>>(P);
  edit_alloc_kernel<<<blocks, 256, 0, st>>>(P);
  ctx->launches.fetch_add(2);
  const meso_status mrc =
      rebuild_macro(ctx, s, d_cells, (uint32_t)nc, st, d_cells3, (uint32_t)nc3);
  MESO_CUDA_TRY(cudaFreeAsync(d, st));
  if (mrc != MESO_OK) return mrc;
  MESO_CUDA_TRY(cudaGetLastError());
  if (h_dirty && chunks.size() > dirty_cap) return fail(MESO_ERR_OVERFLOW, "edit: dirty list overflow");
  return MESO_OK;
}

}  // namespace meso
