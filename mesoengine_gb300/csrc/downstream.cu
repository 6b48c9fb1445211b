// downstream.cu -- the steps either side of the two hot paths:
//   * brick-map files (save / load a resident scene);
//   * quad -> vertex expansion for raster consumers;
//   * the reference's 26-neighbour occupancy erosion pyramid on device.
#include <cstdio>
#include <cstring>
#include <vector>

#include "meso_internal.h"

namespace meso {

namespace {

using namespace ::meso::dev;

constexpr uint32_t kFull = 0xFFFFFFFFu;

// ------------------------------------------------------------ vertices
// Plane axes per face direction: X faces u=y v=z; Y faces u=x v=z; Z faces u=x v=y.
// A CTA of kQvThreads threads writes kQvPer x kQvThreads consecutive
// vertices (4 per quad); in step k thread t makes vertex
// base + k*kQvThreads + t, so every warp store covers 512 contiguous bytes,
// and a thread's kQvPer quad loads are issued before any of them is used.
constexpr int kQvThreads = 256, kQvPer = 8;

__device__ __forceinline__ float4 quad_vertex(uint64_t q, int k, const int32_t* origins, uint32_t n_chunks,
                                              uint32_t* err) {
  const uint32_t chunk = (uint32_t)(q >> 44);
  const int dir = (int)((q >> 41) & 7u);
  const int lz = (int)((q >> 36) & 31u), ly = (int)((q >> 31) & 31u), lx = (int)((q >> 26) & 31u);
  const int w = (int)((q >> 21) & 31u) + 1, h = (int)((q >> 16) & 31u) + 1;
  const uint32_t mat = (uint32_t)(q & 0xFFFFu);
  int ox = 0, oy = 0, oz = 0;
  if (chunk < n_chunks) {
    ox = __ldg(origins + 3 * chunk) * 32;
    oy = __ldg(origins + 3 * chunk + 1) * 32;
    oz = __ldg(origins + 3 * chunk + 2) * 32;
  } else if (k == 0) {
    atomicOr(err, ERR_BAD_INPUT);
  }
  const int a = dir >> 1;
  const int plus = (dir & 1) == 0;
  // voxel origin in (a, u, v) coordinates
  int pa, u0, v0;
  if (a == 0) { pa = lx; u0 = ly; v0 = lz; }
  else if (a == 1) { pa = ly; u0 = lx; v0 = lz; }
  else { pa = lz; u0 = lx; v0 = ly; }
  const int plane = pa + (plus ? 1 : 0);
  // u x v points along +a for X and Z faces and along -a for Y faces; keep
  // the corner order when that matches the face normal, reverse it otherwise
  const bool natural = (a == 1) ? !plus : plus;
  // corners (u0,v0), (u0+w,v0), (u0+w,v0+h), (u0,v0+h)
  const int c = natural ? k : (4 - k) & 3;
  const int cu = (c == 1 || c == 2) ? u0 + w : u0;
  const int cv = c >= 2 ? v0 + h : v0;
  int x, y, z;
  if (a == 0) { x = plane; y = cu; z = cv; }
  else if (a == 1) { y = plane; x = cu; z = cv; }
  else { z = plane; x = cu; y = cv; }
  float4 vtx;
  vtx.x = (float)(ox + x);
  vtx.y = (float)(oy + y);
  vtx.z = (float)(oz + z);
  vtx.w = __uint_as_float(mat | (uint32_t)dir << 16 | (uint32_t)k << 19);
  return vtx;
}

__global__ void __launch_bounds__(kQvThreads) quads_to_vertices_kernel(const uint64_t* __restrict__ quads, uint64_t n,
                                                                     const int32_t* __restrict__ origins,
                                                                     uint32_t n_chunks, meso_vertex* __restrict__ out,
                                                                     uint32_t* err) {
  const uint64_t base = (uint64_t)blockIdx.x * (kQvPer * kQvThreads) + threadIdx.x;
  uint64_t q[kQvPer];
#pragma unroll
  for (int k = 0; k < kQvPer; k++) {
    const uint64_t i = (base + (uint64_t)k * kQvThreads) >> 2;
    q[k] = i < n ? __ldg(quads + i) : 0ull;
  }
#pragma unroll
  for (int k = 0; k < kQvPer; k++) {
    const uint64_t vi = base + (uint64_t)k * kQvThreads;
    if ((vi >> 2) < n) __stcs(reinterpret_cast<float4*>(out) + vi, quad_vertex(q[k], (int)(vi & 3u), origins, n_chunks, err));
  }
}

// ------------------------------------------------------------ erosion
struct ErodeParams {
  const uint8_t* data;
  int32_t nx, ny, nz;
  const uint32_t* bptr;
  const uint64_t* bocc;
  int32_t bx, by, bz;
  const int32_t* coords;
  uint32_t n;
  uint32_t depth;
  uint32_t* out;
  uint32_t* err;
};

// Bits of the nonzero voxels of 16 bytes: 8 (16-bit) or 16 (8-bit).
template <bool k16>
__device__ __forceinline__ uint32_t solid_bits(const uint4& v) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t b = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if constexpr (k16) {
      const uint32_t t = (((w[k] & 0x7FFF7FFFu) + 0x7FFF7FFFu) | w[k]) & 0x80008000u;  // a bit per half, no carry leaves it
      b |= (t >> 15 | t >> 30) << (2 * k) & 3u << (2 * k);
    } else {
      const uint32_t t = (((w[k] & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w[k]) >> 7 & 0x01010101u;
      b |= (t * 0x01020408u >> 24) << (4 * k);  // bits 0, 8, 16, 24 to 24 .. 27; nothing else lands there
    }
  }
  return b;
}

// One CTA of 8 warps per chunk.  The occupancy bits of its rows (z, y) come from
// 16-byte loads (chunk arrays, and grids that start on 16 bytes; nx is a multiple
// of 32, so their rows then do too), from the bricks' occupancy words, each byte
// of which is a quarter of a row, or voxel by voxel (grids that do not).  Then
// lane = y and a warp has four layers z in registers: mip d from mip d-1, with
// the y neighbours by shuffles and the layers of the neighbouring warps by shared
// memory.  P = R & (R << 1) & (R >> 1) covers the three x positions of each of the
// 8 other rows, (R << 1) & (R >> 1) the two x neighbours of the own row.
//
// Bound by DRAM: 4096 uint16 chunks, depth 4, 268 MB read and 67 written in 55 us
// (63 with the rows in shared memory and nine reads of them per row and step; 62
// at 32 registers, which leave too few loads in flight), uint8 chunks 34 (55),
// and chunks of a grid or a scene, which went voxel by voxel through ballots:
// uint8 grid 45 (202), uint16 grid 62 (205), 1024^3 terrain 29 (190).
constexpr int kErodeThreads = 256;
constexpr int kErodeBatch = 8;  // 16-byte loads a thread has in flight at once
static_assert(2048 % (kErodeBatch * kErodeThreads) == 0, "a chunk is whole batches of loads");

template <int KIND, bool kWide>
__global__ void __launch_bounds__(kErodeThreads, 4) erode_kernel(const ErodeParams p) {
  constexpr bool kBrick = KIND == MESO_SRC_BRICKMAP;
  constexpr bool kGrid = KIND == MESO_SRC_GRID_U8 || KIND == MESO_SRC_GRID_U16;
  constexpr bool k16 = KIND == MESO_SRC_GRID_U16 || KIND == MESO_SRC_CHUNKS_U16;
  __shared__ uint32_t rows[1024];
  __shared__ uint32_t edge[2][16][32];  // first and last layer of each warp, of the last step and this one
  const uint32_t c = blockIdx.x;
  const int t = (int)threadIdx.x, warp = t >> 5, lane = t & 31;
  int cx = 0, cy = 0, cz = 0;
  uint32_t idx = c;
  bool ok = true;
  if constexpr (kGrid || kBrick) {
    cx = p.coords[3 * c];
    cy = p.coords[3 * c + 1];
    cz = p.coords[3 * c + 2];
    const int lx = kBrick ? p.bx / 4 : p.nx / 32, ly = kBrick ? p.by / 4 : p.ny / 32, lz = kBrick ? p.bz / 4 : p.nz / 32;
    ok = cx >= 0 && cy >= 0 && cz >= 0 && cx < lx && cy < ly && cz < lz;
  } else if (p.coords) {
    idx = (uint32_t)p.coords[c];
    ok = idx < (uint32_t)p.nx;
  }
  uint32_t* out = p.out + (size_t)c * p.depth * 1024;
  if (!ok) {
    if (t == 0) atomicOr(p.err, ERR_BAD_INPUT);
    for (uint32_t i = t; i < p.depth * 1024; i += kErodeThreads) out[i] = 0;
    return;
  }
  if constexpr (kBrick) {
    // word (brick, z) holds rows y of 8 voxels, a byte each
#pragma unroll
    for (int i = t; i < 512; i += kErodeThreads) {
      const int b = i >> 3, z = i & 7;  // brick b of the chunk: bit x + 4y + 16z
      const uint32_t slot = __ldg(p.bptr + (size_t)(4 * cx + (b & 3)) +
                                  (size_t)p.bx * ((size_t)(4 * cy + ((b >> 2) & 3)) + (size_t)p.by * (size_t)(4 * cz + (b >> 4))));
      const uint64_t w = slot != MESO_EMPTY_BRICK ? __ldg(p.bocc + (size_t)slot * 8 + z) : 0ull;
      uint8_t* dst = reinterpret_cast<uint8_t*>(rows) + (32 * (8 * (b >> 4) + z) + 8 * ((b >> 2) & 3)) * 4 + (b & 3);
#pragma unroll
      for (int y = 0; y < 8; y++) dst[4 * y] = (uint8_t)(w >> (8 * y));
    }
  } else if constexpr (kWide) {
    constexpr int kPer = k16 ? 4 : 2;  // loads per row
    const size_t pitch_y = kGrid ? (size_t)p.nx * (k16 ? 2 : 1) : 16 * kPer,
                 pitch_z = kGrid ? pitch_y * (size_t)p.ny : 32 * 16 * kPer;
    const uint8_t* src = kGrid ? p.data + (size_t)cx * (16 * kPer) + (size_t)cy * 32 * pitch_y + (size_t)cz * 32 * pitch_z
                               : p.data + (size_t)idx * (32 * 32 * 16 * kPer);
#pragma unroll 1
    for (int i0 = t; i0 < 1024 * kPer; i0 += kErodeBatch * kErodeThreads) {
      uint4 v[kErodeBatch];
#pragma unroll
      for (int j = 0; j < kErodeBatch; j++) {
        const int i = i0 + j * kErodeThreads, row = i / kPer;
        v[j] = __ldcs(reinterpret_cast<const uint4*>(src + (size_t)(row & 31) * pitch_y + (size_t)(row >> 5) * pitch_z) + i % kPer);
      }
#pragma unroll
      for (int j = 0; j < kErodeBatch; j++) {
        const uint32_t b = solid_bits<k16>(v[j]);
        if constexpr (k16) reinterpret_cast<uint8_t*>(rows)[i0 + j * kErodeThreads] = (uint8_t)b;
        else reinterpret_cast<uint16_t*>(rows)[i0 + j * kErodeThreads] = (uint16_t)b;
      }
    }
  } else {
#pragma unroll 4
    for (int row = warp; row < 1024; row += kErodeThreads / 32) {
      const int z = row >> 5, y = row & 31;
      const size_t g = (size_t)(cx * 32 + lane) + (size_t)p.nx * ((size_t)(cy * 32 + y) + (size_t)p.ny * (size_t)(cz * 32 + z));
      const uint32_t w = __ballot_sync(kFull, (k16 ? reinterpret_cast<const uint16_t*>(p.data)[g] : p.data[g]) != 0);
      if (lane == 0) rows[row] = w;
    }
  }
  __syncthreads();
  uint32_t mip0[4], R[6];  // this warp's layers 4 warp .. + 3, and R also the ones around them
#pragma unroll
  for (int j = 0; j < 4; j++) {
    mip0[j] = R[j + 1] = rows[32 * (4 * warp + j) + lane];
    out[32 * (4 * warp + j) + lane] = mip0[j];
    // the chunk's first and last voxels have neighbours outside it
    const bool border = lane == 0 || lane == 31 || (warp == 0 && j == 0) || (warp == 7 && j == 3);
    mip0[j] = border ? 0u : mip0[j] & 0x7FFFFFFEu;
  }
  for (uint32_t d = 1; d < p.depth; d++) {
    uint32_t(*const e)[32] = edge[d & 1];
    e[2 * warp][lane] = R[1];
    e[2 * warp + 1][lane] = R[4];
    __syncthreads();
    R[0] = e[warp > 0 ? 2 * warp - 1 : 0][lane];
    R[5] = e[warp < 7 ? 2 * warp + 2 : 15][lane];
    uint32_t sides[6], all[6];  // rows y - 1 and y + 1, and the three of them
#pragma unroll
    for (int j = 0; j < 6; j++) {
      const uint32_t P = R[j] & (R[j] << 1) & (R[j] >> 1);
      sides[j] = __shfl_up_sync(kFull, P, 1) & __shfl_down_sync(kFull, P, 1);
      all[j] = sides[j] & P;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t r = R[j + 1];
      R[j + 1] = all[j] & all[j + 2] & sides[j + 1] & (r << 1) & (r >> 1) & mip0[j];
      out[(size_t)d * 1024 + 32 * (4 * warp + j) + lane] = R[j + 1];
    }
  }
}

}  // namespace
}  // namespace meso

using namespace meso;

extern "C" {

meso_status meso_quads_to_vertices(meso_ctx* ctx, const uint64_t* d_quads, uint64_t n, const int32_t* d_origins,
                                   uint32_t n_chunks, meso_vertex* d_out, void* stream) {
  if (!ctx || (n && (!d_quads || !d_origins || !d_out)))
    return fail(MESO_ERR_INVALID_ARG, "quads_to_vertices: null argument");
  if (n == 0) return MESO_OK;
  if (reinterpret_cast<uintptr_t>(d_out) & 15u)
    return fail(MESO_ERR_INVALID_ARG, "quads_to_vertices: output must be 16-byte aligned");
  const cudaStream_t st = pick_stream(ctx, stream);
  const uint64_t per_block = (uint64_t)kQvPer * kQvThreads;
  const uint64_t blocks = (4 * n + per_block - 1) / per_block;
  if (blocks > 0x7FFFFFFFull) return fail(MESO_ERR_INVALID_ARG, "quads_to_vertices: too many quads");
  quads_to_vertices_kernel<<<(unsigned)blocks, kQvThreads, 0, st>>>(d_quads, n, d_origins, n_chunks, d_out,
                                                                    ctx->d_scratch + 1);
  ctx->launches.fetch_add(1);
  MESO_CUDA_TRY(cudaGetLastError());
  return MESO_OK;
}

meso_status meso_erode_mips(meso_ctx* ctx, const meso_mesh_source* src, const int32_t* d_coords, uint32_t n,
                            uint32_t depth, uint32_t* d_out, void* stream) {
  if (!ctx || !src || (n && !d_out)) return fail(MESO_ERR_INVALID_ARG, "erode_mips: null argument");
  if (depth < 1 || depth > 8) return fail(MESO_ERR_INVALID_ARG, "erode_mips: depth must be 1..8");
  if (n == 0) return MESO_OK;
  if (n > 0x7FFFFFFFu) return fail(MESO_ERR_INVALID_ARG, "erode_mips: too many chunks");
  ErodeParams p;
  memset(&p, 0, sizeof(p));
  p.coords = d_coords;
  p.n = n;
  p.depth = depth;
  p.out = d_out;
  p.err = ctx->d_scratch + 1;
  if (src->kind == MESO_SRC_BRICKMAP) {
    if (!src->scene || !d_coords) return fail(MESO_ERR_INVALID_ARG, "erode_mips: brick map needs scene + coords");
    p.bptr = src->scene->d_ptr;
    p.bocc = src->scene->d_occ;
    p.bx = src->scene->bx;
    p.by = src->scene->by;
    p.bz = src->scene->bz;
  } else if (src->kind >= MESO_SRC_GRID_U8 && src->kind <= MESO_SRC_CHUNKS_U8) {
    if (!src->d_data) return fail(MESO_ERR_INVALID_ARG, "erode_mips: null data");
    const bool grid = src->kind == MESO_SRC_GRID_U8 || src->kind == MESO_SRC_GRID_U16;
    if (grid && (!d_coords || src->nx % 32 || src->ny % 32 || src->nz % 32))
      return fail(MESO_ERR_INVALID_ARG, "erode_mips: grid needs coords and dims multiple of 32");
    if (!grid && d_coords && src->nx <= 0)
      return fail(MESO_ERR_INVALID_ARG, "erode_mips: an index list needs nx = chunks in the array");
    if (!grid && (reinterpret_cast<uintptr_t>(src->d_data) & 15u))
      return fail(MESO_ERR_INVALID_ARG, "erode_mips: chunk array must be 16-byte aligned");
    p.data = static_cast<const uint8_t*>(src->d_data);
    p.nx = src->nx;
    p.ny = src->ny;
    p.nz = src->nz;
  } else {
    return fail(MESO_ERR_INVALID_ARG, "erode_mips: unknown source kind");
  }
  const cudaStream_t st = pick_stream(ctx, stream);
  const bool wide = (reinterpret_cast<uintptr_t>(p.data) & 15u) == 0;
  switch (src->kind) {
    case MESO_SRC_CHUNKS_U16: erode_kernel<MESO_SRC_CHUNKS_U16, true><<<n, kErodeThreads, 0, st>>>(p); break;
    case MESO_SRC_CHUNKS_U8: erode_kernel<MESO_SRC_CHUNKS_U8, true><<<n, kErodeThreads, 0, st>>>(p); break;
    case MESO_SRC_GRID_U8:
      if (wide) erode_kernel<MESO_SRC_GRID_U8, true><<<n, kErodeThreads, 0, st>>>(p);
      else erode_kernel<MESO_SRC_GRID_U8, false><<<n, kErodeThreads, 0, st>>>(p);
      break;
    case MESO_SRC_GRID_U16:
      if (wide) erode_kernel<MESO_SRC_GRID_U16, true><<<n, kErodeThreads, 0, st>>>(p);
      else erode_kernel<MESO_SRC_GRID_U16, false><<<n, kErodeThreads, 0, st>>>(p);
      break;
    default: erode_kernel<MESO_SRC_BRICKMAP, false><<<n, kErodeThreads, 0, st>>>(p);
  }
  ctx->launches.fetch_add(1);
  MESO_CUDA_TRY(cudaGetLastError());
  return MESO_OK;
}

meso_status meso_scene_save(meso_ctx* ctx, const meso_scene* s, const char* path) {
  if (!ctx || !s || !path) return fail(MESO_ERR_INVALID_ARG, "scene_save: null argument");
  const uint64_t nb = n_bricks_of(s);
  std::vector<uint32_t> ptr(nb);
  std::vector<uint64_t> occ(s->capacity * 8);
  std::vector<uint16_t> mat(s->capacity * 512);
  MESO_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  MESO_CUDA_TRY(cudaMemcpy(ptr.data(), s->d_ptr, nb * 4, cudaMemcpyDeviceToHost));
  MESO_CUDA_TRY(cudaMemcpy(occ.data(), s->d_occ, occ.size() * 8, cudaMemcpyDeviceToHost));
  MESO_CUDA_TRY(cudaMemcpy(mat.data(), s->d_mat, mat.size() * 2, cudaMemcpyDeviceToHost));
  FILE* f = fopen(path, "wb");
  if (!f) return fail(MESO_ERR_INVALID_ARG, std::string("scene_save: cannot open ") + path);
  uint64_t n = 0;
  for (uint64_t b = 0; b < nb; b++) n += ptr[b] != MESO_EMPTY_BRICK;
  char hdr[32];
  memset(hdr, 0, sizeof(hdr));
  memcpy(hdr, "MESOBRK1", 8);
  const uint32_t version = 1;
  memcpy(hdr + 8, &version, 4);
  memcpy(hdr + 12, &s->nx, 4);
  memcpy(hdr + 16, &s->ny, 4);
  memcpy(hdr + 20, &s->nz, 4);
  memcpy(hdr + 24, &n, 8);
  bool ok = fwrite(hdr, 1, 32, f) == 32;
  std::vector<uint32_t> order;
  order.reserve(n);
  std::vector<uint32_t> canon(nb);
  for (uint64_t b = 0; b < nb; b++) {
    if (ptr[b] == MESO_EMPTY_BRICK) {
      canon[b] = MESO_EMPTY_BRICK;
    } else {
      canon[b] = (uint32_t)order.size();
      order.push_back(ptr[b]);
    }
  }
  ok = ok && fwrite(canon.data(), 4, nb, f) == nb;
  for (uint64_t k = 0; ok && k < n; k++) ok = fwrite(&occ[(size_t)order[k] * 8], 8, 8, f) == 8;
  for (uint64_t k = 0; ok && k < n; k++) ok = fwrite(&mat[(size_t)order[k] * 512], 2, 512, f) == 512;
  ok = (fclose(f) == 0) && ok;
  return ok ? MESO_OK : fail(MESO_ERR_INVALID_ARG, std::string("scene_save: write failed: ") + path);
}

meso_status meso_scene_load(meso_ctx* ctx, const char* path, uint64_t spare, meso_scene** out) {
  if (!ctx || !path || !out) return fail(MESO_ERR_INVALID_ARG, "scene_load: null argument");
  FILE* f = fopen(path, "rb");
  if (!f) return fail(MESO_ERR_INVALID_ARG, std::string("scene_load: cannot open ") + path);
  char hdr[32];
  if (fread(hdr, 1, 32, f) != 32 || memcmp(hdr, "MESOBRK1", 8) != 0) {
    fclose(f);
    return fail(MESO_ERR_INVALID_ARG, "scene_load: not a brick-map file");
  }
  uint32_t version;
  int32_t nx, ny, nz;
  uint64_t n;
  memcpy(&version, hdr + 8, 4);
  memcpy(&nx, hdr + 12, 4);
  memcpy(&ny, hdr + 16, 4);
  memcpy(&nz, hdr + 20, 4);
  memcpy(&n, hdr + 24, 8);
  if (version != 1 || nx <= 0 || ny <= 0 || nz <= 0 || nx % 32 || ny % 32 || nz % 32 || nx > 8192 || ny > 8192 ||
      nz > 8192) {
    fclose(f);
    return fail(MESO_ERR_INVALID_ARG, "scene_load: unsupported header");
  }
  const uint64_t nb = (uint64_t)(nx / 8) * (ny / 8) * (nz / 8);
  if (n > nb) {
    fclose(f);
    return fail(MESO_ERR_INVALID_ARG, "scene_load: corrupt brick count");
  }
  std::vector<uint32_t> ptr(nb);
  std::vector<uint64_t> occ(n * 8);
  std::vector<uint16_t> mat(n * 512);
  bool ok = fread(ptr.data(), 4, nb, f) == nb && fread(occ.data(), 8, n * 8, f) == n * 8 &&
            fread(mat.data(), 2, n * 512, f) == n * 512;
  fclose(f);
  if (!ok) return fail(MESO_ERR_INVALID_ARG, "scene_load: truncated file");
  for (uint64_t b = 0; b < nb; b++)
    if (ptr[b] != MESO_EMPTY_BRICK && ptr[b] >= n) return fail(MESO_ERR_INVALID_ARG, "scene_load: bad brick pointer");
  meso_scene* s = nullptr;
  MESO_TRY(scene_alloc(ctx, nx, ny, nz, n + spare, &s));
  // All on ctx->stream, as the arrays' allocation and the maps' kernels are: a
  // pageable copy on the default stream may return before its data has reached
  // the device, and ctx->stream does not wait for that one.
  const cudaStream_t st = ctx->stream;
  const int32_t alloc[4] = {(int32_t)n, 0, 0, 0};
  cudaError_t e = cudaMemcpyAsync(s->d_ptr, ptr.data(), nb * 4, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && n) e = cudaMemcpyAsync(s->d_occ, occ.data(), n * 64, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && n) e = cudaMemcpyAsync(s->d_mat, mat.data(), n * 1024, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(s->d_alloc, alloc, 16, cudaMemcpyHostToDevice, st);
  meso_status rc = e == cudaSuccess ? MESO_OK : cuda_fail(e, "scene_load: upload");
  if (rc == MESO_OK) rc = rebuild_macro(ctx, s, nullptr, 0, st);
  if (rc == MESO_OK) rc = rebuild_sub(ctx, s, n, st);
  e = cudaStreamSynchronize(st);  // also after a failure: the copies read this call's memory
  if (rc == MESO_OK && e != cudaSuccess) rc = cuda_fail(e, "scene_load: macro map");
  if (rc != MESO_OK) {
    scene_release(ctx, s);
    return rc;
  }
  s->live_bricks_host = n;
  *out = s;
  return MESO_OK;
}

}  // extern "C"
