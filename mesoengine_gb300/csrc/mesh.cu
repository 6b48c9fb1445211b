// mesh.cu -- greedy chunk meshing on sm_103a.
//
// Replaces the reference's per-chunk host work: the 26-neighbour erosion cull
// (Runtimes/Voxel/Occupancy/BinaryOccupancyVolume.h:76-99, run from
// Runtimes/Voxel/Chunk/Chunk.h:73-100) and the one-instance-per-visible-block
// emission of FChunkPool::PushToBlockPool (Runtimes/Voxel/Chunk/ChunkPool.h:381-445),
// dispatched 8 chunks per host task by FChunkManage::MultiThreadGeneratorBatched
// (Runtimes/Voxel/Chunk/ChunkManager.h:183-210).  Here a persistent kernel
// pulls chunks from a device ticket queue and emits greedy quads.
//
// Two CTAs of 16 warps share each SM (64 registers per thread), each meshing
// its own chunk, so one CTA's barrier-separated phases overlap the other's
// work; the kernel is latency bound and 32 resident warps hide more of it
// than 16 or 24 did.  Per chunk:
//  1. staging: the 32^3 materials arrive in shared memory asynchronously
//     (TMA: one bulk copy per chunk of a chunk array, one 3-D tensor box per
//     chunk of a dense grid; for a brick map 16-byte copies of the occupied
//     bricks by the whole CTA, after the chunk has been picked out of a
//     ticket of chunks tested together against the scene's cell map); the
//     one-voxel occupancy halo is read with plain loads while it lands (the
//     columns beside a grid chunk's X faces arrive by TMA too);
//  2. masks: a lane takes 8 voxels of a row with one wide load, a warp 8 rows;
//     packed 16-bit (8-bit) operations give the byte of the row's occupancy
//     word and of its material-equality words with the -x, -y and -z
//     neighbour; warp-transposed copies (bits over y) serve the X faces;
//     face masks occ & ~shift(occ) are recomputed from these where needed;
//  3. sweep: one warp per face direction, lane = slice, row after row; all quads
//     of a row grow and start in about 30 word operations (see carry_on), and
//     what a row leaves behind is the word of its columns that continue a quad
//     from the row above;
//  4. emission: from those words any warp can tell the quads that start in a
//     row, their widths and heights; a task is 32 of the words that hold any,
//     lane = word, and the output is reserved once per chunk and direction.
#include <cudaTypedefs.h>

#include <cstdio>
#include <cstddef>
#include <cstring>

#include "meso_internal.h"

namespace meso {
namespace {

using namespace ::meso::dev;

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
// In the mask pass warp w takes rows 8 (w mod 4) .. +7 of slabs 8 (w / 4) .. +7.
static_assert(kWarps == 16, "four row groups by four slab groups");
constexpr int kS = 33;               // padded row stride of 32x32 word arrays
constexpr int kArr = 32 * kS;
// Words are emitted by the number of quads that start in them: up to kFew, up
// to kSome (lane = word in both), more (lane = column).
constexpr int kFew = 2, kSome = 8;
// Bytes per staged brick: two rows of each of four bricks side by side, what a
// quarter of a warp loads at once, lie in 32 different banks (with 1040 one row
// met another's: all chunks of the 1024^3 terrain, launches back to back, 330 us
// and 324 so; at another time 288 and 283).
constexpr int kBrickSlot = 1056;
constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr uint32_t kSideBytes = 32 * 32 * 16;  // the column of 16 bytes beside a grid chunk, for its X halo
constexpr uint64_t kWaitLimitNs = 2000000000ull;

// Shared memory of one CTA: these arrays (the words first: see kSideBytes), then
// the staged materials of the chunk (KindTraits::kMatBytes, 128-byte aligned).
struct __align__(128) MeshSmem {
  uint32_t occ[kArr];                     // occupancy, bits over x, [z][y]
  uint32_t occt[kArr];                    // occupancy, bits over y, [z][x]
  uint32_t ex[kArr], ey[kArr], ez[kArr];  // equality with -x / -y / -z neighbour, bits over x, [z][y]
  uint32_t eyt[kArr], ezt[kArr];          // equality with -y / -z neighbour, bits over y, [z][x]
  // columns that continue a quad from the row above, bits and layout as the
  // words of the direction: the odd directions'; the even directions' replace
  // the equality with the row above, which the sweep is the last to read
  uint32_t cont[3][kArr];
  uint32_t halo[6][32];                   // -X,+X: bits y by z; -Y,+Y: bits x by z; -Z,+Z: bits x by y
  uint64_t quad_base[6];                  // per direction: first output index of its quads
  uint32_t quad_next[6];                  // how many of them have their place
  uint32_t start_rows[18][32];            // per class and direction, per row: slices with such a word
  uint16_t start_rank[18][32];            // how many such words the rows before hold
  uint16_t start_words[18];               // how many all rows hold
  uint64_t bar;
  struct {
    int32_t chunk;     // list entry, -1: the queue is empty
    int32_t valid;     // 1: mesh it; 0: bad coordinate or index (flagged); 2: no occupied brick
    int32_t coord[3];  // chunk coordinates; chunk arrays: [0] the chunk's index
    uint32_t bricks[64];  // brick maps: the chunk's 64 brick pointers
  } job[2];  // the chunk being meshed and the one after it, in turn
  uint32_t chunk_quads;
  uint32_t task_next;                     // dynamic task counter of the emission
  uint32_t any_solid;
};

static_assert(offsetof(MeshSmem, halo) >= 2 * kSideBytes, "a grid chunk's two side columns land in the word arrays");

struct MeshParams {
  const uint8_t* data;
  int32_t nx, ny, nz;
  const uint32_t* bptr;
  const uint64_t* bocc;
  const uint16_t* bmat;
  const uint8_t* bcell;  // per 4x4x4-brick cell (one chunk): nonzero iff a brick of it is occupied
  int32_t bx, by, bz;
  const int32_t* coords;
  uint32_t n_chunks;
  uint32_t chunk_id_base;
  uint64_t* quads;
  uint64_t cap;
  unsigned long long* count;
  uint32_t* chunk_counts;
  uint32_t* ticket;
  uint32_t* err;
  uint32_t per_ticket;
  int32_t use_queue;
  uint32_t perm_mul;  // brick maps: ticket t takes list entry (t * perm_mul) mod n_chunks
};

// Per source kind: halo reads, addressing, element size, the staged bytes of
// one chunk, and the CTAs per SM (two of 16 warps: the register file allows
// no more, and 16-bit chunks fill the shared memory of two).
template <int KIND>
struct KindTraits;
template <int KIND>
struct KindBase {
  static constexpr bool kHalo = KIND != MESO_SRC_CHUNKS_U16 && KIND != MESO_SRC_CHUNKS_U8;
  static constexpr bool kGrid = KIND == MESO_SRC_GRID_U8 || KIND == MESO_SRC_GRID_U16;
  static constexpr bool kBrick = KIND == MESO_SRC_BRICKMAP;
  static constexpr int kElem = KIND == MESO_SRC_CHUNKS_U8 || KIND == MESO_SRC_GRID_U8 ? 1 : 2;
  static constexpr int kMatBytes = kBrick ? 64 * kBrickSlot : 32768 * kElem;
  static constexpr int kCtasPerSm = 2;
  static_assert(sizeof(MeshSmem) + kMatBytes + 128 + 1024 <= 228 * 1024 / kCtasPerSm,
                "the mesher's CTAs per SM must fit the shared memory");
};
template <>
struct KindTraits<MESO_SRC_CHUNKS_U16> : KindBase<MESO_SRC_CHUNKS_U16> {};
template <>
struct KindTraits<MESO_SRC_CHUNKS_U8> : KindBase<MESO_SRC_CHUNKS_U8> {};
template <>
struct KindTraits<MESO_SRC_GRID_U8> : KindBase<MESO_SRC_GRID_U8> {};
template <>
struct KindTraits<MESO_SRC_GRID_U16> : KindBase<MESO_SRC_GRID_U16> {};
template <>
struct KindTraits<MESO_SRC_BRICKMAP> : KindBase<MESO_SRC_BRICKMAP> {};

// Material at chunk-local linear index lin = x + 32 y + 1024 z.
template <int KIND>
__device__ __forceinline__ uint32_t load_mat_lin(const uint8_t* buf, uint32_t lin) {
  using T = KindTraits<KIND>;
  if constexpr (T::kBrick) {
    const uint32_t x = lin & 31u, y = (lin >> 5) & 31u, z = lin >> 10;
    const uint32_t b = (x >> 3) + 4 * (y >> 3) + 16 * (z >> 3);
    return reinterpret_cast<const uint16_t*>(buf + b * kBrickSlot)[(x & 7) + 8 * (y & 7) + 64 * (z & 7)];
  } else if constexpr (T::kElem == 2) {
    return reinterpret_cast<const uint16_t*>(buf)[lin];
  } else {
    return buf[lin];
  }
}

// The 8 voxels 8 seg .. of row (y, z): 16-bit materials in 4 registers, 8-bit
// ones in 2.
template <int KIND>
struct Seg {
  static constexpr int kRegs = KindTraits<KIND>::kElem == 2 ? 4 : 2;
  uint32_t w[kRegs];
};
template <int KIND>
__device__ __forceinline__ Seg<KIND> load_seg(const uint8_t* buf, int seg, int y, int z) {
  using T = KindTraits<KIND>;
  Seg<KIND> r;
  if constexpr (T::kElem == 2) {
    const uint8_t* a;
    if constexpr (T::kBrick)
      a = buf + (seg + 4 * (y >> 3) + 16 * (z >> 3)) * kBrickSlot + 128 * (z & 7) + 16 * (y & 7);
    else
      a = buf + (z * 32 + y) * 64 + 16 * seg;
    const uint4 v = *reinterpret_cast<const uint4*>(a);
    r.w[0] = v.x;
    r.w[1] = v.y;
    r.w[2] = v.z;
    r.w[3] = v.w;
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(buf + (z * 32 + y) * 32 + 8 * seg);
    r.w[0] = v.x;
    r.w[1] = v.y;
  }
  return r;
}

// Bit x set iff voxel x of a and of b differ.
template <int KIND>
__device__ __forceinline__ uint32_t differ(const Seg<KIND>& a, const Seg<KIND>& b) {
  if constexpr (KindTraits<KIND>::kElem == 2) {
    uint32_t t = 0;  // even voxels in bits 0, 2, 4, 6, odd ones 16 higher
#pragma unroll
    for (int k = 3; k >= 0; k--) t = t * 4u + __vminu2(a.w[k] ^ b.w[k], 0x00010001u);
    return (t | t >> 15) & 0xFFu;
  } else {
    uint32_t m[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint32_t d = a.w[k] ^ b.w[k];
      const uint32_t f = ((((d & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | d) >> 7) & 0x01010101u;  // bit 0 of each byte
      m[k] = f * 0x01020408u >> 24;                                                    // .. side by side
    }
    return m[0] | m[1] << 4;
  }
}

// Producer side: called by one warp (all lanes), which holds the queue state:
// takes the next chunk off the queue, writes what the CTA needs to know of it
// into `job` and has its data prefetched into L2.  It runs beside the emission
// of the chunk before, so the ticket, the coordinates and the brick pointers,
// loads that wait for one another, cost nothing; taken any earlier, a CTA with
// a slow chunk would hold back work from the others.  All chunks of the 1024^3
// terrain 436 -> 410 us, the 256^3 grid 49 -> 45.
//
// cur .. end is the rest of the current ticket.  Brick maps take a ticket of
// per_ticket (<= 32) list entries at a time, one per lane, through the bijection
// t -> (t * perm_mul) mod n_chunks so that a ticket samples the whole list (runs
// of neighbouring chunks are all air or all terrain), and test them together
// against the scene's cell map: a chunk with no occupied brick has no solid
// voxel and so no face, and is counted (0 quads) and passed over here, without
// a round trip through the CTA.  bc is this lane's entry of the current ticket,
// bmask the lanes whose entry is still to be meshed (an entry with an invalid
// coordinate is meshed, to be flagged there).
template <int KIND, typename Job>
__device__ __forceinline__ void take_chunk(Job& job, const MeshParams& p, const CUtensorMap* tmap, int lane,
                                           uint32_t& cur, uint32_t& end, int& bc, uint32_t& bmask) {
  using T = KindTraits<KIND>;
  int c = -1;
  if (T::kBrick && p.use_queue) {
    const int MX = p.bx >> 2, MY = p.by >> 2, MZ = p.bz >> 2;
    for (;;) {
      if (bmask == 0) {
        uint32_t t0 = 0;
        if (lane == 0) t0 = atomicAdd(p.ticket, p.per_ticket);
        t0 = __shfl_sync(kFull, t0, 0);
        if (t0 >= p.n_chunks) break;
        const uint32_t t = t0 + (uint32_t)lane;
        bool need = false;
        bc = -1;
        if ((uint32_t)lane < p.per_ticket && t < p.n_chunks) {
          bc = (int)(((uint64_t)t * p.perm_mul) % p.n_chunks);
          const int x = p.coords[3 * bc], y = p.coords[3 * bc + 1], z = p.coords[3 * bc + 2];
          const bool ok = x >= 0 && y >= 0 && z >= 0 && x < MX && y < MY && z < MZ;
          need = !ok || __ldg(p.bcell + x + (size_t)MX * (y + (size_t)MY * z)) != 0;
          if (!need && p.chunk_counts) p.chunk_counts[bc] = 0;
        }
        bmask = __ballot_sync(kFull, need);
        continue;
      }
      const int l = __ffs(bmask) - 1;
      bmask &= bmask - 1u;
      c = __shfl_sync(kFull, bc, l);
      break;
    }
  } else {
    if (lane == 0) {
      if (p.use_queue) {
        if (cur >= end) {
          cur = atomicAdd(p.ticket, p.per_ticket);
          end = cur + p.per_ticket;
        }
        if (cur < p.n_chunks) c = (int)cur++;
      } else if (cur < p.n_chunks) {
        c = (int)cur;
        cur += gridDim.x;
      }
    }
    c = __shfl_sync(kFull, c, 0);
  }
  if (lane == 0) job.chunk = c;
  if (c < 0) return;
  if constexpr (!T::kGrid && !T::kBrick) {
    if (lane == 0) {
      // with an index list, p.nx is the number of chunks in the array
      const uint32_t idx = p.coords ? (uint32_t)p.coords[c] : (uint32_t)c;
      const bool ok = !p.coords || idx < (uint32_t)p.nx;
      job.valid = ok ? 1 : 0;
      job.coord[0] = (int32_t)idx;
      if (ok) bulk_prefetch_l2(p.data + (size_t)idx * 32768u * T::kElem, 32768u * T::kElem);
      else atomicOr(p.err, ERR_BAD_INPUT);
    }
  } else {
    const int xyz = lane < 3 ? p.coords[3 * (size_t)c + lane] : 0;
    const int cx = __shfl_sync(kFull, xyz, 0), cy = __shfl_sync(kFull, xyz, 1), cz = __shfl_sync(kFull, xyz, 2);
    const int lim_x = T::kBrick ? p.bx / 4 : p.nx / 32, lim_y = T::kBrick ? p.by / 4 : p.ny / 32,
              lim_z = T::kBrick ? p.bz / 4 : p.nz / 32;
    const bool ok = cx >= 0 && cy >= 0 && cz >= 0 && cx < lim_x && cy < lim_y && cz < lim_z;
    if (lane < 3) job.coord[lane] = xyz;
    if (lane == 0) {
      job.valid = ok ? 1 : 0;
      if (!ok) atomicOr(p.err, ERR_BAD_INPUT);
    }
    if (!ok) return;
    if constexpr (T::kGrid) {
      if (lane == 0) tma_prefetch_3d(tmap, cx * 32, cy * 32, cz * 32);
    } else {
      // 64 bricks, two per lane
      bool any = false;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int b = lane + 32 * k;
        const int gx = cx * 4 + (b & 3), gy = cy * 4 + ((b >> 2) & 3), gz = cz * 4 + (b >> 4);
        const uint32_t slot = __ldg(p.bptr + gx + (size_t)p.bx * (gy + (size_t)p.by * gz));
        job.bricks[b] = slot;
        if (slot != MESO_EMPTY_BRICK) {
          any = true;
          bulk_prefetch_l2(p.bmat + (size_t)slot * 512, 1024);
        }
      }
      // no occupied brick: no solid voxel, so no face and nothing to stage
      any = __any_sync(kFull, any);
      if (lane == 0 && !any) job.valid = 2;
    }
  }
}

// Starts the copy of the job's materials into the staging buffer and, for a
// grid, of the columns beside its X faces into the word arrays (one thread;
// brick maps are copied by the whole CTA, their phase of the barrier completes
// with no bytes).
template <int KIND, typename Job>
__device__ __forceinline__ void stage_chunk(MeshSmem& sm, uint8_t* dst, const Job& job, const MeshParams& p,
                                            const CUtensorMap* tmap, const CUtensorMap* hmap) {
  using T = KindTraits<KIND>;
  uint64_t* bar = &sm.bar;
  if (T::kBrick || job.valid != 1) {
    mbar_arrive_expect_tx(bar, 0);
    return;
  }
  fence_proxy_async_smem();
  const uint32_t bytes = 32768u * T::kElem;
  mbar_arrive_expect_tx(bar, bytes + (T::kGrid ? 2u * kSideBytes : 0u));
  if constexpr (T::kGrid) {
    const int x = job.coord[0] * 32, y = job.coord[1] * 32, z = job.coord[2] * 32;
    uint8_t* const sides = reinterpret_cast<uint8_t*>(&sm);
    tma_load_3d(sides, hmap, x - 16 / T::kElem, y, z, bar);
    tma_load_3d(sides + kSideBytes, hmap, x + 32, y, z, bar);
    tma_load_3d(dst, tmap, x, y, z, bar);
  } else {
    const uint8_t* src = p.data + (size_t)(uint32_t)job.coord[0] * bytes;
    for (uint32_t off = 0; off < bytes; off += 16384u) bulk_g2s(dst + off, src + off, 16384u, bar);
  }
}

// The one-voxel occupancy halo around a chunk of a brick map: each face of the
// chunk meets 16 bricks, whose 8 x 8 voxels there are bytes (or, for the X
// faces, a bit of each byte) of their occupancy words; a lane takes 8 of them.
// (A voxel per lane and a ballot per row took 7 times the instructions: all
// chunks of the 1024^3 terrain 410 us, 292 then.)
__device__ __forceinline__ void brick_halos(MeshSmem& sm, const int32_t (&coord)[3], const MeshParams& p, int warp,
                                            int lane) {
  for (int i = warp; i < 24; i += kWarps) {
    const int f = i >> 2, k = lane + 32 * (i & 3), b = k >> 3, r = k & 7;
    const int side = f & 1 ? 4 : -1, in = f & 1 ? 0 : 7;  // the brick beyond the chunk, its layer next to it
    const int u = b & 3, v = b >> 2;
    const int gx = coord[0] * 4 + (f < 2 ? side : u), gy = coord[1] * 4 + (f < 2 ? u : (f < 4 ? side : v)),
              gz = coord[2] * 4 + (f < 4 ? v : side);
    uint32_t bits = 0;
    if (gx >= 0 && gy >= 0 && gz >= 0 && gx < p.bx && gy < p.by && gz < p.bz) {
      const uint32_t slot = __ldg(p.bptr + gx + (size_t)p.bx * (gy + (size_t)p.by * gz));
      if (slot != MESO_EMPTY_BRICK) {
        const uint64_t w = __ldg(p.bocc + (size_t)slot * 8 + (f < 4 ? r : in));
        if (f < 2) bits = (uint32_t)((((w >> in) & 0x0101010101010101ull) * 0x0102040810204080ull) >> 56);
        else bits = (uint32_t)(w >> (8 * (f < 4 ? in : r))) & 0xFFu;
      }
    }
    reinterpret_cast<uint8_t*>(&sm.halo[f][8 * v + r])[u] = (uint8_t)bits;
  }
}

// The same for the Y and Z faces of a dense grid: 4 faces x 32 rows, 8 rows of a
// face to a warp, 8 voxels of a row to a lane.  (A voxel per lane and a ballot per
// row took several times the instructions: 4096 chunks uint8 196 us, now 192, uint16
// 192 and 188.)
template <int KIND>
__device__ __forceinline__ void grid_halos(MeshSmem& sm, const int32_t (&coord)[3], const MeshParams& p, int warp,
                                           int lane) {
  static_assert(kWarps == 16, "a warp takes 8 of the 128 rows");
  using T = KindTraits<KIND>;
  const int f = 2 + (warp >> 2), k = 8 * (warp & 3) + (lane >> 2), seg = lane & 3;
  const int beyond = f & 1 ? 32 : -1;
  const int y = coord[1] * 32 + (f < 4 ? beyond : k), z = coord[2] * 32 + (f < 4 ? k : beyond);
  uint32_t bits = 0;
  if (y >= 0 && y < p.ny && z >= 0 && z < p.nz) {
    const uint8_t* a =
        p.data + ((size_t)(coord[0] * 32 + 8 * seg) + (size_t)p.nx * ((size_t)y + (size_t)p.ny * (size_t)z)) * T::kElem;
    Seg<KIND> v, none;
#pragma unroll
    for (int i = 0; i < Seg<KIND>::kRegs; i++) none.w[i] = 0;
    if constexpr (T::kElem == 2) {
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(a));
      v.w[0] = w.x;
      v.w[1] = w.y;
      v.w[2] = w.z;
      v.w[3] = w.w;
    } else {
      const uint2 w = __ldg(reinterpret_cast<const uint2*>(a));
      v.w[0] = w.x;
      v.w[1] = w.y;
    }
    bits = differ<KIND>(v, none);
  }
  reinterpret_cast<uint8_t*>(sm.halo[f])[4 * k + seg] = (uint8_t)bits;
}

// In-register 32x32 bit transpose across a warp: lane r holds row r (bit c =
// element (r, c)); afterwards lane c holds column c (bit r).  Five butterfly
// stages swap the off-diagonal blocks of size 16, 8, 4, 2, 1.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
  for (int j = 16; j >= 1; j >>= 1) {
    const uint32_t lo = j == 16 ? 0x0000FFFFu : j == 8 ? 0x00FF00FFu : j == 4 ? 0x0F0F0F0Fu : j == 2 ? 0x33333333u
                                                                                                      : 0x55555555u;
    const uint32_t t = __shfl_xor_sync(kFull, x, j);
    x = (lane & j) ? ((x & ~lo) | ((t & ~lo) >> j)) : ((x & lo) | ((t & lo) << j));
  }
  return x;
}

// Array addressing of direction d: (slice s, row v) -> word offset.
__device__ __forceinline__ int word_off(int d, int s, int v) { return d < 4 ? v * kS + s : s * kS + v; }

// In-plane equality arrays of direction d: E along u, V along v.
__device__ __forceinline__ const uint32_t* e_arr(const MeshSmem& sm, int d) { return d < 2 ? sm.eyt : sm.ex; }
__device__ __forceinline__ uint32_t* v_arr(MeshSmem& sm, int d) { return d < 2 ? sm.ezt : (d < 4 ? sm.ez : sm.ey); }
// After the sweep: the words of the columns that continue from the row above.
__device__ __forceinline__ uint32_t* c_arr(MeshSmem& sm, int d) { return d & 1 ? sm.cont[d >> 1] : v_arr(sm, d); }

// Face word of direction d, slice s, row r: the occupancy word of the slice
// minus that of the next slice along the face normal, or of the halo.
__device__ __forceinline__ uint32_t face_col(const MeshSmem& sm, int d, int s, int r) {
  const bool pos = (d & 1) == 0;
  const int sn = pos ? s + 1 : s - 1;
  const bool edge = pos ? s == 31 : s == 0;
  // halo[d ^ 1] is the layer beyond the chunk on the side the face points to
  if (d < 2) return sm.occt[r * kS + s] & ~(edge ? sm.halo[d ^ 1][r] : sm.occt[r * kS + sn]);
  if (d < 4) return sm.occ[r * kS + s] & ~(edge ? sm.halo[d ^ 1][r] : sm.occ[r * kS + sn]);
  return sm.occ[s * kS + r] & ~(edge ? sm.halo[d ^ 1][r] : sm.occ[sn * kS + r]);
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Barrier of a pair of warps (ids 1.. ; 0 is __syncthreads).
__device__ __forceinline__ void pair_sync(int g) {
  asm volatile("bar.sync %0, 64;" ::"r"(1 + g) : "memory");
}

// The columns of a row in which the quads of the row above go on.  A: the
// faces of the row above (each belongs to a quad), J: its columns that belong to
// the same quad as the one before, G: the columns whose face continues the one
// above in material.  A quad goes on iff all of its columns are in G.
//
// A carry runs through consecutive ones: adding the columns above those that
// fail to J marks the rest of their quads upwards, and the same in reversed bits
// marks it downwards.  The two halves do not wait for one another: marking the
// quads that start well upwards and then, from their last columns, downwards
// made the sweep of 4096 chunks 5.6 us a chunk, this 5.4.
__device__ __forceinline__ uint32_t carry_on(uint32_t A, uint32_t J, uint32_t G) {
  const uint32_t fail = A & ~G, up = (fail << 1) & J;
  const uint32_t rJ = __brev(J) << 1, down = (__brev(fail) << 1) & rJ;  // rJ: same quad as the one after
  const uint32_t above = (((J + up) ^ J) | up) & J, below = (((rJ + down) ^ rJ) | down) & rJ;
  return A & G & ~(above | __brev(below));
}

// The sweep of direction d (one warp, lane = slice; the warps of directions 2k
// and 2k + 1 run together): Lysenko's scan takes the first face that no quad
// has, widens it along u while the material matches and grows it along v while
// the whole run matches.  Row by row that is: the quads of the row above whose
// columns all continue go on (they were started earlier and come first), and
// every maximal run of the faces that are left starts a quad.  Words of the
// columns that go on are left in c_arr; the slices' quads are counted, the
// direction's output range reserved.
//
// Some 35 instructions per row and 32 slices, whatever the faces look like.  It
// replaces a warp per slice that grew the runs of one row at a time, some 1300
// instructions for a slice of the 256^3 noise grid, on which its chunks spent
// 40 us of 58 (now 4 of 16).
template <bool kHalo>
__device__ __forceinline__ void sweep(MeshSmem& sm, const MeshParams& p, int d, int lane) {
  const int st = d < 4 ? kS : 1, base = d < 4 ? lane : lane * kS;  // word_off(d, lane, v) = base + v * st
  const uint32_t* occ = d < 2 ? sm.occt : sm.occ;
  const uint32_t* eq = e_arr(sm, d);
  const uint32_t* up = v_arr(sm, d);
  uint32_t* out = c_arr(sm, d);
  const bool plus = (d & 1) == 0;
  const bool edge = lane == (plus ? 31 : 0);
  const int src = (lane + (plus ? 1 : 31)) & 31;
  uint32_t A = 0, J = 0, n = 0;
#pragma unroll 1
  for (int v0 = 0; v0 < 32; v0 += 8) {
    uint32_t F[8], G[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int o = base + (v0 + k) * st;
      const uint32_t c = occ[o];
      uint32_t beyond = __shfl_sync(kFull, c, src);
      if (edge) beyond = kHalo ? sm.halo[d ^ 1][v0 + k] : 0u;
      F[k] = c & ~beyond;
      G[k] = F[k] & up[o];
    }
    // both directions have read these rows of `up` before one overwrites them
    pair_sync(d >> 1);
    uint32_t any = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) any |= F[k];
    if (!__any_sync(kFull, any != 0)) {
#pragma unroll
      for (int k = 0; k < 8; k++) out[base + (v0 + k) * st] = 0;
      if (lane < 24) sm.start_rows[d + 6 * (lane >> 3)][v0 + (lane & 7)] = 0;
      A = J = 0;
      continue;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int o = base + (v0 + k) * st;
      const uint32_t C = carry_on(A, J, G[k]);
      const uint32_t left = F[k] & ~C;
      const uint32_t link = left & eq[o] & (left << 1), starts = left & ~link;
      out[o] = C;
      const uint32_t m = __popc(starts);
      n += m;
      const uint32_t any = __ballot_sync(kFull, m != 0), some = __ballot_sync(kFull, m > (uint32_t)kFew),
                     many = __ballot_sync(kFull, m > (uint32_t)kSome);
      // (a store by one lane takes no turn of the ALU pipe; keeping each row's words
      // in its lane's registers took six: 4096 chunks 216 us, now 208)
      if (lane == 0) {
        sm.start_rows[d][v0 + k] = any;
        sm.start_rows[6 + d][v0 + k] = some;
        sm.start_rows[12 + d][v0 + k] = many;
      }
      A = F[k];
      J = (J & C) | link;
    }
  }
  const uint32_t total = __reduce_add_sync(kFull, n);
  __syncwarp();
  uint32_t rows[3];  // of row `lane`, the classes apart
  rows[2] = sm.start_rows[12 + d][lane];
  rows[1] = sm.start_rows[6 + d][lane] & ~rows[2];
  rows[0] = sm.start_rows[d][lane] & ~(rows[1] | rows[2]);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    uint32_t rank = __popc(rows[k]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, rank, o);
      if (lane >= o) rank += y;
    }
    const int i = 6 * k + d;
    sm.start_rows[i][lane] = rows[k];
    sm.start_rank[i][lane] = (uint16_t)(rank - __popc(rows[k]));
    if (lane == 31) sm.start_words[i] = (uint16_t)rank;
  }
  if (lane == 0) {
    sm.quad_next[d] = 0;
    if (total) {
      sm.quad_base[d] = atomicAdd(p.count, (unsigned long long)total);
      atomicAdd(&sm.chunk_quads, total);
    }
  }
}

// What the emission of a direction needs of it.
struct EmitDir {
  const uint32_t* C;       // columns that continue
  int dir;
  int sh_s, sh_u, sh_v;    // bit offsets of slice, column and row in the linear voxel index
  uint32_t hi_bits;        // chunk and direction in a quad's upper word
};

// Starts of quads in row v of the slice, and the columns that widen them.
__device__ __forceinline__ void row_words(uint32_t faces, uint32_t C, uint32_t E, uint32_t& starts, uint32_t& link) {
  const uint32_t left = faces & ~C;
  link = left & E & (left << 1);
  starts = left & ~link;
}

// Where the quads of some words go: `to` is the place of the first in the
// output, `room` the places that are left there (all of them, as a rule).
struct Places {
  uint2* to;
  uint32_t room;
};

// Writes the quad that starts in column u of a word; lin0: the word's voxel of
// column 0, link: its columns that widen a quad, below: the columns of the next
// row that continue one.
template <int KIND>
__device__ __forceinline__ void put_quad(const uint8_t* mb, const EmitDir& D, uint32_t lin0, int sl, int v, uint32_t u,
                                         uint32_t link, uint32_t below, const Places& at, uint32_t k) {
  const uint32_t lin = lin0 | u << D.sh_u;
  const uint32_t mat = load_mat_lin<KIND>(mb, lin);
  const uint32_t more = (uint32_t)__ffs(~((link >> u) >> 1)) - 1u;  // columns after the first
  uint32_t h = (below >> u) & 1u;                                   // rows after the first
  if (h)
    while (v + 1 + (int)h < 32 && (D.C[word_off(D.dir, sl, v + 1 + (int)h)] >> u) & 1u) h++;
  if (k < at.room) at.to[k] = make_uint2(lin << 26 | more << 21 | h << 16 | mat, D.hi_bits | lin >> 6);
}

// Position of the (r+1)-th set bit of w (r < popc(w)): halving on popcounts.
__device__ __forceinline__ uint32_t select_bit(uint32_t w, uint32_t r) {
  uint32_t pos = 0, c;
  c = __popc(w & 0xFFFFu);
  if (r >= c) { r -= c; w >>= 16; pos = 16; }
  c = __popc(w & 0xFFu);
  if (r >= c) { r -= c; w >>= 8; pos += 8; }
  c = __popc(w & 0xFu);
  if (r >= c) { r -= c; w >>= 4; pos += 4; }
  c = __popc(w & 0x3u);
  if (r >= c) { r -= c; w >>= 2; pos += 2; }
  return pos + (r >= (w & 1u) ? 1u : 0u);
}

// The quads of words j0 .. j0+31 of list i (class i / 6, direction D.dir) of
// the words (slice, row) in which any start, lane = word.  Lanes take their
// words' quads one by one, words with many are taken one at a time, lane =
// column.
//
// On the chunk workload 800 of a chunk's 6144 words hold quads, 3.3 each.
// 4096 chunks: 256 us with all words in one list, 234 by classes (1 and 8: 237,
// 2 and 12: 236, 3 and 10: 236), 220 with the places and the row below of a word
// looked up once per word; a lane per slice taking its quads one by one, 459.
template <int KIND>
__device__ __forceinline__ void emit_words(MeshSmem& sm, const MeshParams& p, const uint8_t* mb, const EmitDir& D,
                                           int i, uint32_t j0, int lane) {
  const uint32_t words = sm.start_words[i];
  const bool mine = j0 + (uint32_t)lane < words;
  const uint32_t j = mine ? j0 + (uint32_t)lane : words - 1u;
  const uint32_t rank = sm.start_rank[i][lane];
  int v = 0;
#pragma unroll
  for (int step = 16; step >= 1; step >>= 1) {
    const uint32_t r = __shfl_sync(kFull, rank, v + step);
    if (r <= j) v += step;
  }
  const int sl = (int)select_bit(sm.start_rows[i][v], j - __shfl_sync(kFull, rank, v));
  const int o = word_off(D.dir, sl, v);
  uint32_t starts, link;
  row_words(face_col(sm, D.dir, sl, v), D.C[o], e_arr(sm, D.dir)[o], starts, link);
  if (!mine) starts = 0;
  const uint32_t below = v < 31 ? D.C[word_off(D.dir, sl, v + 1)] : 0u;
  const uint32_t lin0 = (uint32_t)sl << D.sh_s | (uint32_t)v << D.sh_v;
  const uint32_t sum = __reduce_add_sync(kFull, (uint32_t)__popc(starts));
  uint32_t place = 0;
  if (lane == 0) place = atomicAdd(&sm.quad_next[D.dir], sum);
  const unsigned long long first = sm.quad_base[D.dir] + __shfl_sync(kFull, place, 0);
  Places at;
  at.to = reinterpret_cast<uint2*>(p.quads) + first;
  at.room = first >= p.cap ? 0u : (uint32_t)min(p.cap - first, (unsigned long long)0xFFFFFFFFu);
  uint32_t todo = __ballot_sync(kFull, starts != 0), k = 0;
  if (i < 12) {
    while (todo) {
      if (starts) {
        const uint32_t u = (uint32_t)__ffs(starts) - 1u;
        starts &= starts - 1u;
        put_quad<KIND>(mb, D, lin0, sl, v, u, link, below, at, k + __popc(todo & lanemask_lt()));
      }
      k += __popc(todo);
      todo = __ballot_sync(kFull, starts != 0);
    }
  } else {
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1u;
      const uint32_t word = __shfl_sync(kFull, starts, src), lk = __shfl_sync(kFull, link, src),
                     bl = __shfl_sync(kFull, below, src), l0 = __shfl_sync(kFull, lin0, src);
      const int s1 = __shfl_sync(kFull, sl, src), v1 = __shfl_sync(kFull, v, src);
      if ((word >> lane) & 1u)
        put_quad<KIND>(mb, D, l0, s1, v1, (uint32_t)lane, lk, bl, at, k + __popc(word & lanemask_lt()));
      k += __popc(word);
    }
  }
}

template <int KIND>
__global__ void __launch_bounds__(kThreads, KindTraits<KIND>::kCtasPerSm)
    mesh_kernel(const MeshParams p, const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap hmap) {
  using T = KindTraits<KIND>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base_addr = smem_u32(smem_raw);
  const uint32_t pad = (128u - (base_addr & 127u)) & 127u;
  MeshSmem& sm = *reinterpret_cast<MeshSmem*>(smem_raw + pad);
  uint8_t* const mat = smem_raw + pad + sizeof(MeshSmem);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the queue state, held by the last warp
  uint32_t cur = p.use_queue ? 0u : blockIdx.x, end = 0;
  int bc = -1;  // brick maps: the lanes' ticket entries (see take_chunk)
  uint32_t bmask = 0;

  if (tid == 0) {
    mbar_init(&sm.bar, 1);
    sm.chunk_quads = 0;
    sm.task_next = 0;
    sm.any_solid = 0;
    fence_proxy_async_smem();
  }
  for (int i = tid; i < 6 * 32; i += kThreads) (&sm.halo[0][0])[i] = 0;
  if (warp == kWarps - 1) take_chunk<KIND>(sm.job[0], p, &tmap, lane, cur, end, bc, bmask);
  __syncthreads();

  uint32_t phase = 0;  // of sm.bar, and the job's slot
  for (;;) {
    auto& job = sm.job[phase];
    const int c = job.chunk;
    if (c < 0) break;
    const bool valid = job.valid == 1;
    if (tid == 0) stage_chunk<KIND>(sm, mat, job, p, &tmap, &hmap);
    if constexpr (T::kBrick) {
      if (valid) {
        // 64 bricks x 64 pieces of 16 bytes; a warp covers 512 contiguous
        // bytes of one brick
#pragma unroll
        for (int k = 0; k < 4096 / kThreads; k++) {
          const int i = tid + kThreads * k, b = i >> 6, piece = i & 63;
          const uint32_t bp = job.bricks[b];
          uint8_t* d = mat + b * kBrickSlot + 16 * piece;
          if (bp != MESO_EMPTY_BRICK)
            cp_async16(d, reinterpret_cast<const uint8_t*>(p.bmat) + (size_t)bp * 1024u + 16u * piece);
          else
            *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
        }
        cp_async_commit();
      }
    }
    if constexpr (T::kHalo) {
      if (valid) {
        if constexpr (T::kBrick) brick_halos(sm, job.coord, p, warp, lane);
        else grid_halos<KIND>(sm, job.coord, p, warp, lane);
      }
    }
    if constexpr (T::kBrick) {
      if (valid) cp_async_wait_all();
    }
    const bool ok = mbar_wait_bounded(&sm.bar, phase, kWaitLimitNs);
    if (__syncthreads_or(!ok)) {
      // the copy did not land within the limit: flag it, give it one more
      // bounded wait so nothing is in flight into shared memory, and leave
      if (tid == 0) {
        atomicOr(p.err, ERR_TIMEOUT);
        mbar_wait_bounded(&sm.bar, phase, kWaitLimitNs);
      }
      __syncthreads();
      return;
    }
    if constexpr (T::kGrid) {
      // The X faces' halo from the columns of 16 bytes beside the chunk, one row
      // per ballot.  A voxel there is alone in its line, and as plain loads these
      // 2048 were 12 % of a chunk's time in the load pipe and most of the wait for
      // its data; TMA takes them past it, into the word arrays, which are idle
      // between two chunks, and fills what lies outside of the grid with zeros.
      // 4096 chunks of a grid: uint8 235 -> 196 us, uint16 241 -> 192; with the
      // columns prefetched into L2 like the chunk 204 and 200.
      if (valid) {
        const uint8_t* sides = reinterpret_cast<const uint8_t*>(&sm);
#pragma unroll
        for (int i = 0; i < 64 / kWarps; i++) {
          const int wi = warp + kWarps * i, f = wi >> 5, k = wi & 31;
          const uint8_t* a = sides + f * kSideBytes + (k * 32 + lane) * 16 + (f ? 0 : 16 - T::kElem);
          const uint32_t v = T::kElem == 2 ? *reinterpret_cast<const uint16_t*>(a) : *a;
          const uint32_t w = __ballot_sync(kFull, v != 0);
          if (lane == 0) sm.halo[f][k] = w;
        }
      }
      __syncthreads();
    }
    if (valid) {
      const uint8_t* mb = mat;
      // ---- pass 1: rows y0 .. y0+7 of slabs z0 .. z0+7, lane = 8 voxels (seg)
      // of a row; the slab below stays in registers.  Neighbours outside the
      // chunk need no care: the equality bits of the first column and row and
      // of the first slab meet no face that is joined across them.  Bits of
      // empty voxels are never looked at, so an empty group only clears its
      // occupancy.
      {
        const int y0 = (warp & 3) * 8, z0 = (warp >> 2) * 8;
        const int seg = lane & 3, y = y0 + (lane >> 2), yu = y > 0 ? y - 1 : 0;
        Seg<KIND> below = load_seg<KIND>(mb, seg, y, z0 > 0 ? z0 - 1 : 0);
        Seg<KIND> none;
#pragma unroll
        for (int k = 0; k < Seg<KIND>::kRegs; k++) none.w[k] = 0;
#pragma unroll 2
        for (int z = z0; z < z0 + 8; z++) {
          const Seg<KIND> m = load_seg<KIND>(mb, seg, y, z);
          const int o = (z * kS + y0) * 4 + lane;  // byte seg of row y's word
          uint32_t any = 0;
#pragma unroll
          for (int k = 0; k < Seg<KIND>::kRegs; k++) any |= m.w[k];
          if (!__any_sync(kFull, any != 0)) {
            reinterpret_cast<uint8_t*>(sm.occ)[o] = 0;
          } else {
            const Seg<KIND> up = load_seg<KIND>(mb, seg, yu, z);
            Seg<KIND> left;
            const uint32_t before = __shfl_up_sync(kFull, m.w[Seg<KIND>::kRegs - 1], 1);
#pragma unroll
            for (int k = 0; k < Seg<KIND>::kRegs; k++)
              left.w[k] = __byte_perm(k ? m.w[k ? k - 1 : 0] : before, m.w[k], KindTraits<KIND>::kElem == 2 ? 0x5432 : 0x6543);
            reinterpret_cast<uint8_t*>(sm.occ)[o] = (uint8_t)differ<KIND>(m, none);
            reinterpret_cast<uint8_t*>(sm.ex)[o] = (uint8_t)~differ<KIND>(m, left);
            reinterpret_cast<uint8_t*>(sm.ey)[o] = (uint8_t)~differ<KIND>(m, up);
            reinterpret_cast<uint8_t*>(sm.ez)[o] = (uint8_t)~differ<KIND>(m, below);
          }
          below = m;
        }
        // the four warps of these slabs' rows; then two slabs' transposes each
        asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp >> 2)) : "memory");
#pragma unroll 1
        for (int j = 2 * (warp & 3); j < 2 * (warp & 3) + 2; j++) {
          const int o = (z0 + j) * kS + lane;
          const uint32_t r_occ = sm.occ[o];
          uint32_t occT = 0, eyT = 0, ezT = 0;
          if (__any_sync(kFull, r_occ != 0)) {  // an empty slab needs no transposes
            occT = transpose32(r_occ, lane);
            eyT = transpose32(sm.ey[o], lane);
            ezT = transpose32(sm.ez[o], lane);
            if (lane == 0) sm.any_solid = 1;
          }
          sm.occt[o] = occT;
          sm.eyt[o] = eyT;
          sm.ezt[o] = ezT;
        }
      }
      __syncthreads();
      // ---- pass 2: the sweep, one warp per direction
      if (sm.any_solid) {
        if (warp < 6) sweep<T::kHalo>(sm, p, warp, lane);
        __syncthreads();
      }
    }
    // the next chunk is chosen beside the emission of this one
    if (warp == kWarps - 1) take_chunk<KIND>(sm.job[phase ^ 1u], p, &tmap, lane, cur, end, bc, bmask);
    if (valid) {
      const uint8_t* mb = mat;
      if (sm.any_solid) {
        // ---- pass 3: emission
        const uint32_t chunk_hi = ((p.chunk_id_base + (uint32_t)c) & 0xFFFFFu) << 12;
        // the 18 lists' tasks, longest first: lane l holds list 17 - l and the
        // number of tasks before it
        const uint32_t mine = lane < 18 ? ((uint32_t)sm.start_words[lane < 18 ? 17 - lane : 0] + 31u) >> 5 : 0u;
        uint32_t until = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(kFull, until, o);
          if (lane >= o) until += y;
        }
        const uint32_t n_tasks = __shfl_sync(kFull, until, 31);
#pragma unroll 1
        for (;;) {
          uint32_t t = 0;
          if (lane == 0) t = atomicAdd(&sm.task_next, 1u);
          t = __shfl_sync(kFull, t, 0);
          if (t >= n_tasks) break;
          const int l = __ffs(__ballot_sync(kFull, until > t)) - 1;
          const uint32_t before = __shfl_sync(kFull, until - mine, l);
          const int list = 17 - l;
          EmitDir D;
          D.dir = list >= 12 ? list - 12 : (list >= 6 ? list - 6 : list);
          D.C = c_arr(sm, D.dir);
          D.sh_s = D.dir < 2 ? 0 : (D.dir < 4 ? 5 : 10);
          D.sh_u = D.dir < 2 ? 5 : 0;
          D.sh_v = D.dir < 4 ? 10 : 5;
          D.hi_bits = chunk_hi | (uint32_t)D.dir << 9;
          emit_words<KIND>(sm, p, mb, D, list, (t - before) * 32u, lane);
        }
      }
    }
    __syncthreads();
    if (tid == 0) {
      if (p.chunk_counts) p.chunk_counts[c] = valid ? sm.chunk_quads : 0u;
      sm.chunk_quads = 0;
      sm.task_next = 0;
      sm.any_solid = 0;
    }
    phase ^= 1u;
  }
}

// --------------------------------------------------------------- host side

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  });
  return fn;
}

meso_status make_grid_map(const meso_mesh_source* src, int elem, uint32_t width, CUtensorMap* map) {
  auto enc = get_encode_fn();
  if (!enc) return fail(MESO_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[3] = {(cuuint64_t)src->nx, (cuuint64_t)src->ny, (cuuint64_t)src->nz};
  cuuint64_t strides[2] = {(cuuint64_t)src->nx * elem, (cuuint64_t)src->nx * src->ny * elem};
  cuuint32_t box[3] = {width, 32, 32};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3,
                   const_cast<void*>(src->d_data), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MESO_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return MESO_OK;
}

template <int KIND>
meso_status launch_kind(meso_ctx* ctx, const MeshParams& base, const CUtensorMap& tmap, const CUtensorMap& hmap, uint32_t n_chunks,
                        cudaStream_t st, bool per_launch) {
  const size_t smem = sizeof(MeshSmem) + KindTraits<KIND>::kMatBytes + 128;
  static bool attr_set[64] = {false};
  if (!attr_set[ctx->device & 63]) {
    MESO_CUDA_TRY(cudaFuncSetAttribute(mesh_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    MESO_CUDA_TRY(cudaFuncSetAttribute(mesh_kernel<KIND>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared));
    attr_set[ctx->device & 63] = true;
  }
  constexpr bool kCoords3 = KindTraits<KIND>::kGrid || KindTraits<KIND>::kBrick;
  if (per_launch) {
    for (uint32_t i = 0; i < n_chunks; i++) {
      MeshParams p = base;
      p.n_chunks = 1;
      p.chunk_id_base = base.chunk_id_base + i;
      p.use_queue = 0;
      if (kCoords3) p.coords = base.coords + 3 * (size_t)i;
      else if (base.coords) p.coords = base.coords + i;
      else p.data = base.data + (size_t)i * 32768u * KindTraits<KIND>::kElem;
      if (p.chunk_counts) p.chunk_counts = base.chunk_counts + i;
      mesh_kernel<KIND><<<1, kThreads, smem, st>>>(p, tmap, hmap);
      ctx->launches.fetch_add(1);
    }
    MESO_CUDA_TRY(cudaGetLastError());
    return MESO_OK;
  }
  MeshParams p = base;
  p.use_queue = 1;
  // CTAs per SM: the tuned value, at most (and by default) what fits the SM
  constexpr uint32_t kMaxCtas = KindTraits<KIND>::kCtasPerSm;
  const uint32_t tuned = ctx->tuning.mesh_ctas_per_sm;
  uint32_t grid = ctx->sm_count * (tuned && tuned < kMaxCtas ? tuned : kMaxCtas);
  if constexpr (KindTraits<KIND>::kBrick) {
    // tickets of up to 8 list entries (tested together against the cell map) as
    // long as a CTA gets 8 of them, fewer to a ticket on shorter lists: what a CTA
    // still holds when the queue runs out, the others wait for.  (us, with up to 8
    // as soon as there are as many entries per CTA, and so: 4096 chunks at a
    // terrain's ground 209 and 170, 2500 of them 150 and 109, 1200 76 and 61, all
    // 8000 of a 640^3 terrain 130 and 104, all 32,768 of a 1024^3 one, 80 % of
    // them air, alike: 324, and with tickets of 2, 4 and 16 345, 328 and 333.  A
    // list of nothing but air pays for its smaller tickets, 4096 entries 17 us
    // after 8; larger ones after a ticket of air took a list of 4096 entries with
    // one chunk in 20 from 37 to 43, with one in 5 from 60 to 68.)
    // 7919 and 104729 are primes, and no list of at most 2^20 entries is a
    // multiple of both, so t -> (t * perm_mul) mod n is a bijection
    const uint32_t b = n_chunks / (grid * 8u);
    p.per_ticket = b < 1 ? 1 : (b > 8 ? 8 : b);
    p.perm_mul = n_chunks % 7919u ? 7919u : 104729u;
  }
  const uint32_t per = p.per_ticket ? p.per_ticket : 1;
  const uint32_t need = (n_chunks + per - 1) / per;
  if (grid > need) grid = need;
  if (grid == 0) grid = 1;
  MESO_CUDA_TRY(cudaMemsetAsync(p.ticket, 0, sizeof(uint32_t), st));
  mesh_kernel<KIND><<<grid, kThreads, smem, st>>>(p, tmap, hmap);
  ctx->launches.fetch_add(1);
  MESO_CUDA_TRY(cudaGetLastError());
  return MESO_OK;
}

}  // namespace

meso_status launch_mesh(meso_ctx* ctx, const meso_mesh_source* src, const int32_t* d_coords, uint32_t n_chunks,
                        const meso_mesh_output* out, cudaStream_t st, bool per_launch, uint32_t chunk_id_base,
                        bool accumulate) {
  if (!src || !out || !out->d_quad_count) return fail(MESO_ERR_INVALID_ARG, "mesh: null source/output");
  if ((uint64_t)chunk_id_base + n_chunks > MESO_MAX_CHUNKS_PER_CALL)
    return fail(MESO_ERR_INVALID_ARG, "mesh: more than 2^20 chunks");
  if (out->capacity && !out->d_quads) return fail(MESO_ERR_INVALID_ARG, "mesh: capacity without buffer");
  MeshParams p;
  memset(&p, 0, sizeof(p));
  p.coords = d_coords;
  p.n_chunks = n_chunks;
  p.quads = out->d_quads;
  p.cap = out->capacity;
  p.count = reinterpret_cast<unsigned long long*>(out->d_quad_count);
  p.chunk_counts = out->d_chunk_quad_counts;
  p.ticket = ctx->d_tickets + (ctx->next_ticket.fetch_add(1) % meso_ctx::kTicketRing);
  p.err = ctx->d_scratch + 1;
  p.per_ticket = ctx->tuning.mesh_chunks_per_ticket ? ctx->tuning.mesh_chunks_per_ticket : 1;
  p.chunk_id_base = chunk_id_base;
  CUtensorMap tmap, hmap;
  memset(&tmap, 0, sizeof(tmap));
  memset(&hmap, 0, sizeof(hmap));
  const int kind = src->kind;
  if (kind == MESO_SRC_BRICKMAP) {
    const meso_scene* s = src->scene;
    if (!s) return fail(MESO_ERR_INVALID_ARG, "mesh: brick-map source without scene");
    if (s->nx % 32 || s->ny % 32 || s->nz % 32) return fail(MESO_ERR_INVALID_ARG, "mesh: scene dims not multiples of 32");
    if (!d_coords && n_chunks) return fail(MESO_ERR_INVALID_ARG, "mesh: brick-map source needs chunk coordinates");
    p.bptr = s->d_ptr;
    p.bocc = s->d_occ;
    p.bmat = s->d_mat;
    p.bcell = s->d_macro;
    p.bx = s->bx;
    p.by = s->by;
    p.bz = s->bz;
  } else {
    if (!src->d_data && n_chunks) return fail(MESO_ERR_INVALID_ARG, "mesh: null data");
    p.data = static_cast<const uint8_t*>(src->d_data);
    p.nx = src->nx;
    p.ny = src->ny;
    p.nz = src->nz;
    if (kind == MESO_SRC_GRID_U8 || kind == MESO_SRC_GRID_U16) {
      if (src->nx <= 0 || src->ny <= 0 || src->nz <= 0 || src->nx % 32 || src->ny % 32 || src->nz % 32)
        return fail(MESO_ERR_INVALID_ARG, "mesh: grid dims must be positive multiples of 32");
      if (!d_coords && n_chunks) return fail(MESO_ERR_INVALID_ARG, "mesh: grid source needs chunk coordinates");
      if ((reinterpret_cast<uintptr_t>(src->d_data) & 15u) != 0)
        return fail(MESO_ERR_INVALID_ARG, "mesh: grid base must be 16-byte aligned");
      const int elem = kind == MESO_SRC_GRID_U16 ? 2 : 1;
      MESO_TRY(make_grid_map(src, elem, 32, &tmap));
      MESO_TRY(make_grid_map(src, elem, 16 / elem, &hmap));
    } else if (kind == MESO_SRC_CHUNKS_U16 || kind == MESO_SRC_CHUNKS_U8) {
      if ((reinterpret_cast<uintptr_t>(src->d_data) & 15u) != 0)
        return fail(MESO_ERR_INVALID_ARG, "mesh: chunk array must be 16-byte aligned");
      if (d_coords && src->nx <= 0)
        return fail(MESO_ERR_INVALID_ARG, "mesh: an index list needs nx = number of chunks in the array");
    } else {
      return fail(MESO_ERR_INVALID_ARG, "mesh: unknown source kind");
    }
  }
  if (!accumulate) MESO_CUDA_TRY(cudaMemsetAsync(out->d_quad_count, 0, sizeof(uint64_t), st));
  if (n_chunks == 0) return MESO_OK;
  switch (kind) {
    case MESO_SRC_CHUNKS_U16: return launch_kind<MESO_SRC_CHUNKS_U16>(ctx, p, tmap, hmap, n_chunks, st, per_launch);
    case MESO_SRC_CHUNKS_U8: return launch_kind<MESO_SRC_CHUNKS_U8>(ctx, p, tmap, hmap, n_chunks, st, per_launch);
    case MESO_SRC_GRID_U8: return launch_kind<MESO_SRC_GRID_U8>(ctx, p, tmap, hmap, n_chunks, st, per_launch);
    case MESO_SRC_GRID_U16: return launch_kind<MESO_SRC_GRID_U16>(ctx, p, tmap, hmap, n_chunks, st, per_launch);
    default: return launch_kind<MESO_SRC_BRICKMAP>(ctx, p, tmap, hmap, n_chunks, st, per_launch);
  }
}


}  // namespace meso
