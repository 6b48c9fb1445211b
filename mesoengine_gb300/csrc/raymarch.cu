// raymarch.cu -- two-level brick-map DDA with a fused shadow ray, sm_103a.
//
// Replaces the reference's render step: an instanced draw of MaxBlockCount
// 7-vertex imposter cubes whose vertex shader places each visible block
// relative to the chunk-rebased camera (Samples/SimpleVoxel.cpp:146-192, draw
// at :383-387).  Here every pixel is one thread; a warp covers a tw x (32/tw)
// pixel tile so neighbouring rays walk the same bricks; many views (cameras,
// scenes) share one launch through a per-view descriptor table.
//
// Traversal (Amanatides & Woo 1987, at two levels): bricks whose pointer is
// empty are crossed in one coarse step; inside an occupied brick every voxel
// advance is a fine step over the brick's 8x8x8 occupancy bits.  Boundary
// times are computed from integer coordinates, t = (b - o) * (1/d), with
// correctly rounded single operations (__fsub_rn/__fmul_rn...) so the results
// are bit-identical to a host evaluation of the same sequence.  Equal boundary
// times break x < y < z.  walk_steps is that definition; walk_regions, which
// nearly all rays take, crosses empty space of any size in one turn of one
// loop and gives the same bytes.
//
// What bounds it: the instructions of the loop (141 per warp and turn, 45 % of
// them on the half-rate ALU pipe) and, for small images and at the end of a
// launch, the longest ray's chain of up to about 100 turns of some 0.3 us.
// 1920x1080, primary and shadow rays, 1024^3 terrain: 102 M warp instructions
// with 23.8 of 32 lanes active in 132 us, where separate loops for cell jumps,
// brick steps and voxel steps took 290 M with 16.6 lanes in 384 us; DRAM is
// idle (1 %).
#include <cmath>
#include <cstring>

#include "meso_internal.h"

namespace meso {

struct RayView {
  const uint32_t* ptr;
  const uint64_t* occ;
  const uint16_t* mat;
  const uint8_t* level;  // per brick: log2 of the edge (voxels) of the largest aligned empty cube it is part of, 0 if it is occupied
  const int4* bounds;    // of the occupied cells (voxels): minus the lowest, and the highest coordinates
  const uint64_t* sub;   // per pool slot: the brick's non-empty 2x2x2-voxel blocks, bit x + 4y + 16z; [-1]: none
  int32_t nx, ny, nz;
  int32_t cam_chunk[3];
  float o[3];
  float fwd[3], right[3], up[3];
  float tan_half;
  float aspect;  // width / height, correctly rounded
  uint32_t width, height;
  float margin;          // region walk: distance (voxels) at which a position estimate settles a boundary; 0: step by step
  uint32_t block_start;  // the launch's first block of this view
  meso_hit* out;  // this view's width*height hit records, row major
};

namespace {

using namespace ::meso::dev;

constexpr int kInlineViews = 32;
constexpr int kPlain = 0, kStatsMode = 1, kHashMode = 2;
constexpr int kByRegion = 0, kEither = 1, kBySteps = 2;  // which walk a launch's rays take (see raymarch_kernel)
constexpr uint32_t kFullMask = 0xFFFFFFFFu;
constexpr float kInf = __builtin_huge_valf();

// splitmix64 finaliser (the hit checksum's mixing function)
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 30;
  x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27;
  x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return x;
}

// The views of a launch as kernel parameters (one entry and no use where the
// descriptors come from a device table).
template <int kViews>
struct Views {
  RayView v[kViews];
};

struct RayParams {
  const RayView* table;  // device table (n_views > kInlineViews) or null
  uint32_t n_views;
  uint32_t tile_w, tile_h;
  uint32_t tile_shift;   // log2 of tile_w
  uint32_t block_shift;  // log2 of a block's tiles side by side
  float light[3];
  float inv_light[3];  // 1 / light per axis, correctly rounded (0 for a zero component)
  uint32_t shadow;
  uint64_t* stats;
  unsigned long long* hash;  // checksum instantiation: partial sums per view (see launch_raymarch)
  uint32_t order_mul;  // CTA b takes block (b * order_mul) mod gridDim.x (0: block b)
  uint32_t cta_rows;   // 1: the output is host memory; write whole CTA rows (see the kernel)
};

struct Trav {
  int hit;
  int vx, vy, vz;
  float t;
  int axis;
  uint32_t slot;  // pool slot of the brick that was hit
  uint32_t coarse, fine;
  uint32_t fetches, bricks;  // pointer fetches and occupied bricks entered (statistics only)
};

__device__ __forceinline__ float bound_time(int b, float o, float inv) {
  return __fmul_rn(__fsub_rn(__int2float_rn(b), o), inv);
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// ------------------------------------------------------- step by step
// Brick steps that the walk takes along one axis (sign s, brick B, next brick
// boundary nb) while it crosses an empty cube of mask + 1 bricks on a side, up to
// the step that leaves the cube through another axis at time tE (`first`: this
// axis wins ties with that one).  They are the axis's inner boundaries that
// precede the exit in (time, axis) order: a prefix, whose length is estimated
// from the position at tE and settled by the boundaries' own times.
__device__ __forceinline__ int inner_steps(int s, int B, int mask, int nb, float o, float d, float inv, float tE,
                                           bool first) {
  if (s == 0) return 0;
  const int inner = s > 0 ? mask - (B & mask) : (B & mask);
  const float pos = __fmaf_rn(d, tE, o), b = __int2float_rn(nb);
  const float q = s > 0 ? __fsub_rn(pos, b) : __fsub_rn(b, pos);
  int k = clampi((int)ceilf(__fmul_rn(q, 0.125f)), 0, inner);
  auto taken = [&](int i) {  // boundary i of the inner ones
    const float tb = bound_time(nb + 8 * s * i, o, inv);
    return tb < tE || (tb == tE && first);
  };
  while (k > 0 && !taken(k - 1)) k--;
  while (k < inner && taken(k)) k++;
  return k;
}

// The walk as it is defined, from voxel (vx,vy,vz) (absolute, inside the
// grid) at time t, entered through axis ea (-1 none).  Ray coordinates are
// relative to the absolute voxel (bx0,by0,bz0); ix, iy, iz are 1/d per axis
// (0 where d is 0).  A step cap ends the walk of a ray that makes no
// progress (a direction of zeros or NaNs).  The statistics instantiation
// takes this path to count its fetches, and so does any ray whose values lie
// outside what the region walk below was proven for.  kCubes: an empty cube of
// bricks is crossed in one step.  kKeep: the boundary times and the occupancy word
// are kept from voxel to voxel, as only a stepped axis has another time and only a
// step along z another word (256^3 random voxels, 10 % solid, 1280x720: 79.6 us
// without, 69.3 so); where the walk is out of line it has no registers for them.
template <bool kStats, bool kCubes, bool kKeep>
__device__ __forceinline__ void walk_steps(const RayView& V, int bx0, int by0, int bz0, float ox, float oy, float oz,
                                        float dx, float dy, float dz, float ix, float iy, float iz, int vx, int vy,
                                        int vz, float t, int ea, Trav& r) {
  uint32_t n_fetch = 0, n_brick = 0;
  const int sx = dx > 0.0f ? 1 : (dx < 0.0f ? -1 : 0);
  const int sy = dy > 0.0f ? 1 : (dy < 0.0f ? -1 : 0);
  const int sz = dz > 0.0f ? 1 : (dz < 0.0f ? -1 : 0);
  const int px = sx > 0 ? 1 : 0, py = sy > 0 ? 1 : 0, pz = sz > 0 ? 1 : 0;
  const int NBx = V.nx >> 3, NBy = V.ny >> 3, NBz = V.nz >> 3;
  int Bx = vx >> 3, By = vy >> 3, Bz = vz >> 3;
  uint32_t cs = 0, fs = 0;
  const uint32_t cap = (uint32_t)(4 * (V.nx + V.ny + V.nz) + 64);
  uint32_t p = MESO_EMPTY_BRICK;
  bool entered = false;  // into this brick from an empty one
  r.hit = 0;
  for (;;) {
    if (cs + fs > cap) break;
    const uint32_t brick = (uint32_t)Bx + (uint32_t)NBx * ((uint32_t)By + (uint32_t)NBy * (uint32_t)Bz);
    p = __ldg(V.ptr + brick);
    if (kStats) {
      n_fetch++;
      n_brick += p != MESO_EMPTY_BRICK;
    }
    const bool coarse = p == MESO_EMPTY_BRICK;
    if (coarse) {
      const int sh = kCubes ? (int)__ldg(V.level + brick) - 3 : 0;
      if (sh > 2) {
        // an empty cube of 2^sh bricks on a side, unless that would pass the cap;
        // smaller cubes are faster by the brick (the far view below, out of line: 175
        // us, with cubes of 4 188, of 2 as well 197)
        const int mask = (1 << sh) - 1;
        const float tx = sx ? bound_time((((Bx >> sh) + px) << (sh + 3)) - bx0, ox, ix) : kInf;
        const float ty = sy ? bound_time((((By >> sh) + py) << (sh + 3)) - by0, oy, iy) : kInf;
        const float tz = sz ? bound_time((((Bz >> sh) + pz) << (sh + 3)) - bz0, oz, iz) : kInf;
        const bool cy = ty < tx;
        float tm = cy ? ty : tx;
        const bool cz = tz < tm;
        tm = cz ? tz : tm;
        const int a = cz ? 2 : (cy ? 1 : 0);
        const int Ba = a == 0 ? Bx : (a == 1 ? By : Bz), sa = a == 0 ? sx : (a == 1 ? sy : sz);
        const int out = (sa > 0 ? mask - (Ba & mask) : (Ba & mask)) + 1;
        const int kx = a == 0 ? out : inner_steps(sx, Bx, mask, (Bx + px) * 8 - bx0, ox, dx, ix, tm, true);
        const int ky = a == 1 ? out : inner_steps(sy, By, mask, (By + py) * 8 - by0, oy, dy, iy, tm, a == 2);
        const int kz = a == 2 ? out : inner_steps(sz, Bz, mask, (Bz + pz) * 8 - bz0, oz, dz, iz, tm, false);
        const uint32_t k = (uint32_t)(kx + ky + kz);
        if (cs + fs + k <= cap) {
          cs += k;
          t = tm;
          ea = a;
          Bx += sx * kx;
          By += sy * ky;
          Bz += sz * kz;
          if (((unsigned)Bx >= (unsigned)NBx) | ((unsigned)By >= (unsigned)NBy) | ((unsigned)Bz >= (unsigned)NBz)) break;
          entered = true;
          continue;
        }
      }
      // one step per empty brick
      const float tx = sx ? bound_time((Bx + px) * 8 - bx0, ox, ix) : kInf;
      const float ty = sy ? bound_time((By + py) * 8 - by0, oy, iy) : kInf;
      const float tz = sz ? bound_time((Bz + pz) * 8 - bz0, oz, iz) : kInf;
      const bool cy = ty < tx;
      float tm = cy ? ty : tx;
      const bool cz = tz < tm;
      tm = cz ? tz : tm;
      const int a = cz ? 2 : (cy ? 1 : 0);
      cs++;
      t = tm;
      ea = a;
      Bx += a == 0 ? sx : 0;
      By += a == 1 ? sy : 0;
      Bz += a == 2 ? sz : 0;
      if (((unsigned)Bx >= (unsigned)NBx) | ((unsigned)By >= (unsigned)NBy) | ((unsigned)Bz >= (unsigned)NBz)) break;
      entered = true;
      continue;
    }
    if (entered) {
      // the voxel entered: exact along the stepped axis, floor of the entry
      // point (clamped into the brick) along the others
      const int fx = clampi((int)floorf(__fadd_rn(ox, __fmul_rn(dx, t))) + bx0, Bx * 8, Bx * 8 + 7);
      const int fy = clampi((int)floorf(__fadd_rn(oy, __fmul_rn(dy, t))) + by0, By * 8, By * 8 + 7);
      const int fz = clampi((int)floorf(__fadd_rn(oz, __fmul_rn(dz, t))) + bz0, Bz * 8, Bz * 8 + 7);
      vx = ea == 0 ? (sx > 0 ? Bx * 8 : Bx * 8 + 7) : fx;
      vy = ea == 1 ? (sy > 0 ? By * 8 : By * 8 + 7) : fy;
      vz = ea == 2 ? (sz > 0 ? Bz * 8 : Bz * 8 + 7) : fz;
      entered = false;
    }
    // voxel steps inside occupied brick p
    const uint64_t* occ = V.occ + (size_t)p * 8;
    uint64_t w = 0;
    int nvx = 0, nvy = 0, nvz = 0;  // next voxel boundary (relative) along each axis, and its time
    float tx = kInf, ty = kInf, tz = kInf;
    auto look = [&] {
      w = __ldg(occ + (vz & 7));
      nvx = vx + px - bx0;
      nvy = vy + py - by0;
      nvz = vz + pz - bz0;
      tx = sx ? bound_time(nvx, ox, ix) : kInf;
      ty = sy ? bound_time(nvy, oy, iy) : kInf;
      tz = sz ? bound_time(nvz, oz, iz) : kInf;
    };
    bool left = false;
    if (kKeep) look();
    for (;;) {
      if (!kKeep) look();
      if ((w >> ((vx & 7) + 8 * (vy & 7))) & 1ull) {
        r.hit = 1;
        break;
      }
      const bool cy = ty < tx;
      float tm = cy ? ty : tx;
      const bool cz = tz < tm;
      tm = cz ? tz : tm;
      const bool a2 = cz, a1 = cy && !cz, a0 = !cy && !cz;
      fs++;
      t = tm;
      ea = a2 ? 2 : (a1 ? 1 : 0);
      vx += a0 ? sx : 0;
      vy += a1 ? sy : 0;
      vz += a2 ? sz : 0;
      if (kKeep && a2) w = __ldg(occ + (vz & 7));  // (a word of this brick, unused, where the step leaves it)
      const int c = a0 ? vx : (a1 ? vy : vz);
      const int cb = a0 ? Bx : (a1 ? By : Bz);
      if ((c >> 3) != cb) {
        Bx = vx >> 3;
        By = vy >> 3;
        Bz = vz >> 3;
        left = ((unsigned)Bx >= (unsigned)NBx) | ((unsigned)By >= (unsigned)NBy) | ((unsigned)Bz >= (unsigned)NBz);
        break;
      }
      if (cs + fs > cap) {
        left = true;
        break;
      }
      if (kKeep) {
        nvx += a0 ? sx : 0;
        nvy += a1 ? sy : 0;
        nvz += a2 ? sz : 0;
        const float tn = bound_time(a0 ? nvx : (a1 ? nvy : nvz), a0 ? ox : (a1 ? oy : oz), a0 ? ix : (a1 ? iy : iz));
        tx = a0 ? tn : tx;
        ty = a1 ? tn : ty;
        tz = a2 ? tn : tz;
      }
    }
    if (r.hit || left) break;
  }
  r.vx = vx;
  r.vy = vy;
  r.vz = vz;
  r.t = t;
  r.axis = ea;
  r.slot = p;
  r.coarse = cs;
  r.fine = fs;
  r.fetches = n_fetch;
  r.bricks = n_brick;
}

// Out of line where few rays take it: it shares no registers with the region walk.
template <bool kCubes>
__device__ __noinline__ void walk_steps_apart(const RayView& V, int bx0, int by0, int bz0, float ox, float oy, float oz,
                                              float dx, float dy, float dz, float ix, float iy, float iz, int vx, int vy,
                                              int vz, float t, int ea, Trav& r) {
  walk_steps<false, kCubes, false>(V, bx0, by0, bz0, ox, oy, oz, dx, dy, dz, ix, iy, iz, vx, vy, vz, t, ea, r);
}

// ---------------------------------------------------------- region walk
// The same walk, taken a region at a time, with the same results bit for bit.
//
// A region is an aligned empty cube of 2^l voxels around the ray's position:
// l = 3..9 one brick to 64^3 bricks (a level byte per brick), l = 1, 2 blocks of 2^3 or 4^3 voxels of an occupied brick (a 64-bit mask of
// its 2^3-voxel blocks), l = 0 one voxel.  Every kind is left by one and the
// same piece of code, so the lanes of a warp stay together whatever each is
// crossing; the former loops for cell jumps, brick steps and voxel steps ran
// one after the other with half of the lanes idle.
//
// Why it is the same walk.  Each axis's boundary times never decrease along
// the ray, and the walk takes all axes' boundaries merged in (time, axis x<y<z)
// order.  So it leaves a region through the face with the smallest (time,
// axis); the boundaries of another axis that it takes before are those whose
// (time, axis) precede the face's, a prefix; and the steps it makes are the
// voxels (inside a brick) or bricks it moves by, whatever their order, so they
// are counted from the positions where a run of either kind begins and ends.
//
// The position along the other axes.  A boundary at relative coordinate b is
// taken iff its computed time (b - o) * (1/d) precedes the face's time tE.
// The computed time differs from the real (b - o) / d by at most 3 roundings,
// the position o + d * tE below by a few more: less than 8 * 2^-24 of the
// largest coordinate R in all.  Where the position lies further than twice
// that (margin = R * 2^-20) from a boundary, the boundary's side of it
// decides; else the boundary's own time is computed and compared.
//
// Directions are mirrored so that every ray moves up: an axis with d < 0
// counts voxels as ~v and uses -o, -d and -1/d, which rounds the same way
// and keeps the regions' alignment.  An axis with d = 0 gets an infinite
// 1/d, so its faces lie at infinite time and are never chosen.
//
constexpr float kRoundMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to the nearest integer
constexpr int kRoundBits = 0x4B400000;      // its bits

struct RayAxis {
  float o, d, i;  // mirrored origin, |d| and 1/|d| (infinite for d = 0)
  float a;        // o plus the base voxel: absolute origin, for estimates
  int b1;         // 1 - mirrored base voxel, plus kRoundBits
  int m;          // -1 for a mirrored axis, else 0
  int lo, hi;     // mirrored bounds of the occupied cells
};

__device__ __forceinline__ RayAxis ray_axis(int b0, float o, float d, float inv, int nlo, int hi) {
  RayAxis A;
  A.m = d < 0.0f ? -1 : 0;
  A.o = d < 0.0f ? -o : o;
  A.d = fabsf(d);
  A.i = d == 0.0f ? kInf : fabsf(inv);
  const int b = d < 0.0f ? -b0 : b0;
  A.a = A.o + __int2float_rn(b);
  A.b1 = kRoundBits + 1 - b;
  A.lo = d < 0.0f ? ~hi : -nlo;
  A.hi = d < 0.0f ? nlo - 1 : hi;
  return A;
}

// d is 0, or of a size at which 1/d and the boundary times are normal numbers
__host__ __device__ __forceinline__ bool regular_axis(float d) {
  const float m = fabsf(d);
  return m == 0.0f || (m > 1e-30f && m < 1e30f);
}

// Time of the mirrored absolute boundary last + 1.  The conversion to float
// (exact: the coordinate is below 2^22) is an addition in a float whose unit
// is one, which takes the FMA pipe and 4 cycles where the convert instruction
// takes a quarter-rate pipe.
__device__ __forceinline__ float face_time(const RayAxis& A, int last) {
  const float b = __fsub_rn(__int_as_float(last + A.b1), kRoundMagic);
  return __fmul_rn(__fsub_rn(b, A.o), A.i);
}

// Voxel (mirrored) at time t along an axis that was not stepped, by the
// definition's own operations: floor(o + d*t).
__device__ __forceinline__ int entry_voxel(const RayAxis& A, float t) {
  const float x = __fadd_rn(A.o, __fmul_rn(A.d, t));
  return (__float2int_rd(A.m ? -x : x) ^ A.m) + kRoundBits + 1 - A.b1;
}

// Position along one axis at time t in units of 1 / inv_unit voxels: the unit
// that the estimate lies in (its first voxel), and how far the estimate is
// from that unit's middle.
__device__ __forceinline__ int estimate(const RayAxis& A, float t, float inv_unit, uint32_t unit, uint32_t bias,
                                       float& off) {
  const float q = __fmaf_rn(__fmaf_rn(A.d, t, A.a), inv_unit, -0.5f);
  const float s = __fadd_rn(q, kRoundMagic);
  off = __fsub_rn(q, __fsub_rn(s, kRoundMagic));
  return (int)((uint32_t)__float_as_int(s) * unit + bias);
}

// An estimate too close to a unit boundary: the boundary's own time decides
// on which side of it the ray is at tE (`first`: this axis wins ties).
__device__ __forceinline__ int settle(const RayAxis& A, int e, int unit, float off, float tE, bool first) {
  const int b = off > 0.0f ? e + unit : e;  // the boundary next to the estimate
  const float tb = face_time(A, b - 1);
  return (tb < tE || (tb == tE && first)) ? b : b - unit;
}

// The position (nx, ny, nz) at time t on the two axes that are not stepped
// (ax, ay, az says which is), in units of voxels or bricks.
struct Unit {
  float inv;           // 1 / its voxels
  uint32_t voxels, bias;
};
__device__ __forceinline__ Unit voxel_unit() { return {1.0f, 1u, 0u - (uint32_t)kRoundBits}; }
__device__ __forceinline__ Unit brick_unit() { return {0.125f, 8u, 0u - 8u * (uint32_t)kRoundBits}; }

__device__ __forceinline__ void locate(const RayAxis& X, const RayAxis& Y, const RayAxis& Z, float margin,
                                       const Unit& U, float t, bool ax, bool ay, bool az, int& nx, int& ny, int& nz) {
  const float lim = __fmaf_rn(-margin, U.inv, 0.5f);
  float gx, gy, gz;
  nx = estimate(X, t, U.inv, U.voxels, U.bias, gx);
  ny = estimate(Y, t, U.inv, U.voxels, U.bias, gy);
  nz = estimate(Z, t, U.inv, U.voxels, U.bias, gz);
  const bool qx = !ax && fabsf(gx) > lim, qy = !ay && fabsf(gy) > lim, qz = !az && fabsf(gz) > lim;
  if (qx | qy | qz) {
    if (qx) nx = settle(X, nx, (int)U.voxels, gx, t, true);
    if (qy) ny = settle(Y, ny, (int)U.voxels, gy, t, az);
    if (qz) nz = settle(Z, nz, (int)U.voxels, gz, t, false);
  }
}

__device__ __forceinline__ void walk_regions(const RayView& V, const RayAxis& X, const RayAxis& Y, const RayAxis& Z,
                                             float margin, int vx, int vy, int vz, float t, int ea, Trav& r) {
  const uint32_t NBX = (uint32_t)V.nx >> 3, NBY = (uint32_t)V.ny >> 3;
  const uint32_t flip = (X.m & 7) | (Y.m & 56) | (Z.m & 448);  // the same, of a voxel's 3+3+3 bits in its brick
  int x = vx ^ X.m, y = vy ^ Y.m, z = vz ^ Z.m;            // mirrored position
  // steps: += position where a run of its kind ends, -= where it begins
  int cs = 0, fs = -(x + y + z);
  // the unit of the position estimates (a voxel in an occupied brick, a brick
  // elsewhere), kept and not derived from l: 6 instructions of each turn
  Unit U = voxel_unit();
  bool fine = true;   // in an occupied brick (the first position counts as one until looked up)
  bool look = true;   // the brick at the position has not been looked up
  uint32_t p = 0;
  uint2 blocks = make_uint2(0u, 0u);  // 2^3-voxel blocks of the current brick
  r.hit = 0;
  // All space outside the bounds of the occupied cells is one region: before
  // the loop the ray moves up to the bounds, behind it out of the grid.  (1080p
  // frame of the 1024^3 terrain, whose upper two thirds are sky: 15 % fewer
  // turns and 142 -> 132 us; a 256^2 view 31.6 -> 30.3.)
  bool past = (x > X.hi) | (y > Y.hi) | (z > Z.hi);
  if (!past && ((x < X.lo) | (y < Y.lo) | (z < Z.lo))) {
    // the last of the axes' entries; the ray misses the bounds if it leaves
    // them along another axis before
    const float tx = x < X.lo ? face_time(X, X.lo - 1) : -kInf, ty = y < Y.lo ? face_time(Y, Y.lo - 1) : -kInf,
                tz = z < Z.lo ? face_time(Z, Z.lo - 1) : -kInf;
    const float txy = fmaxf(tx, ty);
    const bool az = tz >= txy, ay = !az && ty >= tx, ax = !az && !ay;
    const float tE = fmaxf(txy, tz);
    const float ux = face_time(X, X.hi), uy = face_time(Y, Y.hi), uz = face_time(Z, Z.hi);
    past = ux < tE || (ux == tE && !ax) || uy < tE || (uy == tE && az) || uz < tE;
    if (!past) {
      fs = 0;
      cs = -((x >> 3) + (y >> 3) + (z >> 3));
      fine = false;
      U = brick_unit();
      int nx, ny, nz;
      locate(X, Y, Z, margin, U, tE, ax, ay, az, nx, ny, nz);
      x = ax ? X.lo : max(x, nx);
      y = ay ? Y.lo : max(y, ny);
      z = az ? Z.lo : max(z, nz);
      t = tE;
      ea = az ? 2 : (ay ? 1 : 0);
    }
  }
  while (!past) {
    int l = 0;
    if (look) {
      if ((x > X.hi) | (y > Y.hi) | (z > Z.hi)) break;
      const uint32_t brick = (uint32_t)((x ^ X.m) >> 3) +
                             NBX * ((uint32_t)((y ^ Y.m) >> 3) + NBY * (uint32_t)((z ^ Z.m) >> 3));
      l = __ldg(V.level + brick);
      p = __ldg(V.ptr + brick);  // fetched beside the level: one latency instead of two where it is needed
      if (l == 0) {
        // Signed: an edit on a stream that this launch is not ordered with may
        // have unlinked the brick and not reached its level byte yet.  The empty
        // pointer is then -1, before the first slot, where no block is set (slots
        // are below 2^31, their materials alone would be 2 TiB).  A comparison
        // here instead took a 1080p frame from 129.1 to 130.4 us, this nothing.
        blocks = __ldg(reinterpret_cast<const uint2*>(V.sub) + (int32_t)p);
        if (!fine) {
          cs += (x >> 3) + (y >> 3) + (z >> 3);
          // floor of the entry point, in the brick (along the stepped axis
          // that is the brick's first voxel: the point lies on its face)
          x = clampi(entry_voxel(X, t), x & ~7, x | 7);
          y = clampi(entry_voxel(Y, t), y & ~7, y | 7);
          z = clampi(entry_voxel(Z, t), z & ~7, z | 7);
          fs -= x + y + z;
          fine = true;
          U = voxel_unit();
        }
      } else if (fine) {
        fs += x + y + z;
        cs -= (x >> 3) + (y >> 3) + (z >> 3);
        fine = false;
        U = brick_unit();
      }
    }
    if (fine) {
      const uint32_t v = ((x & 7) | ((y << 3) & 56) | ((z << 6) & 448)) ^ flip;  // voxel of the brick
      const uint32_t k = ((v >> 1) & 3u) | ((v >> 2) & 12u) | ((v >> 3) & 16u);  // its block, of half the brick
      const uint32_t half = v & 256u ? blocks.y : blocks.x;
      l = ((half >> (k & 10u)) & 0x330033u) == 0 ? 2 : 1;
      if ((half >> (k & 31u)) & 1u) {
        const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(V.occ) + ((size_t)p * 16 + (v >> 5)));
        if ((w >> (v & 31u)) & 1u) {
          r.hit = 1;
          break;
        }
        l = 0;
      }
    }
    // ---- leave the region of 2^l voxels
    const int in = (1 << l) - 1;
    const int lx = x | in, ly = y | in, lz = z | in;  // the region's last voxels
    const float tx = face_time(X, lx), ty = face_time(Y, ly), tz = face_time(Z, lz);
    const float txy = fminf(tx, ty);
    const bool az = tz < txy, ay = ty < tx && !az, ax = !az && !(ty < tx);
    const float tE = fminf(txy, tz);
    int nx, ny, nz;
    locate(X, Y, Z, margin, U, tE, ax, ay, az, nx, ny, nz);
    if (ax) nx = lx + 1;
    if (ay) ny = ly + 1;
    if (az) nz = lz + 1;
    // an entry point rounded up may lie ahead of the estimate; past the
    // region's face it cannot be, as that face's own time is not before tE
    x = max(x, nx);
    y = max(y, ny);
    z = max(z, nz);
    t = tE;
    ea = az ? 2 : (ay ? 1 : 0);
    look = !fine || ((az ? lz : (ay ? ly : lx)) & 7) == 7;
  }
  const int ex = V.nx & ~X.m, ey = V.ny & ~Y.m, ez = V.nz & ~Z.m;  // first mirrored voxels beyond the grid
  if (!r.hit && (x < ex) & (y < ey) & (z < ez)) {
    if (fine) {
      fs += x + y + z;
      cs -= (x >> 3) + (y >> 3) + (z >> 3);
      fine = false;
    }
    const float tx = face_time(X, ex - 1), ty = face_time(Y, ey - 1), tz = face_time(Z, ez - 1);
    const float txy = fminf(tx, ty);
    const bool az = tz < txy, ay = ty < tx && !az, ax = !az && !(ty < tx);
    int nx, ny, nz;
    locate(X, Y, Z, margin, brick_unit(), fminf(txy, tz), ax, ay, az, nx, ny, nz);
    x = ax ? ex : max(x, nx);
    y = ay ? ey : max(y, ny);
    z = az ? ez : max(z, nz);
  }
  if (fine) fs += x + y + z;
  else cs += (x >> 3) + (y >> 3) + (z >> 3);
  // a mirrored boundary that passes through the origin: (b - o) * (1/d) is
  // minus zero there
  if (t == 0.0f && ea >= 0) {
    const int f = (ea == 0 ? x + X.b1 : (ea == 1 ? y + Y.b1 : z + Z.b1)) - kRoundBits, m = ea == 0 ? X.m : (ea == 1 ? Y.m : Z.m);
    const float o = ea == 0 ? X.o : (ea == 1 ? Y.o : Z.o);
    if (m && __int2float_rn(f - 1) == o) t = -0.0f;
  }
  r.vx = x ^ X.m;
  r.vy = y ^ Y.m;
  r.vz = z ^ Z.m;
  r.t = t;
  r.axis = ea;
  r.slot = p;
  r.coarse = (uint32_t)cs;
  r.fine = (uint32_t)fs;
}

// Traces a ray by regions where its values allow, else step by step.
template <bool kStats, int kWalk>
__device__ __forceinline__ void trace(const RayView& V, float margin, int bx0, int by0, int bz0, float ox, float oy,
                                      float oz, float dx, float dy, float dz, float ix, float iy, float iz, int vx,
                                      int vy, int vz, float t, int ea, Trav& r) {
  if constexpr (kStats) {
    walk_steps<true, false, false>(V, bx0, by0, bz0, ox, oy, oz, dx, dy, dz, ix, iy, iz, vx, vy, vz, t, ea, r);
  } else if constexpr (kWalk == kBySteps) {
    walk_steps<false, true, true>(V, bx0, by0, bz0, ox, oy, oz, dx, dy, dz, ix, iy, iz, vx, vy, vz, t, ea, r);
  } else if (margin > 0.0f && regular_axis(dx) && regular_axis(dy) && regular_axis(dz) &&
             (dx != 0.0f || dy != 0.0f || dz != 0.0f)) {
    const int4 nlo = __ldg(V.bounds), hi = __ldg(V.bounds + 1);
    const RayAxis X = ray_axis(bx0, ox, dx, ix, nlo.x, hi.x), Y = ray_axis(by0, oy, dy, iy, nlo.y, hi.y),
                  Z = ray_axis(bz0, oz, dz, iz, nlo.z, hi.z);
    walk_regions(V, X, Y, Z, margin, vx, vy, vz, t, ea, r);
  } else {
    Trav q;
    walk_steps_apart<kWalk == kEither>(V, bx0, by0, bz0, ox, oy, oz, dx, dy, dz, ix, iy, iz, vx, vy, vz, t, ea, q);
    r = q;
  }
}

__device__ __forceinline__ void camera_ray(const RayView& V, uint32_t px, uint32_t py, float& dx, float& dy,
                                           float& dz) {
  float sxv = __fdiv_rn(__uint2float_rn(2u * px + 1u), __uint2float_rn(V.width));
  sxv = __fsub_rn(sxv, 1.0f);
  sxv = __fmul_rn(sxv, V.tan_half);
  sxv = __fmul_rn(sxv, V.aspect);
  float syv = __fdiv_rn(__uint2float_rn(2u * py + 1u), __uint2float_rn(V.height));
  syv = __fsub_rn(1.0f, syv);
  syv = __fmul_rn(syv, V.tan_half);
  const float d0 = __fadd_rn(__fadd_rn(V.fwd[0], __fmul_rn(V.right[0], sxv)), __fmul_rn(V.up[0], syv));
  const float d1 = __fadd_rn(__fadd_rn(V.fwd[1], __fmul_rn(V.right[1], sxv)), __fmul_rn(V.up[1], syv));
  const float d2 = __fadd_rn(__fadd_rn(V.fwd[2], __fmul_rn(V.right[2], sxv)), __fmul_rn(V.up[2], syv));
  float n2 = __fmul_rn(d0, d0);
  n2 = __fadd_rn(n2, __fmul_rn(d1, d1));
  n2 = __fadd_rn(n2, __fmul_rn(d2, d2));
  const float len = __fsqrt_rn(n2);
  dx = __fdiv_rn(d0, len);
  dy = __fdiv_rn(d1, len);
  dz = __fdiv_rn(d2, len);
}

template <bool kStats, int kWalk>
__device__ __forceinline__ void trace_pixel(const RayView& V, uint32_t px, uint32_t py, const RayParams& P,
                                            meso_hit& h, uint32_t* st) {
  h.voxel = ~0ull;
  h.t = kInf;
  h.material = 0;
  h.face = 6;
  h.shadow = 255;
  h.steps = 0;
  h.shadow_steps = 0;
  float dx, dy, dz;
  camera_ray(V, px, py, dx, dy, dz);
  const int bx0 = V.cam_chunk[0] * 32, by0 = V.cam_chunk[1] * 32, bz0 = V.cam_chunk[2] * 32;
  const float ox = V.o[0], oy = V.o[1], oz = V.o[2];
  const int sx = dx > 0.0f ? 1 : (dx < 0.0f ? -1 : 0);
  const int sy = dy > 0.0f ? 1 : (dy < 0.0f ? -1 : 0);
  const int sz = dz > 0.0f ? 1 : (dz < 0.0f ? -1 : 0);
  const float ix = sx ? __frcp_rn(dx) : 0.0f;
  const float iy = sy ? __frcp_rn(dy) : 0.0f;
  const float iz = sz ? __frcp_rn(dz) : 0.0f;
  // slab test against [-base, N - base)
  float tnear = -kInf, tfar = kInf;
  int ea = -1;
  {
    const float lo = __int2float_rn(-bx0), hi = __int2float_rn(V.nx - bx0);
    if (!sx) {
      if (ox < lo || ox >= hi) return;
    } else {
      const float inv = ix;
      const float t1 = __fmul_rn(__fsub_rn(lo, ox), inv), t2 = __fmul_rn(__fsub_rn(hi, ox), inv);
      const float tn = sx > 0 ? t1 : t2, tf = sx > 0 ? t2 : t1;
      if (tn > tnear) { tnear = tn; ea = 0; }
      if (tf < tfar) tfar = tf;
    }
  }
  {
    const float lo = __int2float_rn(-by0), hi = __int2float_rn(V.ny - by0);
    if (!sy) {
      if (oy < lo || oy >= hi) return;
    } else {
      const float inv = iy;
      const float t1 = __fmul_rn(__fsub_rn(lo, oy), inv), t2 = __fmul_rn(__fsub_rn(hi, oy), inv);
      const float tn = sy > 0 ? t1 : t2, tf = sy > 0 ? t2 : t1;
      if (tn > tnear) { tnear = tn; ea = 1; }
      if (tf < tfar) tfar = tf;
    }
  }
  {
    const float lo = __int2float_rn(-bz0), hi = __int2float_rn(V.nz - bz0);
    if (!sz) {
      if (oz < lo || oz >= hi) return;
    } else {
      const float inv = iz;
      const float t1 = __fmul_rn(__fsub_rn(lo, oz), inv), t2 = __fmul_rn(__fsub_rn(hi, oz), inv);
      const float tn = sz > 0 ? t1 : t2, tf = sz > 0 ? t2 : t1;
      if (tn > tnear) { tnear = tn; ea = 2; }
      if (tf < tfar) tfar = tf;
    }
  }
  if (!(tnear < tfar) || !(tfar > 0.0f)) return;
  int vx, vy, vz;
  float t0;
  if (tnear > 0.0f) {
    t0 = tnear;
    vx = ea == 0 ? (sx > 0 ? 0 : V.nx - 1)
                 : clampi((int)floorf(__fadd_rn(ox, __fmul_rn(dx, t0))) + bx0, 0, V.nx - 1);
    vy = ea == 1 ? (sy > 0 ? 0 : V.ny - 1)
                 : clampi((int)floorf(__fadd_rn(oy, __fmul_rn(dy, t0))) + by0, 0, V.ny - 1);
    vz = ea == 2 ? (sz > 0 ? 0 : V.nz - 1)
                 : clampi((int)floorf(__fadd_rn(oz, __fmul_rn(dz, t0))) + bz0, 0, V.nz - 1);
  } else {
    t0 = 0.0f;
    ea = -1;
    vx = clampi((int)floorf(ox) + bx0, 0, V.nx - 1);
    vy = clampi((int)floorf(oy) + by0, 0, V.ny - 1);
    vz = clampi((int)floorf(oz) + bz0, 0, V.nz - 1);
  }
  // pass 0 the primary ray, pass 1 the shadow ray of a hit: one copy of the
  // walk's code for both
  int base_x = bx0, base_y = by0, base_z = bz0;
  float rox = ox, roy = oy, roz = oz, rdx = dx, rdy = dy, rdz = dz, rix = ix, riy = iy, riz = iz;
#pragma unroll 1
  for (int pass = 0;; pass++) {
    Trav r;
    trace<kStats, kWalk>(V, V.margin, base_x, base_y, base_z, rox, roy, roz, rdx, rdy, rdz, rix, riy, riz, vx, vy, vz,
                          t0, ea, r);
    if (kStats) {
      st[0] += r.fetches;
      st[1] += r.bricks;
      st[3] += 1;
    }
    if (pass) {
      h.shadow = (uint8_t)(r.hit ? 1 : 0);
      h.shadow_steps = r.fine | (r.coarse << 16);
      return;
    }
    h.steps = r.fine | (r.coarse << 16);
    if (!r.hit) return;
    if (kStats) st[2] += 1;
    h.voxel = (uint64_t)r.vx + (uint64_t)V.nx * ((uint64_t)r.vy + (uint64_t)V.ny * (uint64_t)r.vz);
    h.t = r.t;
    h.material = __ldg(V.mat + (size_t)r.slot * 512 + (r.vx & 7) + 8 * (r.vy & 7) + 64 * (r.vz & 7));
    if (r.axis < 0) return;
    const float da = r.axis == 0 ? rdx : (r.axis == 1 ? rdy : rdz);
    const int sa = da > 0.0f ? 1 : (da < 0.0f ? -1 : 0);
    h.face = (uint8_t)(2 * r.axis + (sa > 0 ? 1 : 0));
    if (!P.shadow) return;
    // the shadow ray starts at the centre of the empty voxel across the face
    vx = r.vx - (r.axis == 0 ? sa : 0);
    vy = r.vy - (r.axis == 1 ? sa : 0);
    vz = r.vz - (r.axis == 2 ? sa : 0);
    if (((unsigned)vx >= (unsigned)V.nx) | ((unsigned)vy >= (unsigned)V.ny) | ((unsigned)vz >= (unsigned)V.nz)) {
      h.shadow = 0;
      return;
    }
    base_x = vx;
    base_y = vy;
    base_z = vz;
    rox = roy = roz = 0.5f;
    rdx = P.light[0];
    rdy = P.light[1];
    rdz = P.light[2];
    rix = P.inv_light[0];
    riy = P.inv_light[1];
    riz = P.inv_light[2];
    t0 = 0.0f;
    ea = -1;
  }
}

// kMode: kPlain; kStatsMode also accumulates {pointer fetches, occupied
// bricks entered, hits, rays} into P.stats; kHashMode also adds each view's
// order-sensitive hit checksum and its traced shadow rays into P.hash (the
// serving loop's per-request summary, so the hits need not be read again).
// Each is a separate instantiation; the timed path has none of it.
// At most 128 threads per CTA; 8 resident CTAs per SM cap registers at 64
// (1080p frame 149 us; 7 CTAs 154, 6 152, 9 with 56 registers 151).
// kViews: 1 = one view and 32 = up to 32 views as kernel parameters, 0 = a
// device table.  A block belongs to one view (a view's last block may have
// idle warps), so the descriptor's index depends on the block alone and its
// fields are read through the uniform path; one view's are operands in the
// parameter bank, with no load at all.
// kWalk: kByRegion where the region walk takes all views (single rays that it does
// not take step by the brick).  kBySteps where it takes none: views from beyond its
// coordinates (1080p view of the 1024^3 terrain from 140,000 voxels away: 342 us by
// the brick, 148 so) and of rough scenes (see set_rough), whose rays have no empty
// space to skip (256^3 random voxels, 25 % solid, 1280x720 with shadow rays: 75 us
// by region, 51 so).  kEither where the views or the shadow rays' light differ in
// this; an instantiation of its own, as a step over cubes out of line costs the
// region walk registers (256^2 view 30.7 us, and 31.4; 40 served requests 4.16 and
// 4.20 ms).
template <int kViews, int kMode, int kWalk>
__global__ void __launch_bounds__(128, 8)
    raymarch_kernel(const RayParams P, const __grid_constant__ Views<kViews ? kViews : 1> iv) {
  constexpr bool kStats = kMode == kStatsMode;
  const uint32_t warps = blockDim.x >> 5;
  const uint32_t bid = P.order_mul ? (blockIdx.x * P.order_mul) % gridDim.x : blockIdx.x;
  const RayView* views = kViews ? iv.v : P.table;
  uint32_t lo = 0;
  if constexpr (kViews != 1) {
    // view lookup: last view whose block_start <= bid
    uint32_t hi = P.n_views;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (views[mid].block_start <= bid) lo = mid;
      else hi = mid;
    }
  }
  const RayView& V = kViews == 1 ? iv.v[0] : views[lo];
  const uint32_t lb = bid - V.block_start;
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t tiles_x = (V.width + P.tile_w - 1u) >> P.tile_shift;
  const uint32_t tiles_y = (V.height + P.tile_h - 1u) >> (5u - P.tile_shift);
  const uint32_t blocks_x = (tiles_x + (1u << P.block_shift) - 1u) >> P.block_shift;
  const uint32_t by = lb / blocks_x, bx = lb - by * blocks_x;
  const uint32_t tx = (bx << P.block_shift) + (warp & ((1u << P.block_shift) - 1u));
  const uint32_t ty = by * (warps >> P.block_shift) + (warp >> P.block_shift);
  if (tx >= tiles_x || ty >= tiles_y) return;
  const int lane = threadIdx.x & 31;
  const uint32_t px0 = tx * P.tile_w, py0 = ty * P.tile_h;
  const uint32_t px = px0 + ((uint32_t)lane & (P.tile_w - 1u));
  const uint32_t py = py0 + ((uint32_t)lane >> P.tile_shift);
  uint32_t st[4] = {0, 0, 0, 0};
  // The tile's hit records (24 B each) are staged in shared memory and
  // written back as runs of consecutive 8-byte words, one run per tile row,
  // so every store instruction fills whole sectors (this matters most when
  // the output is page-locked host memory written over the CPU-GPU link).
  __shared__ __align__(16) uint64_t stage[4][96];
  uint64_t* sw = stage[threadIdx.x >> 5];
  if (px < V.width && py < V.height) {
    meso_hit h;
    trace_pixel<kStats, kWalk>(V, px, py, P, h, st);
    sw[3 * lane] = h.voxel;
    sw[3 * lane + 1] = (uint64_t)__float_as_uint(h.t) | (uint64_t)h.material << 32 | (uint64_t)h.face << 48 |
                       (uint64_t)h.shadow << 56;
    sw[3 * lane + 2] = (uint64_t)h.steps | (uint64_t)h.shadow_steps << 32;
  }
  __syncwarp();
  const uint32_t row_words = 3 * P.tile_w;
  uint64_t* base = reinterpret_cast<uint64_t*>(V.out);
  // Output in host memory, a CTA of four 8x4 tiles side by side, all inside
  // the image: after one barrier each warp writes one 32-pixel row of the
  // CTA (768 contiguous bytes, whole 128-byte lines when the row starts on
  // one), so no line crosses the CPU-GPU link in two pieces.  (Into device
  // memory the barrier costs more than it saves.)
  bool done = false;
  if (P.cta_rows && warps == 4 && P.tile_w == 8 && P.tile_h == 4 && (bx + 1) * 4 <= tiles_x) {
    const uint32_t x0 = px0 - 8u * (threadIdx.x >> 5);  // the CTA's first pixel column
    const bool ok = px0 + 8 <= V.width && py0 + 4 <= V.height &&
                    ((reinterpret_cast<uintptr_t>(base) + (((uint64_t)py0 * V.width + x0) * 24)) & 15u) == 0 &&
                    (V.width & 1u) == 0;
    if (__syncthreads_and(ok)) {
      const uint32_t row = threadIdx.x >> 5;
      uint4* dst = reinterpret_cast<uint4*>(base + ((uint64_t)(py0 + row) * V.width + x0) * 3);
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint32_t c = (uint32_t)lane + 32u * r;  // 16-byte chunk c of the row (48 in all)
        if (c < 48u) dst[c] = reinterpret_cast<const uint4*>(stage[c / 12u])[12u * row + c % 12u];
      }
      done = true;
    }
  }
  if (!done) {
    // a whole tile whose rows all start on 16 bytes goes out in 16-byte
    // stores, any other tile word by word
    const bool vec = ((reinterpret_cast<uintptr_t>(base) + (((uint64_t)py0 * V.width + px0) * 24)) & 15u) == 0 &&
                     (V.width & 1u) == 0 && (P.tile_w & 1u) == 0 && px0 + P.tile_w <= V.width &&
                     py0 + P.tile_h <= V.height;
    if (vec) {
      // the usual 8-pixel tile with its 12 chunks per row known at compile time
      const uint32_t row_vecs = row_words / 2;
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint32_t c = (uint32_t)lane + 32u * r;  // 16-byte chunk c of the tile (48 in all)
        if (c < 48u) {
          const uint32_t row = P.tile_w == 8 ? c / 12u : c / row_vecs, q = c - row * row_vecs;
          const uint4 v = reinterpret_cast<const uint4*>(sw)[c];
          reinterpret_cast<uint4*>(base + ((uint64_t)(py0 + row) * V.width + px0) * 3)[q] = v;
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < 3; r++) {
        const uint32_t c = (uint32_t)lane + 32u * r;  // word c of the tile: row c / row_words
        const uint32_t row = c / row_words, w = c % row_words;
        const uint32_t x = px0 + w / 3, y = py0 + row;
        if (x < V.width && y < V.height) base[((uint64_t)y * V.width + px0) * 3 + w] = sw[c];
      }
    }
  }
  if (kStats) {
    for (int k = 0; k < 4; k++) {
      const uint32_t tot = __reduce_add_sync(0xFFFFFFFFu, st[k]);
      if (lane == 0) atomicAdd(reinterpret_cast<unsigned long long*>(P.stats) + k, (unsigned long long)tot);
    }
  }
  if constexpr (kMode == kHashMode) {
    unsigned long long term = 0;
    uint32_t shadow = 0;
    if (px < V.width && py < V.height) {
      const uint64_t i = (uint64_t)py * V.width + px;
      const uint64_t w0 = sw[3 * lane], w1 = sw[3 * lane + 1], w2 = sw[3 * lane + 2];
      term = mix64(w0 ^ mix64(w1 ^ mix64(w2 ^ (i * 0x9E3779B97F4A7C15ull + 1ull))));
      shadow = (w2 >> 32) != 0;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) term += __shfl_down_sync(kFullMask, term, o);
    shadow = __reduce_add_sync(kFullMask, shadow);
    if (lane == 0) {
      const uint32_t slot = lo * kRayHashSlots + (bid & (kRayHashSlots - 1u));
      atomicAdd(P.hash + slot, term);
      if (shadow) atomicAdd(P.hash + kRayHashShadow + slot, (unsigned long long)shadow);
    }
  }
}

}  // namespace

size_t raymarch_view_table_bytes(uint32_t n_views) { return sizeof(RayView) * (size_t)n_views; }

// Into page-locked host memory the CTAs take their blocks in a strided order,
// b * 7919 mod blocks (a bijection unless blocks is a multiple of the prime
// 7919), so the cheap sky tiles and the expensive terrain tiles of a frame mix
// over the whole launch and the hit records leave at an even rate, which the
// CPU-GPU link needs (1080p end to end 0.48 -> 0.39 ms).  Into device memory
// they go in their own order: neighbouring blocks run at the same time and
// share what they fetch (1080p with shadow rays 149.5 us strided, 141.7 us in
// order; 40 served requests 4.53 and 4.45 ms).  Launches of 2^32 / 7919 blocks and
// more (69 Mpixel at 128 a block) keep their order, as the product must fit 32 bits:
// 16384x4864 takes 9.92 ms into host memory in either, the link's 193 GB/s.
static uint32_t block_order_mul(uint32_t blocks, bool host_out) {
  return host_out && blocks > 1 && blocks < 542000u && blocks % 7919u ? 7919u : 0u;
}

// A view's margin in the region walk: 2^-20 of the largest coordinate that its
// rays reach (twice the error bound derived at walk_regions), or 0 (every ray
// step by step) outside what that bound was derived for: coordinates beyond
// 2^17 voxels, an origin that is not finite.
static float region_margin(const meso_scene* s, const meso_camera& c) {
  const int32_t n[3] = {s->nx, s->ny, s->nz};
  float R = 0.0f;
  for (int a = 0; a < 3; a++) {
    const float r = 32.0f * fabsf((float)c.origin_chunk[a]) + (float)n[a] + fabsf(c.origin_frac[a]) + 64.0f;
    if (!(r < 131072.0f)) return 0.0f;
    R = r > R ? r : R;
  }
  return R * 4.76837158203125e-7f;
}

// Tiles of a block side by side, as a power of two: two by two for four warps
// (the block's rays stay in a squarer patch of the scene and share more of its
// lines in L1: 1080p 155.6 -> 151.3 us, 40 served requests 4.85 -> 4.59 ms);
// four in a row where whole rows of the block are written at once (host output).
static uint32_t block_tiles_shift(uint32_t wpc, bool rows) { return wpc == 4 ? (rows ? 2u : 1u) : (wpc == 2 ? 1u : 0u); }

// Running totals over the views of a launch.
struct ViewTotals {
  uint64_t tiles = 0, blocks = 0, hits = 0;
  uint32_t stepped = 0;  // views that the region walk does not take
};

// Fills the host descriptors out[0 .. n) of views scenes/cams[0 .. n) for
// blocks of wpc warps, after those that the totals count already.
static void fill_views(const meso_scene* const* scenes, const meso_camera* cams, uint32_t n, uint32_t tw, uint32_t th,
                       uint32_t wpc, uint32_t bsh, meso_hit* d_hits, meso_hit* const* view_out, RayView* out,
                       ViewTotals& tot) {
  for (uint32_t v = 0; v < n; v++) {
    const meso_scene* s = scenes[v];
    const meso_camera& c = cams[v];
    RayView& V = out[v];
    memset(&V, 0, sizeof(V));
    V.ptr = s->d_ptr;
    V.level = s->d_level;
    V.bounds = reinterpret_cast<const int4*>(s->d_bounds);
    V.sub = s->d_sub;
    V.occ = s->d_occ;
    V.mat = s->d_mat;
    V.nx = s->nx;
    V.ny = s->ny;
    V.nz = s->nz;
    for (int a = 0; a < 3; a++) {
      V.cam_chunk[a] = c.origin_chunk[a];
      V.o[a] = c.origin_frac[a];
      V.fwd[a] = c.forward[a];
      V.right[a] = c.right[a];
      V.up[a] = c.up[a];
    }
    V.tan_half = c.tan_half_fov_y;
    V.aspect = (float)c.width / (float)c.height;  // IEEE conversions and division, as on the device
    V.width = c.width;
    V.height = c.height;
    V.margin = s->rough ? 0.0f : region_margin(s, c);
    if (!regular_axis(c.forward[0]) || !regular_axis(c.forward[1]) || !regular_axis(c.forward[2])) V.margin = 0.0f;
    tot.stepped += V.margin == 0.0f;
    V.block_start = (uint32_t)tot.blocks;
    V.out = view_out && view_out[v] ? view_out[v] : d_hits + tot.hits;
    const uint32_t tiles_x = (c.width + tw - 1) / tw, tiles_y = (c.height + th - 1) / th;
    const uint32_t bw = 1u << bsh, bh = wpc >> bsh;
    tot.tiles += (uint64_t)tiles_x * tiles_y;
    tot.blocks += (uint64_t)((tiles_x + bw - 1) / bw) * ((tiles_y + bh - 1) / bh);
    tot.hits += (uint64_t)c.width * c.height;
  }
}

}  // namespace meso

namespace meso {
namespace {

// Descriptors of up to kFillViews views, passed by value to the kernel that
// writes them into a device view table.  Kernel parameters are copied when
// the launch is issued (and kept by value in a captured graph node), so no
// host buffer has to outlive the call; 64 views are 9.5 KiB of parameters
// and of the caller's stack.
constexpr uint32_t kFillViews = 64;
struct ViewBatch {
  RayView v[kFillViews];
};
static_assert(sizeof(ViewBatch) <= 32000, "a view batch must fit the kernel parameter space");

__global__ void view_fill_kernel(const __grid_constant__ ViewBatch b, uint32_t n, RayView* dst) {
  const uint32_t words = n * (uint32_t)(sizeof(RayView) / 8);
  const uint64_t* src = reinterpret_cast<const uint64_t*>(b.v);
  uint64_t* d = reinterpret_cast<uint64_t*>(dst);
  for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) d[i] = src[i];
}

}  // namespace

// Writes the descriptors of n_views views into the device table d_table,
// stream-ordered before the launch that reads it: one small kernel per 64
// views, the descriptors travelling as its parameters.
static meso_status stage_view_table(const meso_scene* const* scenes, const meso_camera* cams, uint32_t n_views,
                                    uint32_t tw, uint32_t th, uint32_t wpc, uint32_t bsh,
                                    meso_hit* d_hits, meso_hit* const* view_out, RayView* d_table, cudaStream_t st, ViewTotals& tot) {
  ViewBatch batch;
  for (uint32_t v0 = 0; v0 < n_views; v0 += kFillViews) {
    const uint32_t n = n_views - v0 < kFillViews ? n_views - v0 : kFillViews;
    fill_views(scenes + v0, cams + v0, n, tw, th, wpc, bsh, d_hits, view_out ? view_out + v0 : nullptr, batch.v, tot);
    view_fill_kernel<<<1, 128, 0, st>>>(batch, n, d_table + v0);
    MESO_CUDA_TRY(cudaGetLastError());
  }
  return MESO_OK;
}

// Launches one mode's kernel over the totals' blocks.
template <int kViews, int kWalk>
static void launch_walk(const RayParams& P, const Views<kViews ? kViews : 1>& iv, uint32_t blocks, uint32_t wpc,
                        cudaStream_t st) {
  if (P.hash) raymarch_kernel<kViews, kHashMode, kWalk><<<blocks, wpc * 32, 0, st>>>(P, iv);
  else raymarch_kernel<kViews, kPlain, kWalk><<<blocks, wpc * 32, 0, st>>>(P, iv);
}
template <int kViews>
static void launch_mode(const RayParams& P, const Views<kViews ? kViews : 1>& iv, const ViewTotals& tot, uint32_t wpc,
                        cudaStream_t st) {
  const uint32_t blocks = (uint32_t)tot.blocks;
  const float* L = P.light;
  const bool light = regular_axis(L[0]) && regular_axis(L[1]) && regular_axis(L[2]) && (L[0] != 0.0f || L[1] != 0.0f || L[2] != 0.0f);
  if (P.stats) raymarch_kernel<kViews, kStatsMode, kByRegion><<<blocks, wpc * 32, 0, st>>>(P, iv);
  else if (tot.stepped == P.n_views) launch_walk<kViews, kBySteps>(P, iv, blocks, wpc, st);
  else if (tot.stepped || (P.shadow && !light)) launch_walk<kViews, kEither>(P, iv, blocks, wpc, st);
  else launch_walk<kViews, kByRegion>(P, iv, blocks, wpc, st);
}

meso_status launch_raymarch(meso_ctx* ctx, const meso_scene* const* scenes, const meso_camera* cams,
                            uint32_t n_views, const float light[3], uint32_t flags, meso_hit* d_hits,
                            cudaStream_t st, void* d_view_table, size_t view_table_bytes, uint64_t* d_stats,
                            meso_hit* const* view_out, unsigned long long* d_hash, bool host_out) {
  if (!scenes || !cams || !d_hits) return fail(MESO_ERR_INVALID_ARG, "raymarch: null argument");
  if (n_views == 0) return MESO_OK;
  for (uint32_t v = 0; v < n_views; v++) {
    if (!scenes[v]) return fail(MESO_ERR_INVALID_ARG, "raymarch: null scene");
    if (cams[v].width == 0 || cams[v].height == 0 || cams[v].width > 16384 || cams[v].height > 16384)
      return fail(MESO_ERR_INVALID_ARG, "raymarch: image size out of range");
    if (view_out && (reinterpret_cast<uintptr_t>(view_out[v]) & 7u))
      return fail(MESO_ERR_INVALID_ARG, "raymarch: view output not 8-byte aligned");
  }
  if (d_hash && (d_stats || n_views > kRayHashViews))
    return fail(MESO_ERR_INVALID_ARG, "raymarch: checksums need at most 64 views and no statistics");
  if ((flags & MESO_RAY_SHADOW) && !light) return fail(MESO_ERR_INVALID_ARG, "raymarch: shadow without light");
  const uint32_t tw = ctx->tuning.ray_tile_w ? ctx->tuning.ray_tile_w : 8;
  if (32 % tw) return fail(MESO_ERR_INVALID_ARG, "raymarch: tile width must divide 32");
  const uint32_t th = 32 / tw;
  const uint32_t wpc = ctx->tuning.ray_warps_per_cta ? ctx->tuning.ray_warps_per_cta : 4;
  RayParams P;
  memset(&P, 0, sizeof(P));
  P.n_views = n_views;
  P.tile_w = tw;
  P.tile_h = th;
  P.tile_shift = (uint32_t)__builtin_ctz(tw);
  P.block_shift = block_tiles_shift(wpc, host_out);
  P.shadow = (flags & MESO_RAY_SHADOW) ? 1u : 0u;
  if (light)
    for (int a = 0; a < 3; a++) {
      P.light[a] = light[a];
      P.inv_light[a] = light[a] != 0.0f ? 1.0f / light[a] : 0.0f;  // IEEE division, as __fdiv_rn
    }
  P.stats = d_stats;
  P.hash = d_hash;
  P.cta_rows = host_out ? 1u : 0u;
  ViewTotals tot;
  if (n_views <= (uint32_t)kInlineViews) {
    Views<kInlineViews> iv;
    fill_views(scenes, cams, n_views, tw, th, wpc, P.block_shift, d_hits, view_out, iv.v, tot);
    if (tot.tiles >= (1ull << 31)) return fail(MESO_ERR_INVALID_ARG, "raymarch: too many tiles");
    P.order_mul = block_order_mul((uint32_t)tot.blocks, P.cta_rows != 0);
    if (n_views == 1) {
      Views<1> one;
      one.v[0] = iv.v[0];
      launch_mode<1>(P, one, tot, wpc, st);
    } else {
      launch_mode<kInlineViews>(P, iv, tot, wpc, st);
    }
  } else {
    if (!d_view_table || view_table_bytes < raymarch_view_table_bytes(n_views))
      return fail(MESO_ERR_INVALID_ARG, "raymarch: view table too small");
    MESO_TRY(stage_view_table(scenes, cams, n_views, tw, th, wpc, P.block_shift, d_hits, view_out,
                              static_cast<RayView*>(d_view_table), st, tot));
    if (tot.tiles >= (1ull << 31)) return fail(MESO_ERR_INVALID_ARG, "raymarch: too many tiles");
    P.table = static_cast<const RayView*>(d_view_table);
    P.order_mul = block_order_mul((uint32_t)tot.blocks, P.cta_rows != 0);
    static Views<1> unused;  // zero-initialised; the table path does not read it
    launch_mode<0>(P, unused, tot, wpc, st);
  }
  ctx->launches.fetch_add(1);
  MESO_CUDA_TRY(cudaGetLastError());
  return MESO_OK;
}

}  // namespace meso

// ---------------------------------------------------------------------------
// Multi-view raymarch that allocates nothing.
//
// meso_raymarch stages the descriptor table of more than 32 views in device
// memory it allocates per call.  Some callers cannot allocate device memory
// at that point: a frame loop running on a fixed device-memory budget that
// must not allocate mid-frame (an allocation can synchronise the device and
// stall the frame), or a host application whose own memory manager owns all
// device memory.  This entry point keeps the table in a fixed file-scope
// device array instead; the descriptors reach it as kernel parameters, 64
// views at a time, through a 9.5 KiB batch on the caller's stack.
//
// Limits and behaviour:
//  - at most kNoAllocViews (512) views per call; more is rejected with
//    MESO_ERR_INVALID_ARG;
//  - the array (512 x 152 B = 76 KiB) stays resident on every device that
//    loads the library until the process exits;
//  - the calling thread's current device must be the context's device;
//  - the first call on a device looks up the array's device address (with
//    that device current) and caches it; make that first call before any
//    stream capture;
//  - every call reuses the same array and overwrites the entries it uses, so
//    calls whose kernels overlap on the GPU race on it: issue them on one
//    stream, or order them with events.
namespace meso {
namespace {

constexpr uint32_t kNoAllocViews = 512;
static_assert(sizeof(RayView) == 152, "the documented size of the fixed view table is 512 x 152 bytes");
static __device__ __align__(256) unsigned char g_noalloc_views[kNoAllocViews * sizeof(RayView)];

std::mutex g_noalloc_mu;
void* g_noalloc_ptr[64] = {};

// Device address of g_noalloc_views on `device` (looked up once per device;
// `device` is current when this is called).
meso_status noalloc_table(int device, void** out) {
  if (device < 0 || device >= 64) return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: device ordinal >= 64");
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[device]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_views);
    if (e != cudaSuccess) return cuda_fail(e, "raymarch_noalloc: cudaGetSymbolAddress");
    g_noalloc_ptr[device] = p;
  }
  *out = g_noalloc_ptr[device];
  return MESO_OK;
}

}  // namespace
}  // namespace meso

extern "C" meso_status meso_raymarch_noalloc(meso_ctx* ctx, const meso_scene* const* scenes,
                                             const meso_camera* h_cams, uint32_t n_views, const float light[3],
                                             uint32_t flags, meso_hit* d_hits, void* stream) {
  using namespace meso;
  if (!ctx || !scenes || !h_cams || !d_hits) return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: null argument");
  if (n_views > kNoAllocViews)
    return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: at most 512 views per call (fixed device view table)");
  if (n_views == 0) return MESO_OK;
  for (uint32_t v = 0; v < n_views; v++) {
    if (!scenes[v]) return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: null scene");
    if (h_cams[v].width == 0 || h_cams[v].height == 0 || h_cams[v].width > 16384 || h_cams[v].height > 16384)
      return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: image size out of range");
  }
  if ((flags & MESO_RAY_SHADOW) && !light) return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: shadow without light");
  const uint32_t tw = ctx->tuning.ray_tile_w ? ctx->tuning.ray_tile_w : 8;
  if (32 % tw) return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: tile width must divide 32");
  const uint32_t th = 32 / tw;
  const uint32_t wpc = ctx->tuning.ray_warps_per_cta ? ctx->tuning.ray_warps_per_cta : 4;
  int cur = -1;
  MESO_CUDA_TRY(cudaGetDevice(&cur));
  if (cur != ctx->device)
    return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: the current device is not the context's device");
  void* table = nullptr;
  MESO_TRY(noalloc_table(ctx->device, &table));
  // the same validation as meso_raymarch, before any work is issued
  uint64_t tiles = 0;
  for (uint32_t v = 0; v < n_views; v++)
    tiles += (uint64_t)((h_cams[v].width + tw - 1) / tw) * ((h_cams[v].height + th - 1) / th);
  if (tiles >= (1ull << 31)) return fail(MESO_ERR_INVALID_ARG, "raymarch_noalloc: too many tiles");
  RayParams P;
  memset(&P, 0, sizeof(P));
  P.table = static_cast<const RayView*>(table);
  P.n_views = n_views;
  P.tile_w = tw;
  P.tile_h = th;
  P.tile_shift = (uint32_t)__builtin_ctz(tw);
  P.block_shift = block_tiles_shift(wpc, false);
  P.shadow = (flags & MESO_RAY_SHADOW) ? 1u : 0u;
  if (light)
    for (int a = 0; a < 3; a++) {
      P.light[a] = light[a];
      P.inv_light[a] = light[a] != 0.0f ? 1.0f / light[a] : 0.0f;  // IEEE division, as __fdiv_rn
    }
  const cudaStream_t st = pick_stream(ctx, stream);
  ViewTotals tot;
  MESO_TRY(stage_view_table(scenes, h_cams, n_views, tw, th, wpc, P.block_shift, d_hits, nullptr,
                            static_cast<RayView*>(table), st, tot));
  P.order_mul = block_order_mul((uint32_t)tot.blocks, P.cta_rows != 0);
  static Views<1> unused;  // zero-initialised; the table path does not read it
  launch_mode<0>(P, unused, tot, wpc, st);
  ctx->launches.fetch_add(1);
  MESO_CUDA_TRY(cudaGetLastError());
  return MESO_OK;
}
