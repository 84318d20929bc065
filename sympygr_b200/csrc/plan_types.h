// Work-plan descriptors shared by the host planner and the kernels.
//
// A plan covers a list of octree blocks.  Each block's interior (sz-6)^3 is cut into
// z-slabs and each slab into column tiles of at most 16x8 points (cut_start).  The slabs are
// packed into chunks whose points fit the derivative scratch; each chunk is evaluated by
// derivative launches (one CTA per tile and variable, streaming along z) followed by one
// algebra launch (runs of points along the block's rows).
//
// Scratch points.  Every tile owns 128 scratch points per plane, planes one after another;
// row y of the tile sits at row_off(y), 16 points.  So a store of the derivative stage fills
// whole 32-byte sectors, and a 32-point block of the scratch (scr_index) belongs to one tile.
// That matters more than the padding it costs: with points numbered densely over the slab,
// rows of different tiles shared sectors, and the stores -- not the arithmetic, nor the
// bytes -- set the derivative stage's time.  On 16 blocks of 69^3 (4.0 M points) the stage
// took 1.43 ms (MIXED) and 2.00 ms (FP64), 0.67 and 0.72 ms with its stores switched off;
// with whole sectors, and the rest of the rewrite, 0.83 and 1.14 ms.
//
// The algebra takes 32 points at a time along the block's rows (slab_point): two neighbouring
// tiles' parts of a row, and, where a row has an odd number of tiles, its last part together
// with those of the next rows.  Its accesses to the state and the right-hand side are then
// runs of up to 32 points, and no two warps share a sector of the scratch.  (Groups of four
// points taken densely along the rows instead left fewer lanes idle, but on 135^3 blocks,
// whose rows of 129 points then straddle the tiles or leave a group of one point, the algebra
// took 1.64 instead of 1.38 ms, MIXED, and 2.69 instead of 2.38 ms, FP64, on 6.4 M points.
// Two rows of one tile, whose 32 points are one block of the scratch: 1.52 and 2.46 ms.)
#pragma once
#include <stdint.h>

namespace b200bssn {

constexpr int kNumVars = 24;
constexpr int kNumDerivs = 138;  // algebra inputs: 72 first + 66 second derivatives
constexpr int kTileX = 16, kTileY = 8;
constexpr int kTilePlane = kTileX * kTileY;  // scratch points of a tile per plane
constexpr int kHalo = 3;         // staged points beyond a tile or slab on each side
constexpr int kGroup = 4;        // points that never lie in different tiles or rows: lanes 4g .. 4g+3 of a task
constexpr int kAlgebraThreads = 128;
constexpr int kRangeTasks = kAlgebraThreads / 32;

// Cuts of `n` interior points (7 or more) of one axis into pieces of `size` (a multiple of
// four, 8 or more): all full but the last -- and, where that would hold fewer than three
// points, the last but one, which hands it four.  The three points next to a flagged face
// then always share a piece, and their closure rows reach no further than three points
// beyond it.
__host__ __device__ inline int num_cuts(int n, int size) { return (n + size - 1) / size; }
__host__ __device__ inline int cut_start(int n, int size, int k) {
  const int last = num_cuts(n, size) - 1, rest = n - last * size;
  if (k > last) return n;
  return k * size - (k == last && last > 0 && rest < 3 ? 4 : 0);
}
// the piece that holds point `pos`
__host__ __device__ inline int cut_of(int n, int size, int pos) {
  const int last = num_cuts(n, size) - 1, k = pos / size;
  return k + 1 == last && pos >= cut_start(n, size, last) ? last : k;
}
// Scratch offset of row y of a tile within its plane: rows y and y + 2 share a 32-point
// block, so that the derivative stage's stores, two rows apart in a warp, fill it.
__host__ __device__ inline int row_off(int y) { return ((y & 1) << 5) | ((y & 2) << 3) | ((y & 4) << 4); }

struct BlockDev {
  uint64_t offset;   // element offset in every variable array
  int32_t sz[3];
  uint32_t bflag;
  double pmin[3];    // ghost-inclusive corner
  double h[3];       // (pmax - pmin)/(sz - 1), computed on the host as bssnrhs does
};

struct SlabDev {
  int32_t block;
  int32_t k0, nz;     // first interior plane (0-based interior index), planes
  int32_t sbase;      // first scratch point of the slab within its chunk (a multiple of 128)
  // a strip of the planes' rows (whole tiles) where the planes are too large for the scratch:
  // first row, and how many of the block's rows it leaves out
  int32_t j0 = 0, jcut = 0;
};
// tile rows of a slab: the first one's number in the block, and how many
__host__ __device__ inline int first_cut(const SlabDev& s) { return (s.j0 + kTileY / 2) / kTileY; }
__host__ __device__ inline int cut_rows(int n, const SlabDev& s) {
  return cut_of(n, kTileY, s.j0 + n - s.jcut - 1) - first_cut(s) + 1;
}

// A column tile of a slab.
struct TileDev {
  int32_t block;
  int32_t sbase;      // first scratch point of the tile within its chunk
  int32_t k0, nz;     // of its slab
  int16_t i0, j0;     // interior-relative origin of the x-y tile
  int16_t ex, ey;     // extents (<= kTileX, kTileY)
};

// Padded block coordinates of an interior point, and its scratch point; `valid` is false for
// lanes that pad a task (their scratch points lie in the tile's padding or on another row).
struct SlabPoint {
  int i, j, k, lp;
  bool valid;
};
// How the rows of a slab of block B are cut into tasks: `tiles` parts per row, in pairs; with
// an odd number of tiles the last parts (`lanes` lanes each) of `rows` rows share a task, which
// follows the rows' other tasks, so that the sectors of the state and of the right-hand side
// that it shares with them are still in L2.
struct RowTasks {
  int tiles, pairs, lanes, rows, tasks;  // tasks per `rows` rows
};
__host__ __device__ inline RowTasks row_tasks(int I0) {
  const int tiles = num_cuts(I0, kTileX), pairs = tiles / 2;
  if (tiles % 2 == 0) return {tiles, pairs, 0, 1, pairs};
  const int lanes = (I0 - cut_start(I0, kTileX, tiles - 1) + kGroup - 1) / kGroup * kGroup, rows = 32 / lanes;
  return {tiles, pairs, lanes, rows, rows * pairs + 1};
}
// Tasks of a slab of nz planes of block B that leaves out jcut of its rows.
__host__ __device__ inline int64_t slab_tasks(const BlockDev& B, int nz, int jcut = 0) {
  const RowTasks t = row_tasks(B.sz[0] - 6);
  return ((int64_t)(B.sz[1] - 6 - jcut) * nz + t.rows - 1) / t.rows * t.tasks;
}
// The point of lane `lane` of a task of slab s.
__host__ __device__ inline SlabPoint slab_point(const BlockDev& B, const SlabDev& s, int task, int lane) {
  const int I0 = B.sz[0] - 6, I1 = B.sz[1] - 6, J = I1 - s.jcut, rows = J * s.nz;
  const RowTasks t = row_tasks(I0);
  const int set = task / t.tasks, k = task - set * t.tasks;
  int r = set * t.rows, cx, x;  // row, its tile, point in the tile
  if (k < t.rows * t.pairs) {
    const int q = k / t.pairs;
    r += q;
    cx = 2 * (k - q * t.pairs) + lane / kTileX;
    x = lane % kTileX;
  } else {
    const int q = lane / t.lanes;
    r = q < t.rows ? r + q : rows;
    cx = t.tiles - 1;
    x = lane - q * t.lanes;
  }
  const int x0 = cut_start(I0, kTileX, cx);
  const bool valid = r < rows && x0 + x < cut_start(I0, kTileX, cx + 1);
  r = r < rows ? r : rows - 1;
  const int z = r / J, y = s.j0 + r - z * J, cy = cut_of(I1, kTileY, y);
  return {3 + x0 + x, 3 + y, 3 + s.k0 + z,
          s.sbase + (((cy - first_cut(s)) * t.tiles + cx) * s.nz + z) * kTilePlane + row_off(y - cut_start(I1, kTileY, cy)) + x, valid};
}

// Which closure rows a tile's output points take: those within three points of a flagged face.
enum TileClosure : int { kClosureNone = 0, kClosureZ = 1, kClosureXY = 2 };  // none; along z only; along x or y
__host__ __device__ inline bool near_face(int p0, int e, int n, bool lo, bool hi) {
  return (lo && p0 < 6) || (hi && p0 + e - 1 >= n - 6);
}
__host__ __device__ inline TileClosure tile_closure(const BlockDev& B, const TileDev& t) {
  const uint32_t bf = B.bflag;
  if (near_face(3 + t.i0, t.ex, B.sz[0], bf & 1u, bf & 2u) || near_face(3 + t.j0, t.ey, B.sz[1], bf & 4u, bf & 8u))
    return kClosureXY;
  return near_face(3 + t.k0, t.nz, B.sz[2], bf & 16u, bf & 32u) ? kClosureZ : kClosureNone;
}

// One tile-slab of the one-pass kernel: a 16x8 column tile of a block over a z-slab
// of at most kFusedSlab interior planes.
struct FusedTileDev {
  int32_t block;
  int16_t i0, j0;     // interior-relative x-y origin of the tile
  int16_t ex, ey;     // extents (<= kTileX, kTileY)
  int16_t k0, nz;     // interior-relative first plane and planes (<= kFusedSlab)
  int32_t pad;
};
constexpr int kFusedSlab = 24;                               // max interior planes per tile-slab
constexpr int kFusedSlotPts = kTileX * kTileY * kFusedSlab;  // 3072 points per ring slot
constexpr int kFusedRingDefault = 128;                       // slots: 256 MB in MIXED

// A run of consecutive tasks of a slab: the points of one CTA of kAlgebraThreads.
struct RangeDev {
  int32_t slab;
  int32_t start;     // first task
  int32_t count;     // tasks, <= kRangeTasks
};

// Classic RK4 stage update fused into the algebra kernel's epilogue.  With k the
// right-hand side at a point (in FP64, KO included) and u^n the state at the start
// of the step:
//   RK_FIRST   acc  = w k          next = u^n + c k      (stage 1)
//   RK_MIDDLE  acc += w k          next = u^n + c k      (stages 2, 3)
//   RK_LAST    u^n  = u^n + acc + w k                     (stage 4)
// with w = dt/6, dt/3, dt/3, dt/6 and c = dt/2, dt/2, dt.  Every array is read and
// written at the thread's own point only, so the kernel's inputs (the stage state
// `u`, read at the point and by the derivative kernel) never alias its outputs.
enum RkMode : int32_t { RK_NONE = 0, RK_FIRST = 1, RK_MIDDLE = 2, RK_LAST = 3 };

struct RkStage {
  int32_t mode;
  double w, c;
  double* acc[kNumVars];
  double* next[kNumVars];
  double* base[kNumVars];  // u^n: read in every stage, written in RK_LAST
};

// Scratch slots of a point: the 138 derivatives, the 24 KO sums, then in the upwind mode the
// 72 advective derivatives.
constexpr int kKoSlot = kNumDerivs;                        // KO sum of variable v: kKoSlot + v
constexpr int kAdvSlot = kNumDerivs + kNumVars;            // advective derivative 3v + axis: kAdvSlot + 3v + axis
__host__ __device__ constexpr int num_slots(bool adv) { return kAdvSlot + (adv ? 3 * kNumVars : 0); }

// Scratch layout: blocks of 32 scratch points
// (chunk-relative index lp), each block holding its NS slots one after another --
// value (slot s, point lp) at ((lp / 32) * NS + s) * 32 + lp % 32.  A 32-point task
// of the algebra kernel then reads one contiguous run of NS * 32 values instead of
// NS columns far apart (a copy of that shape reaches the full HBM read rate; 138
// scattered 128-byte pieces per task reach about two thirds of it).
template <int NS>
__device__ __forceinline__ int scr_index(int s, int lp) {
  return ((lp >> 5) * NS + s) * 32 + (lp & 31);
}
__device__ __forceinline__ int scr_index(int ns, int s, int lp) {
  return ((lp >> 5) * ns + s) * 32 + (lp & 31);
}

}  // namespace b200bssn
