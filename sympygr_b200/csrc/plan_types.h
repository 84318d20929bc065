// Work-plan descriptors shared by the host planner and the kernels.
//
// A plan covers a list of octree blocks.  Each block's interior (sz-6)^3 is cut into
// z-slabs and each slab into column tiles of at most 16x8 points (cut_start).  The slabs are
// packed into chunks whose points fit the derivative scratch; each chunk is evaluated by
// derivative launches (one CTA per tile and variable, streaming along z) followed by one
// algebra launch (runs of points along the block's rows).
//
// Scratch points.  Every tile owns 128 scratch points per plane, planes one after another;
// row y of the tile sits at row_off(y), 16 points (narrow tiles: see kNarrow).  So a store of
// the derivative stage fills whole 32-byte sectors, and a 32-point block of the scratch
// (scr_index) belongs to one tile.
// That matters more than the padding it costs: with points numbered densely over the slab,
// rows of different tiles shared sectors, and the stores -- not the arithmetic, nor the
// bytes -- set the derivative stage's time.  On 16 blocks of 69^3 (4.0 M points) the stage
// took 1.43 ms (MIXED) and 2.00 ms (FP64), 0.67 and 0.72 ms with its stores switched off;
// with whole sectors, and the rest of the rewrite, 0.83 and 1.14 ms.
//
// The algebra takes 32 points at a time along the block's rows (slab_point): two neighbouring
// tiles' parts of a row, and tiles left over together with those of the next rows (RowTasks).
// Its accesses to the state and the right-hand side are then runs of up to 32 points, and no two
// warps share a sector of the scratch.  (Groups of four points taken densely along the rows
// instead left fewer lanes idle, but on 135^3 blocks, whose rows of 129 points then straddle the
// tiles or leave a group of one point, the algebra took 1.64 instead of 1.38 ms, MIXED, and 2.69
// instead of 2.38 ms, FP64, on 6.4 M points.
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
// Narrow tiles, of at most kNarrow columns (the last of a row can be that narrow), have rows of
// kNarrow points, in the first half of the planes' points, the even rows before the odd ones:
// with rows of 16, half of each 128-byte line would be unused, and memory is read by such lines.
// (4373 blocks of 13^3, 1.5 M points, whose only tiles are 7 wide: the algebra takes 0.89 instead
// of 1.25 ms in FP64, 0.56 instead of 0.74 ms in MIXED.  Parts of 8 and 4 columns for tiles of
// 9 to 12 as well scattered a task's rows over more lines: 15^3 blocks took 24 % longer.)
constexpr int kNarrow = 8;
// Scratch offset of point (x, y) of a tile within its plane: row_off(y) + x, or the same with
// narrow rows.
__host__ __device__ inline int point_off(bool narrow, int x, int y) {
  return ((y & 1) << 5) + (y >> 1 & 1) * (narrow ? kNarrow : kTileX) + (y >> 2) * (narrow ? 2 * kNarrow : 4 * kTileX) + x;
}

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
  int32_t narrow = 0; // its last column of tiles is narrow
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
// How the rows of a slab are cut into tasks, in sets of kTaskRows rows: `pairs` pairs of tiles
// per row; then the tiles left over, one column of them after the other -- the last, where the
// row has an odd number of tiles or the last is narrow, and in the latter case of an even number
// the last but one --, `lanes` lanes (0: no such column) to a row and 2^shift rows to a task.
// They follow the set's pairs, so that the sectors of the state and of the right-hand side that
// they share with them are still in L2.  (A narrow tile paired with the one before left up to 15
// of 32 lanes idle: 257 blocks of 24^3, rows of 12 + 6, FP64: algebra 0.88 ms, now 0.77.)
constexpr int kTaskRows = 8;
struct ColumnTasks {
  int lanes, shift;
};
__host__ __device__ inline ColumnTasks column(int ex) {
  const int lanes = (ex + kGroup - 1) / kGroup * kGroup;
  return {lanes, lanes <= 4 ? 3 : (lanes <= 8 ? 2 : 1)};
}
struct RowTasks {
  int tiles, pairs;
  ColumnTasks c0, c1;  // of the last tile but one, of the last one
};
__host__ __device__ inline RowTasks row_tasks(int I0) {
  const int tiles = num_cuts(I0, kTileX), last = cut_start(I0, kTileX, tiles - 1);
  if (tiles % 2) return {tiles, tiles / 2, {0, 0}, column(I0 - last)};
  if (I0 - last > kNarrow) return {tiles, tiles / 2, {0, 0}, {0, 0}};
  return {tiles, tiles / 2 - 1, column(last - cut_start(I0, kTileX, tiles - 2)), column(I0 - last)};
}
// tasks of `rows` rows of a left-over column, and of `rows` rows of a set
__host__ __device__ inline int column_tasks(const ColumnTasks& c, int rows) {
  return c.lanes ? (rows + (1 << c.shift) - 1) >> c.shift : 0;
}
__host__ __device__ inline int set_tasks(const RowTasks& t, int rows) {
  return rows * t.pairs + column_tasks(t.c0, rows) + column_tasks(t.c1, rows);
}
// Tasks of a slab of nz planes of block B that leaves out jcut of its rows.
__host__ __device__ inline int64_t slab_tasks(const BlockDev& B, int nz, int jcut = 0) {
  const RowTasks t = row_tasks(B.sz[0] - 6);
  const int64_t rows = (int64_t)(B.sz[1] - 6 - jcut) * nz;
  return rows / kTaskRows * set_tasks(t, kTaskRows) + set_tasks(t, (int)(rows % kTaskRows));
}
// The point of lane `lane` of a task of slab s.
__host__ __device__ inline SlabPoint slab_point(const BlockDev& B, const SlabDev& s, int task, int lane) {
  const int I0 = B.sz[0] - 6, I1 = B.sz[1] - 6, J = I1 - s.jcut;
  const RowTasks t = row_tasks(I0);
  const int per_set = set_tasks(t, kTaskRows), set = task / per_set, r0 = set * kTaskRows;
  const int rows = J * s.nz - r0 < kTaskRows ? J * s.nz - r0 : kTaskRows;  // of this set
  int k = task - set * per_set, q, cx, x;  // row of the set, its tile, point in the tile
  bool valid = true;
  if (k < rows * t.pairs) {
    q = k / t.pairs;
    cx = 2 * (k - q * t.pairs) + lane / kTileX;
    x = lane % kTileX;
  } else {
    k -= rows * t.pairs;
    const int first = column_tasks(t.c0, rows);
    const bool last = k >= first;
    const ColumnTasks c = last ? t.c1 : t.c0;
    const int p = c.lanes == 12 ? (lane >= 12 ? 1 : 0) + (lane >= 24 ? 1 : 0) : lane >> (5 - c.shift);  // lane / lanes
    valid = p >> c.shift == 0;
    q = ((last ? k - first : k) << c.shift) + (valid ? p : 0);
    cx = t.tiles - (last ? 1 : 2);
    x = lane - p * c.lanes;
  }
  valid = valid && q < rows;
  const int x0 = cut_start(I0, kTileX, cx), ex = cut_start(I0, kTileX, cx + 1) - x0;
  const int r = r0 + (q < rows ? q : rows - 1), z = r / J, y = s.j0 + r - z * J, cy = cut_of(I1, kTileY, y);
  return {3 + x0 + x, 3 + y, 3 + s.k0 + z,
          s.sbase + (((cy - first_cut(s)) * t.tiles + cx) * s.nz + z) * kTilePlane +
              point_off(s.narrow && cx == t.tiles - 1, x, y - cut_start(I1, kTileY, cy)), valid && x < ex};
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
