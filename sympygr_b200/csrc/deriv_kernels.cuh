// The derivative stage: a 2.5-D streaming stencil.
//
// A work item is one column tile (16 x 8 columns of a z-slab of one block) and one variable.
// A CTA of two warps marches along z; thread (tx, g) owns columns (tx, 2g) and (tx, 2g + 1).
//
//   * Planes of the tile plus a 3-point halo (22 x 14 points) arrive in a ring of kRing
//     shared-memory buffers by 16-byte cp.async.  A block's rows have an odd pitch as a rule,
//     so a row need not start on a 16-byte boundary: its copy starts at the boundary before
//     it, and the row then sits one element further right in its buffer (its shift).
//   * Per plane a thread reads the 8 values along y that the windows of its two points share
//     and their 6 x neighbours, and forms D_x, D_y, D_xx, D_yy and ko_x + ko_y.  For the 11
//     variables with second derivatives (DD) it also leaves D_x in shared memory, the threads
//     share out the D_x rows of the y halo, and D_y(D_x) follows from them (the reference's
//     composition, bssn/scripts/bssnrhs_derivs.h).
//   * The last six planes of u, D_x u and D_y u of each column stay in registers; the plane
//     three behind then has its z neighbourhood complete: D_z, D_zz, ko_z, D_z(D_x),
//     D_z(D_y).  unroll_planes planes are processed per loop pass, so the register windows
//     move once per pass.
//
// What bounds it: see plan_types.h for the stores.  With one column per thread, CTAs of 4
// warps, 8-byte copies and one plane per barrier and pass, the shared-memory data pipe is 81 /
// 70 % busy (without / with second derivatives) once the stores fill whole sectors; sharing the
// y windows, 16-byte copies and the unrolled passes bring that to 59 %, the issue slots to 65 /
// 60 % and DRAM to 52 / 44 % of its peak (64 blocks of 37^3, MIXED): no single resource is full,
// and what is left is the latency of 16 / 12 warps per SM.  16 blocks of 69^3 (4.0 M points):
// 0.83 ms (MIXED) and 1.14 ms (FP64), in that other form 1.46 and 2.00 ms.
//
// Closure rows (within three points of a flagged face) reach no further than three points
// beyond a tile or slab (cut_start).  Along z the three rows of a face are formed together,
// at the plane whose window holds the six that they read.  The item's code is instantiated
// without closure rows, with those along z (a branch that all threads take together) and with
// all (TileClosure), in kernels of their own: compiled into the common path the z branch alone
// cost it 18 % (16 blocks of 69^3, MIXED: 1.01 against 0.86 ms).  One code runs for all six
// rows, their weights in shared memory: a copy per row, inlined for each of a pass's planes
// and columns, left the kernel waiting for instructions a fifth of its time.  The closure rows
// along x and y are spread over all threads first: evaluated where they occur, by a few lanes
// of every warp, they took tiles at such faces 3.5 times as long as others.  64 blocks of 37^3
// with all faces flagged: 0.93 ms (MIXED) and 1.03 ms (FP64); with the z rows copied out and
// every thread working out its closure points anew in each plane 1.10 and 1.25 ms; 0.46 and
// 0.60 ms without faces.  16 blocks of 69^3: 1.39 and 1.62 ms.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "plan_types.h"
#include "stencils.cuh"

namespace b200bssn {

// VAR index -> position in the second-derivative list (gt0..gt5, chi, alpha,
// beta0..2; bssn/scripts/gen_bssnrhs_code:31-32), -1 if none.
__device__ __forceinline__ int dd_index(int v) {
  switch (v) {
    case 12: return 0; case 13: return 1; case 14: return 2;
    case 15: return 3; case 16: return 4; case 17: return 5;
    case 1: return 6;  case 0: return 7;
    case 6: return 8;  case 7: return 9;  case 8: return 10;
    default: return -1;
  }
}

struct DerivArgs {
  const double* u[kNumVars];
  const BlockDev* blocks;
  const TileDev* tiles;
  const int32_t* order;  // this launch's tiles, longest first
  void* scr;             // num_slots(ADV) slots per scratch point (double or float), layout scr_index
  const uint8_t* up;     // upwind mode: per scratch point bit a set where beta_a > 0
  int32_t tile_count;
  int* counter;          // work counter of this launch, zero at launch
};

constexpr int kRing = 4;                          // planes in flight or in use
constexpr int kRows = 2;                          // columns per thread, consecutive along y
constexpr int kItemThreads = kTilePlane / kRows;  // 64
constexpr int kPlaneW = kTileX + 2 * kHalo + 2;   // 24: staged row, with room for its shift
constexpr int kPlaneRows = kTileY + 2 * kHalo;    // 14
constexpr int kPlane = kPlaneW * kPlaneRows;      // doubles per buffer
constexpr int kDxPlane = kPlaneRows * kTileX;     // D_x rows of a plane, y halo included

// Shared memory of one item.
template <bool DD>
struct alignas(16) DerivSmem {
  double plane[kRing][kPlane];
  double dx[DD ? kDxPlane : 1];
  LineScales sc[3];
};
// Closure values of a plane: d1, ko, d2 of the columns next to faces flagged along x (staged
// row by staged row, three columns a face), then of the rows next to faces flagged along y
// (row by row); and where each one's points lie (closure_point).  Before them ko_x + ko_y of
// the last kKoPlanes planes, which the closure rows along z take from here.
constexpr int kKoPlanes = 8;
constexpr int kClosurePoints = 2 * 3 * kPlaneRows + 2 * 3 * kTileX;
struct ClosureValues {
  double ko[kKoPlanes][kTilePlane];
  double v[3][kClosurePoints];
  int32_t point[kClosurePoints];
};
struct ClosureRow;

__device__ __forceinline__ void cp_async16(uint32_t smem_dst, uint64_t gmem_src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Closure row of plane zo along z: -1 centred, 0..2 the low-side rows (zo = 3, 4, 5),
// 3..5 the high-side rows (zo = n-6, n-5, n-4).
__device__ __forceinline__ int z_case(int zo, int n, bool lo, bool hi) {
  if (hi && zo >= n - 6) return 3 + (zo - (n - 6));
  if (lo && zo < 6) return zo - 3;
  return -1;
}

// Centred-row arithmetic of the derivative kernel, by precision mode.
//
// ExactRows (FP64 mode): the reference's operations and order, each rounded
// (the win_* rows), so every derivative equals the reference's bit for bit.
//
// SplitRows (MIXED mode): the split-precision stencil.  Neighbour values enter
// only through FP64 differences taken before any downcast -- antisymmetric
// a_k = u(+k) - u(-k) for first derivatives, symmetric s_k = u(+k) + u(-k) - 2u
// for second derivatives (the centre weight cancels exactly since the weights
// sum to zero) -- whose weighted sum (fused multiply-adds allowed) is rounded once
// to FP32, the precision the derivative is stored in.  The Kreiss-Oliger row, a
// sixth difference that cancels all lower orders, stays in FP64 (from the same
// symmetric sums).
struct ExactRows {
  using D = double;
  template <typename T, int N>
  static __device__ __forceinline__ D d1(const T (&w)[N], int C, const LineScales& c) {
    return win_d1(w, C, c);
  }
  // first derivative kept for composition (D_x, D_y fields)
  template <int N>
  static __device__ __forceinline__ double d1_field(const double (&w)[N], int C, const LineScales& c) {
    return win_d1(w, C, c);
  }
  template <int N>
  static __device__ __forceinline__ D d2(const double (&w)[N], int C, const LineScales& c) {
    return win_d2(w, C, c);
  }
  template <int N>
  static __device__ __forceinline__ double ko(const double (&w)[N], int C, const LineScales& c) {
    return win_ko(w, C, c);
  }
  // upwind advective row `row` (adv_row_id) in the reference's order, each op rounded
  template <int N>
  static __device__ __forceinline__ D adv(const double (&w)[N], int C, int row, const LineScales& c) {
    double a;
    switch (row) {
      case 0:
        a = __dmul_rn(-3.0, w[C - 1]); a = mad_rn(a, -10.0, w[C]); a = mad_rn(a, 18.0, w[C + 1]);
        a = mad_rn(a, -6.0, w[C + 2]); a = mad_rn(a, 1.0, w[C + 3]);
        return __dmul_rn(a, c.d1_b);
      case 1:
        a = __dmul_rn(-1.0, w[C - 3]); a = mad_rn(a, 6.0, w[C - 2]); a = mad_rn(a, -18.0, w[C - 1]);
        a = mad_rn(a, 10.0, w[C]); a = mad_rn(a, 3.0, w[C + 1]);
        return __dmul_rn(a, c.d1_b);
      case 2:
        a = __dmul_rn(-3.0, w[C]); a = mad_rn(a, 4.0, w[C + 1]); a = mad_rn(a, -1.0, w[C + 2]);
        return __dmul_rn(a, c.adv_b2);
      case 3:
        a = __dmul_rn(-1.0, w[C - 1]); a = mad_rn(a, 1.0, w[C + 1]);
        return __dmul_rn(a, c.adv_b2);
      default:
        a = __dmul_rn(1.0, w[C - 2]); a = mad_rn(a, -4.0, w[C - 1]); a = mad_rn(a, 3.0, w[C]);
        return __dmul_rn(a, c.adv_b2);
    }
  }
};

struct SplitRows {
  using D = float;
  // the weighted sum of the FP64 differences is formed in FP64 and rounded once to the
  // FP32 of the slot: one rounding instead of four, and no conversion per difference
  template <typename T, int N>
  static __device__ __forceinline__ D d1(const T (&w)[N], int C, const LineScales& c) {
    const double a1 = (double)w[C + 1] - (double)w[C - 1];
    const double a2 = (double)w[C + 2] - (double)w[C - 2];
    const double a3 = (double)w[C + 3] - (double)w[C - 3];
    return (float)(fma(45.0, a1, fma(-9.0, a2, a3)) * c.d1_c);
  }
  // D_x / D_y fields that feed the mixed derivatives stay FP64: differencing
  // FP32-rounded first derivatives would cancel their leading digits
  template <int N>
  static __device__ __forceinline__ double d1_field(const double (&w)[N], int C, const LineScales& c) {
    const double a1 = w[C + 1] - w[C - 1];
    const double a2 = w[C + 2] - w[C - 2];
    const double a3 = w[C + 3] - w[C - 3];
    return fma(45.0, a1, fma(-9.0, a2, a3)) * c.d1_c;
  }
  template <int N>
  static __device__ __forceinline__ D d2(const double (&w)[N], int C, const LineScales& c) {
    const double u2 = 2.0 * w[C];
    const double s1 = (w[C + 1] + w[C - 1]) - u2;
    const double s2 = (w[C + 2] + w[C - 2]) - u2;
    const double s3 = (w[C + 3] + w[C - 3]) - u2;
    return (float)(fma(270.0, s1, fma(-27.0, s2, 2.0 * s3)) * c.d2_c);
  }
  template <int N>
  static __device__ __forceinline__ double ko(const double (&w)[N], int C, const LineScales& c) {
    const double u2 = 2.0 * w[C];
    const double s1 = (w[C + 1] + w[C - 1]) - u2;
    const double s2 = (w[C + 2] + w[C - 2]) - u2;
    const double s3 = (w[C + 3] + w[C - 3]) - u2;
    return c.ko_c * fma(-15.0, s1, fma(6.0, s2, -s3));
  }
  // upwind advective rows: the weights sum to zero, so the row is a weighted sum of FP64
  // differences from the centre value, summed in FP32
  template <int N>
  static __device__ __forceinline__ D adv(const double (&w)[N], int C, int row, const LineScales& c) {
    auto dd = [&](int k) { return (float)(w[C + k] - w[C]); };
    switch (row) {
      case 0:
        return fmaf(-3.0f, dd(-1), fmaf(18.0f, dd(1), fmaf(-6.0f, dd(2), dd(3)))) * (float)c.d1_b;
      case 1:
        return fmaf(6.0f, dd(-2), fmaf(-18.0f, dd(-1), fmaf(3.0f, dd(1), -dd(-3)))) * (float)c.d1_b;
      case 2:
        return fmaf(4.0f, dd(1), -dd(2)) * (float)c.adv_b2;
      case 3:
        return (float)(w[C + 1] - w[C - 1]) * (float)c.adv_b2;
      default:
        return fmaf(-4.0f, dd(-1), dd(-2)) * (float)c.adv_b2;
    }
  }
};
template <typename ST>
struct RowsFor { using type = ExactRows; };
template <>
struct RowsFor<float> { using type = SplitRows; };

// The closure rows of a line, for the points next to a flagged face.  Row id: 0..2
// the points 3, 4, 5 at a low face, 3..5 the points n-6, n-5, n-4 at a high one (closure_id).
// A row reads the values m[k], k points from the face point inwards.  d1 and d2 sum five of
// them in ascending index order, with the row's weights; ko sums from the far point inwards,
// with weights by distance from the face.  Operations and order are the reference's: the weights
// come from a table (in shared memory), so that lanes at different rows run one code.
struct ClosureRow {
  double d1[5], d2[5];  // ascending index
  double ko[4];         // m3, m2, m1, m0
};
static __constant__ ClosureRow kClosureRows[6] = {
    {{-25, 48, -36, 16, -3}, {35, -104, 114, -56, 11}, {1, -3, 3, -1}},
    {{-3, -10, 18, -6, 1}, {11, -20, 6, 4, -1}, {-6, 12, -10, 3}},
    {{1, -8, 0, 8, -1}, {-1, 16, -30, 16, -1}, {15, -19, 12, -3}},
    {{1, -8, 0, 8, -1}, {-1, 16, -30, 16, -1}, {15, -19, 12, -3}},
    {{-1, 6, -18, 10, 3}, {-1, 4, 6, -20, 11}, {-6, 12, -10, 3}},
    {{3, -16, 36, -48, 25}, {11, -56, 114, -104, 35}, {1, -3, 3, -1}},
};
// (-1: none, also past the last interior point, where only lanes that pad a tile stand)
__device__ __forceinline__ int closure_id(int pos, int n, bool lo, bool hi) {
  if (hi && pos >= n - 6) return pos <= n - 4 ? 3 + (pos - (n - 6)) : -1;
  return lo && pos < 6 ? pos - 3 : -1;
}
// (the caller's next barrier makes the copy visible)
__device__ __forceinline__ void load_closure_rows(ClosureRow* dst) {
  for (int k = threadIdx.x; k < 6 * (int)(sizeof(ClosureRow) / sizeof(double)); k += blockDim.x)
    reinterpret_cast<double*>(dst)[k] = reinterpret_cast<const double*>(kClosureRows)[k];
}
__device__ __forceinline__ double closure_d1(const double (&m)[6], int id, const ClosureRow& c, const LineScales& sc) {
  const bool hi = id >= 3, skip = id == 2 || id == 3;  // those rows have no term at the point itself
  double a = __dmul_rn(c.d1[0], hi ? m[4] : m[0]);
  a = mad_rn(a, c.d1[1], hi ? m[3] : m[1]);
  const double b = mad_rn(a, c.d1[2], m[2]);
  a = skip ? a : b;
  a = mad_rn(a, c.d1[3], hi ? m[1] : m[3]);
  a = mad_rn(a, c.d1[4], hi ? m[0] : m[4]);
  return __dmul_rn(a, sc.d1_b);
}
__device__ __forceinline__ double closure_d2(const double (&m)[6], int id, const ClosureRow& c, const LineScales& sc) {
  const bool hi = id >= 3;
  double a = __dmul_rn(c.d2[0], hi ? m[4] : m[0]);
  a = mad_rn(a, c.d2[1], hi ? m[3] : m[1]);
  a = mad_rn(a, c.d2[2], m[2]);
  a = mad_rn(a, c.d2[3], hi ? m[1] : m[3]);
  a = mad_rn(a, c.d2[4], hi ? m[0] : m[4]);
  return __dmul_rn(a, sc.d2_b);
}
__device__ __forceinline__ double closure_ko(const double (&m)[6], int id, const ClosureRow& c, const LineScales& sc) {
  const int dist = id < 3 ? id : 5 - id;  // points from the face
  double a = dist == 2 ? mad_rn(m[5], -6.0, m[4]) : m[4];
  a = dist == 0 ? m[3] : mad_rn(a, c.ko[0], m[3]);
  a = mad_rn(a, c.ko[1], m[2]);
  a = mad_rn(a, c.ko[2], m[1]);
  a = mad_rn(a, c.ko[3], m[0]);
  return __ddiv_rn(a, dist == 0 ? sc.ko_s3 : (dist == 1 ? sc.ko_s2 : sc.ko_s1));
}

// Where an item's outputs go.  FULL: a tile of the plan's scratch (planes 128 scratch points
// apart, rows by point_off; whole sectors stored: the lanes that pad a row write values
// nobody reads).  Else points numbered densely (the allocation-free entry point, whose fixed
// array has no room for the padding): lp = base + tx + row_stride * ty + plane_pts * plane.
struct ScratchMap {
  int32_t base;
  bool narrow;
  int32_t row_stride, plane_pts;
};

// Planes per loop pass (measured on 16 blocks of 69^3, MIXED / FP64 ms: without second
// derivatives 2 planes 0.322 / 0.451, 4 planes 0.314 / 0.418; with them 2 planes 0.553 /
// 0.770, 4 planes 0.675 / 0.903: the longer pass spills).
__host__ __device__ constexpr int unroll_planes(bool dd, bool cl, bool adv) { return dd || cl || adv ? 2 : 4; }

// Where the points of a closure row lie in a staged plane: the offset of the face point, the
// parity of its staged row, whether the row runs along y, and the row id.
__device__ __forceinline__ int closure_point(int offset, int row, bool along_y, int id) {
  return offset | (row & 1) << 9 | (int)along_y << 10 | id << 11;
}
static_assert(kPlane <= 512, "closure_point holds nine bits of offset");

// Barrier over the kItemThreads threads of an item; `id` names it where a CTA runs several.
__device__ __forceinline__ void item_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kItemThreads) : "memory");
}

// One (column tile, variable) work item; DD: the variable has second derivatives; ADV: also
// the upwind advective derivatives (slots kAdvSlot + 3v + axis, upwinded by the sign of the
// matching shift component at the point); CLOSURE: which closure rows the item may take
// (tile_closure).  Those along x and y have their weights at `closure`; the threads share the
// points out before they form a plane's derivatives, and leave the values in `fix`.
template <typename ST, bool DD, bool ADV, int CLOSURE, bool FULL>
__device__ __forceinline__ void derive_item(const DerivArgs& a, const BlockDev& Bk, const TileDev& t, const ScratchMap sm, const int v,
                                            DerivSmem<DD>& S, const ClosureRow* closure, ClosureValues* fix,
                                            const int barrier) {
  using Rows = typename RowsFor<ST>::type;
  constexpr int NS = num_slots(ADV);
  constexpr int R = kRows;
  constexpr bool CL = CLOSURE == kClosureXY, CLZ = CLOSURE != kClosureNone;
  constexpr int B = unroll_planes(DD, CL, ADV);
  constexpr int NK = 3;  // planes of ko_x + ko_y kept
  const int tid = threadIdx.x % kItemThreads;
  const int nx = Bk.sz[0], ny = Bk.sz[1], nz = Bk.sz[2];
  const int i0 = 3 + t.i0, j0 = 3 + t.j0, k0 = 3 + t.k0;
  const int ex = t.ex, ey = t.ey, ez = t.nz;
  const uint32_t bf = Bk.bflag;
  const bool lox = CL && (bf & 1u), hix = CL && (bf & 2u), loy = CL && (bf & 4u),
             hiy = CL && (bf & 8u), loz = CLZ && (bf & 16u), hiz = CLZ && (bf & 32u);
  const int tx = tid & 15, ty0 = R * (tid >> 4);
  const int gi = i0 + tx, gj0 = j0 + ty0;
  // closure rows of this thread's column and rows, -1 for none; the tile's faces
  const int idx = closure_id(gi, nx, lox, hix);
  int idy[R];
#pragma unroll
  for (int r = 0; r < R; ++r) idy[r] = closure_id(gj0 + r, ny, loy, hiy);
  // Closure points along x and y (ClosureValues): per = those of a face along x -- all staged
  // rows with second derivatives, whose D_y(D_x) reads them, else the tile's own --, npx of both.
  constexpr int kRow0 = DD ? 0 : kHalo;
  const bool flx = lox && i0 == 3, fhx = hix && i0 + ex == nx - 3, fly = loy && j0 == 3, fhy = hiy && j0 + ey == ny - 3;
  const uint32_t plane_elems = (uint32_t)nx * (uint32_t)ny;
  const int np = ez + 2 * kHalo;  // planes streamed: k0 - 3 .. k0 + ez + 2, all inside the block
  const int rows = ey + 2 * kHalo;
  const int per = 3 * (DD ? rows : ey), npx = per * ((int)flx + (int)fhx), npc = npx + 3 * kTileX * ((int)fly + (int)fhy);
  // this thread's values: along x of staged row w at fx + 3 w, along y of its row r at fy[r]
  int fx = 0, fy[R] = {};
  if constexpr (CL) {
    fx = (idx >= 3 ? idx - 3 + (flx ? per : 0) : idx) - 3 * kRow0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      fy[r] = npx + (idy[r] >= 3 ? kTileX * (idy[r] - 3) + (fly ? 3 * kTileX : 0) : kTileX * idy[r]) + tx;
    for (int e = tid; e < npc; e += kItemThreads) {
      const bool along_y = e >= npx, first = along_y ? fly : flx;
      const int each = along_y ? 3 * kTileX : per, f = along_y ? e - npx : e;
      const bool hi = !first || f >= each;
      const int g = first && hi ? f - each : f, k = along_y ? g / kTileX : g % 3;
      const int row = along_y ? (hi ? ey - 1 : 0) + kHalo : kRow0 + g / 3, x = along_y ? g % kTileX : (hi ? ex - 1 : 0);
      fix->point[e] = closure_point(row * kPlaneW + x + kHalo, row, along_y, hi ? k + 3 : k);
    }
  }

  // Copies: a plane is 14 rows of 12 sixteen-byte pieces, piece e (row e / 12) by thread
  // e % 64.  A row's pieces start at the 16-byte boundary at or before its first element.
  // Pieces without a needed element are left out.  Rows of the y halo in planes of the z
  // halo are read in the tile's columns only, and there the pieces at both ends are left out
  // too: with that no piece leaves the block.
  const double* const f = a.u[v] + Bk.offset + (i0 - kHalo) + (int64_t)nx * (j0 - kHalo) + (int64_t)plane_elems * (k0 - kHalo);
  constexpr int kPieces = kPlaneRows * (kPlaneW / 2), kCopies = (kPieces + kItemThreads - 1) / kItemThreads;
  uint32_t off[kCopies], want = 0, want_halo = 0;
#pragma unroll
  for (int k = 0; k < kCopies; ++k) {
    const int e = tid + kItemThreads * k, row = e / (kPlaneW / 2), c = e - row * (kPlaneW / 2), w = ex + 2 * kHalo;
    const bool in = row < rows && 2 * c <= w;
    off[k] = 8u * ((uint32_t)nx * (uint32_t)row);  // bytes; the piece is added after rounding the row down
    want |= in ? 1u << k : 0u;
    const bool halo_row = row < kHalo || row >= ey + kHalo;
    want_halo |= in && (!halo_row || (c > 0 && 2 * c + 2 <= w)) ? 1u << k : 0u;
  }
  const uint32_t dst0 = static_cast<uint32_t>(__cvta_generic_to_shared(&S.plane[0][0])) + (uint32_t)tid * 16u;
  auto stage = [&](int s) {
    if (s < np) {
      const uint32_t m = s < kHalo || s >= np - kHalo ? want_halo : want;
      const uint64_t src = reinterpret_cast<uint64_t>(f + plane_elems * (uint32_t)s);
      const uint32_t dst = dst0 + ((uint32_t)s % kRing) * (uint32_t)(kPlane * 8);
#pragma unroll
      for (int k = 0; k < kCopies; ++k) {
        const uint32_t c = (uint32_t)(tid + kItemThreads * k) % (kPlaneW / 2);
        if (m & (1u << k)) cp_async16(dst + 16u * kItemThreads * k, ((src + off[k]) & ~uint64_t(15)) + 16u * c);
      }
    }
    cp_async_commit();
  };

  // Outputs: slot s of scratch point lp sits at (lp / 32) * 32 NS + s * 32 + lp % 32; scratch
  // offsets fit in 32 bits (NS * points < 2^31).  `at(r, o)`: row r of the thread, slab plane o.
  const int q = DD ? dd_index(v) : -1;
  ST* const sd_first = static_cast<ST*>(a.scr) + (3 * v) * 32;                   // D_x, D_y, D_z
  ST* const sd_second = static_cast<ST*>(a.scr) + (72 + 6 * (DD ? q : 0)) * 32;  // the 6 second
  ST* const sd_ko = static_cast<ST*>(a.scr) + (kKoSlot + v) * 32;                // KO sum
  ST* const sd_adv = static_cast<ST*>(a.scr) + (kAdvSlot + 3 * v) * 32;          // upwind mode
  auto col = [](int lp) { return (lp >> 5) * (NS * 32) + (lp & 31); };
  const int full0 = col(sm.base + point_off(sm.narrow, tx, ty0));
  static_assert(kRows == 2, "point_off puts a thread's second row 32 scratch points after its first");
  const int lp0 = sm.base + tx + sm.row_stride * ty0;
  auto at = [&](int r, int o) {
    if constexpr (FULL) return full0 + o * (kTilePlane / 32 * NS * 32) + r * (NS * 32);
    return col(lp0 + sm.row_stride * r + sm.plane_pts * o);
  };
  // rows r < nr of this thread are stored: whole sectors when FULL, so up to 7 (MIXED) or 3
  // lanes past the tile's last column
  constexpr int kSector = 32 / (int)sizeof(ST);
  const int exs = FULL ? (ex + kSector - 1) / kSector * kSector : ex;
  const int nr = tx < exs ? max(0, min(R, ey - ty0)) : 0;
  // address of the first staged element in units of 8 bytes: its parity, and how it
  // alternates with rows and planes, gives each row's shift (ty0 is even)
  const uint32_t par0 = (uint32_t)(reinterpret_cast<uint64_t>(f) >> 3);

#pragma unroll
  for (int s = 0; s < kRing - 1; ++s) stage(s);
  if (tid < 3) S.sc[tid] = make_line_scales(Bk.h[tid]);
  const LineScales& cx = S.sc[0];
  const LineScales& cy = S.sc[1];
  const LineScales& cz = S.sc[2];

  double U[R][6 + B], X[DD ? R : 1][6 + B], Y[DD ? R : 1][6 + B], K[R][NK + B];  // (K: without closure rows along z)
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int k = 0; k < 6 + B; ++k) {
      U[r][k] = 0.0;
      if (DD) X[r][k] = Y[r][k] = 0.0;
    }
#pragma unroll
    for (int k = 0; k < NK + B; ++k) K[r][k] = 0.0;
  }

  // upwind mode: the sign bits of the thread's points, read one plane ahead (up_next); the
  // last four planes' in up_bits, the newest lowest
  const uint8_t* const up0 = ADV ? a.up + sm.base + point_off(sm.narrow, tx, ty0) : nullptr;
  uint32_t up_bits[R] = {}, up_next[R] = {};
  auto load_up = [&](int o) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (ADV && r < nr && o < ez) up_next[r] = __ldg(up0 + o * kTilePlane + r * 32);
  };
  load_up(0);

  for (int s0 = 0; s0 < np; s0 += B) {
#pragma unroll
    for (int p = 0; p < B; ++p) {
      const int s = s0 + p;
      if (s < np) {
        const uint32_t slot = (uint32_t)s % kRing;
        cp_async_wait<kRing - 2>();
        item_sync(barrier);  // plane s is visible, and every thread is done with the one before, whose buffer is refilled
        stage(s + kRing - 1);
        // rows ty0 + even of this plane sit at pe, rows ty0 + odd at po
        const uint32_t sh = (par0 + plane_elems * (uint32_t)s) & 1u;
        const double* const P = S.plane[0] + slot * kPlane + ty0 * kPlaneW + tx;
        const double* const pe = P + sh;
        const double* const po = P + (sh ^ ((uint32_t)nx & 1u));
        const int o = s - kHalo;
        const bool out = (unsigned)o < (unsigned)ez;
        if constexpr (ADV) {
#pragma unroll
          for (int r = 0; r < R; ++r) up_bits[r] = (up_bits[r] << 8) | (out ? up_next[r] : 0u);
          if (out) load_up(o + 1);
        }
        if (CL && (DD || out)) {
          for (int e = tid; e < npc; e += kItemThreads) {
            const int pt = fix->point[e], id = pt >> 11;
            const bool along_y = pt >> 10 & 1;
            const uint32_t nxo = (uint32_t)nx & 1u, even = sh ^ (nxo & (uint32_t)(pt >> 9)), odd = even ^ (along_y ? nxo : 0u);
            const int step = (along_y ? kPlaneW : 1) * (id >= 3 ? -1 : 1);
            const double* const q = S.plane[0] + slot * kPlane + (pt & 511);
            double m[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) m[k] = q[k * step + (int)((k & 1) ? odd : even)];
            const LineScales& sc = along_y ? cy : cx;
            fix->v[0][e] = closure_d1(m, id, closure[id], sc);
            if (out) {
              fix->v[1][e] = closure_ko(m, id, closure[id], sc);
              if (DD) fix->v[2][e] = closure_d2(m, id, closure[id], sc);
            }
          }
          item_sync(barrier);
        }
        double yv[R + 6];
#pragma unroll
        for (int m = 0; m < R + 6; ++m) yv[m] = ((m & 1) ? po : pe)[m * kPlaneW + kHalo];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          U[r][6 + p] = yv[r + 3];
          K[r][NK + p] = 0.0;
          if (DD || out) {
            const double* px = (((r + 3) & 1) ? po : pe) + (r + 3) * kPlaneW + kHalo;
            double wx[7], wy[7];
#pragma unroll
            for (int k = 0; k < 7; ++k) {
              wx[k] = k == 3 ? yv[r + 3] : px[k - 3];
              wy[k] = yv[r + k];
            }
            double dx = Rows::d1_field(wx, 3, cx), dy = Rows::d1_field(wy, 3, cy);
            double kx = Rows::ko(wx, 3, cx), ky = Rows::ko(wy, 3, cy);
            ST dxx = ST(0), dyy = ST(0);
            if (DD) {
              dxx = (ST)Rows::d2(wx, 3, cx);
              dyy = (ST)Rows::d2(wy, 3, cy);
            }
            if (CL && idx >= 0) {
              const int e = fx + 3 * (ty0 + r + kHalo);
              dx = fix->v[0][e];
              kx = fix->v[1][e];
              if (DD) dxx = (ST)fix->v[2][e];
            }
            if (CL && idy[r] >= 0) {
              dy = fix->v[0][fy[r]];
              ky = fix->v[1][fy[r]];
              if (DD) dyy = (ST)fix->v[2][fy[r]];
            }
            if (CLZ)
              fix->ko[o & (kKoPlanes - 1)][tid + kItemThreads * r] = __dadd_rn(kx, ky);
            else
              K[r][NK + p] = __dadd_rn(kx, ky);
            if (DD) {
              X[r][6 + p] = dx;
              Y[r][6 + p] = dy;
              S.dx[(ty0 + r + kHalo) * kTileX + tx] = dx;
            }
            if (out && r < nr) {
              const int c = at(r, o);
              sd_first[c] = (ST)dx;
              sd_first[c + 32] = (ST)dy;
              if (DD) {
                sd_second[c + 0 * 32] = dxx;
                sd_second[c + 3 * 32] = dyy;
              }
              if constexpr (ADV) {
                // deriv42adv_x / _y (derivs.cpp:495-775) by the signs of beta0 / beta1 at the point
                const bool upx = up_bits[r] & 1u, upy = up_bits[r] & 2u;
                sd_adv[c] = (ST)(double)Rows::adv(wx, 3, adv_row_id(gi, nx, lox, hix, upx), cx);
                sd_adv[c + 32] = (ST)(double)Rows::adv(wy, 3, adv_row_id(gj0 + r, ny, loy, hiy, upy), cy);
              }
            }
          }
        }
        if constexpr (DD) {
          if (out) {
            // D_x on the three rows above and below the tile: 96 values
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const int h = 4 * k + (tid >> 4);
              if (h < 2 * kHalo) {
                const int row = h < kHalo ? h : ey + h;
                const uint32_t shr = (sh + ((uint32_t)nx & (uint32_t)row)) & 1u;
                const double* px = S.plane[0] + slot * kPlane + row * kPlaneW + tx + kHalo + shr;
                double w[7];
#pragma unroll
                for (int m = 0; m < 7; ++m) w[m] = px[m - 3];
                double dx = Rows::d1_field(w, 3, cx);
                if (CL && idx >= 0) dx = fix->v[0][fx + 3 * row];
                S.dx[row * kTileX + tx] = dx;
              }
            }
            item_sync(barrier);  // the plane's D_x rows are visible
            const double* pd = S.dx + ty0 * kTileX + tx;
            double dv[R + 6];
#pragma unroll
            for (int m = 0; m < R + 6; ++m) dv[m] = m >= 3 && m < R + 3 ? X[m >= 3 && m < R + 3 ? m - 3 : 0][6 + p] : pd[m * kTileX];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              double w[7];
#pragma unroll
              for (int k = 0; k < 7; ++k) w[k] = dv[r + k];
              ST dxy = (ST)Rows::d1(w, 3, cy);
              if (CL && idy[r] >= 0) {
                double m[6];
#pragma unroll
                for (int k = 0; k < 6; ++k) m[k] = pd[((idy[r] >= 3 ? ny - 4 - k : 3 + k) - gj0 + 3) * kTileX];
                dxy = (ST)closure_d1(m, idy[r], closure[idy[r]], cy);
              }
              if (r < nr) sd_second[at(r, o) + 1 * 32] = dxy;
            }
          }
        }
        // z rows of slab plane o - 3; window index 3 + p is its plane
        const int oz = s - 2 * kHalo;
        if ((unsigned)oz < (unsigned)ez) {
          const int zc = CLZ ? z_case(k0 + oz, nz, loz, hiz) : -1;
          if (!CLZ || zc < 0) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              // rhs.cpp:332-369 sums (ko_x + ko_y) + ko_z; summed in FP64, stored like the
              // slots (FP32 in MIXED: the term enters the output scaled by sigma)
              const ST dz = (ST)Rows::d1(U[r], 3 + p, cz);
              const double kxy = CLZ ? fix->ko[oz & (kKoPlanes - 1)][tid + kItemThreads * r] : K[r][NK + p - 3];
              const ST ks = (ST)__dadd_rn(kxy, Rows::ko(U[r], 3 + p, cz));
              ST dzz = ST(0), dxz = ST(0), dyz = ST(0);
              if (DD) {
                dzz = (ST)Rows::d2(U[r], 3 + p, cz);
                dxz = (ST)Rows::d1(X[r], 3 + p, cz);
                dyz = (ST)Rows::d1(Y[r], 3 + p, cz);
              }
              if (r < nr) {
                const int c = at(r, oz);
                sd_first[c + 2 * 32] = dz;
                sd_ko[c] = ks;
                if (DD) {
                  sd_second[c + 5 * 32] = dzz;
                  sd_second[c + 2 * 32] = dxz;
                  sd_second[c + 4 * 32] = dyz;
                }
              }
            }
          } else if (zc == 2 || zc == 3) {
            // The three closure rows of a face, with the one farthest from it: the window then
            // holds the six planes that they read, m[k] the one k from the face plane.
            const bool hi = zc == 3;
            const int o0 = hi ? oz : oz - 2, id0 = hi ? 3 : 0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
              auto inwards = [&](const double (&w)[6 + B], double (&m)[6]) {
#pragma unroll
                for (int k = 0; k < 6; ++k) m[k] = hi ? w[5 + p - k] : w[1 + p + k];
              };
              if (r < nr) {
                double m[6];
                inwards(U[r], m);
#pragma unroll 1
                for (int k = 0; k < 3; ++k) {
                  const int id = id0 + k, c = at(r, o0 + k);
                  const double kxy = fix->ko[(o0 + k) & (kKoPlanes - 1)][tid + kItemThreads * r];
                  sd_first[c + 2 * 32] = (ST)closure_d1(m, id, closure[id], cz);
                  sd_ko[c] = (ST)__dadd_rn(kxy, closure_ko(m, id, closure[id], cz));
                  if (DD) sd_second[c + 5 * 32] = (ST)closure_d2(m, id, closure[id], cz);
                }
                if constexpr (DD) {
                  double mx[6], my[6];
                  inwards(X[r], mx);
                  inwards(Y[r], my);
#pragma unroll 1
                  for (int k = 0; k < 3; ++k) {
                    const int id = id0 + k, c = at(r, o0 + k);
                    sd_second[c + 2 * 32] = (ST)closure_d1(mx, id, closure[id], cz);
                    sd_second[c + 4 * 32] = (ST)closure_d1(my, id, closure[id], cz);
                  }
                }
              }
            }
          }
          if constexpr (ADV) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              if (r < nr) {
                // deriv42adv_z (derivs.cpp:776-900) by the sign of beta2 at the point
                const bool upz = up_bits[r] >> 24 & 4u;
                sd_adv[at(r, oz) + 2 * 32] = (ST)(double)Rows::adv(U[r], 3 + p, adv_row_id(k0 + oz, nz, loz, hiz, upz), cz);
              }
            }
          }
        }
      }
    }
    // the windows move on
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        U[r][k] = U[r][k + B];
        if (DD) {
          X[r][k] = X[r][k + B];
          Y[r][k] = Y[r][k + B];
        }
      }
#pragma unroll
      for (int k = 0; k < NK; ++k) K[r][k] = K[r][k + B];
    }
  }
  cp_async_wait<0>();
}

// Upwind mode: the signs of the shift at every scratch point of a chunk's tiles, one CTA of
// kTilePlane threads per tile.  (A derivative item that reads the shift itself has
// three loads of 8 bytes per point, direction and variable, waited for at once; this way it has
// a byte per point, a plane ahead.)  Columns that pad a tile take its last one's.
static __global__ void __launch_bounds__(kTilePlane)
bssn_shift_signs_kernel(const double* b0, const double* b1, const double* b2, const BlockDev* blocks, const TileDev* tiles,
                        uint8_t* up) {
  const TileDev t = tiles[blockIdx.x];
  const BlockDev& B = blocks[t.block];
  const int x = threadIdx.x % kTileX, y = threadIdx.x / kTileX;
  const bool narrow = t.ex <= kNarrow;
  if (y >= t.ey || (narrow && x >= kNarrow)) return;
  const int64_t plane = (int64_t)B.sz[0] * B.sz[1];
  int64_t p = B.offset + (3 + t.i0 + min(x, t.ex - 1)) + (int64_t)B.sz[0] * (3 + t.j0 + y) + plane * (3 + t.k0);
  uint8_t* const out = up + t.sbase + point_off(narrow, x, y);
#pragma unroll 4
  for (int z = 0; z < t.nz; ++z, p += plane)
    out[z * kTilePlane] = (uint8_t)((__ldg(b0 + p) > 0.0) | (__ldg(b1 + p) > 0.0) << 1 | (__ldg(b2 + p) > 0.0) << 2);
}

// The variables of each kind: 13 without second derivatives (K Gt B At), 11 with
// (alpha chi beta gt).
__device__ __forceinline__ int kind_var(bool dd, int i) {
  // 2 3 4 5 9 10 11 18 19 20 21 22 23
  if (!dd) return i < 4 ? i + 2 : (i < 7 ? i + 5 : i + 11);
  // 0 1 6 7 8 12 13 14 15 16 17
  return i < 2 ? i : (i < 5 ? i + 4 : i + 7);
}
constexpr int kKindVars[2] = {13, 11};        // [DD]

// Persistent derivative kernels: the grid holds as many CTAs as fit on the GPU at once, and
// each takes the next (tile, variable) item of its list from a device counter (the planner
// lists a chunk's tiles longest first).  CTAs of two warps per SM, and so the registers:
// 8 (128 registers) without second derivatives, 6 (168) with.
//
// The launches of a chunk's derivative stage depend on nothing of each other: each but the
// first is launched as a programmatic dependent of the one before (launch_deriv), which lets
// it start at once, so its CTAs fill the SMs as the ones before run out of items, and the
// launches of a small plan run side by side.  A CTA ends only when the launch before has
// ended, so that the last launch's end is the stage's.  (A call on one 21^3 block with all
// faces flagged, MIXED, whose launches last 20-30 us each, takes 80 us.)
constexpr int kind_ctas_per_sm(bool dd, bool adv, int closure) {
  return dd ? (adv ? 4 : 6) : (closure == kClosureXY ? 6 : 8);
}

template <typename ST, bool DD, bool ADV, int CLOSURE>
__global__ void __launch_bounds__(kItemThreads, kind_ctas_per_sm(DD, ADV, CLOSURE))
bssn_derivs_kind_kernel(const __grid_constant__ DerivArgs a) {
  constexpr int NV = kKindVars[DD];
  constexpr bool CL = CLOSURE == kClosureXY, CLZ = CLOSURE != kClosureNone;
  __shared__ DerivSmem<DD> S;
  __shared__ ClosureRow s_closure[CLZ ? 6 : 1];
  __shared__ __align__(8) unsigned char s_fix[CL ? sizeof(ClosureValues) : CLZ ? sizeof(ClosureValues::ko) : 8];
  __shared__ int s_item;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (CLZ) load_closure_rows(s_closure);
  for (;;) {
    __syncthreads();  // the previous item is finished with the shared memory
    if (threadIdx.x == 0) s_item = atomicAdd(a.counter, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= a.tile_count * NV) break;
    const TileDev t = a.tiles[a.order[item / NV]];
    const ScratchMap sm{t.sbase, t.ex <= kNarrow, 0, 0};
    derive_item<ST, DD, ADV, CLOSURE, true>(a, a.blocks[t.block], t, sm, kind_var(DD, item % NV), S, s_closure,
                                        reinterpret_cast<ClosureValues*>(s_fix), 1);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launches a derivative kernel; `follows`: right behind another one of its stage, see above.
inline cudaError_t launch_deriv(const void* fn, int grid, void** arg, bool follows, cudaStream_t s) {
  cudaLaunchAttribute dependent;
  dependent.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  dependent.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kItemThreads);
  cfg.stream = s;
  cfg.attrs = &dependent;
  cfg.numAttrs = follows ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, fn, arg);
}

}  // namespace b200bssn
