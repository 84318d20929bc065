// How a plan cuts its blocks into z-slabs, column tiles, runs of algebra tasks and chunks, and
// how large its derivative scratch is.  Host code without CUDA calls.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "b200bssn.h"
#include "plan_types.h"

namespace b200bssn {

constexpr int64_t kDefaultChunkPoints = int64_t(1) << 23, kSmallScratch = int64_t(1) << 20;
// A plan is refused when a z-slab of the depth asked for (kNominalDepth planes where none is)
// holds more interior points than max_chunk_points.  The slabs that are made may be thinner.
constexpr int64_t kNominalDepth = 48;
constexpr int64_t max_chunk_points(bool adv) { return (int64_t(1) << 31) / (kNumDerivs + (adv ? 3 * kNumVars : 0) + 1) - 1; }
// Scratch slots are addressed with 32-bit offsets: slots * scratch points < 2^31.
constexpr int64_t max_scratch_points(int slots) { return ((int64_t(1) << 31) / slots - 1) / kTilePlane * kTilePlane; }

struct ChunkRec {
  int32_t tile_begin, tile_count;
  int32_t list[3];  // how many of them take which closure rows (TileClosure): the plan's `order` holds them so
  int32_t range_begin, range_count;
  int64_t points;
};

struct PlanLayout {
  std::vector<SlabDev> slabs;
  std::vector<TileDev> tiles;
  std::vector<RangeDev> ranges;
  std::vector<ChunkRec> chunks;
  int64_t cap = 0;  // scratch points of a buffer
};

// Interior extents of a block, its rows and columns of tiles, and the scratch points of a plane.
struct Interior {
  int64_t n[3];
  int cutx, cuty;
  int64_t plane;
  explicit Interior(const b200bssn_block& b) : n{(int64_t)b.sz[0] - 6, (int64_t)b.sz[1] - 6, (int64_t)b.sz[2] - 6} {
    cutx = num_cuts((int)n[0], kTileX);
    cuty = num_cuts((int)n[1], kTileY);
    plane = (int64_t)cutx * cuty * kTilePlane;
  }
  bool narrow() const { return n[0] - cut_start((int)n[0], kTileX, cutx - 1) <= kNarrow; }  // the last column of tiles
  int64_t points(int64_t planes) const { return n[0] * n[1] * planes; }
  // Slabs of nearly equal depth, of at most `depth` planes and `limit` scratch points each but
  // never fewer than three planes (see cut_start).
  int64_t slabs(int64_t depth, int64_t limit) const {
    const int64_t d = std::min(depth, std::max<int64_t>(3, limit / plane));
    return std::min((n[2] + d - 1) / d, n[2] / 3);
  }
};

// Default z-slab depth of a plan, from a model of the derivative stage: a tile costs its
// planes, the 6 halo planes and about 4 planes' worth of start-up; the 11 variables with second
// derivatives (the longer kernel) share out 6 CTAs per SM, and each launch ends with one
// tile's time.  Deep slabs pay the halo less often, shallow ones give small plans enough
// items and every launch a shorter tail.  (16 blocks of 69^3 as one slab each, or in slabs of
// 48, 24, 12, 6, 3 planes, MIXED: 0.86, 0.91, 0.93, 1.07, 1.32, 1.76 ms.)
inline int64_t default_depth(const b200bssn_block* blocks, size_t nblocks, int64_t capacity, int64_t limit, int sms) {
  constexpr int kLongerKindVars = 11;
  const double resident = 6.0 * std::max(1, sms);
  int64_t best = 3;
  double best_cost = 0.0;
  for (const int64_t depth : {3, 4, 5, 6, 8, 11, 16, 22, 33, 44, 66, 99, 132}) {
    double work = 0.0, points = 0.0, scratch = 0.0;
    int64_t longest = 0;
    for (size_t b = 0; b < nblocks; ++b) {
      const Interior in(blocks[b]);
      const int64_t n = in.slabs(depth, limit);
      work += (double)(in.cutx * in.cuty) * (double)(in.n[2] + 10 * n);
      points += (double)in.points(in.n[2]);
      scratch += (double)(in.plane * in.n[2]);
      longest = std::max(longest, (in.n[2] + n - 1) / n + 10);
    }
    const double launches = std::max({1.0, points / (double)capacity, scratch / (double)limit});
    const double cost = work * kLongerKindVars / resident + launches * (double)longest;
    if (best_cost == 0.0 || cost < best_cost) {
      best_cost = cost;
      best = depth;
    }
  }
  return best;
}

// Cuts valid blocks (13 or more points per axis) into slabs, packs these into chunks and lists
// their tiles and runs.  `max_scratch`: max_scratch_points of the plan's slots.
inline int lay_out(PlanLayout& L, const b200bssn_block* blocks, const std::vector<BlockDev>& dev,
                   const b200bssn_plan_options& o, int64_t max_scratch, int sms) {
  const size_t nblocks = dev.size();
  auto depth_asked = [&](size_t b) {
    return o.block_slab_depth && o.block_slab_depth[b] ? (int64_t)o.block_slab_depth[b] : (int64_t)o.slab_depth;
  };
  const int64_t kMaxChunkPoints = max_chunk_points(o.advective != 0);
  int64_t max_slab = 0;  // interior points
  for (size_t b = 0; b < nblocks; ++b) {
    const Interior in(blocks[b]);
    const int64_t depth = depth_asked(b) ? depth_asked(b) : kNominalDepth, n = (in.n[2] + depth - 1) / depth;
    const int64_t points = in.points((in.n[2] + n - 1) / n);
    if (points > INT32_MAX) return B200BSSN_ERR_INVALID_ARGUMENT;
    max_slab = std::max(max_slab, points);
  }
  if (max_slab > kMaxChunkPoints) return B200BSSN_ERR_SIZE_LIMIT;
  // Interior points of a chunk, and the scratch points of a buffer.  Padding takes part of the
  // latter: a plan of several chunks has two buffers of at most `capacity` scratch points each,
  // and a plan whose interior points fit one chunk no more than that in all -- in two buffers
  // where its scratch points do not fit one --, but for whole blocks and slabs of the depth asked
  // for, which are not cut for this, and for kSmallScratch points, which padding may always take:
  // smaller chunks cost more time than the memory is worth (305 blocks of 23^3, MIXED, chunks
  // of 60,000 points: 2.69 ms when these include the padding, 2.08 ms when they do not).
  const int64_t capacity = std::min(std::max(o.chunk_points ? (int64_t)o.chunk_points : kDefaultChunkPoints, max_slab), kMaxChunkPoints);
  int64_t limit = std::min(capacity, max_scratch), all_points = 0, all_need = 0, whole = 0;
  for (size_t b = 0; b < nblocks; ++b) {
    const Interior in(blocks[b]);
    const int64_t points = in.points(in.n[2]), need = in.plane * in.n[2];
    all_points += points;
    all_need += need;
    if (points <= capacity && need <= max_scratch) whole = std::max(whole, need);
    const int64_t depth = depth_asked(b) ? depth_asked(b) : kNominalDepth, n = (in.n[2] + depth - 1) / depth;
    const int64_t slab = in.plane * ((in.n[2] + n - 1) / n);
    if (slab <= max_scratch) whole = std::max(whole, slab);
  }
  if (all_points <= capacity && all_need > limit) limit /= 2;
  limit = std::max({limit, whole, std::min(kSmallScratch, max_scratch)});
  if (all_points <= capacity && all_need <= std::min(2 * limit, max_scratch)) limit = std::max(limit, all_need);

  // The slabs; in planes of which no three fit the scratch, strips of a slab's tile rows.
  const int64_t model_depth = default_depth(blocks, nblocks, capacity, limit, sms);
  for (size_t b = 0; b < nblocks; ++b) {
    const Interior in(blocks[b]);
    const int64_t n = in.slabs(depth_asked(b) ? depth_asked(b) : model_depth, limit);
    for (int64_t sl = 0; sl < n; ++sl) {
      const int64_t k0 = sl * in.n[2] / n, nz = (sl + 1) * in.n[2] / n - k0;
      int per = in.cuty;  // rows of tiles per strip
      if (in.plane * nz > max_scratch) per = (int)std::max<int64_t>(1, max_scratch / (in.cutx * kTilePlane * nz));
      const int I1 = (int)in.n[1];
      for (int c = 0; c < in.cuty; c += per) {
        const int j0 = cut_start(I1, kTileY, c), j1 = cut_start(I1, kTileY, std::min(c + per, in.cuty));
        L.slabs.push_back({(int32_t)b, (int32_t)k0, (int32_t)nz, 0, j0, I1 - (j1 - j0), in.narrow()});
        limit = std::max(limit, (int64_t)in.cutx * std::min(per, in.cuty - c) * kTilePlane * nz);
      }
    }
  }

  ChunkRec cur{0, 0, {0, 0, 0}, 0, 0, 0};
  int64_t used = 0;  // scratch points of the current chunk
  auto flush = [&]() {
    if (cur.points > 0) {
      cur.tile_count = (int32_t)L.tiles.size() - cur.tile_begin;
      cur.range_count = (int32_t)L.ranges.size() - cur.range_begin;
      L.chunks.push_back(cur);
      L.cap = std::max<int64_t>(L.cap, used);
    }
    cur = ChunkRec{(int32_t)L.tiles.size(), 0, {0, 0, 0}, (int32_t)L.ranges.size(), 0, 0};
    used = 0;
  };
  for (size_t si = 0; si < L.slabs.size(); ++si) {
    SlabDev& u = L.slabs[si];
    const BlockDev& B = dev[u.block];
    const int I0 = B.sz[0] - 6, I1 = B.sz[1] - 6;
    const int cutx = num_cuts(I0, kTileX), c0 = first_cut(u), cuty = cut_rows(I1, u);
    const int64_t points = (int64_t)I0 * (I1 - u.jcut) * u.nz, need = (int64_t)cutx * cuty * u.nz * kTilePlane;
    // a block's slabs stay in one chunk when the whole block fits in one
    const Interior in(blocks[u.block]);
    const int64_t block_pts = in.points(in.n[2]), block_need = in.plane * in.n[2];
    const bool first = si == 0 || L.slabs[si - 1].block != u.block;
    if (first && block_pts <= capacity && block_need <= limit &&
        (cur.points + block_pts > capacity || used + block_need > limit))
      flush();
    if (cur.points + points > capacity || used + need > limit) flush();
    cur.points += points;
    u.sbase = (int32_t)used;
    for (int ty = 0; ty < cuty; ++ty)
      for (int tx = 0; tx < cutx; ++tx) {
        TileDev t;
        t.block = u.block;
        t.sbase = u.sbase + (ty * cutx + tx) * u.nz * kTilePlane;
        t.k0 = u.k0;
        t.nz = u.nz;
        t.i0 = (int16_t)cut_start(I0, kTileX, tx);
        t.j0 = (int16_t)cut_start(I1, kTileY, c0 + ty);
        t.ex = (int16_t)(cut_start(I0, kTileX, tx + 1) - t.i0);
        t.ey = (int16_t)(cut_start(I1, kTileY, c0 + ty + 1) - t.j0);
        L.tiles.push_back(t);
      }
    used += need;
    const int tasks = (int)slab_tasks(B, u.nz, u.jcut);
    for (int s = 0; s < tasks; s += kRangeTasks)
      L.ranges.push_back({(int32_t)si, s, std::min(kRangeTasks, tasks - s)});
  }
  flush();
  return B200BSSN_OK;
}

}  // namespace b200bssn
