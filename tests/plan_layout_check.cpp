// Host check of how a plan cuts blocks (plan_layout.h); the argument names the check.
#include <cstdio>
#include <cstring>
#include <string>

#define __host__
#define __device__
#define __forceinline__ inline
#include "plan_layout.h"

using namespace b200bssn;

static const int kSms = 148;

static b200bssn_block block_of(uint32_t nx, uint32_t ny, uint32_t nz) {
  b200bssn_block b{};
  b.sz[0] = nx, b.sz[1] = ny, b.sz[2] = nz;
  for (int a = 0; a < 3; ++a) b.pmax[a] = 1.0;
  return b;
}

static std::vector<BlockDev> devices(const std::vector<b200bssn_block>& blocks) {
  std::vector<BlockDev> d(blocks.size());
  for (size_t b = 0; b < blocks.size(); ++b)
    for (int a = 0; a < 3; ++a) d[b].sz[a] = (int32_t)blocks[b].sz[a];
  return d;
}

static std::string text(const std::vector<b200bssn_block>& v, const b200bssn_plan_options& o) {
  char s[200];
  std::snprintf(s, sizeof(s), "%zu blocks, the first %u x %u x %u, slab depth %u, chunk points %llu%s", v.size(), v[0].sz[0],
                v[0].sz[1], v[0].sz[2], o.slab_depth, (unsigned long long)o.chunk_points, o.advective ? ", upwind" : "");
  return s;
}

static int fail(const char* what, const std::vector<b200bssn_block>& v, const b200bssn_plan_options& o) {
  std::printf("%s: %s\n", what, text(v, o).c_str());
  return 1;
}

// Whether slabs of the depth asked for (48 planes by default) fit a scratch without padding.
static bool expected(const std::vector<b200bssn_block>& v, const b200bssn_plan_options& o) {
  const int64_t depth = o.slab_depth ? o.slab_depth : 48, limit = (int64_t(1) << 31) / (o.advective ? 211 : 139) - 1;
  for (const b200bssn_block& b : v) {
    const int64_t I2 = b.sz[2] - 6, n = (I2 + depth - 1) / depth;
    if ((int64_t)(b.sz[0] - 6) * (b.sz[1] - 6) * ((I2 + n - 1) / n) > limit) return false;
  }
  return true;
}

// A plan of valid blocks is accepted exactly when expected, and then every buffer offset fits
// 32 bits, slabs hold three planes or more, and tiles and runs cover every point.
static int check_limits(const std::vector<b200bssn_block>& v, const b200bssn_plan_options& o) {
  PlanLayout L;
  const int slots = num_slots(o.advective != 0);
  const int rc = lay_out(L, v.data(), devices(v), o, max_scratch_points(slots), kSms);
  if ((rc == B200BSSN_OK) != expected(v, o)) return fail(rc == B200BSSN_OK ? "accepted" : "refused", v, o);
  if (rc != B200BSSN_OK) return 0;
  if (L.cap * slots >= int64_t(1) << 31) return fail("scratch offsets exceed 32 bits", v, o);
  int64_t points = 0, all = 0;
  for (const SlabDev& s : L.slabs)
    if (s.nz < 3) return fail("slab below three planes", v, o);
  for (const ChunkRec& c : L.chunks)
    for (int t = c.tile_begin; t < c.tile_begin + c.tile_count; ++t) {
      const TileDev& T = L.tiles[t];
      if (T.sbase < 0 || T.sbase + (int64_t)T.nz * kTilePlane > L.cap) return fail("tile outside the scratch", v, o);
      points += (int64_t)T.ex * T.ey * T.nz;
    }
  for (const b200bssn_block& b : v) all += Interior(b).points(b.sz[2] - 6);
  return points == all ? 0 : fail("tiles leave points out", v, o);
}

static int limits() {
  for (int adv = 0; adv < 2; ++adv) {
    b200bssn_plan_options o{};
    o.advective = adv;
    for (uint32_t n = 13; n <= 600; ++n)
      if (check_limits({block_of(n, n, n)}, o)) return 1;
    const uint32_t flat[][3] = {{300, 500, 100}, {1483, 1483, 13}, {1483, 1484, 14}, {32767, 300, 13}, {300, 32767, 13}, {15, 32767, 60},
                                {32767, 15, 60}, {700, 640, 40}, {1200, 13, 900}, {13, 1200, 900}, {561, 561, 54}, {3000, 700, 13}};
    for (const auto& f : flat) {
      for (const uint32_t depth : {0u, 1u, 2u, 3u, 5u, 16u, 48u, 100u, 4000u}) {
        o.slab_depth = depth;
        if (check_limits({block_of(f[0], f[1], f[2])}, o)) return 1;
      }
      o.slab_depth = 0;
      if (check_limits({block_of(21, 21, 21), block_of(f[0], f[1], f[2]), block_of(375, 375, 375)}, o)) return 1;
    }
    // planes of which three do not fit the scratch
    for (const uint32_t n : {2000u, 2105u, 3200u, 3930u})
      for (o.slab_depth = 1; o.slab_depth < 4; ++o.slab_depth)
        if (check_limits({block_of(n, n + 3, 14)}, o)) return 1;
  }
  return 0;
}

// Every point has one scratch point, inside its buffer and no other point's, which is the one that
// the algebra's tasks read it from, in groups of four that never straddle 32-point blocks.
static int check_points(const std::vector<b200bssn_block>& v, const b200bssn_plan_options& o, int64_t max_scratch) {
  const std::vector<BlockDev> dev = devices(v);
  PlanLayout L;
  if (lay_out(L, v.data(), dev, o, max_scratch, kSms) != B200BSSN_OK) return fail("refused", v, o);
  std::vector<std::vector<char>> seen(v.size());
  for (size_t b = 0; b < v.size(); ++b) seen[b].assign(Interior(v[b]).points(v[b].sz[2] - 6), 0);
  auto id = [&](int b, int i, int j, int k) {  // interior-relative
    return (int64_t)b << 32 | (i + Interior(v[b]).n[0] * (j + Interior(v[b]).n[1] * k));
  };
  for (const ChunkRec& c : L.chunks) {
    std::vector<int64_t> owner(L.cap, -1);
    for (int t = c.tile_begin; t < c.tile_begin + c.tile_count; ++t) {
      const TileDev& T = L.tiles[t];
      if (T.ex < 3 || T.ey < 3 || T.ex > kTileX || T.ey > kTileY || T.sbase % 32) return fail("tile", v, o);
      for (int z = 0; z < T.nz; ++z)
        for (int y = 0; y < T.ey; ++y)
          for (int x = 0; x < T.ex; ++x) {
            const int64_t lp = T.sbase + z * kTilePlane + point_off(T.ex <= kNarrow, x, y);
            if (lp < 0 || lp >= L.cap) return fail("scratch point outside the buffer", v, o);
            if (owner[lp] != -1) return fail("scratch point used twice", v, o);
            owner[lp] = id(T.block, T.i0 + x, T.j0 + y, T.k0 + z);
          }
    }
    for (int r = c.range_begin; r < c.range_begin + c.range_count; ++r)
      for (int k = 0; k < 32 * L.ranges[r].count; ++k) {
        const SlabDev& s = L.slabs[L.ranges[r].slab];
        const SlabPoint p = slab_point(dev[s.block], s, L.ranges[r].start + k / 32, k % 32);
        if (p.lp < 0 || p.lp >= L.cap) return fail("task outside the buffer", v, o);
        if ((p.lp - k % kGroup) % kGroup) return fail("group split", v, o);
        if (!p.valid) continue;
        const int64_t q = id(s.block, p.i - 3, p.j - 3, p.k - 3);
        if (owner[p.lp] != q) return fail("the algebra reads another point", v, o);
        if (seen[s.block][(int32_t)q]++) return fail("point taken twice", v, o);
      }
  }
  for (const auto& w : seen)
    for (const char s : w)
      if (!s) return fail("point left out", v, o);
  return 0;
}

static int points() {
  b200bssn_plan_options o{};
  for (uint32_t n = 13; n <= 151; ++n) {  // every width of the last tiles, whole and ragged rows
    o.slab_depth = n % 7;
    if (check_points({block_of(n, 13 + n * 5 % 29, 13 + n * 3 % 17), block_of(13 + n % 19, n, 14)}, o, max_scratch_points(162))) return 1;
  }
  return 0;
}

// planes of which no three fit the scratch
static int strips() {
  for (const int I1 : {7, 9, 17, 18, 31, 64, 65, 66})
    for (const int64_t rows : {1, 2, 3})
      for (const int I0 : {40, 44, 48})
        if (check_points({block_of(I0 + 6, I1 + 6, 19), block_of(19, 23, 17)}, {}, rows * 3 * 4 * kTilePlane)) return 1;
  return 0;
}

// Blocks that fit a chunk are not split between chunks (the host-array path overlaps its copies
// only then).
static int check_whole(const std::vector<b200bssn_block>& v, const b200bssn_plan_options& o) {
  PlanLayout L;
  const int64_t max_scratch = max_scratch_points(num_slots(o.advective != 0));
  if (lay_out(L, v.data(), devices(v), o, max_scratch, kSms) != B200BSSN_OK) return fail("refused", v, o);
  std::vector<int> chunk(v.size(), -1);
  for (size_t c = 0; c < L.chunks.size(); ++c)
    for (int t = L.chunks[c].tile_begin; t < L.chunks[c].tile_begin + L.chunks[c].tile_count; ++t) {
      const int b = L.tiles[t].block;
      const Interior in(v[b]);
      const int64_t capacity = o.chunk_points ? (int64_t)o.chunk_points : int64_t(1) << 23;
      if (chunk[b] >= 0 && chunk[b] != (int)c && in.points(in.n[2]) <= capacity && in.plane * in.n[2] <= max_scratch)
        return fail("block split between chunks", v, o);
      chunk[b] = (int)c;
    }
  return 0;
}

static int whole() {
  for (int adv = 0; adv < 2; ++adv) {
    b200bssn_plan_options o{};
    o.advective = adv;
    for (const int count : {4, 23})
      for (const uint32_t n : {135u, 151u, 167u, 175u, 200u})
        if (check_whole(std::vector<b200bssn_block>(count, block_of(n, n, n)), o)) return 1;
    std::vector<b200bssn_block> mixed;
    for (int k = 0; k < 3000; ++k) mixed.push_back(block_of(13 + k % 3, 13 + k % 5, 13));
    for (int k = 0; k < 12; ++k) mixed.push_back(block_of(135 + 9 * (k % 4), 140, 130));
    for (const uint64_t points : {0, 2200000, 3000000, 5000000}) {
      o.chunk_points = points;
      if (check_whole(mixed, o)) return 1;
    }
  }
  return 0;
}

// The scratch of lists of small blocks, whose padding weighs most: as many scratch points as
// chunk_points for a plan whose interior points fit one chunk, twice as many for others.
static int memory() {
  for (int adv = 0; adv < 2; ++adv)
    for (const uint32_t n : {13u, 14u, 15u, 17u, 21u, 23u, 37u})
      for (const int64_t points : {30000, 2000000, 6860000, 12000000})
        for (const int64_t chunk : {0, 20000, 300000, 3000000}) {
          b200bssn_plan_options o{};
          o.advective = adv;
          o.chunk_points = chunk;
          const Interior in(block_of(n, n, n));
          const std::vector<b200bssn_block> v(points / in.points(in.n[2]) + 1, block_of(n, n, n));
          PlanLayout L;
          if (lay_out(L, v.data(), devices(v), o, max_scratch_points(num_slots(adv != 0)), kSms) != B200BSSN_OK) return fail("refused", v, o);
          const int64_t capacity = chunk ? chunk : int64_t(1) << 23, all = in.points(in.n[2]) * (int64_t)v.size();
          int64_t bound = all <= capacity ? capacity : 2 * capacity;
          bound = std::max(bound, int64_t(2) << 20);  // small scratch buffers may be padded beyond it
          if (L.cap * (L.chunks.size() > 1 ? 2 : 1) > bound) return fail("scratch larger than asked for", v, o);
        }
  return 0;
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  int rc = 2;
  if (what == "limits") rc = limits();
  if (what == "points") rc = points();
  if (what == "strips") rc = strips();
  if (what == "whole") rc = whole();
  if (what == "memory") rc = memory();
  if (rc == 0) std::puts("ok");
  return rc;
}
