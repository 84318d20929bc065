// Host check of the plan's index arithmetic (plan_types.h), over many block shapes: tiles and
// slabs cover every interior point once, never thinner than three points; the scratch point
// that the derivative stage gives a point is the one the algebra's tasks read it from; and
// the derivative stage's 16-byte copies stay inside the block and bring every element that
// the stencils read, whatever the alignment of the block's first element.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#define __host__
#define __device__
#define __forceinline__ inline
#include "plan_types.h"

using namespace b200bssn;

static int fail(const char* what, const int* n) {
  std::printf("%s: block %d x %d x %d\n", what, n[0], n[1], n[2]);
  return 1;
}

// The copies of one tile (deriv_kernels.cuh, `stage`): rows of 12 pieces of two elements.
static const char* check_copies(const BlockDev& B, int i0, int j0, int k0, int ex, int ey, int nz, int parity) {
  const long nx = B.sz[0], plane = nx * B.sz[1], total = plane * B.sz[2];
  const int w = ex + 2 * kHalo, rows = ey + 2 * kHalo;
  for (int s = 0; s < nz + 2 * kHalo; ++s) {
    const bool halo_plane = s < kHalo || s >= nz + kHalo;
    for (int row = 0; row < rows; ++row) {
      const bool halo_row = row < kHalo || row >= ey + kHalo;
      const long first = i0 + nx * (j0 + row) + plane * (k0 + s);  // padded coordinates i0, j0, k0 less the halo
      const long shift = (first + parity) & 1;
      std::vector<char> got(w, 0);
      for (int c = 0; c < 12; ++c) {
        const bool in = 2 * c <= w, clipped = halo_row && !(c > 0 && 2 * c + 2 <= w);
        if (!in || (halo_plane && clipped)) continue;
        for (int h = 0; h < 2; ++h) {
          const long e = first - shift + 2 * c + h;
          if (e < 0 || e >= total) return "copy leaves the block";
          if (e >= first && e < first + w) got[e - first] = 1;
        }
      }
      const bool inner = halo_plane && halo_row;  // such rows are read in the tile's columns only
      for (int x = inner ? kHalo : 0; x < (inner ? kHalo + ex : w); ++x)
        if (!got[x]) return "element not copied";
    }
  }
  return nullptr;
}

int main() {
  std::srand(1);
  for (int it = 0; it < 600; ++it) {
    int n[3];
    for (int a = 0; a < 3; ++a) n[a] = 13 + std::rand() % 44;
    if (it < 60) n[0] = 13 + it;
    if (it >= 60 && it < 120) n[1] = 13 + it - 60;
    BlockDev B{};
    for (int a = 0; a < 3; ++a) B.sz[a] = n[a];
    const int I0 = n[0] - 6, I1 = n[1] - 6, I2 = n[2] - 6, depth = 1 + std::rand() % 70;
    const int slabs = std::min((I2 + depth - 1) / depth, I2 / 3), cx = num_cuts(I0, kTileX), cy = num_cuts(I1, kTileY);
    std::vector<char> seen((size_t)I0 * I1 * I2, 0);
    int base = 0;
    for (int u = 0; u < slabs; ++u) {
      const int k0 = u * I2 / slabs, nz = (u + 1) * I2 / slabs - k0, need = cx * cy * nz * kTilePlane;
      if (nz < 3) return fail("slab below three planes", n);
      const SlabDev slab{0, k0, nz, base};
      std::vector<int> owner(need, -1);
      for (int t = 0; t < cx * cy; ++t) {
        const int i0 = cut_start(I0, kTileX, t % cx), ex = cut_start(I0, kTileX, t % cx + 1) - i0;
        const int j0 = cut_start(I1, kTileY, t / cx), ey = cut_start(I1, kTileY, t / cx + 1) - j0;
        if (ex < 3 || ey < 3 || ex > kTileX || ey > kTileY || i0 % kGroup) return fail("tile extents", n);
        for (int z = 0; z < nz; ++z)
          for (int y = 0; y < ey; ++y)
            for (int x = 0; x < ex; ++x) {
              int& o = owner[(t * nz + z) * kTilePlane + row_off(y) + x];
              if (o != -1) return fail("scratch point used twice", n);
              o = (i0 + x) + I0 * ((j0 + y) + I1 * (k0 + z));
            }
        for (int parity = 0; parity < 2; ++parity)
          if (const char* why = check_copies(B, i0, j0, k0, ex, ey, nz, parity)) return fail(why, n);
      }
      for (int task = 0; task < slab_tasks(B, nz); ++task)
        for (int lane = 0; lane < 32; ++lane) {
          const SlabPoint p = slab_point(B, slab, task, lane);
          if (p.lp < base || p.lp >= base + need) return fail("scratch point outside the slab", n);
          if (p.lp / 32 != (p.lp - lane % kGroup) / 32 || (p.lp - lane % kGroup) % kGroup) return fail("group split", n);
          if (!p.valid) continue;
          const int id = (p.i - 3) + I0 * ((p.j - 3) + I1 * (p.k - 3));
          if (owner[p.lp - base] != id) return fail("the algebra reads another point", n);
          if (seen[id]++) return fail("point taken twice", n);
        }
      base += need;
    }
    for (char c : seen)
      if (!c) return fail("point left out", n);
  }
  std::puts("ok");
  return 0;
}
