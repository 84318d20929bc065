// b200bssn_rhs_noalloc: the right-hand side of one block with no device
// allocation at all.
//
// Who needs this: a solver framework that hands the whole GPU memory to its own
// pool allocator at start-up (so a library cudaMalloc would fail or fragment that
// pool), and a time-step loop that must not call cudaMalloc/cudaFree because they
// can synchronise the whole device.  Such callers own the input and output arrays;
// the only other memory this path needs -- the derivative scratch -- lives in one fixed
// array below, reserved when the library is loaded and held by every GPU that loads it
// until the process exits; the work descriptors are kernel arguments.
//
// Limits and sharing:
//  * at most kNoallocMaxPoints interior points per call (a block with a 32^3
//    interior, i.e. 38^3 padded, is the largest cube that fits); larger blocks
//    are rejected with B200BSSN_ERR_SIZE_LIMIT before anything is launched;
//  * every call on a device uses the same array, which keeps whatever the last
//    call left in it.  Each call rewrites every word it later reads (every
//    derivative slot of every interior point), so nothing has to start at zero -- but two calls whose work overlaps on the GPU (different
//    streams, or host threads racing) overwrite each other's scratch and give
//    wrong results.  Serialise calls per device;
//  * the first call on each device looks up the array's device address with
//    cudaGetSymbolAddress, with that device current; make that first call before any
//    stream capture.  The address is kept for the life of the process, so calls after
//    a cudaDeviceReset of that device (which reloads the library's device code at a
//    new address) are not supported.
//
// The derivatives come from the plans' kernels in a form that numbers scratch points
// densely, tile after tile: the array has no room for the plans' padding.  Every tile takes
// the form with closure rows when the block has a flagged face.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "b200bssn.h"
#include "rhs_kernels.cuh"

using namespace b200bssn;

namespace {

constexpr int64_t kNoallocMaxPoints = B200BSSN_NOALLOC_MAX_POINTS;
constexpr int kMaxDevices = 64;
constexpr int kNoallocSlab = 48;  // greatest z-slab depth of this path

// the derivative scratch
constexpr size_t kNoallocBytes = sizeof(double) * num_slots(false) * kNoallocMaxPoints;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocBytes];

// Per-device address of g_noalloc_scratch (host-side handle -> device address) and the
// SM count.
struct DeviceSetup {
  void* addr = nullptr;
  int sms = 0;
};
std::mutex g_setup_mutex;
DeviceSetup g_setup[kMaxDevices];

int setup_device(int dev, DeviceSetup* out) {
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  DeviceSetup& d = g_setup[dev];
  if (!d.addr) {
    void* p = nullptr;
    int sms = 0;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || p == nullptr ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
      cudaGetLastError();
      return B200BSSN_ERR_CUDA;
    }
    d.sms = sms;
    d.addr = p;
  }
  *out = d;
  return B200BSSN_OK;
}

// The one block of a call, as kernel arguments: its tiles are numbered slab by slab, and
// their scratch points lie densely, tile after tile.
struct NoallocGeom {
  BlockDev block;
  int tiles_x, tiles_y, slabs;
  int runs;  // runs of kAlgebraThreads points per tile, of the largest one
};
__device__ __forceinline__ TileDev noalloc_tile(const NoallocGeom& g, int k) {
  const int I0 = g.block.sz[0] - 6, I1 = g.block.sz[1] - 6, I2 = g.block.sz[2] - 6;
  const int u = k / (g.tiles_x * g.tiles_y), ty = k / g.tiles_x % g.tiles_y, tx = k % g.tiles_x;
  TileDev t;
  t.block = 0;
  t.k0 = u * I2 / g.slabs;  // near-equal slabs (never below three planes)
  t.nz = (u + 1) * I2 / g.slabs - t.k0;
  t.i0 = (int16_t)cut_start(I0, kTileX, tx);
  t.j0 = (int16_t)cut_start(I1, kTileY, ty);
  t.ex = (int16_t)(cut_start(I0, kTileX, tx + 1) - t.i0);
  t.ey = (int16_t)(cut_start(I1, kTileY, ty + 1) - t.j0);
  t.sbase = I0 * I1 * t.k0 + t.nz * (I0 * t.j0 + t.i0 * t.ey);  // points of the tiles before
  return t;
}

// One (tile, variable) item per CTA.
template <typename ST, bool DD, int CLOSURE>
__global__ void __launch_bounds__(kItemThreads, kind_ctas_per_sm(DD, false, CLOSURE))
noalloc_derivs(const __grid_constant__ DerivArgs a, const __grid_constant__ NoallocGeom g) {
  constexpr int NV = kKindVars[DD];
  __shared__ DerivSmem<DD> S;
  __shared__ ClosureRow s_closure[CLOSURE == kClosureXY ? 6 : 1];
  __shared__ __align__(8) unsigned char s_fix[CLOSURE == kClosureXY ? sizeof(ClosureValues) : 8];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (CLOSURE == kClosureXY) {
    load_closure_rows(s_closure);
    __syncthreads();
  }
  const TileDev t = noalloc_tile(g, blockIdx.x / NV);
  const ScratchMap sm{t.sbase, false, t.ex, t.ex * t.ey};
  derive_item<ST, DD, false, CLOSURE, false>(a, g.block, t, sm, kind_var(DD, blockIdx.x % NV), S, s_closure,
                                             reinterpret_cast<ClosureValues*>(s_fix), 1);
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename ST>
const void* derivs_kernel(bool dd, bool closure) {
  if (dd)
    return closure ? (const void*)noalloc_derivs<ST, true, kClosureXY> : (const void*)noalloc_derivs<ST, true, kClosureNone>;
  return closure ? (const void*)noalloc_derivs<ST, false, kClosureXY> : (const void*)noalloc_derivs<ST, false, kClosureNone>;
}

template <typename ST>
struct GlobalScratch {
  static constexpr bool kHolds = false;
  const ST* d;       // slot 0 of the point
  __device__ __forceinline__ ST dv(int s) const { return __ldg(d + s * 32); }
  __device__ __forceinline__ double kov(int v) const { return (double)__ldg(d + (kKoSlot + v) * 32); }
};

// The algebra: one CTA per run of up to 128 points of a tile, one thread per point, inputs
// loaded from global memory as the generated code needs them.
template <typename ST>
__global__ void __launch_bounds__(kAlgebraThreads, 2)
noalloc_algebra(const __grid_constant__ AlgebraArgs a, const __grid_constant__ NoallocGeom g) {
  constexpr int NS = num_slots(false);
  const int tile = blockIdx.x / g.runs, start = (blockIdx.x - tile * g.runs) * kAlgebraThreads;
  const TileDev t = noalloc_tile(g, tile);
  const int count = min(kAlgebraThreads, t.ex * t.ey * t.nz - start);
  if (count <= 0) return;
  // pull this CTA's scratch into L2 first, so the per-point loads below hit L2 instead of
  // waiting on DRAM: the 32-point blocks its points fall in are one contiguous run (every
  // block starts on a 16-byte boundary), in pieces of at most 4 KB
  const int lp0 = t.sbase + start;
  const int b0 = lp0 >> 5, nblk = ((lp0 + count - 1) >> 5) - b0 + 1;
  const char* pd = reinterpret_cast<const char*>(static_cast<const ST*>(a.scr) + (size_t)b0 * NS * 32);
  const uint32_t td = (uint32_t)nblk * NS * 32 * sizeof(ST);
  for (uint32_t off = 4096u * threadIdx.x; off < td; off += 4096u * kAlgebraThreads)
    prefetch_l2_bulk(pd + off, min(4096u, td - off));
  const bool valid = (int)threadIdx.x < count;
  const int lp = start + (valid ? threadIdx.x : 0), r = lp / t.ex, z = r / t.ey;
  const int i = 3 + t.i0 + (lp - r * t.ex), j = 3 + t.j0 + (r - z * t.ey), k = 3 + t.k0 + z;
  const ST* const scr = static_cast<const ST*>(a.scr);
  const bool face = face_points<RK_NONE, kFaceBatch<ST, RK_NONE>>(a, g.block, i, j, k, valid, [&](int l) {
    return GlobalScratch<ST>{scr + scr_index<NS>(0, __shfl_sync(0xffffffffu, t.sbase + lp, l))};
  });
  if (valid && !face)
    algebra_point_at<ST, RK_NONE>(a, g.block, i, j, k, GlobalScratch<ST>{scr + scr_index<NS>(0, t.sbase + lp)});
}

}  // namespace

extern "C" int b200bssn_rhs_noalloc(double* const* rhs_dev, const double* const* u_dev,
                                    const b200bssn_block* block, const b200bssn_params* prm,
                                    void* stream) {
  if (!rhs_dev || !u_dev || !block || !prm) return B200BSSN_ERR_INVALID_ARGUMENT;
  if (prm->precision != B200BSSN_FP64 && prm->precision != B200BSSN_MIXED)
    return B200BSSN_ERR_INVALID_ARGUMENT;
  for (int v = 0; v < kNumVars; ++v)
    if (!rhs_dev[v] || !u_dev[v]) return B200BSSN_ERR_INVALID_ARGUMENT;
  for (int a = 0; a < 3; ++a) {
    if (block->sz[a] < 13) return B200BSSN_ERR_BLOCK_TOO_SMALL;
    if (!(block->pmax[a] > block->pmin[a])) return B200BSSN_ERR_INVALID_ARGUMENT;
  }
  if (block->bflag >> 6) return B200BSSN_ERR_INVALID_ARGUMENT;
  const int64_t I0 = block->sz[0] - 6, I1 = block->sz[1] - 6, I2 = block->sz[2] - 6;
  const int64_t npts = I0 * I1 * I2;
  const int64_t tiles_x = (I0 + kTileX - 1) / kTileX, tiles_y = (I1 + kTileY - 1) / kTileY;
  const auto pieces = [](int64_t n, int64_t size) { return (n + size - 1) / size; };
  // (the limits of descriptor arrays that are gone; kept so that the same blocks are refused)
  const int64_t fewest = pieces(I2, kNoallocSlab);
  if (npts > kNoallocMaxPoints || fewest > 1024 || fewest * tiles_x * tiles_y > 4096 ||
      fewest * pieces(I0 * I1 * kNoallocSlab, kAlgebraThreads) > 2048)
    return B200BSSN_ERR_SIZE_LIMIT;

  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return B200BSSN_ERR_NO_DEVICE;
  }
  DeviceSetup setup;
  const int rc = setup_device(dev, &setup);
  if (rc != B200BSSN_OK) return rc;
  // as many slabs as fill the GPU with one wave of the 11 variables with second derivatives (6
  // CTAs per SM), but none below three planes (38^3: ten slabs)
  const int64_t columns = tiles_x * tiles_y;
  const int64_t slabs = std::max(fewest, std::min<int64_t>(I2 / 3, 6 * setup.sms / (columns * kKindVars[1])));
  const int64_t n_tiles = slabs * columns;
  NoallocGeom g;
  BlockDev& blk = g.block;
  blk.offset = block->offset;
  blk.bflag = block->bflag;
  for (int a = 0; a < 3; ++a) {
    blk.sz[a] = (int32_t)block->sz[a];
    blk.pmin[a] = block->pmin[a];
    blk.h[a] = (block->pmax[a] - block->pmin[a]) / (block->sz[a] - 1);  // rhs.cpp:144-146
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  g.tiles_x = (int)tiles_x;
  g.tiles_y = (int)tiles_y;
  g.slabs = (int)slabs;
  g.runs = (int)pieces(std::min<int64_t>(I0, kTileX) * std::min<int64_t>(I1, kTileY) * pieces(I2, slabs), kAlgebraThreads);

  DerivArgs da;
  AlgebraArgs aa;
  std::memset(&da, 0, sizeof(da));
  std::memset(&aa, 0, sizeof(aa));  // aa.rk.mode = RK_NONE: store the RHS
  for (int v = 0; v < kNumVars; ++v) {
    da.u[v] = u_dev[v];
    aa.u[v] = u_dev[v];
    aa.rhs[v] = rhs_dev[v];
  }
  da.scr = setup.addr;
  aa.scr = setup.addr;
  aa.prm64 = {(double)prm->lambda[0], (double)prm->lambda[1], (double)prm->lambda[2],
              (double)prm->lambda[3], prm->lambda_f[0], prm->lambda_f[1]};
  aa.prm32 = {(float)prm->lambda[0], (float)prm->lambda[1], (float)prm->lambda[2],
              (float)prm->lambda[3], (float)prm->lambda_f[0], (float)prm->lambda_f[1]};
  aa.eta_const = prm->eta_const;
  aa.eta_r0 = prm->eta_r0;
  aa.eta_damping_exp = prm->eta_damping_exp;
  aa.ko_sigma = prm->ko_sigma;

  const bool mixed = prm->precision == B200BSSN_MIXED;
  const bool closure = blk.bflag != 0;
  for (int k = 1; k >= 0; --k) {
    void* arg[] = {&da, &g};
    const void* fn = mixed ? derivs_kernel<float>(k == 1, closure) : derivs_kernel<double>(k == 1, closure);
    if (launch_deriv(fn, (int)n_tiles * kKindVars[k], arg, k == 0, s) != cudaSuccess) {
      cudaGetLastError();
      return B200BSSN_ERR_CUDA;
    }
  }
  const unsigned grid = (unsigned)(n_tiles * g.runs);
  if (mixed)
    noalloc_algebra<float><<<grid, kAlgebraThreads, 0, s>>>(aa, g);
  else
    noalloc_algebra<double><<<grid, kAlgebraThreads, 0, s>>>(aa, g);
  if (cudaGetLastError() != cudaSuccess) return B200BSSN_ERR_CUDA;
  return B200BSSN_OK;
}
