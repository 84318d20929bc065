// The algebra stage of one right-hand-side evaluation of a chunk of blocks: per interior
// point the generated BSSN algebra (or, on a flagged face plane, the Sommerfeld value of
// bssn/src/rhs.cpp:833-977), plus sigma times the KO sum (bssn/src/rhs.cpp:332-369),
// written to the RHS arrays -- or, in an RK4 stage, folded straight into the stage update
// (see RkStage) so the RHS never goes to memory.  The derivatives come from the scratch
// that the derivative stage (deriv_kernels.cuh) wrote.
//
// bssn_algebra_staged_kernel: persistent warps reading their points' scratch from shared
// memory.  (The allocation-free entry point has a kernel of its own around the same algebra.)
#pragma once
#include <stdint.h>

#include "deriv_kernels.cuh"
#include "generated/bssn_rhs_algebra.cuh"
#include "generated/bssn_rhs_algebra_adv.cuh"
#include "generated/bssn_rhs_algebra_split.cuh"
#include "plan_types.h"

namespace b200bssn {

// Staged algebra kernel geometry: 32-point tasks (one warp each); a warp's buffer
// holds its task's staged slots, 32 values per slot.  MIXED stages all slots in FP32
// (20,736 B), 4 warps per CTA, 2 CTAs per SM (the register limit of the 254-register
// algebra).  FP64 stages the 72 first derivatives and the KO sums (24,576 B) and reads the 66
// second derivatives, which the Ricci stage and the outputs use, from global memory
// after an L2 prefetch: one-warp CTAs, 8 per SM (the register limit; staging all 138 slots
// fitted only 5).  In the upwind mode (ADV) the scratch also holds the 72 advective
// derivatives: MIXED stages them too (2 warps per CTA, 3 CTAs per SM), FP64 reads them from
// global memory like the second derivatives.
constexpr int kStageW = 32;
template <typename ST, bool ADV = false>
struct StageCfg {
  static constexpr int kSlots = num_slots(ADV);  // 234 / 162
  // slots copied to shared memory: all in MIXED; in FP64 the first kFirst and the KO sums (the
  // rest, prefetched into L2, is read from global memory), so 8 warps fit per SM
  static constexpr bool kAll = sizeof(ST) == 4;
  static constexpr int kFirst = 72;
  static constexpr int kStaged = kAll ? kSlots : kFirst + kNumVars;
  static constexpr int kWarps = sizeof(ST) == 4 ? (ADV ? 2 : 4) : 1;
  static constexpr int kThreads = 32 * kWarps;
  static constexpr int kMinBlocks = sizeof(ST) == 4 ? (ADV ? 3 : 2) : 8;
  static constexpr size_t kBytesPerWarp = (size_t)kStaged * kStageW * sizeof(ST);
  static constexpr size_t kSmemBytes = kWarps * kBytesPerWarp;
};

struct AlgebraArgs {
  const double* u[kNumVars];
  double* rhs[kNumVars];
  RkStage rk;
  const BlockDev* blocks;
  const SlabDev* slabs;
  const RangeDev* ranges;
  const void* scr;
  int32_t range_base;
  AlgebraParams<double> prm64;
  AlgebraParams<float> prm32;
  double eta_const, eta_r0, eta_damping_exp, ko_sigma;
};

// Sommerfeld falloff / asymptotic value per VAR index (bssn/src/rhs.cpp:263-318).
__device__ __forceinline__ double bc_falloff(int v) {
  return (v >= 3 && v <= 5) || v >= 18 ? 2.0 : 1.0;
}
__device__ __forceinline__ double bc_asymptotic(int v) {
  return (v == 0 || v == 1 || v == 12 || v == 15 || v == 17) ? 1.0 : 0.0;
}

// Where an algebra thread reads its point's slots: from a copy its warp staged in shared
// memory (one 32-point column per slot), some from the scratch in global memory.
// Derivative s of the algebra's numbering (72 first, 66 second, 72 advective); KO sums.
__device__ __forceinline__ int deriv_slot(int s) { return s < kNumDerivs ? s : s + kNumVars; }

template <typename ST, bool ALL>
struct SharedScratch {
  const ST* d;       // this lane's column: all slots, or the first 72 and the KO sums
  const ST* g;       // this lane's slot 0 in the scratch
  __device__ __forceinline__ ST dv(int s) const {
    return ALL ? d[deriv_slot(s) * kStageW] : (s < 72 ? d[s * kStageW] : __ldg(g + deriv_slot(s) * kStageW));
  }
  __device__ __forceinline__ double kov(int v) const { return (double)d[((ALL ? kKoSlot : 72) + v) * kStageW]; }
};

template <typename RT, class Src>
struct PointIn {
  const AlgebraArgs* a;
  int64_t pp;   // element index of the point in the variable arrays
  Src src;
  __device__ __forceinline__ RT u(int v) const { return (RT)__ldg(a->u[v] + pp); }
  __device__ __forceinline__ RT d(int s) const { return (RT)src.dv(s); }
};

// Stores the right-hand side k of variable v at element pp: to the RHS arrays
// (MODE RK_NONE) or through one RK4 stage update.  The mode is a template
// parameter so each instantiation is straight-line code: a run-time branch per
// output splits the generated algebra into basic blocks the scheduler cannot
// interleave across (measured: the algebra kernel ran 2x slower).
template <int MODE>
__device__ __forceinline__ void store_rhs(const AlgebraArgs& a, int v, int64_t pp, double k) {
  const RkStage& rk = a.rk;
  if constexpr (MODE == RK_LAST) {
    rk.base[v][pp] = rk.base[v][pp] + rk.acc[v][pp] + rk.w * k;
  } else if constexpr (MODE == RK_FIRST) {
    rk.acc[v][pp] = rk.w * k;
    rk.next[v][pp] = __ldg(rk.base[v] + pp) + rk.c * k;
  } else if constexpr (MODE == RK_MIDDLE) {
    rk.acc[v][pp] = rk.acc[v][pp] + rk.w * k;
    rk.next[v][pp] = __ldg(rk.base[v] + pp) + rk.c * k;
  } else {
    a.rhs[v][pp] = k;
  }
}

template <int MODE, class Src>
struct PointSink {
  const AlgebraArgs* a;
  int64_t pp;
  Src src;
  template <typename RT>
  __device__ __forceinline__ void put(int v, RT val) {
    // rhs += sigma * (ko_x + ko_y + ko_z), rounded as rhs.cpp:332-369 rounds it
    store_rhs<MODE>(*a, v, pp, __dadd_rn((double)val, __dmul_rn(a->ko_sigma, src.kov(v))));
  }
};

__device__ __forceinline__ void prefetch_l2_bulk(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// FP64 algebra as the two-part split of bssn_rhs_algebra_split.cuh
constexpr bool kSplitAlgebra64 = true;

// The right-hand side of interior point (i, j, k) (padded coordinates) of block B,
// inputs through `src`.
template <typename RT, int MODE, class Src, bool ADV = false>
__device__ __forceinline__ void algebra_point_at(const AlgebraArgs& a, const BlockDev& B, int i, int j,
                                                 int k, const Src& src) {
  const int nx = B.sz[0], ny = B.sz[1];
  const int64_t pp = B.offset + i + (int64_t)nx * (j + (int64_t)ny * k);
  // coordinates as bssnrhs forms them (pmin + i*h, two roundings, rhs.cpp:207-213)
  const double x = __dadd_rn(B.pmin[0], __dmul_rn((double)i, B.h[0]));
  const double y = __dadd_rn(B.pmin[1], __dmul_rn((double)j, B.h[1]));
  const double z = __dadd_rn(B.pmin[2], __dmul_rn((double)k, B.h[2]));
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
  const uint32_t bf = B.bflag;
  const bool on_face = ((bf & 1u) && i == 3) || ((bf & 2u) && i == nx - 4) ||
                       ((bf & 4u) && j == 3) || ((bf & 8u) && j == ny - 4) ||
                       ((bf & 16u) && k == 3) || ((bf & 32u) && k == B.sz[2] - 4);
  if (on_face) {
    // bssn_bcs (rhs.cpp:833-977) replaces the algebra on face planes; KO is added
    // afterwards (rhs.cpp:323-369).
    const double inv_r = 1.0 / sqrt(r2);
#pragma unroll 1
    for (int v = 0; v < kNumVars; ++v) {
      const double f = __ldg(a.u[v] + pp);
      const double dxf = (double)src.dv(3 * v + 0);
      const double dyf = (double)src.dv(3 * v + 1);
      const double dzf = (double)src.dv(3 * v + 2);
      double t = __dmul_rn(x, dxf);
      t = __dadd_rn(t, __dmul_rn(y, dyf));
      t = __dadd_rn(t, __dmul_rn(z, dzf));
      t = __dadd_rn(t, __dmul_rn(bc_falloff(v), __dsub_rn(f, bc_asymptotic(v))));
      const double val = __dmul_rn(-inv_r, t);
      store_rhs<MODE>(a, v, pp, __dadd_rn(val, __dmul_rn(a.ko_sigma, src.kov(v))));
    }
    return;
  }
  // eta damping, rhs.cpp:213-219
  const double r_coord = sqrt(r2);
  double eta = a.eta_const;
  if (r_coord >= a.eta_r0) eta *= pow(a.eta_r0 / r_coord, a.eta_damping_exp);

  PointIn<RT, Src> in{&a, pp, src};
  PointSink<MODE, Src> sink{&a, pp, src};
  const AlgebraParams<RT>* prm;
  if constexpr (sizeof(RT) == 8)
    prm = &a.prm64;
  else
    prm = &a.prm32;
  if constexpr (ADV) {
    bssn_rhs_algebra_adv<RT>(in, sink, *prm, (RT)eta);
  } else if constexpr (sizeof(RT) == 8 && kSplitAlgebra64) {
    // FP64: the algebra in two parts (the six At_rhs with the Ricci tensor, then the
    // rest), each with its own live set
    RhsAlgebraPart<0>::run<RT>(in, sink, *prm, (RT)eta);
    RhsAlgebraPart<1>::run<RT>(in, sink, *prm, (RT)eta);
  } else {
    bssn_rhs_algebra<RT>(in, sink, *prm, (RT)eta);
  }
}

__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Staged algebra kernel: persistent warps, each taking 32-point tasks (slab_point)
// round-robin.  A task first copies its points' slots into the
// warp's shared-memory buffer with 16-byte cp.async -- lane l always the same piece of the 32
// points, of every second (FP64) or fourth (MIXED) slot, so its addresses step by a
// constant -- and prefetches the 24 state values into L2, then runs the algebra reading
// shared memory: the loads that kept the one-CTA-per-range version waiting on L2/DRAM become
// shared-memory loads, and while one warp waits for its copies the others compute.
template <typename ST, int MODE, bool ADV = false>
__global__ void __launch_bounds__(StageCfg<ST, ADV>::kThreads, StageCfg<ST, ADV>::kMinBlocks)
bssn_algebra_staged_kernel(const __grid_constant__ AlgebraArgs a, int ntasks) {
  using Cfg = StageCfg<ST, ADV>;
  using RT = ST;  // FP32 algebra in MIXED, FP64 in FP64
  constexpr int NS = Cfg::kSlots;
  constexpr int kPieces = kStageW * (int)sizeof(ST) / 16;            // 16-byte pieces of 32 values: 16 / 8
  constexpr int kPerPass = 32 / kPieces;                             // slots copied per instruction: 2 / 4
  extern __shared__ __align__(16) unsigned char s_stage[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ST* sd = reinterpret_cast<ST*>(s_stage + warp * Cfg::kBytesPerWarp);
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(sd)) + 16u * (uint32_t)lane;
  const int nwarps = gridDim.x * Cfg::kWarps;
  for (int task = blockIdx.x * Cfg::kWarps + warp; task < ntasks; task += nwarps) {
    const RangeDev rg = a.ranges[a.range_base + task / kRangeTasks];
    if ((task & (kRangeTasks - 1)) >= rg.count) continue;
    const SlabDev slab = a.slabs[rg.slab];
    const BlockDev& B = a.blocks[slab.block];
    const SlabPoint p = slab_point(B, slab, rg.start + (task & (kRangeTasks - 1)), lane);
    const int64_t pp = B.offset + p.i + (int64_t)B.sz[0] * (p.j + (int64_t)B.sz[1] * p.k);
    if (p.valid) {
#pragma unroll
      for (int v = 0; v < kNumVars; ++v) prefetch_l2(a.u[v] + pp);
      if constexpr (MODE == RK_MIDDLE || MODE == RK_LAST) {
        // the stage update reads u^n and the accumulator at every output
#pragma unroll
        for (int v = 0; v < kNumVars; ++v) {
          prefetch_l2(a.rk.base[v] + pp);
          prefetch_l2(a.rk.acc[v] + pp);
        }
      }
    }
    const ST* const scr = static_cast<const ST*>(a.scr);
    const ST* const own = scr + scr_index<NS>(0, p.lp);
    __syncwarp();  // every lane is done reading the previous task's buffer
    {
      // piece lane % kPieces of the 32 points: group piece * 8 / kPieces, its first or second half
      const int piece = lane % kPieces;
      const int lp = __shfl_sync(0xffffffffu, p.lp, piece * (32 / kPieces) / kGroup * kGroup) + piece * (32 / kPieces) % kGroup;
      const uint64_t src = reinterpret_cast<uint64_t>(scr + scr_index<NS>(lane / kPieces, lp));
      constexpr int kLead = Cfg::kAll ? NS : Cfg::kFirst;  // slots from slot 0 on
#pragma unroll 6
      for (int k = 0; k < (kLead + kPerPass - 1) / kPerPass; ++k)
        if (kLead % kPerPass == 0 || k * kPerPass + lane / kPieces < kLead)
          cp_async16(dst + 512u * k, src + (uint64_t)k * (kPerPass * 32 * sizeof(ST)));
      if constexpr (!Cfg::kAll) {
#pragma unroll 4
        for (int k = 0; k < kNumVars / kPerPass; ++k)
          cp_async16(dst + 512u * (kLead / kPerPass + k), src + (uint64_t)(kKoSlot + k * kPerPass) * 32 * sizeof(ST));
        // the slots read from global memory, into L2: one sector per group and slot
        constexpr int kGroups = kStageW / kGroup;
        const ST* const pg = scr + scr_index<NS>(0, __shfl_sync(0xffffffffu, p.lp, lane % kGroups * kGroup));
        for (int k = Cfg::kFirst + lane / kGroups; k < kNumDerivs; k += 32 / kGroups) prefetch_l2(pg + k * 32);
        if constexpr (ADV)
          for (int k = kAdvSlot + lane / kGroups; k < NS; k += 32 / kGroups) prefetch_l2(pg + k * 32);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();  // the copies of every lane are visible to the whole warp
    if (p.valid) {
      using Src = SharedScratch<ST, Cfg::kAll>;
      const Src src{sd + lane, own};
      algebra_point_at<RT, MODE, Src, ADV>(a, B, p.i, p.j, p.k, src);
    }
  }
}

}  // namespace b200bssn
