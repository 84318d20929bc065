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
// RK4 stages that read the accumulator: their outputs are held back in shared memory until the
// algebra is through, and the stage's update then follows for kUpdateBatch variables at a time.
// Done output by output, each waited for its own load of the accumulator, which no compiler may
// move ahead of the stores before it: an RK4 step on 64 blocks of 37^3 took 5.08 (MIXED) and 7.31
// ms (FP64) instead of 4.46 and 6.63.  (The first stage, which writes the accumulator only,
// gains nothing from it: 4.49 and 6.67 ms.)
__host__ __device__ constexpr bool held_back(int mode) { return mode == RK_MIDDLE || mode == RK_LAST; }
constexpr int kUpdateBatch = 8;
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
  // and the outputs that an RK4 stage holds back (held_back): in FP64 over the KO sums
  static __host__ __device__ constexpr int slots(int mode) { return kStaged + (kAll && held_back(mode) ? kNumVars : 0); }
  static __host__ __device__ constexpr size_t bytes_per_warp(int mode) { return (size_t)slots(mode) * kStageW * sizeof(ST); }
  static __host__ __device__ constexpr size_t smem_bytes(int mode) { return kWarps * bytes_per_warp(mode); }
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

template <typename ST, bool ALL, int SLOTS>
struct SharedScratch {
  static constexpr bool kHolds = true;
  ST* d;             // this lane's column: all slots, or the first 72 and the KO sums
  const ST* g;       // this lane's slot 0 in the scratch
  __device__ __forceinline__ ST dv(int s) const {
    return ALL ? d[deriv_slot(s) * kStageW] : (s < 72 ? d[s * kStageW] : __ldg(g + deriv_slot(s) * kStageW));
  }
  __device__ __forceinline__ double kov(int v) const { return (double)d[((ALL ? kKoSlot : 72) + v) * kStageW]; }
  // keeps output v of the algebra; the right-hand side that follows from it
  __device__ __forceinline__ void hold(int v, ST val, double sigma) const {
    if constexpr (ALL)
      d[(SLOTS + v) * kStageW] = val;
    else
      d[(72 + v) * kStageW] = __dadd_rn(val, __dmul_rn(sigma, kov(v)));
  }
  __device__ __forceinline__ double held(int v, double sigma) const {
    if constexpr (ALL)
      return __dadd_rn((double)d[(SLOTS + v) * kStageW], __dmul_rn(sigma, kov(v)));
    else
      return d[(72 + v) * kStageW];
  }
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
struct StageIn { double base, acc; };  // what the update reads: u^n and the accumulator
template <int MODE>
__device__ __forceinline__ StageIn stage_in(const AlgebraArgs& a, int v, int64_t pp) {
  StageIn in{};
  if constexpr (MODE == RK_FIRST || MODE == RK_MIDDLE) in.base = __ldg(a.rk.base[v] + pp);
  if constexpr (MODE == RK_LAST) in.base = a.rk.base[v][pp];
  if constexpr (MODE == RK_MIDDLE || MODE == RK_LAST) in.acc = a.rk.acc[v][pp];
  return in;
}
template <int MODE>
__device__ __forceinline__ void store_rhs(const AlgebraArgs& a, int v, int64_t pp, double k, const StageIn& in) {
  const RkStage& rk = a.rk;
  if constexpr (MODE == RK_LAST) {
    rk.base[v][pp] = in.base + in.acc + rk.w * k;
  } else if constexpr (MODE == RK_FIRST) {
    rk.acc[v][pp] = rk.w * k;
    rk.next[v][pp] = in.base + rk.c * k;
  } else if constexpr (MODE == RK_MIDDLE) {
    rk.acc[v][pp] = in.acc + rk.w * k;
    rk.next[v][pp] = in.base + rk.c * k;
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
    if constexpr (held_back(MODE) && Src::kHolds)
      src.hold(v, val, a->ko_sigma);
    else
      store_rhs<MODE>(*a, v, pp, __dadd_rn((double)val, __dmul_rn(a->ko_sigma, src.kov(v))), stage_in<MODE>(*a, v, pp));
  }
};

__device__ __forceinline__ void prefetch_l2_bulk(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool on_flagged_face(const BlockDev& B, int i, int j, int k) {
  const uint32_t bf = B.bflag;
  return ((bf & 1u) && i == 3) || ((bf & 2u) && i == B.sz[0] - 4) || ((bf & 4u) && j == 3) ||
         ((bf & 8u) && j == B.sz[1] - 4) || ((bf & 16u) && k == 3) || ((bf & 32u) && k == B.sz[2] - 4);
}

// coordinates as bssnrhs forms them (pmin + i*h, two roundings, rhs.cpp:207-213)
struct PointPos {
  double x, y, z, r2;
};
__device__ __forceinline__ PointPos point_pos(const BlockDev& B, int i, int j, int k) {
  const double x = __dadd_rn(B.pmin[0], __dmul_rn((double)i, B.h[0]));
  const double y = __dadd_rn(B.pmin[1], __dmul_rn((double)j, B.h[1]));
  const double z = __dadd_rn(B.pmin[2], __dmul_rn((double)k, B.h[2]));
  return {x, y, z, __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z))};
}

// The face planes of a warp's points: bssn_bcs (rhs.cpp:833-977) replaces the algebra there,
// KO is added afterwards (rhs.cpp:323-369).  The whole warp calls it, each lane with its own
// point (`valid`: it has one); `at(l)` is the scratch of lane l's point.  Returns whether
// the lane's point lies on a face, and so is done.
// A row meets the two x faces with one point each, so nearly every warp of a flagged block has
// one such lane, and its 24 variables one after another -- a load from L2 and a chain of
// FP64 operations each -- took as long as the algebra of all the others.  The (face point,
// variable) pairs are therefore shared out over the lanes, BATCH of them in flight per lane.
// Per evaluation of 64 blocks of 37^3 with all faces flagged (1.9 M points) the algebra took
// 0.91 ms (MIXED) and 1.19 ms (FP64) with each lane looping over its own variables, 0.43 and
// 0.69 ms without faces; so shared out 0.49 and 0.76 ms.
// In FP64, at 255 registers, what a batch holds is paid for in spills of the whole kernel: with
// batches of four the RK4 stages spilled 144-268 bytes per thread, with one 24-48; the plain
// right-hand side 72, with two 40; the upwind mode 376, with two 312.  An RK4 step on 50 blocks
// of 37^3 takes 7 % less with batches of one than of four (6 % with all faces flagged), a
// right-hand side 4 % less with batches of two.
template <typename ST, int MODE>
constexpr int kFaceBatch = sizeof(ST) == 4 ? 4 : (MODE == RK_NONE ? 2 : 1);
template <int MODE, int BATCH, class At>
__device__ __forceinline__ bool face_points(const AlgebraArgs& a, const BlockDev& B, int i, int j, int k, bool valid,
                                            const At& at) {
  if (B.bflag == 0) return false;
  const bool mine = valid && on_flagged_face(B, i, j, k);
  const uint32_t mask = __ballot_sync(0xffffffffu, mine);
  if (mask == 0) return false;
  const int lane = threadIdx.x & 31, n = __popc(mask);
  // the lane of face point `lane`
  int owner = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1)
    if (__popc(mask & ((1u << (owner + step)) - 1u)) <= lane) owner += step;
  const PointPos P = point_pos(B, i, j, k);
  const double inv_r = mine ? 1.0 / sqrt(P.r2) : 0.0;
  const int64_t pp = B.offset + i + (int64_t)B.sz[0] * (j + (int64_t)B.sz[1] * k);
  const int dv = 32 / n, dq = 32 - dv * n;
  int v = lane / n, q = lane - v * n;  // this lane's variable and face point
  for (int pass = 0; pass < (kNumVars * n + 31) / 32; pass += BATCH) {
    int va[BATCH], from[BATCH];
    int64_t pa[BATCH];
    double f[BATCH], d[BATCH][3], ko[BATCH];
    StageIn in[BATCH];
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      from[b] = __shfl_sync(0xffffffffu, owner, q);
      pa[b] = __shfl_sync(0xffffffffu, pp, from[b]);
      const auto src = at(from[b]);
      va[b] = v;
      if (v < kNumVars) {
        f[b] = __ldg(a.u[v] + pa[b]);
        in[b] = stage_in<MODE>(a, v, pa[b]);
#pragma unroll
        for (int x = 0; x < 3; ++x) d[b][x] = (double)src.dv(3 * v + x);
        ko[b] = src.kov(v);
      }
      v += dv;
      q += dq;
      if (q >= n) q -= n, ++v;
    }
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const double x = __shfl_sync(0xffffffffu, P.x, from[b]), y = __shfl_sync(0xffffffffu, P.y, from[b]);
      const double z = __shfl_sync(0xffffffffu, P.z, from[b]), ir = __shfl_sync(0xffffffffu, inv_r, from[b]);
      if (va[b] < kNumVars) {
        double t = __dmul_rn(x, d[b][0]);
        t = __dadd_rn(t, __dmul_rn(y, d[b][1]));
        t = __dadd_rn(t, __dmul_rn(z, d[b][2]));
        t = __dadd_rn(t, __dmul_rn(bc_falloff(va[b]), __dsub_rn(f[b], bc_asymptotic(va[b]))));
        const double val = __dmul_rn(-ir, t);
        store_rhs<MODE>(a, va[b], pa[b], __dadd_rn(val, __dmul_rn(a.ko_sigma, ko[b])), in[b]);
      }
    }
  }
  return mine;
}

// The right-hand side of interior point (i, j, k) (padded coordinates) of block B, off its
// flagged faces, inputs through `src`.
template <typename RT, int MODE, class Src, bool ADV = false>
__device__ __forceinline__ void algebra_point_at(const AlgebraArgs& a, const BlockDev& B, int i, int j,
                                                 int k, const Src& src) {
  const int64_t pp = B.offset + i + (int64_t)B.sz[0] * (j + (int64_t)B.sz[1] * k);
  const double r2 = point_pos(B, i, j, k).r2;
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
  } else if constexpr (sizeof(RT) == 8) {
    // FP64: the algebra in two parts (the six At_rhs with the Ricci tensor, then the
    // rest), each with its own live set: the opaque offset between them keeps the compiler from
    // holding values of the first for the second.  At 255 registers what spills -- 40 bytes --
    // counts: shared memory leaves little L1, and the same kernel with 72 and 340 bytes took
    // 1.36 and 1.60 instead of 1.32 ms on 16 blocks of 69^3
    RhsAlgebraPart<0>::run<RT>(in, sink, *prm, (RT)eta);
    asm volatile("" : "+l"(in.pp));
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
  ST* sd = reinterpret_cast<ST*>(s_stage + warp * Cfg::bytes_per_warp(MODE));
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(sd)) + 16u * (uint32_t)lane;
  const int nwarps = gridDim.x * Cfg::kWarps;
  // Neighbouring tasks share state and scratch lines and go to one CTA; fewer tasks than warps
  // are spread over the SMs first.  From one round of tasks to the next every warp's place moves
  // on by one: tasks with face points take longer and recur with the rows, and at the same place
  // half of the warps could meet nearly all of them (135^3, MIXED, all faces flagged, where
  // they recur every 34 tasks: a call took 4 % longer).
  int place = ntasks < nwarps ? warp * gridDim.x + blockIdx.x : blockIdx.x * Cfg::kWarps + warp;
  for (int round = 0; round < ntasks; round += nwarps, place = place + 1 < nwarps ? place + 1 : 0) {
    const int task = round + place;
    if (task >= ntasks) continue;
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
      // (FP64, bound by memory, leaves out groups without points: their first lane has none)
      const int piece = lane % kPieces, from = piece * (32 / kPieces) / kGroup * kGroup;
      const int lp = __shfl_sync(0xffffffffu, p.lp, from) + piece * (32 / kPieces) % kGroup;
      const bool any = Cfg::kAll || __shfl_sync(0xffffffffu, p.valid, from);
      const uint64_t src = reinterpret_cast<uint64_t>(scr + scr_index<NS>(lane / kPieces, lp));
      constexpr int kLead = Cfg::kAll ? NS : Cfg::kFirst;  // slots from slot 0 on
#pragma unroll 6
      for (int k = 0; k < (kLead + kPerPass - 1) / kPerPass; ++k)
        if (any && (kLead % kPerPass == 0 || k * kPerPass + lane / kPieces < kLead))
          cp_async16(dst + 512u * k, src + (uint64_t)k * (kPerPass * 32 * sizeof(ST)));
      if constexpr (!Cfg::kAll) {
#pragma unroll 4
        for (int k = 0; k < kNumVars / kPerPass; ++k)
          if (any) cp_async16(dst + 512u * (kLead / kPerPass + k), src + (uint64_t)(kKoSlot + k * kPerPass) * 32 * sizeof(ST));
        // the slots read from global memory, into L2: one sector per group and slot
        constexpr int kGroups = kStageW / kGroup;
        const ST* const pg = scr + scr_index<NS>(0, __shfl_sync(0xffffffffu, p.lp, lane % kGroups * kGroup));
        if (__shfl_sync(0xffffffffu, p.valid, lane % kGroups * kGroup)) {
          for (int k = Cfg::kFirst + lane / kGroups; k < kNumDerivs; k += 32 / kGroups) prefetch_l2(pg + k * 32);
          if constexpr (ADV)
            for (int k = kAdvSlot + lane / kGroups; k < NS; k += 32 / kGroups) prefetch_l2(pg + k * 32);
        }
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();  // the copies of every lane are visible to the whole warp
    using Src = SharedScratch<ST, Cfg::kAll, Cfg::kStaged>;
    const bool face = face_points<MODE, kFaceBatch<ST, MODE>>(a, B, p.i, p.j, p.k, p.valid, [sd, own](int l) { return Src{sd + l, own}; });
    if (p.valid && !face) {
      const Src src{sd + lane, own};
      algebra_point_at<RT, MODE, Src, ADV>(a, B, p.i, p.j, p.k, src);
      if constexpr (held_back(MODE)) {
#pragma unroll 1
        for (int v0 = 0; v0 < kNumVars; v0 += kUpdateBatch) {
          StageIn in[kUpdateBatch];
#pragma unroll
          for (int b = 0; b < kUpdateBatch; ++b) in[b] = stage_in<MODE>(a, v0 + b, pp);
#pragma unroll
          for (int b = 0; b < kUpdateBatch; ++b) store_rhs<MODE>(a, v0 + b, pp, src.held(v0 + b, a.ko_sigma), in[b]);
        }
      }
    }
  }
}

}  // namespace b200bssn
