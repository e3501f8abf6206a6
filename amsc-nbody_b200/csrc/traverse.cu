// traverse.cu -- Barnes-Hut force evaluation on sm_100a.
//
//  traverse_fp64_kernel   plain form of barnes_hut.cu:164-322 (paths relative
//                         to the sytrams/AMSC-Nbody project root): per-target
//                         acceptance test and interaction order identical to
//                         the reference, FP64 throughout.
//  traverse_mixed_kernel  mixed form: warp-group acceptance test, shared
//                         interaction lists evaluated in FP32.
//  direct_kernel          FP64 direct summation (theta-error oracle).
//  ref_octree_kernel      traversal of a caller octree in the reference's own
//                         node numbering (function-level API).
//  kick / kick_drift      integrator.cu:51-106.
#include "nbb_internal.cuh"
#include "walk_fp64.cuh"
#include "walk_list.cuh"

#include <algorithm>
#include <climits>
#include <cmath>

namespace nbb {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ long long warp_sum_ll(long long v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Plain FP64 traversal on the ordered interaction lists of walk_list.cuh, for
// sets of at most kTargets Morton-consecutive targets.  Every target sees its
// own node sequence of the reference's stackless walk (barnes_hut.cu:90-162):
// a list entry counts for a target when its preorder index has reached the
// target's resume index, and an undecided cell that the target accepts moves
// that index past the cell's subtree.
//
// With 32 targets a lane holds one target and the warp takes the entries in
// order, four in flight.  With one target the 32 lanes form the terms of 32
// consecutive entries at once; the terms are then added in entry order, each
// component's sum by one lane, so the result has the same bits.  One target
// per set wastes the walk on a single target but fills the GPU from small
// systems (see fp64_targets).
//
// With kPair a set is two warps' work: one walks and fills the list, the other
// evaluates it, with two buffers between them.  That is for systems whose sets
// all run at once, where the time is that of one set: its round trips and its
// FP64 chains then overlap (walk at 2000, 12000, 24000 particles 120, 540, 582
// us by one warp, 86, 348, 390 by two; alike at 65536).  Where sets wait for
// warps, a warp for each has the FP64 pipe busier: 10.7 against 11.9 ms at 2^20
// (see pair_sets).
//
// Bound at 2^20 particles: instruction issue and FP64 latency (FP64 pipe 49 %,
// issue 61 % busy at 16 warps per SM; an entry takes 23 FP64 operations of
// 2.2 cycles).  16 warps with 128 registers, four entries in flight, beat 20
// warps of 96 registers and 24 of 80 (10.7, 11.8 and 12.4 ms).
constexpr int kFp64Warps = 2;  // sets of a block, one warp each
constexpr int kFp64Pairs = 4;  // sets of a block, two warps each: w walks, w + 4 evaluates (one of each per SM quarter)
template <bool kPair>
__host__ __device__ constexpr int fp64_threads() {
  return kPair ? 64 * kFp64Pairs : 32 * kFp64Warps;
}

// One warp's targets and their sums.
template <int kTargets>
struct Fp64Targets {
  int s, resume;
  unsigned count;  // interactions
  bool valid, in_range, singular = false;
  double4 t;
  double soft2, ax, ay, az;

  // set g0 .. g1 - 1
  __device__ __forceinline__ void load(const Workspace &ws, const TraversalParams &p, int g0, int g1, int sys) {
    s = g0 + ((threadIdx.x & 31) & (kTargets - 1));
    valid = s < g1;
    t = ws.pm4[valid ? s : g0];
    const double soft = ws.sys_eps ? ws.sys_eps[sys] : p.soft;
    soft2 = __dmul_rn(soft, soft);
    // no squared distance of the system leaves inv_sqrt_core's range; without
    // softening each is looked at
    in_range = soft2 > 0x1p-900 && soft2 < 0x1p900 && ws.sys_box[4 * sys + 3] < 0x1p400;
    resume = valid ? 0 : INT_MAX;
    ax = ay = az = 0.0;
    count = 0;
  }

  // Entries [0, n) of the list for 32 targets.  kLook: a squared distance may
  // leave inv_sqrt_core's range (no softening, or extreme units), so each is
  // looked at.  A loop of its own: the look as a branch inside one loop slows
  // the softened form by 4 %.  Step of 2^20 particles: 11.1 ms softened, 12.2
  // without softening (20.5 with the general form for every term).
  template <bool kLook, int kCap>
  __device__ __forceinline__ void eval_sets(const Workspace &ws, const ListBuffer<kCap> &list, int n) {
    for (int j = 0; j < n; j += 4) {
      double dx[4], dy[4], dz[4], r2[4], f[4];
      int pre[4], aux[4];
      bool act[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double4 v = list.src[j + q];
        const int2 tag = list.tag[j + q];
        pre[q] = tag.x;
        aux[q] = tag.y;
        dx[q] = __dsub_rn(v.x, t.x);
        dy[q] = __dsub_rn(v.y, t.y);
        dz[q] = __dsub_rn(v.z, t.z);
        f[q] = v.w;
        r2[q] = sqdist(dx[q], dy[q], dz[q]);
        act[q] = pre[q] >= resume && aux[q] != s;
      }
      if (min(min(aux[0], aux[1]), min(aux[2], aux[3])) < -1) {
        // undecided cells: a target that accepts one resumes past it
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          act[q] = act[q] && pre[q] >= resume;
          if (aux[q] < -1) {
            act[q] = act[q] && accept_entry(list, j + q, ws, pre[q], t, r2[q]);
            if (act[q]) resume = -aux[q];
          }
        }
      }
      // all terms are formed before any is added; the sums take them in
      // the reference's order
      bool plain = kLook || in_range;  // inv_sqrt_core gets every term right
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        r2[q] = __dadd_rn(r2[q], soft2);
        plain = plain && inv_sqrt_low_word(r2[q]);
      }
      if constexpr (kLook) {
#pragma unroll
        for (int q = 0; q < 4; ++q) plain = plain && (!act[q] || inv_sqrt_in_range(r2[q]));
      }
      double inv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) inv[q] = inv_sqrt_core(r2[q]);
      if (!plain) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (kLook && (!act[q] || inv_sqrt_in_range(r2[q]))) continue;
          inv[q] = inv_sqrt_general(r2[q]);
          if (act[q] && r2[q] <= 0.0) {
            singular = true;
            act[q] = false;
            ++count;
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) f[q] = __dmul_rn(f[q], __dmul_rn(__dmul_rn(inv[q], inv[q]), inv[q]));
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (act[q]) {
          ax = __fma_rn(f[q], dx[q], ax);
          ay = __fma_rn(f[q], dy[q], ay);
          az = __fma_rn(f[q], dz[q], az);
          ++count;
        }
    }
  }

  // Entries [0, n) of the list; returns the smallest resume index.  term:
  // room for each lane's offset and factor (one target only).
  template <int kCap>
  __device__ __forceinline__ int eval(const Workspace &ws, const ListBuffer<kCap> &list, int n, double4 *term) {
    const int lane = threadIdx.x & 31;
    if constexpr (kTargets == 32) {
      if (in_range)
        eval_sets<false>(ws, list, n);
      else
        eval_sets<true>(ws, list, n);
    } else {
      // lane (el, tl): entry el of each block of kLanes, target tl; lanes
      // el = 0, 1, 2 sum the x, y, z component (in ax)
      constexpr int kLanes = 32 / kTargets;  // lanes per target
      const int tl = lane & (kTargets - 1), el = lane / kTargets, comp = min(el, 2);
      for (int e0 = 0; e0 < n; e0 += kLanes) {
        const bool has = e0 + el < n;
        const int j = has ? e0 + el : e0;
        const double4 q = list.src[j];
        const int2 tg = list.tag[j];
        const double dx = __dsub_rn(q.x, t.x), dy = __dsub_rn(q.y, t.y), dz = __dsub_rn(q.z, t.z);
        const double d2 = sqdist(dx, dy, dz);
        const bool undecided = has && tg.y < -1;
        bool act = has && tg.x >= resume && tg.y != s;
        if (__any_sync(kFull, undecided)) {
          // the entries' decisions in order: each may move the resume
          // index of the target's later entries
          const bool take = act && (!undecided || accept_entry(list, j, ws, tg.x, t, d2));
          act = false;
          for (int e = 0; e < kLanes; ++e) {
            if (e == el) act = take && tg.x >= resume;
            const int moved = (act && undecided) ? -tg.y : resume;
            resume = __shfl_sync(kFull, moved, e * kTargets + tl);
          }
        }
        const double r2 = __dadd_rn(d2, soft2);
        double inv = inv_sqrt_core(r2);
        if (!inv_sqrt_in_range(r2)) inv = inv_sqrt_general(r2);
        const double f = __dmul_rn(q.w, __dmul_rn(__dmul_rn(inv, inv), inv));
        const bool zero = r2 <= 0.0;
        singular |= act && zero;
        count += act ? 1 : 0;
        // an idle lane's term is 0, which leaves a sum's bits alone
        const bool on = act && !zero;
        term[lane] = make_double4(on ? dx : 0.0, on ? dy : 0.0, on ? dz : 0.0, on ? f : 0.0);
        __syncwarp();
#pragma unroll
        for (int e = 0; e < kLanes; ++e) {
          const double *v = reinterpret_cast<const double *>(term + e * kTargets + tl);
          ax = __fma_rn(v[3], v[comp], ax);
        }
        __syncwarp();
      }
    }
    return __reduce_min_sync(kFull, resume);
  }

  // The accelerations, and the second half kick (integrator.cu:86-106).
  __device__ __forceinline__ void store(const Workspace &ws, const TraversalParams &p) const {
    if (!valid) return;
    const uint32_t ti = ws.idx[s];
    if constexpr (kTargets == 32) {
      ws.ax[ti] = ax;
      ws.ay[ti] = ay;
      ws.az[ti] = az;
      if (p.kick) {
        ws.vx[ti] = __fma_rn(p.half_dt, ax, ws.vx[ti]);
        ws.vy[ti] = __fma_rn(p.half_dt, ay, ws.vy[ti]);
        ws.vz[ti] = __fma_rn(p.half_dt, az, ws.vz[ti]);
      }
    } else {
      const int el = (threadIdx.x & 31) / kTargets;
      if (el >= 3) return;
      double *a = el == 0 ? ws.ax : (el == 1 ? ws.ay : ws.az);
      a[ti] = ax;
      if (p.kick) {
        double *v = el == 0 ? ws.vx : (el == 1 ? ws.vy : ws.vz);
        v[ti] = __fma_rn(p.half_dt, ax, v[ti]);
      }
    }
  }
};

// What a set's warp or pair of warps keeps in shared memory.
template <int kTargets, bool kPair>
struct Fp64Shared {
  static constexpr int kCap = kPair ? 64 : 96;
  Frontier walk;
  ListBuffer<kCap> list[kPair ? 2 : 1];
  double4 term[kTargets < 32 ? 32 : 1];
  int set[2], count[2], last[2], done[2];  // per buffer of a pair: see the kernel
};

// Named barriers of a pair: buffer b filled (kFilled + b), buffer b free (kFree
// + b); the two warps use each in turn, one arriving and one waiting.
constexpr int kFilled = 0, kFree = 2, kPairBarriers = 4;
static_assert(kFp64Pairs * kPairBarriers <= 16, "named barriers of a block");
__device__ __forceinline__ void pair_arrive(int id) {
  __syncwarp();
  asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void pair_wait(int id) {
  __syncwarp();
  asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}

template <int kTargets, bool kPair>
__global__ void __launch_bounds__(fp64_threads<kPair>(), kPair ? 2 : 8)
    traverse_fp64_kernel(Workspace ws, TraversalParams p) {
  using Shared = Fp64Shared<kTargets, kPair>;
  constexpr int kSets = kPair ? kFp64Pairs : kFp64Warps;
  __shared__ Shared shared[kSets];
  DevScalars *sc = ws.sc;
  // (one decision for the block: a pair's warps leave together)
  if (__syncthreads_or(sc->error != 0)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Shared &sh = shared[warp % kSets];
  const int n = ws.n;
  const int m = sc->n_nodes;
  const int n_sets = sc->n_tgroups;
  long long inter = 0, tests = 0;
  Fp64Targets<kTargets> targets;
  const auto bounds = [&](int set, int &g0, int &g1, int &sys) {
    g0 = ws.tstart[set];
    g1 = min(set + 1 < n_sets ? ws.tstart[set + 1] : n, g0 + kTargets);
    // a set's targets belong to one system: walk that system's subtree
    sys = ws.n_systems > 1 ? ws.psys[g0] : 0;
  };
  const auto next_set = [&]() {
    int set = 0;
    if (lane == 0) set = (int)atomicAdd(&sc->work_counter, 1u);
    return __shfl_sync(kFull, set, 0);
  };
  int g0, g1, sys;
  if constexpr (!kPair) {
    for (int set = next_set(); set < n_sets; set = next_set()) {
      bounds(set, g0, g1, sys);
      targets.load(ws, p, g0, g1, sys);
      set_target_box(sh.walk, targets.t, ws.sys_box[4 * sys + 3]);
      unsigned set_tests = 0;
      auto *list = &sh.list[0];
      ordered_walk(ws, m, ws.root_pre[sys], p.g, sh.walk, list, set_tests,
                   [&](int count, bool) { return targets.eval(ws, *list, count, sh.term); });
      tests += set_tests;
      inter += targets.count;
      targets.store(ws, p);
    }
  } else if (warp < kSets) {
    // the walking warp: a buffer is its own once the other warp has freed it
    const int filled = warp * kPairBarriers + kFilled, free = warp * kPairBarriers + kFree;
    int b = 0;
    auto *list = &sh.list[0];
    pair_wait(free);
    for (int set = next_set(); set < n_sets; set = next_set()) {
      bounds(set, g0, g1, sys);
      const int s = g0 + (lane & (kTargets - 1));
      set_target_box(sh.walk, ws.pm4[s < g1 ? s : g0], ws.sys_box[4 * sys + 3]);
      unsigned set_tests = 0;
      bool first = true;  // the other buffer holds no entries of this set yet
      const auto hand = [&](int count, bool last) {
        if (lane == 0) {
          sh.set[b] = set;
          sh.count[b] = count;
          sh.last[b] = last ? 1 : 0;
        }
        pair_arrive(filled + b);
        b ^= 1;
        list = &sh.list[b];
        pair_wait(free + b);
        const int done = first ? 0 : sh.done[b];
        first = false;
        return done;
      };
      ordered_walk(ws, m, ws.root_pre[sys], p.g, sh.walk, list, set_tests, hand);
      tests += set_tests;
    }
    if (lane == 0) sh.set[b] = -1;  // no more
    pair_arrive(filled + b);
    pair_wait(free + (b ^ 1));  // every arrival is met
  } else {
    // the evaluating warp
    const int filled = (warp - kSets) * kPairBarriers + kFilled, free = (warp - kSets) * kPairBarriers + kFree;
    pair_arrive(free);
    pair_arrive(free + 1);
    bool fresh = true;
    for (int b = 0;; b ^= 1) {
      pair_wait(filled + b);
      const int set = sh.set[b];
      if (set < 0) break;
      const bool last = sh.last[b] != 0;
      if (fresh) {
        bounds(set, g0, g1, sys);
        targets.load(ws, p, g0, g1, sys);
      }
      const int done = targets.eval(ws, sh.list[b], sh.count[b], sh.term);
      if (lane == 0) sh.done[b] = done;
      pair_arrive(free + b);
      fresh = last;
      if (!last) continue;
      inter += targets.count;
      targets.store(ws, p);
    }
  }
  if (__any_sync(kFull, targets.singular) && lane == 0) record_error(sc, kStageTraversal, 6);
  inter = warp_sum_ll(inter);
  tests = warp_sum_ll(tests);
  if (lane == 0) {
    if (inter) atomicAdd(&sc->interactions, (unsigned long long)inter);
    if (tests) atomicAdd(&sc->mac_tests, (unsigned long long)tests);
  }
}

// ------------------------------------------------------------ mixed ----

// Compile-time tuning of the mixed walk (warps per block, minimum resident
// blocks per SM for the register budget).
#ifndef NBB_MIXED_WARPS
#define NBB_MIXED_WARPS 2
#endif
#ifndef NBB_MIXED_MINBLOCKS
#define NBB_MIXED_MINBLOCKS 10
#endif
// resident blocks per SM for the two- and four-targets-per-lane instances
// (more registers per thread for the targets' sums)
#ifndef NBB_MIXED_MINBLOCKS2
#define NBB_MIXED_MINBLOCKS2 10
#endif
#ifndef NBB_MIXED_MINBLOCKS4
#define NBB_MIXED_MINBLOCKS4 7
#endif
constexpr int kMixedWarps = NBB_MIXED_WARPS;
constexpr int kWalkPop = 64;     // nodes per round: two per lane
constexpr int kStackCap = 1024;  // shared-memory part of a warp's stack
constexpr int kSpill = 512;      // entries moved to / from the global extension at once
// A spill starts above kStackCap - 7 kWalkPop entries and moves the bottom
// kSpill of them, so that threshold must hold at least kSpill entries (and
// the moved-down rest must end below kSpill, where the sources start).
static_assert(kStackCap - 7 * kWalkPop >= kSpill && kStackCap <= 2 * kSpill, "stack spill bounds");
// Entries per evaluated batch of the force walk: the list is evaluated when it
// holds this many, so each batch's set-up and compensated addition are paid
// once per kEvalBatch entries.  A batch's two chains of plain FP32 additions
// are half as long; 96 entries are 1 % faster (2^20 particles: 2.89 against
// 2.92 ms a step) and lose half as many terms again in a chain, so 64.  The
// walks that track sources (zero softening, the adjoint) keep 32-entry batches
// and the smaller list, whose shared memory keeps 10 blocks per SM.
#ifndef NBB_EVAL_BATCH
#define NBB_EVAL_BATCH 64
#endif
constexpr int kEvalBatch = NBB_EVAL_BATCH;
static_assert(kEvalBatch % 32 == 0 && kEvalBatch >= 32 && kEvalBatch <= 128, "batch of whole warps");
template <bool kTrackSource>
__host__ __device__ constexpr int batch_of() {
  return kTrackSource ? 32 : kEvalBatch;
}
// list capacity: < batch left over + 64 cells + up to 96 leaf particles
template <bool kTrackSource>
__host__ __device__ constexpr int list_cap_of() {
  return batch_of<kTrackSource>() + 160;
}

// The interaction list keeps entries in pairs so that packed two-wide FP32
// instructions (sm_100's FADD2 / FMUL2 / FFMA2) evaluate two entries at once
// from one 16-byte load per half: pair p holds entries 2p and 2p + 1 as
// a = {x0, x1, y0, y1} and b = {z0, z1, m0, m1}.
struct PairList {
  float4 *a, *b;
  __device__ __forceinline__ void put(int j, float x, float y, float z, float m) const {
    float *pa = reinterpret_cast<float *>(a + (j >> 1));
    float *pb = reinterpret_cast<float *>(b + (j >> 1));
    const int h = j & 1;
    pa[h] = x;
    pa[2 + h] = y;
    pb[h] = z;
    pb[2 + h] = m;
  }
};

// Warps of a block: kMixedWarps with a group each, or kSplit on one group.
template <int kSplit>
__host__ __device__ constexpr int mixed_warps() {
  return kSplit > 1 ? kSplit : kMixedWarps;
}
template <bool kTrackSource, int kWarps>
struct MixedShared {
  double gbox[kWarps][9];  // group box lo (3), hi (3), centre (3)
  float ghalf[kWarps][4];  // group box half extents, rounded up to FP32
  int stack[kWarps][kStackCap];
  float4 la[kWarps][list_cap_of<kTrackSource>() / 2];
  float4 lb[kWarps][list_cap_of<kTrackSource>() / 2];
  int src[kWarps][kTrackSource ? list_cap_of<kTrackSource>() : 1];
};

// Hardware approximate reciprocal square root (MUFU), subnormal inputs and
// results flushed to zero: r^2 + eps^2 of a force evaluation is never
// subnormal where it matters, and the flush saves the range fix-up that
// rsqrtf adds around the same instruction.
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Evaluate `count` list entries (rounded up to a whole pair; an odd count
// has a zero-mass pad after it) for this lane's kTPL targets: FP32 offsets,
// approximate rsqrt (no refinement), two-wide FP32 partial sums over
// the batch, then one Kahan-compensated addition of each batch partial into
// its running sum.
//
// With positive softening a target's own entry (a leaf particle equal to the
// target) has offset exactly (0, 0, 0) -- both offsets are rounded from the
// same FP64 difference -- and contributes exactly zero, so no source index is
// needed.  With zero softening the source index excludes self and detects
// the reference's singular interaction (returns true).
// Pairs per unrolled block of the evaluation loop, by the walk's target
// slots per lane (its register budget): 8 for one or two slots, 4 for four
// (8 spills there).
#ifndef NBB_EVAL_UNROLL
#define NBB_EVAL_UNROLL 8
#endif
#ifndef NBB_EVAL_UNROLL4
#define NBB_EVAL_UNROLL4 4
#endif
template <int kSlots>
__host__ __device__ constexpr int eval_unroll() {
  return kSlots >= 4 ? NBB_EVAL_UNROLL4 : NBB_EVAL_UNROLL;
}

template <bool kTrackSource, int kTPL, int kUnroll>
__device__ __forceinline__ bool eval_batch(const PairList &list, const int *src, int count, const int *self,
                                           const float2 *ntx, const float2 *nty, const float2 *ntz, float2 eps2,
                                           float3 *sum, float3 *comp) {
  float2 px[kTPL], py[kTPL], pz[kTPL];
#pragma unroll
  for (int q = 0; q < kTPL; ++q) px[q] = py[q] = pz[q] = make_float2(0.f, 0.f);
  bool singular = false;
  const int pairs = (count + 1) >> 1;
#pragma unroll kUnroll
  for (int pr = 0; pr < pairs; ++pr) {
    const float4 ea = list.a[pr], eb = list.b[pr];
    const float2 ex = make_float2(ea.x, ea.y), ey = make_float2(ea.z, ea.w);
    const float2 ez = make_float2(eb.x, eb.y), em = make_float2(eb.z, eb.w);
#pragma unroll
    for (int q = 0; q < kTPL; ++q) {
      const float2 dx = __fadd2_rn(ex, ntx[q]), dy = __fadd2_rn(ey, nty[q]), dz = __fadd2_rn(ez, ntz[q]);
      const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
      const float2 r = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
      // m r^-3 straight from the hardware estimate: its relative error (a few
      // 1e-7 on r^-3) sits far below the Barnes-Hut truncation error this
      // form is held to, and a Newton step would add 3 packed FP32 operations
      // to the 12 of a pair of entries
      const float2 rr = __fmul2_rn(r, r);
      float2 f = __fmul2_rn(__fmul2_rn(em, r), rr);
      if (kTrackSource) {
        const bool o0 = src[2 * pr] != self[q], o1 = src[2 * pr + 1] != self[q];
        singular |= (o0 && !(r2.x > 0.f) && em.x != 0.f) || (o1 && !(r2.y > 0.f) && em.y != 0.f);
        f.x = (o0 && r2.x > 0.f) ? f.x : 0.f;
        f.y = (o1 && r2.y > 0.f) ? f.y : 0.f;
      }
      px[q] = __ffma2_rn(f, dx, px[q]);
      py[q] = __ffma2_rn(f, dy, py[q]);
      pz[q] = __ffma2_rn(f, dz, pz[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < kTPL; ++q) {
    float y, t;
    y = (px[q].x + px[q].y) - comp[q].x; t = sum[q].x + y; comp[q].x = (t - sum[q].x) - y; sum[q].x = t;
    y = (py[q].x + py[q].y) - comp[q].y; t = sum[q].y + y; comp[q].y = (t - sum[q].y) - y; sum[q].y = t;
    y = (pz[q].x + pz[q].y) - comp[q].z; t = sum[q].z + y; comp[q].z = (t - sum[q].z) - y; sum[q].z = t;
  }
  return singular;
}

// Per-lane target state of the mixed walk: negated target offsets from the
// group centre, each duplicated into both halves of a pair.
template <int kTPL>
struct LaneTargets {
  int s[kTPL];
  bool valid[kTPL];
  float2 ntx[kTPL], nty[kTPL], ntz[kTPL];
  float3 sum[kTPL], comp[kTPL];
  long long inter = 0;
  bool singular = false;
};

// Evaluate `count` entries for the first nq (warp-uniform) of the lane's
// kTPL target slots: a group of g targets fills ceil(g / 32) slots, and the
// empty ones cost nothing (the branch is taken once per batch, outside the
// entry loop).
template <bool kTrackSource, int kTPL>
__device__ __forceinline__ bool eval_slots(const PairList &list, const int *src, int count, int nq,
                                           LaneTargets<kTPL> &t, float2 eps2) {
  if (kTPL >= 4 && nq >= 4)
    return eval_batch<kTrackSource, (kTPL >= 4 ? 4 : 1), eval_unroll<kTPL>()>(
        list, src, count, t.s, t.ntx, t.nty, t.ntz, eps2, t.sum, t.comp);
  if (kTPL >= 3 && nq == 3)
    return eval_batch<kTrackSource, (kTPL >= 3 ? 3 : 1), eval_unroll<kTPL>()>(
        list, src, count, t.s, t.ntx, t.nty, t.ntz, eps2, t.sum, t.comp);
  if (kTPL >= 2 && nq == 2)
    return eval_batch<kTrackSource, (kTPL >= 2 ? 2 : 1), eval_unroll<kTPL>()>(
        list, src, count, t.s, t.ntx, t.nty, t.ntz, eps2, t.sum, t.comp);
  return eval_batch<kTrackSource, 1, eval_unroll<kTPL>()>(list, src, count, t.s, t.ntx, t.nty, t.ntz, eps2, t.sum,
                                                          t.comp);
}

// ------------------------------------------------- mixed adjoint walk ----
//
// Vector-Jacobian product of the mixed form's force, on the mixed walk's own
// interaction lists (group-box acceptance, FP32 offsets from the group
// centre).  For target i, entry s (mass mu, offset r = Y_s - x_i) and the
// accelerations cotangent c_i (see adjoint.cu's file comment):
//   u = G mu (inv3 c_i - 3 inv5 (r . c_i) r),  d/dx_i -= u,  d/dY_s += u,
//   d/dmu_s += G inv3 (r . c_i),
// in FP32 with the hardware reciprocal square root.  A source's u is summed
// over the warp's targets before it is added (FP64 atomics) to the cell's or
// particle's cotangent; the list names each entry's source: a particle by its
// Morton slot, a cell by -3 - its level-order index.

// Cotangent state of the adjoint walk's target (one per lane).
struct LaneVjp {
  float cx = 0.f, cy = 0.f, cz = 0.f;  // accelerations cotangent
  double gx = 0.0, gy = 0.0, gz = 0.0;  // position cotangent (running)
};

// VJP of `count` list entries (a multiple of 8; pads have no mass) for the
// lane's target; returns true on a singular pair.
//
// Entries go two to a packed instruction, eight to a reduction over the warp.
// A lane takes the block's four pairs in an order permuted by its bits 4 and 3,
// so that in the butterfly's first two rounds every lane keeps its first
// registers and sends the others, without selects; then it ends with component
// lane & 3 of entry 2 * (lane >> 3) + (lane >> 2 & 1).  Bound by instruction issue
// (61 % of the slots, ~38 instructions per entry, 8 of them the reduction): the
// walk of 65536 particles takes 646 us, 876 with single entries and a
// reduction by selects.  Blocks of 8 to 10 per SM and batches of 32 to 96
// entries measured alike.
__device__ __forceinline__ bool vjp_entries(const PairList &list, const int *src, int count, int self, bool valid,
                                            float2 ntx, float2 nty, float2 ntz, LaneVjp &v, float2 eps2, float g,
                                            const AdjointBuffers &ab) {
  const int lane = threadIdx.x & 31, perm = lane >> 3;
  const bool b4 = lane & 4, b2 = lane & 2, b1 = lane & 1;
  const float2 cx = make_float2(v.cx, v.cx), cy = make_float2(v.cy, v.cy), cz = make_float2(v.cz, v.cz);
  const float2 g2 = make_float2(g, g), m3 = make_float2(-3.f, -3.f);
  float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx;
  bool zero = false;
#pragma unroll 1
  for (int e0 = 0; e0 < count; e0 += 8) {
    float2 ux[4], uy[4], uz[4], uw[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int pr = (e0 >> 1) + (k ^ perm);
      const float4 ea = list.a[pr], eb = list.b[pr];
      const int2 sr = *reinterpret_cast<const int2 *>(src + 2 * pr);
      const float2 dx = __fadd2_rn(make_float2(ea.x, ea.y), ntx), dy = __fadd2_rn(make_float2(ea.z, ea.w), nty),
                   dz = __fadd2_rn(make_float2(eb.x, eb.y), ntz);
      const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
      zero = zero || !(r2.x > 0.f) || !(r2.y > 0.f);
      // a factor of 0 takes an entry (the target itself, one without mass) out
      // of every sum
      float2 r = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
      r.x = sr.x != self && r2.x > 0.f && eb.z != 0.f ? r.x : 0.f;
      r.y = sr.y != self && r2.y > 0.f && eb.w != 0.f ? r.y : 0.f;
      const float2 rr = __fmul2_rn(r, r);
      const float2 gi3 = __fmul2_rn(__fmul2_rn(g2, rr), r);
      const float2 rc = __ffma2_rn(dx, cx, __ffma2_rn(dy, cy, __fmul2_rn(dz, cz)));
      const float2 f = __fmul2_rn(gi3, make_float2(eb.z, eb.w));
      const float2 h = __fmul2_rn(__fmul2_rn(__fmul2_rn(f, m3), rr), rc);
      ux[k] = __ffma2_rn(f, cx, __fmul2_rn(h, dx));
      uy[k] = __ffma2_rn(f, cy, __fmul2_rn(h, dy));
      uz[k] = __ffma2_rn(f, cz, __fmul2_rn(h, dz));
      uw[k] = __fmul2_rn(gi3, rc);
      sx = __fadd2_rn(sx, ux[k]);
      sy = __fadd2_rn(sy, uy[k]);
      sz = __fadd2_rn(sz, uz[k]);
    }
    const auto halves = [&](float2 (&u)[4]) {
      const auto from = [](float2 t, int o) {
        return make_float2(__shfl_xor_sync(kFull, t.x, o), __shfl_xor_sync(kFull, t.y, o));
      };
      u[0] = __fadd2_rn(u[0], from(u[2], 16));
      u[1] = __fadd2_rn(u[1], from(u[3], 16));
      u[0] = __fadd2_rn(u[0], from(u[1], 8));
      return (b4 ? u[0].y : u[0].x) + __shfl_xor_sync(kFull, b4 ? u[0].x : u[0].y, 4);
    };
    const float tx = halves(ux), ty = halves(uy), tz = halves(uz), tw = halves(uw);
    const float ta = (b2 ? tz : tx) + __shfl_xor_sync(kFull, b2 ? tx : tz, 2);
    const float tb = (b2 ? tw : ty) + __shfl_xor_sync(kFull, b2 ? ty : tw, 2);
    const float val = (b1 ? tb : ta) + __shfl_xor_sync(kFull, b1 ? ta : tb, 1);
    const int e = e0 + 2 * perm + (b4 ? 1 : 0);
    if (val != 0.f) {
      const int sr = src[e];
      double *dst = nullptr;
      if (sr >= 0) dst = reinterpret_cast<double *>(ab.part_g + sr);
      else if (sr <= -3) dst = reinterpret_cast<double *>(ab.node_g + (-3 - sr));
      if (dst) atomicAdd(dst + (lane & 3), (double)val);
    }
  }
  v.gx -= sx.x + sx.y;
  v.gy -= sy.x + sy.y;
  v.gz -= sz.x + sz.y;
  bool singular = false;
  if (valid && zero)  // (the target's own entry, or a singular one)
#pragma unroll 1
    for (int e = 0; e < count; ++e) {
      const float4 ea = list.a[e >> 1], eb = list.b[e >> 1];
      const bool hi = e & 1;
      const float dx = (hi ? ea.y : ea.x) + ntx.x, dy = (hi ? ea.w : ea.z) + nty.x, dz = (hi ? eb.y : eb.x) + ntz.x;
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2.x)));
      singular |= src[e] != self && (hi ? eb.w : eb.z) != 0.f && !(r2 > 0.f);
    }
  __syncwarp();
  return singular;
}

template <bool kTrackSource, int kTPL, bool kVjp>
__device__ __forceinline__ void flush_full(const PairList &list, int *src, int &ls, LaneTargets<kTPL> &lt_,
                                           LaneVjp &vj, float2 eps2, int nq, float g, const AdjointBuffers &ab) {
  constexpr int kBatch = batch_of<kTrackSource>();
  const int lane = threadIdx.x & 31;
  int done = 0;
  while (ls - done >= kBatch) {
    const PairList part{list.a + done / 2, list.b + done / 2};
    bool sg;
    if constexpr (kVjp)
      sg = vjp_entries(part, src + done, kBatch, lt_.s[0], lt_.valid[0], lt_.ntx[0], lt_.nty[0], lt_.ntz[0],
                       vj, eps2, g, ab);
    else
      sg = eval_slots<kTrackSource, kTPL>(part, src + (kTrackSource ? done : 0), kBatch, nq, lt_, eps2);
#pragma unroll
    for (int q = 0; q < kTPL; ++q)
      if (lt_.valid[q]) {
        lt_.inter += kBatch;
        lt_.singular |= sg;
      }
    done += kBatch;
  }
  if (done) {
    __syncwarp();
    // fewer than kBatch entries left; the sources start at done >= kBatch,
    // past the destinations
    const int rest = ls - done;
    for (int i = lane; i < (rest + 1) / 2; i += 32) {
      list.a[i] = list.a[done / 2 + i];
      list.b[i] = list.b[done / 2 + i];
    }
    if (kTrackSource)
      for (int i = lane; i < rest; i += 32) src[i] = src[done + i];
    ls = rest;
    __syncwarp();
  }
}

// The group-box acceptance test of the mixed walk, in FP32, of a node with
// list entry e; the squared distance from the
// box (half extents rounded up) to that point is computed in FP32 and shrunk
// by 2^-20 so that it never exceeds the exact FP64 distance, and cr2 is the
// exact squared radius rounded up with a 2^-18 margin.  An accepted node is
// therefore accepted by the exact test for every target in the box; a node
// within the margins is opened instead (more work, never less accuracy).
__device__ __forceinline__ bool accept_box(const float4 &e, const float *ghalf, float cr2) {
  constexpr float kShrink = 1.0f - 0x1p-20f;
  const float ex = fmaxf(0.f, fmaf(fabsf(e.x), kShrink, -ghalf[0]));
  const float ey = fmaxf(0.f, fmaf(fabsf(e.y), kShrink, -ghalf[1]));
  const float ez = fmaxf(0.f, fmaf(fabsf(e.z), kShrink, -ghalf[2]));
  const float d2 = fmaf(ez, ez, fmaf(ey, ey, ex * ex)) * kShrink;
  return d2 > cr2;
}

// The list entry of a source: its offset from the group centre (formed in
// FP64, then rounded) and its mass.
__device__ __forceinline__ float4 list_entry(const double4 &a, const double *gbox) {
  return make_float4((float)(a.x - gbox[6]), (float)(a.y - gbox[7]), (float)(a.z - gbox[8]), (float)a.w);
}

// Mixed-precision traversal, one warp per target group of at most 32 x kTPL
// Morton-consecutive targets inside one parent cell (kTPL targets per lane).
// The group's bounding box (FP64) replaces the target in the reference's
// acceptance test: a node is accepted for the whole group when the
// box-to-centre-of-mass distance exceeds max(crit, sqrt(3) h + |com -
// centre|) (crit = side/theta + |com - centre|, h the cell's half side),
// tested conservatively in FP32 (accept_box).  Every target in the box is
// then farther than crit from the centre of mass and outside the cell, so
// the reference's test accepts the node for each of them.  Nodes are
// examined 64 at a time (two per lane) from a warp-private stack in shared
// memory, each lane fetching both nodes' 48-byte records (MixedNode) in one
// round trip (a node's children are consecutive records); a full stack spills
// its bottom half to a global extension sized for any walk, so every node
// gets the acceptance test.  Accepted nodes and the particles of reached leaves
// go to a shared interaction list as FP32 offsets from the group centre (formed
// in FP64, then rounded) and are evaluated by all lanes in batches of
// kEvalBatch (32 where sources are tracked).  Bound at 2^18 particles by
// instruction issue (60 % of the slots, FMA pipe 57 %).
// With kVjp (one target per lane, sources tracked) the same walk evaluates
// the vector-Jacobian product above instead of the force.
//
// With kSplit > 1 the block's warps share one group: each walks from the root
// until kDeal nodes are pending, then keeps every kSplit-th of them, and the
// targets' sums are added at the end.  This is for systems with too few groups
// to fill the GPU, where a walk is a chain of ~45 rounds of 2 us.
constexpr int kDeal = 48;

template <bool kTrackSource, int kTPL, bool kVjp = false, int kSplit = 1>
__global__ void __launch_bounds__(mixed_warps<kSplit>() * 32,
                                  kSplit > 1 ? 20 / kSplit
                                             : (kTPL >= 4 ? NBB_MIXED_MINBLOCKS4 : (kTPL == 2 ? NBB_MIXED_MINBLOCKS2 : NBB_MIXED_MINBLOCKS)))
    traverse_mixed_kernel(Workspace ws, TraversalParams p, AdjointBuffers ab) {
  static_assert(!kVjp || (kTrackSource && kTPL == 1), "the adjoint walk tracks sources, one target per lane");
  static_assert(kSplit == 1 || kTPL == 1, "a shared group has one target per lane");
  __shared__ MixedShared<kTrackSource, mixed_warps<kSplit>()> sh;
  __shared__ double s_part[kSplit > 1 ? kSplit - 1 : 1][3][kSplit > 1 ? 32 : 1];  // the other warps' sums
  __shared__ int s_group;
  // node cache: the top cache_depth levels below the root (the first entries
  // of the level order), loaded once per block
  __shared__ MixedNode c_rec[kTopMax];
  DevScalars *sc = ws.sc;
  if (kSplit > 1 ? __syncthreads_or(sc->error != 0) != 0 : sc->error != 0) return;
  const int lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  int *stack = sh.stack[wid];
  const PairList list{sh.la[wid], sh.lb[wid]};
  int *src = sh.src[wid];
  const int n = ws.n;
  const int m = sc->n_nodes;
  const int n_groups = sc->n_tgroups;
  const unsigned lt = lanemask_lt();
  int ccount = 0;  // nodes below this index are cached
  if (p.cache_depth > 0 && ws.n_systems == 1) {
    ccount = min(min(sc->level_base[min(p.cache_depth, kTopDepth) + 1], kTopMax), m);
    for (int q = threadIdx.x; q < ccount; q += blockDim.x) c_rec[q] = ws.node_m[q];
    __syncthreads();
  }
  long long tests = 0;
  unsigned overflow = 0;
  long long inter_total = 0;
  bool singular_any = false;
  while (true) {
    int grp = 0;
    if constexpr (kSplit > 1) {
      if (threadIdx.x == 0) s_group = (int)atomicAdd(&sc->work_counter, 1u);
      __syncthreads();
      grp = s_group;
    } else {
      if (lane == 0) grp = (int)atomicAdd(&sc->work_counter, 1u);
      grp = __shfl_sync(kFull, grp, 0);
    }
    if (grp >= n_groups) break;
    const int g0 = ws.tstart[grp];
    const int g1 = (grp + 1 < n_groups) ? ws.tstart[grp + 1] : n;
    bool dealt = kSplit == 1;
    const long long tests_before = tests;
    const int nq = min(kTPL, max(1, (g1 - g0 + 31) >> 5));  // occupied target slots
    LaneTargets<kTPL> T;
    LaneVjp V;
    double4 tp[kTPL];
    double lo[3], hi[3];
#pragma unroll
    for (int q = 0; q < kTPL; ++q) {
      T.s[q] = g0 + lane + 32 * q;
      T.valid[q] = T.s[q] < g1 && T.s[q] < n;
      tp[q] = ws.pm4[T.valid[q] ? T.s[q] : g0];
      // an empty slot is the group's first target once more: that one's own entry
      // must be its own too, or it would be a singular pair without softening, and
      // with a small one m / eps^5 may overflow in the adjoint and 0 times it is NaN
      if (kTrackSource && !T.valid[q]) T.s[q] = g0;
      T.sum[q] = make_float3(0.f, 0.f, 0.f);
      T.comp[q] = make_float3(0.f, 0.f, 0.f);
    }
    if (kVjp && T.valid[0]) {
      const uint32_t ti = ws.idx[T.s[0]];
      V.cx = (float)(ab.coef * ab.gvx[ti]);
      V.cy = (float)(ab.coef * ab.gvy[ti]);
      V.cz = (float)(ab.coef * ab.gvz[ti]);
    }
    lo[0] = hi[0] = tp[0].x;
    lo[1] = hi[1] = tp[0].y;
    lo[2] = hi[2] = tp[0].z;
#pragma unroll
    for (int q = 1; q < kTPL; ++q) {
      lo[0] = fmin(lo[0], tp[q].x); hi[0] = fmax(hi[0], tp[q].x);
      lo[1] = fmin(lo[1], tp[q].y); hi[1] = fmax(hi[1], tp[q].y);
      lo[2] = fmin(lo[2], tp[q].z); hi[2] = fmax(hi[2], tp[q].z);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      for (int o = 16; o > 0; o >>= 1) {
        lo[a] = fmin(lo[a], __shfl_xor_sync(kFull, lo[a], o));
        hi[a] = fmax(hi[a], __shfl_xor_sync(kFull, hi[a], o));
      }
    }
    {
      // the box and centre live in shared memory while the walk runs, so
      // they hold no registers through the evaluation
      volatile double *gb = sh.gbox[wid];
      if (lane == 0) {
        for (int a = 0; a < 3; ++a) {
          gb[a] = lo[a];
          gb[3 + a] = hi[a];
          gb[6 + a] = 0.5 * (lo[a] + hi[a]);
          sh.ghalf[wid][a] = __double2float_ru(0.5 * (hi[a] - lo[a]));
        }
      }
      __syncwarp();
    }
    const double *gbox = sh.gbox[wid];
    const double gcx = 0.5 * (lo[0] + hi[0]), gcy = 0.5 * (lo[1] + hi[1]),
                 gcz = 0.5 * (lo[2] + hi[2]);
    {
      float tx[kTPL], ty[kTPL], tz[kTPL];
#pragma unroll
      for (int q = 0; q < kTPL; ++q) {
        tx[q] = -(float)(tp[q].x - gcx);
        ty[q] = -(float)(tp[q].y - gcy);
        tz[q] = -(float)(tp[q].z - gcz);
      }
#pragma unroll
      for (int q = 0; q < kTPL; ++q) {
        T.ntx[q] = make_float2(tx[q], tx[q]);
        T.nty[q] = make_float2(ty[q], ty[q]);
        T.ntz[q] = make_float2(tz[q], tz[q]);
      }
    }
    // a group's targets belong to one system: walk that system's subtree
    const int sys = ws.n_systems > 1 ? ws.psys[g0] : 0;
    const int root = ws.root_lo[sys];
    const double soft = ws.sys_eps ? ws.sys_eps[sys] : p.soft;
    const float eps2f = (float)(soft * soft);
    const float2 eps2 = make_float2(eps2f, eps2f);
    int ls = 0;
    if (lane == 0) stack[0] = root;
    int sp = (m > 0 && root >= 0 && root < m) ? 1 : 0;
    __syncwarp();
    // this warp's stack extension in global memory: when the shared part
    // fills, its bottom half moves there (the combined stack keeps its
    // order) and comes back when the shared part runs low
    int *ext = nullptr;
    int esp = 0;
    {
      const int gw = blockIdx.x * mixed_warps<kSplit>() + wid;
      if (ws.walk_ext && gw < ws.walk_warps) ext = ws.walk_ext + (size_t)gw * ws.walk_ext_cap;
    }
    while (sp > 0 || esp > 0) {
      if (kSplit > 1 && !dealt && sp >= kDeal) {
        const int own = (sp - wid + kSplit - 1) / kSplit;
        for (int c = 0; c < own; c += 32) {
          // (the sources start at or after the destinations)
          const int i = c + lane;
          const int v = i < own ? stack[i * kSplit + wid] : 0;
          __syncwarp();
          if (i < own) stack[i] = v;
          __syncwarp();
        }
        sp = own;
        dealt = true;
        if (wid > 0) tests = tests_before;
      }
      // until then every warp walks the same nodes, and only the first lists
      const bool mute = kSplit > 1 && !dealt && wid > 0;
      if (sp > kStackCap - 7 * kWalkPop && ext && esp + kSpill <= ws.walk_ext_cap) {
        for (int i = lane; i < kSpill; i += 32) ext[esp + i] = stack[i];
        __syncwarp();
        // the destination ends below kSpill, where the sources start
        for (int i = lane; i < sp - kSpill; i += 32) stack[i] = stack[kSpill + i];
        esp += kSpill;
        sp -= kSpill;
        __syncwarp();
      } else if (sp < kWalkPop && esp > 0) {
        const int r = min(esp, kSpill);
        const int v0 = (lane < sp) ? stack[lane] : 0, v1 = (lane + 32 < sp) ? stack[lane + 32] : 0;
        __syncwarp();
        if (lane < sp) stack[r + lane] = v0;
        if (lane + 32 < sp) stack[r + lane + 32] = v1;
        for (int i = lane; i < r; i += 32) stack[i] = ext[esp - r + i];
        sp += r;
        esp -= r;
        __syncwarp();
      }
      // up to 64 nodes per round, two per lane, fetched in one round trip
      int k = sp < kWalkPop ? sp : kWalkPop;
      const int room = (kStackCap - sp) / 7;
      if (k > room) k = room > 0 ? room : 1;
      const int n0 = (lane < k) ? stack[sp - k + lane] : -1;
      const int n1 = (lane + 32 < k) ? stack[sp - k + 32 + lane] : -1;
      sp -= k;
      __syncwarp();
      int4 m0 = make_int4(0, 0, 0, 0), m1 = m0;  // radius, first, count, nchild
      double4 a0 = make_double4(0.0, 0.0, 0.0, 0.0), a1 = a0;
      if (n0 >= 0) {
        if (n0 < ccount) {
          a0 = c_rec[n0].a;
          m0 = *reinterpret_cast<const int4 *>(&c_rec[n0].cr2);
        } else {
          a0 = ws.node_m[n0].a;
          m0 = *reinterpret_cast<const int4 *>(&ws.node_m[n0].cr2);
        }
      }
      if (n1 >= 0) {
        if (n1 < ccount) {
          a1 = c_rec[n1].a;
          m1 = *reinterpret_cast<const int4 *>(&c_rec[n1].cr2);
        } else {
          a1 = ws.node_m[n1].a;
          m1 = *reinterpret_cast<const int4 *>(&ws.node_m[n1].cr2);
        }
      }
      const float cr0 = __int_as_float(m0.x), cr1 = __int_as_float(m1.x);  // squared acceptance radius for a target box
      // 0 nothing, 1 accepted cell, 2 leaf, 3 open; a leaf's record carries
      // its first particle, so every node has a list entry
      int cat0 = 0, cat1 = 0;
      const float4 e0 = list_entry(a0, gbox), e1 = list_entry(a1, gbox);
      {
        const bool far0 = accept_box(e0, sh.ghalf[wid], cr0), far1 = accept_box(e1, sh.ghalf[wid], cr1);
        const bool cell0 = m0.z <= 0 && a0.w != 0.0, cell1 = m1.z <= 0 && a1.w != 0.0;
        if (n0 >= 0) cat0 = m0.z > 0 ? 2 : (cell0 ? (far0 ? 1 : 3) : 0);
        if (n1 >= 0) cat1 = m1.z > 0 ? 2 : (cell1 ? (far1 ? 1 : 3) : 0);
        tests += (n0 >= 0 && cell0 ? 1 : 0) + (n1 >= 0 && cell1 ? 1 : 0);
      }
      // opened nodes push their children (node 0's, then node 1's), which are
      // consecutive and come after them in the level order; a push that would
      // end past the stack accepts the node instead
      int nc0 = (cat0 == 3) ? min(max(m0.w, 0), 8) : 0;
      int nc1 = (cat1 == 3) ? min(max(m1.w, 0), 8) : 0;
      if (m0.y <= n0 || m0.y > m - nc0) nc0 = 0;
      if (m1.y <= n1 || m1.y > m - nc1) nc1 = 0;
      // list entries: a cell's, or a leaf's particles
      int cnt0 = mute ? 0 : (cat0 == 1 ? 1 : (cat0 == 2 ? m0.z : 0));
      int cnt1 = mute ? 0 : (cat1 == 1 ? 1 : (cat1 == 2 ? m1.z : 0));
      // both prefix sums in one scan: children (at most 16 a lane) and list
      // entries (capped: a round with that many takes the slow path)
      constexpr int kCap = list_cap_of<kTrackSource>();
      const int own = (nc0 + nc1) | (min(cnt0 + cnt1, 2 * kCap) << 16);
      int scan = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, scan, o);
        if (lane >= o) scan += v;
      }
      const int totals = __shfl_sync(kFull, scan, 31);
      const int all_children = totals & 0xffff, entries = totals >> 16;
      const int excl = (scan - own) & 0xffff;
      int pushed = all_children;
      bool relisted = false;
      if (sp + all_children > kStackCap) {
        relisted = true;  // the scan's list offsets may no longer hold
        if (nc0 > 0 && sp + excl + nc0 > kStackCap) {
          cat0 = 1;
          nc0 = 0;
          ++overflow;
        }
        if (nc1 > 0 && sp + excl + nc0 + nc1 > kStackCap) {
          cat1 = 1;
          nc1 = 0;
          ++overflow;
        }
        pushed = __reduce_max_sync(kFull, (nc0 + nc1 > 0) ? excl + nc0 + nc1 : 0);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < nc0) stack[sp + excl + j] = m0.y + j;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < nc1) stack[sp + excl + nc0 + j] = m1.y + j;
      sp += pushed;
      if (ls + entries <= kCap && !relisted) {
        const int base = ls + ((scan - own) >> 16);
        if (cnt0 > 0) {
          list.put(base, e0.x, e0.y, e0.z, e0.w);
          if (kTrackSource) src[base] = cat0 == 2 ? m0.y : (kVjp ? -3 - n0 : -1);
        }
        if (cnt1 > 0) {
          list.put(base + cnt0, e1.x, e1.y, e1.z, e1.w);
          if (kTrackSource) src[base + cnt0] = cat1 == 2 ? m1.y : (kVjp ? -3 - n1 : -1);
        }
        for (int j = 1; j < cnt0; ++j) {
          const float4 e = list_entry(ws.pm4[m0.y + j], gbox);
          list.put(base + j, e.x, e.y, e.z, e.w);
          if (kTrackSource) src[base + j] = m0.y + j;
        }
        for (int j = 1; j < cnt1; ++j) {
          const float4 e = list_entry(ws.pm4[m1.y + j], gbox);
          list.put(base + cnt0 + j, e.x, e.y, e.z, e.w);
          if (kTrackSource) src[base + cnt0 + j] = m1.y + j;
        }
        ls += entries;
        __syncwarp();
        flush_full<kTrackSource, kTPL, kVjp>(list, src, ls, T, V, eps2, nq, (float)p.g, ab);
      } else {
        // rare: the leaves' particles do not fit behind the list, or a node
        // was accepted for want of stack; the cells first (at most 64)
        const unsigned cm0 = __ballot_sync(kFull, cat0 == 1 && !mute), cm1 = __ballot_sync(kFull, cat1 == 1 && !mute);
        if (cat0 == 1 && !mute) {
          const int pos = ls + __popc(cm0 & lt);
          list.put(pos, e0.x, e0.y, e0.z, e0.w);
          if (kTrackSource) src[pos] = kVjp ? -3 - n0 : -1;
        }
        if (cat1 == 1 && !mute) {
          const int pos = ls + __popc(cm0) + __popc(cm1 & lt);
          list.put(pos, e1.x, e1.y, e1.z, e1.w);
          if (kTrackSource) src[pos] = kVjp ? -3 - n1 : -1;
        }
        ls += __popc(cm0) + __popc(cm1);
        const int lc0 = cat0 == 2 ? cnt0 : 0, lc1 = cat1 == 2 ? cnt1 : 0;
        __syncwarp();
        flush_full<kTrackSource, kTPL, kVjp>(list, src, ls, T, V, eps2, nq, (float)p.g, ab);
        for (int h = 0; h < 2; ++h) {
          unsigned lm = __ballot_sync(kFull, (h == 0 ? lc0 : lc1) > 0);
          while (lm) {
            const int l = __ffs(lm) - 1;
            lm &= lm - 1;
            const int first = __shfl_sync(kFull, h == 0 ? m0.y : m1.y, l);
            const int cnt = __shfl_sync(kFull, h == 0 ? lc0 : lc1, l);
            for (int b0 = 0; b0 < cnt; b0 += 32) {
              const int j = b0 + lane;
              if (j < cnt) {
                const double4 q = ws.pm4[first + j];
                const float4 e = list_entry(q, gbox);
                list.put(ls + lane, e.x, e.y, e.z, e.w);
                if (kTrackSource) src[ls + lane] = first + j;
              }
              ls += (cnt - b0 < 32) ? (cnt - b0) : 32;
              __syncwarp();
              flush_full<kTrackSource, kTPL, kVjp>(list, src, ls, T, V, eps2, nq, (float)p.g, ab);
            }
          }
        }
      }
    }
    if (kSplit > 1 && !dealt && wid > 0) tests = tests_before;
    if (ls > 0) {
      if (kVjp && (ls & 7)) {
        // complete the last block of eight with zero-mass entries
        if (lane < (-ls & 7)) {
          list.put(ls + lane, 0.f, 0.f, 0.f, 0.f);
          src[ls + lane] = -2;
        }
        __syncwarp();
      } else if (ls & 1) {
        // complete the last pair with a zero-mass entry far away (its
        // offset squared stays finite in FP32 and it contributes exactly 0)
        if (lane == 0) {
          list.put(ls, 1.0e18f, 1.0e18f, 1.0e18f, 0.f);
          if (kTrackSource) src[ls] = -2;
        }
        __syncwarp();
      }
      bool sg;
      if constexpr (kVjp)
        sg = vjp_entries(list, src, (ls + 7) & ~7, T.s[0], T.valid[0], T.ntx[0], T.nty[0], T.ntz[0], V, eps2,
                         (float)p.g, ab);
      else
        sg = eval_slots<kTrackSource, kTPL>(list, src, ls, nq, T, eps2);
#pragma unroll
      for (int q = 0; q < kTPL; ++q)
        if (T.valid[q]) {
          T.inter += ls;
          T.singular |= sg;
        }
    }
    __syncwarp();
    // the targets' sums; a shared group's are added in warp order
    double own[kTPL][3];
#pragma unroll
    for (int q = 0; q < kTPL; ++q) {
      own[q][0] = kVjp ? V.gx : (double)T.sum[q].x - (double)T.comp[q].x;
      own[q][1] = kVjp ? V.gy : (double)T.sum[q].y - (double)T.comp[q].y;
      own[q][2] = kVjp ? V.gz : (double)T.sum[q].z - (double)T.comp[q].z;
    }
    if constexpr (kSplit > 1) {
      if (wid > 0)
        for (int c = 0; c < 3; ++c) s_part[wid - 1][c][lane] = own[0][c];
      __syncthreads();
      if (wid == 0)
        for (int w = 0; w < kSplit - 1; ++w)
          for (int c = 0; c < 3; ++c) own[0][c] += s_part[w][c][lane];
    }
#pragma unroll
    for (int q = 0; q < kTPL; ++q) {
      if (!T.valid[q] || (kSplit > 1 && wid > 0)) continue;
      if constexpr (kVjp) {
        ab.tgt_g[T.s[q]] = make_double4(own[q][0], own[q][1], own[q][2], 0.0);
      } else {
        const double ax = p.g * own[q][0], ay = p.g * own[q][1], az = p.g * own[q][2];
        const uint32_t ti = ws.idx[T.s[q]];
        ws.ax[ti] = ax;
        ws.ay[ti] = ay;
        ws.az[ti] = az;
        if (p.kick) {
          ws.vx[ti] = __fma_rn(p.half_dt, ax, ws.vx[ti]);
          ws.vy[ti] = __fma_rn(p.half_dt, ay, ws.vy[ti]);
          ws.vz[ti] = __fma_rn(p.half_dt, az, ws.vz[ti]);
        }
      }
    }
    inter_total += T.inter;
    singular_any |= T.singular;
  }
  if (__any_sync(kFull, singular_any) && lane == 0) record_error(sc, kStageTraversal, 6);
  inter_total = warp_sum_ll(inter_total);
  tests = warp_sum_ll(tests);
  unsigned ov = overflow;
  for (int o = 16; o > 0; o >>= 1) ov += __shfl_xor_sync(kFull, ov, o);
  if (lane == 0) {
    atomicAdd(&sc->interactions, (unsigned long long)inter_total);
    atomicAdd(&sc->mac_tests, (unsigned long long)tests);
    if (ov) {
      // the extension is sized for any walk, so this is a broken invariant:
      // the accepted nodes skipped their acceptance test, and the call fails
      atomicAdd(&sc->stack_overflow, ov);
      record_error(sc, kStageTraversal, 9);
    }
  }
}

// ------------------------------------------------------------ direct ----

constexpr int kDirectThreads = 128;

// barnes_hut_accuracy_test.cu:101-172: each thread sums every other particle
// in index order; sources are staged through shared memory in tiles.  With
// chunked sources (blockIdx.y of gridDim.y chunks, partial sums to
// part[chunk][3][n_targets]) few targets still fill the GPU; the partials are
// then added in chunk order by direct_combine_kernel.
__global__ void __launch_bounds__(kDirectThreads)
    direct_kernel(int n, const double *__restrict__ m, const double *__restrict__ x,
                  const double *__restrict__ y, const double *__restrict__ z, int n_targets,
                  const int *__restrict__ targets, double g, double soft2, double *ax, double *ay,
                  double *az, double *part) {
  __shared__ double4 tile[kDirectThreads];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int chunks = gridDim.y;
  const long long span = ((long long)n + chunks - 1) / chunks;
  const int j0 = (int)min((long long)n, span * blockIdx.y);
  const int j1 = (int)min((long long)n, span * (blockIdx.y + 1));
  int t = (k < n_targets) ? (targets ? targets[k] : k) : 0;
  const bool active = k < n_targets && t >= 0 && t < n;
  if (!active) t = 0;
  const double tx = active ? x[t] : 0.0, ty = active ? y[t] : 0.0, tz = active ? z[t] : 0.0;
  double rx = 0.0, ry = 0.0, rz = 0.0;
  for (int base = j0; base < j1; base += kDirectThreads) {
    const int j = base + threadIdx.x;
    tile[threadIdx.x] = (j < j1) ? make_double4(x[j], y[j], z[j], m[j]) : make_double4(0, 0, 0, 0);
    __syncthreads();
    const int lim = (j1 - base < kDirectThreads) ? j1 - base : kDirectThreads;
    if (active) {
      for (int q = 0; q < lim; ++q) {
        if (base + q == t) continue;
        const double4 s = tile[q];
        const double dx = __dsub_rn(s.x, tx), dy = __dsub_rn(s.y, ty), dz = __dsub_rn(s.z, tz);
        const double d2 = __dadd_rn(sqdist(dx, dy, dz), soft2);
        const double inv = __drcp_rn(__dsqrt_rn(d2));
        const double f = __dmul_rn(__dmul_rn(g, s.w), __dmul_rn(__dmul_rn(inv, inv), inv));
        rx = __fma_rn(f, dx, rx);
        ry = __fma_rn(f, dy, ry);
        rz = __fma_rn(f, dz, rz);
      }
    }
    __syncthreads();
  }
  if (k < n_targets) {
    if (chunks == 1) {
      ax[k] = active ? rx : NAN;
      ay[k] = active ? ry : NAN;
      az[k] = active ? rz : NAN;
    } else {
      double *pc = part + (size_t)blockIdx.y * 3 * n_targets;
      pc[k] = active ? rx : NAN;
      pc[n_targets + k] = active ? ry : NAN;
      pc[2 * (size_t)n_targets + k] = active ? rz : NAN;
    }
  }
}

__global__ void __launch_bounds__(kDirectThreads)
    direct_combine_kernel(const double *__restrict__ part, int chunks, int n_targets, double *ax, double *ay,
                          double *az) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_targets) return;
  double rx = 0.0, ry = 0.0, rz = 0.0;
  for (int c = 0; c < chunks; ++c) {
    const double *pc = part + (size_t)c * 3 * n_targets;
    rx = __dadd_rn(rx, pc[k]);
    ry = __dadd_rn(ry, pc[n_targets + k]);
    rz = __dadd_rn(rz, pc[2 * (size_t)n_targets + k]);
  }
  ax[k] = rx;
  ay[k] = ry;
  az[k] = rz;
}

// ------------------------------------------- reference-layout octree ----

// barnes_hut.cu:90-162 on a caller octree in the reference numbering.
__device__ int ref_first_child(const RefOctree &o, int node, int &err) {
  for (int oc = 7; oc >= 0; --oc) {
    const int c = o.children[node * 8 + oc];
    if (c == -1) continue;
    if (c <= 0 || c >= o.n_nodes) {
      err = 1;
      return -2;
    }
    return c;
  }
  err = 5;
  return -2;
}

__device__ int ref_next(const RefOctree &o, int node, int &err) {
  int climbs = 0;
  while (node != 0) {
    if (++climbs > o.n_nodes) {
      err = 4;
      return -2;
    }
    const int par = o.parent[node];
    if (par < 0 || par >= o.n_nodes) {
      err = 4;
      return -2;
    }
    bool found = false;
    for (int oc = 7; oc >= 0; --oc) {
      const int c = o.children[par * 8 + oc];
      if (c == -1) continue;
      if (c <= 0 || c >= o.n_nodes) {
        err = 1;
        return -2;
      }
      if (found) return c;
      if (c == node) found = true;
    }
    if (!found) {
      err = 4;
      return -2;
    }
    node = par;
  }
  return -1;
}

__global__ void ref_octree_kernel(RefOctree o, const uint32_t *idx, const double *pm,
                                  const double *px, const double *py, const double *pz, double *ax,
                                  double *ay, double *az, double theta, double soft2, double g,
                                  int morton, int *err_out) {
  const int st = blockIdx.x * blockDim.x + threadIdx.x;
  if (st >= o.n_particles) return;
  int err = 0;
  const uint32_t tu = idx[st];
  if (tu >= (uint32_t)o.n_particles) {
    atomicCAS(err_out, 0, 3);
    return;
  }
  const int target = (int)tu;
  const int ti = morton ? st : target;
  const double tx = px[ti], ty = py[ti], tz = pz[ti];
  double rx = 0.0, ry = 0.0, rz = 0.0;
  int node = 0;
  long long visits = 0;
  const long long max_visits = 2ll * o.n_nodes + 8;
  while (node >= 0) {
    if (++visits > max_visits) {  // a cyclic caller octree never ends
      atomicCAS(err_out, 0, 4);
      return;
    }
    const double h = o.half[node];
    if (h <= 0.0) {
      atomicCAS(err_out, 0, 8);
      return;
    }
    const int cnt = o.count[node];
    if (cnt > 0) {
      for (int oc = 0; oc < 8; ++oc)
        if (o.children[node * 8 + oc] != -1) {
          atomicCAS(err_out, 0, 7);
          return;
        }
      const int f = o.first[node];
      if (f < 0 || cnt > o.n_particles || f > o.n_particles - cnt) {
        atomicCAS(err_out, 0, 2);
        return;
      }
      for (int k = 0; k < cnt; ++k) {
        const int sp = f + k;
        const uint32_t su = idx[sp];
        if (su >= (uint32_t)o.n_particles) {
          atomicCAS(err_out, 0, 3);
          return;
        }
        if (su == tu) continue;
        const int si = morton ? sp : (int)su;
        if (pm[si] == 0.0) continue;
        const double dx = __dsub_rn(px[si], tx), dy = __dsub_rn(py[si], ty), dz = __dsub_rn(pz[si], tz);
        if (!point_mass_fp64(dx, dy, dz, sqdist(dx, dy, dz), pm[si], g, soft2, rx, ry, rz)) {
          atomicCAS(err_out, 0, 6);
          return;
        }
      }
      node = ref_next(o, node, err);
      if (node == -2) {
        atomicCAS(err_out, 0, err);
        return;
      }
      continue;
    }
    const double nm = o.mass[node];
    if (nm == 0.0) {
      node = ref_next(o, node, err);
      if (node == -2) {
        atomicCAS(err_out, 0, err);
        return;
      }
      continue;
    }
    const double dx = __dsub_rn(o.comx[node], tx), dy = __dsub_rn(o.comy[node], ty),
                 dz = __dsub_rn(o.comz[node], tz);
    const double d2 = sqdist(dx, dy, dz);
    const bool contains = fabs(__dsub_rn(tx, o.cx[node])) <= h && fabs(__dsub_rn(ty, o.cy[node])) <= h &&
                          fabs(__dsub_rn(tz, o.cz[node])) <= h;
    bool accept = false;
    if (!contains && d2 > 0.0 && theta > 0.0) {
      const double ox = __dsub_rn(o.comx[node], o.cx[node]), oy = __dsub_rn(o.comy[node], o.cy[node]),
                   oz = __dsub_rn(o.comz[node], o.cz[node]);
      const double crit = __dadd_rn(__ddiv_rn(__dmul_rn(2.0, h), theta), __dsqrt_rn(sqdist(ox, oy, oz)));
      accept = __dsqrt_rn(d2) > crit;
    }
    if (accept) {
      if (!point_mass_fp64(dx, dy, dz, d2, nm, g, soft2, rx, ry, rz)) {
        atomicCAS(err_out, 0, 6);
        return;
      }
      node = ref_next(o, node, err);
    } else {
      node = ref_first_child(o, node, err);
    }
    if (node == -2) {
      atomicCAS(err_out, 0, err);
      return;
    }
  }
  ax[target] = rx;
  ay[target] = ry;
  az[target] = rz;
}

// ---------------------------------------------------------- integrator --

__global__ void kick_drift_kernel(double *x, double *y, double *z, double *vx, double *vy, double *vz,
                                  const double *ax, const double *ay, const double *az, size_t n,
                                  double dt) {
  const double hdt = 0.5 * dt;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double nvx = __fma_rn(hdt, ax[i], vx[i]);
    const double nvy = __fma_rn(hdt, ay[i], vy[i]);
    const double nvz = __fma_rn(hdt, az[i], vz[i]);
    vx[i] = nvx;
    vy[i] = nvy;
    vz[i] = nvz;
    x[i] = __fma_rn(dt, nvx, x[i]);
    y[i] = __fma_rn(dt, nvy, y[i]);
    z[i] = __fma_rn(dt, nvz, z[i]);
  }
}

__global__ void kick_kernel(double *vx, double *vy, double *vz, const double *ax, const double *ay,
                            const double *az, size_t n, double dt) {
  const double hdt = 0.5 * dt;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    vx[i] = __fma_rn(hdt, ax[i], vx[i]);
    vy[i] = __fma_rn(hdt, ay[i], vy[i]);
    vz[i] = __fma_rn(hdt, az[i], vz[i]);
  }
}

// Diagnostic: SIMT FMA throughput (8 independent chains per thread).
template <typename T>
__global__ void __launch_bounds__(256) fma_peak_kernel(T *out, int iters, T a, T b) {
  T x0 = (T)threadIdx.x * (T)1e-3, x1 = x0 + (T)1, x2 = x0 + (T)2, x3 = x0 + (T)3;
  T x4 = x0 + (T)4, x5 = x0 + (T)5, x6 = x0 + (T)6, x7 = x0 + (T)7;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  const T s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  if (s == (T)-12345) out[threadIdx.x] = s;
}

// Packed two-wide FP32 variant (sm_100 FFMA2): 8 independent float2 chains.
__global__ void __launch_bounds__(256) fma2_peak_kernel(float *out, int iters, float a, float b) {
  const float2 a2 = make_float2(a, a), b2 = make_float2(b, b);
  float2 x[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] = make_float2(threadIdx.x * 1e-3f + k, threadIdx.x * 1e-3f - k);
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = __ffma2_rn(x[k], a2, b2);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += x[k].x + x[k].y;
  if (s == -12345.f) out[threadIdx.x] = s;
}

inline int stream_grid(size_t n, int num_sms) {
  size_t b = (n + 255) / 256;
  const size_t cap = (size_t)(num_sms > 0 ? num_sms : 148) * 8;
  if (b > cap) b = cap;
  return b < 1 ? 1 : (int)b;
}

int device_sms() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace

// Persistent grids: as many resident blocks as the occupancy calculator
// allows on every SM; warps then pull target groups from a work counter.
template <typename K>
static cudaError_t grid_of(K kernel, int threads, int sms, int &grid) {
  int per_sm = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0);
  grid = sms * (per_sm > 0 ? per_sm : 1);
  return e;
}

// Whether the mixed walk in groups of at most 32 gives a group to four warps:
// while one warp each leaves the GPU unfilled.  Walk of Plummer spheres, one /
// four warps: 44 / 28 us at 1000 particles, 86 / 48 at 4000, 153 / 122 at 20000,
// 208 / 165 at 32768, 232 / 337 at 65536.  An ensemble's small systems split into
// many groups of few particles, each of which would be walked from the root by
// four warps: 2 systems of 10000 155 / 95 us, 8 of 2000 83 / 66, 12 of 1300 67 /
// 65, 12 of 3300 118 / 124, 16 of 2400 101 / 126, 64 of 64 20 / 36, 512 of 64 63 /
// 196.
constexpr int kMixedSplit = 4;
static bool split_group(const Workspace &ws) { return ws.n < 40000 && ws.n_systems <= 12; }

// Whether two warps share a set of the FP64 walk of n particles: up to a few
// sets per pair of warps that fits (figures at the kernel).
static bool pair_sets(int n) { return n < 65536; }

cudaError_t configure_traversal(Workspace &ws) {
  const int sms = ws.num_sms > 0 ? ws.num_sms : 148;
  cudaError_t e = grid_of(traverse_fp64_kernel<32, false>, fp64_threads<false>(), sms, ws.fp64_grid[0]);
  if (e == cudaSuccess) e = grid_of(traverse_fp64_kernel<32, true>, fp64_threads<true>(), sms, ws.fp64_grid[1]);
  if (e == cudaSuccess) e = grid_of(traverse_fp64_kernel<1, true>, fp64_threads<true>(), sms, ws.fp64_grid[2]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<false, 1>, kMixedWarps * 32, sms, ws.mixed_grid[0][0]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<true, 1>, kMixedWarps * 32, sms, ws.mixed_grid[1][0]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<false, 2>, kMixedWarps * 32, sms, ws.mixed_grid[0][1]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<true, 2>, kMixedWarps * 32, sms, ws.mixed_grid[1][1]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<false, 4>, kMixedWarps * 32, sms, ws.mixed_grid[0][2]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<true, 4>, kMixedWarps * 32, sms, ws.mixed_grid[1][2]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<true, 1, true>, kMixedWarps * 32, sms, ws.vjp_grid);
  constexpr int kSplitThreads = 32 * kMixedSplit;
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<false, 1, false, kMixedSplit>, kSplitThreads, sms, ws.split_grid[0]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<true, 1, false, kMixedSplit>, kSplitThreads, sms, ws.split_grid[1]);
  if (e == cudaSuccess) e = grid_of(traverse_mixed_kernel<true, 1, true, kMixedSplit>, kSplitThreads, sms, ws.split_grid[2]);
  // The stack extension holds a whole walk: the stack stays sorted by tree
  // level (a round pops the top and pushes children one level deeper), and
  // a level's entries are pushed only after every older entry of that level
  // has been popped, so at most 8 x kWalkPop entries per level are pending;
  // and a walk pushes each node at most once, so never more than the tree's
  // node capacity either (small systems take a small extension).
  int blocks = 148;
  for (int t = 0; t < 2; ++t)
    for (int q = 0; q < 3; ++q) blocks = std::max(blocks, ws.mixed_grid[t][q]);
  ws.walk_warps = blocks * kMixedWarps;
  for (int t = 0; t < 3; ++t) ws.walk_warps = std::max(ws.walk_warps, ws.split_grid[t] * kMixedSplit);
  ws.walk_ext_cap = std::min(8 * kWalkPop * (ws.max_level + 1), std::max(ws.cap_nodes, 1));
  return e;
}

cudaError_t launch_traversal(Workspace &ws, const TraversalParams &p, cudaStream_t s) {
  // target slots per lane: 1, 2 or 4 for groups of at most 32, 64 or 128
  const int slot = p.group_size > 64 ? 2 : (p.group_size > 32 ? 1 : 0);
  const int track = p.soft > 0.0 ? 0 : 1;
  const int grid = ws.mixed_grid[track][slot] > 0 ? ws.mixed_grid[track][slot] : 148;
  if (p.precision == 0) {
    const int form = p.targets > 1 ? (pair_sets(ws.n) ? 1 : 0) : 2;
    const int blocks = ws.fp64_grid[form] > 0 ? ws.fp64_grid[form] : 148;
    if (form == 2)
      traverse_fp64_kernel<1, true><<<blocks, fp64_threads<true>(), 0, s>>>(ws, p);
    else if (form == 1)
      traverse_fp64_kernel<32, true><<<blocks, fp64_threads<true>(), 0, s>>>(ws, p);
    else
      traverse_fp64_kernel<32, false><<<blocks, fp64_threads<false>(), 0, s>>>(ws, p);
  } else if (slot == 0 && split_group(ws))
    (track ? traverse_mixed_kernel<true, 1, false, kMixedSplit> : traverse_mixed_kernel<false, 1, false, kMixedSplit>)
        <<<ws.split_grid[track] > 0 ? ws.split_grid[track] : 148, 32 * kMixedSplit, 0, s>>>(ws, p, AdjointBuffers{});
  else if (slot == 0)
    (track ? traverse_mixed_kernel<true, 1> : traverse_mixed_kernel<false, 1>)<<<grid, kMixedWarps * 32, 0, s>>>(
        ws, p, AdjointBuffers{});
  else if (slot == 1)
    (track ? traverse_mixed_kernel<true, 2> : traverse_mixed_kernel<false, 2>)<<<grid, kMixedWarps * 32, 0, s>>>(
        ws, p, AdjointBuffers{});
  else
    (track ? traverse_mixed_kernel<true, 4> : traverse_mixed_kernel<false, 4>)<<<grid, kMixedWarps * 32, 0, s>>>(
        ws, p, AdjointBuffers{});
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_adjoint_mixed(Workspace &ws, const TraversalParams &p, const AdjointBuffers &ab,
                                 cudaStream_t s) {
  // the stack extension is sized for the largest mixed grid
  int grid = ws.vjp_grid > 0 ? ws.vjp_grid : 148;
  if (ws.walk_warps > 0 && grid * kMixedWarps > ws.walk_warps) grid = ws.walk_warps / kMixedWarps;
  TraversalParams q = p;
  q.cache_depth = 0;
  if (split_group(ws))
    traverse_mixed_kernel<true, 1, true, kMixedSplit>
        <<<ws.split_grid[2] > 0 ? ws.split_grid[2] : 148, 32 * kMixedSplit, 0, s>>>(ws, q, ab);
  else
    traverse_mixed_kernel<true, 1, true><<<grid, kMixedWarps * 32, 0, s>>>(ws, q, ab);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t measure_fma_tflops(int precision, double *tflops) {
  const int sms = device_sms();
  const int blocks = sms * 8, threads = 256, iters = 1 << 14;
  void *out = nullptr;
  cudaError_t e = cudaMalloc(&out, 256 * sizeof(double));
  if (e != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 4 && e == cudaSuccess; ++rep) {
    cudaEventRecord(e0);
    if (precision == 0)
      fma_peak_kernel<double><<<blocks, threads>>>((double *)out, iters, 0.9999999, 1e-9);
    else if (precision == 1)
      fma_peak_kernel<float><<<blocks, threads>>>((float *)out, iters * 2, 0.9999f, 1e-6f);
    else
      fma2_peak_kernel<<<blocks, threads>>>((float *)out, iters, 0.9999f, 1e-6f);
    cudaEventRecord(e1);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rep > 0 && ms < best) best = ms;
  }
  count_launches(4);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (e != cudaSuccess) return e;
  // FP64: iters x 8 FMAs; FP32: 2 iters x 8; packed: iters x 8 x 2 lanes
  const double flops = 2.0 * 8.0 * (double)iters * (precision == 0 ? 1.0 : 2.0) * blocks * threads;
  *tflops = flops / (best * 1e-3) / 1e12;
  return cudaSuccess;
}

cudaError_t launch_kick(double *vx, double *vy, double *vz, const double *ax, const double *ay,
                        const double *az, size_t n, double dt, cudaStream_t s) {
  kick_kernel<<<stream_grid(n, device_sms()), 256, 0, s>>>(vx, vy, vz, ax, ay, az, n, dt);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_kick_drift(double *x, double *y, double *z, double *vx, double *vy, double *vz,
                              const double *ax, const double *ay, const double *az, size_t n,
                              double dt, cudaStream_t s) {
  kick_drift_kernel<<<stream_grid(n, device_sms()), 256, 0, s>>>(x, y, z, vx, vy, vz, ax, ay, az, n, dt);
  count_launches(1);
  return cudaGetLastError();
}

int direct_chunks(size_t n, int n_targets) {
  const int blocks = (n_targets + kDirectThreads - 1) / kDirectThreads;
  const int want = device_sms() * 8;  // blocks that keep every SM busy
  if (blocks >= want || n < 65536) return 1;
  const long long c = std::min<long long>((want + blocks - 1) / blocks, (long long)(n / 4096));
  return (int)std::max(1ll, std::min(c, 256ll));
}

cudaError_t launch_direct(size_t n, const double *m, const double *x, const double *y, const double *z,
                          int n_targets, const int *targets, double g, double soft, double *ax,
                          double *ay, double *az, double *part, cudaStream_t s) {
  const int blocks = std::max(1, (n_targets + kDirectThreads - 1) / kDirectThreads);
  const int chunks = part ? direct_chunks(n, n_targets) : 1;
  direct_kernel<<<dim3(blocks, chunks), kDirectThreads, 0, s>>>((int)n, m, x, y, z, n_targets, targets, g,
                                                                soft * soft, ax, ay, az, part);
  if (chunks > 1) direct_combine_kernel<<<blocks, kDirectThreads, 0, s>>>(part, chunks, n_targets, ax, ay, az);
  count_launches(chunks > 1 ? 2 : 1);
  return cudaGetLastError();
}

cudaError_t launch_ref_octree_traversal(const RefOctree &o, const uint32_t *idx, const double *m,
                                        const double *x, const double *y, const double *z, double *ax,
                                        double *ay, double *az, double theta, double soft, double g,
                                        int morton_order, int *err, cudaStream_t s) {
  const int blocks = (o.n_particles + 127) / 128;
  ref_octree_kernel<<<blocks > 0 ? blocks : 1, 128, 0, s>>>(o, idx, m, x, y, z, ax, ay, az, theta,
                                                            soft * soft, g, morton_order, err);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace nbb
