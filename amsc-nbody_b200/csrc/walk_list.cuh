// walk_list.cuh -- the tree walk of one warp's targets as an ordered list of
// interactions, for the walks that keep the reference's per-target sequence
// (plain FP64 force) or its interaction sets (its adjoint).
//
// A warp walks for a few targets in a small box and hands their interactions
// out in depth-first preorder (children octant 7 -> 0, the reference's order,
// barnes_hut.cu:90-162).  A cell is judged against the targets' bounding box:
// accepted by every target, opened by every target (it leaves no trace), or
// undecided: then the list has the cell and, after it, its descendants, and
// each target decides at the cell whether it takes the cell or what follows
// it.  The box tests are conservative, so every target keeps its own
// interaction set, and preorder keeps its order: results have the bits of a
// target walking alone.
//
// Why: a warp that visits one node after another waits for a dependent load
// per visit (~4000 of them at 2^20 particles), which bound the plain walk at
// every size.  Here 32 nodes are loaded and judged per round: the warp's
// stack holds the frontier in preorder, a round takes its first 32 entries,
// replaces every cell that some target opens by its children, appends the
// leading run of finished entries to the list and puts the rest back (~170
// rounds for the ~3400 entries of a warp at 2^20 particles).
#pragma once

#include "nbb_internal.cuh"
#include "walk_fp64.cuh"

namespace nbb {

constexpr int kFrontier = 1024;            // stack entries per warp
// With fewer free entries than this a round takes one node only: plain
// depth-first order, which adds at most 7 entries per tree level.
constexpr int kFrontierReserve = 8 * (kMaxLevels + 1);
static_assert(kFrontierReserve + 64 <= kFrontier, "frontier bounds");

// Stack entry: node index (30 bits) and what is known about it.
constexpr unsigned kNodeBits = 0x3fffffffu;
enum EntryState : unsigned { kUntested = 0u, kAccepted = 1u, kLeaf = 2u, kUndecided = 3u };

// Up to kCap interactions to evaluate, in order.  The list is handed out when
// no round of single entries (32) fits any more.
template <int kCap>
struct ListBuffer {
  static_assert(kCap % 4 == 0 && kCap >= 64, "entries are evaluated in fours");
  static constexpr int kListCap = kCap;
  double4 src[kListCap];   // position and scaled mass
  int2 band[kListCap];     // undecided cells: high words of the squared box radius, of the crit^2 band's lower end
  int2 tag[kListCap];      // preorder index (-1: a zero mass); particle's Morton slot, -1 cell, -skip undecided
};
// What one walk keeps beside its list.
struct Frontier {
  unsigned stack[kFrontier];
  double centre[3], scale;  // the targets' box, in units of 1 / scale
  float half[3];
};

// 1 / side rounded to a power of two, so that box tests in FP32 neither
// overflow nor underflow whatever the unit of length.
__device__ __forceinline__ double box_scale(double side) {
  const int e = min(max((__double2hiint(side) >> 20) & 0x7ff, 64), 1980);
  return __hiloint2double((2046 - e) << 20, 0);
}

// The bounding box of the warp's targets (every lane passes a target): centre
// and half extents, these rounded up.
__device__ __forceinline__ void set_target_box(Frontier &sh, const double4 &t, double side) {
  const double v[3] = {t.x, t.y, t.z};
  const double scale = box_scale(side);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double lo = v[a], hi = v[a];
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
      const double c = 0.5 * lo + 0.5 * hi;
      sh.centre[a] = c;
      sh.half[a] = __double2float_ru(fmax(__dsub_ru(hi, c), __dsub_ru(c, lo)) * scale);
    }
  }
  if ((threadIdx.x & 31) == 0) sh.scale = scale;
  __syncwarp();
}

// A cell (centre of mass a, squared acceptance radius c.w, lower crit^2 band
// c.y) against the box: kAccepted or kUndecided, or kUntested when every
// target opens it.  In FP32 with margins that cover every rounding: an offset
// is off by less than 2^-22 of itself, a square by less than 2^-20.
__device__ __forceinline__ unsigned judge_cell(const Frontier &sh, const double4 &a, const double4 &c) {
  const double scale = sh.scale;
  const float ox = fabsf((float)((a.x - sh.centre[0]) * scale)), oy = fabsf((float)((a.y - sh.centre[1]) * scale)),
              oz = fabsf((float)((a.z - sh.centre[2]) * scale));
  const float hx = sh.half[0], hy = sh.half[1], hz = sh.half[2];
  constexpr float kDown = 1.0f - 0x1p-21f, kUp = 1.0f + 0x1p-21f;
  const float nx = fmaxf(0.f, fmaf(ox, kDown, -hx)), ny = fmaxf(0.f, fmaf(oy, kDown, -hy)),
              nz = fmaxf(0.f, fmaf(oz, kDown, -hz));
  const float fx = fmaf(ox, kUp, hx), fy = fmaf(oy, kUp, hy), fz = fmaf(oz, kUp, hz);
  const float near2 = fmaf(nz, nz, fmaf(ny, ny, nx * nx)), far2 = fmaf(fz, fz, fmaf(fy, fy, fx * fx));
  const float outer = __fmul_ru(__double2float_ru(c.w * scale * scale), 1.0f + 0x1p-18f);
  const float inner = __fmul_rd(__double2float_rd(c.y * scale * scale), 1.0f - 0x1p-18f);
  return near2 > outer ? kAccepted : (far2 < inner ? kUntested : kUndecided);
}

// The acceptance test of a target at squared distance d2 from an undecided
// cell: accept_fp64's decision.  The high words decide nearly always (both
// numbers are not negative, so they order as integers): accepted past the box
// radius, which is above the crit^2 band, and opened below that band.  What
// they leave open is decided out of line.
__device__ __forceinline__ bool band_accepts(int2 band, double d2) {
  const int h = __double2hiint(d2);
  return h > band.x && h < 0x7ff00000;
}
__device__ __forceinline__ bool band_opens(int2 band, double d2) { return __double2hiint(d2) < band.y; }
static __device__ __noinline__ bool accept_exact(const double4 *c, const double4 *bp, double tx, double ty, double tz,
                                                 double d2) {
  bool accept = (d2 > c->z) ? true : (d2 < c->y) ? false : (__dsqrt_rn(d2) > c->x);
  if (accept && !(d2 > c->w)) {
    const double4 b = *bp;
    const bool contains =
        fabs(__dsub_rn(tx, b.x)) <= b.w && fabs(__dsub_rn(ty, b.y)) <= b.w && fabs(__dsub_rn(tz, b.z)) <= b.w;
    accept = !contains && d2 > 0.0;
  }
  return accept;
}
template <int kCap>
__device__ __forceinline__ bool accept_entry(const ListBuffer<kCap> &list, int j, const Workspace &ws, int pre, const double4 &t,
                                             double d2) {
  const int2 band = list.band[j];
  if (band_accepts(band, d2)) return true;
  if (band_opens(band, d2)) return false;
  return accept_exact(ws.node_c + pre, ws.node_b + pre, t.x, t.y, t.z, d2);
}

// Walk the subtree of `root` for the targets in the box of sh.  hand(count,
// last) is called by the whole warp with entries [0, count) of *list, in
// preorder, each time the list is full and, with last, at the end (inactive
// entries fill the last block of four); it may move `list` to another buffer,
// and returns a resume index that all of the warp's targets have reached
// (frontier entries before it are dropped: a box that spans distant targets
// leaves cells undecided that every one of them accepts).  Masses are stored
// times mscale.  Cells judged are added to `tests`.
template <int kListCap, class Hand>
__device__ __forceinline__ void ordered_walk(const Workspace &ws, int m, int root, double mscale, Frontier &sh,
                                             ListBuffer<kListCap> *&list, unsigned &tests, Hand &&hand) {
  constexpr int kListFull = kListCap - 32;
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  int sp = (root >= 0 && root < m) ? 1 : 0;
  int ls = 0;                    // list entries
  int done = 0;                  // every target's walk has passed the nodes before this one
  int part_node = -1, part = 0;  // a leaf at the front of the frontier, its first `part` particles listed
  if (lane == 0) sh.stack[0] = (unsigned)root;
  __syncwarp();
  // every round finishes or expands the first node of the frontier (or lists
  // a part of a leaf): the limit only ends a walk over inconsistent records,
  // with an error (one test at the frontier's own: 0.3 % of a walk at 2^20
  // particles; an error of its own at the end of the loop took 1.2 %)
  unsigned rounds = 2u * (unsigned)m + (unsigned)ws.n + 2u;
  while (true) {
    const bool last = sp == 0;
    if (ls > kListFull || last) {
      if (ls + lane < ((ls + 3) & ~3)) list->tag[ls + lane] = make_int2(-1, 0);
      __syncwarp();
      done = hand(ls, last);
      __syncwarp();
      ls = 0;
    }
    if (last) break;
    // the first k entries of the frontier, lane 0 the first in preorder; a
    // round adds at most 8 entries per node taken
    const int k = min(min(32, sp), max(1, (kFrontier - kFrontierReserve - sp) >> 3));
    unsigned state = kUntested;
    int node = -1;
    int nc = 0;  // children that replace or follow the entry; more than the frontier holds: not a tree's node
    if (lane < k) {
      const unsigned ent = sh.stack[sp - 1 - lane];
      node = (int)(ent & kNodeBits);
      state = ent >> 30;
      if (node >= m) nc = kFrontier + 1;
      if (node < done || node >= m) node = -1;
    }
    sp -= k;
    double4 a = make_double4(0.0, 0.0, 0.0, 0.0), c = a;
    int4 meta = make_int4(0, 0, 0, 0), k0 = make_int4(0, 0, 0, 0), k1 = k0;
    bool keep = false;  // an entry that stays or is listed
    if (node >= 0) {
      a = ws.node_a[node];
      c = ws.node_c[node];
      meta = ws.node_meta[node];
      keep = true;
      if (state == kUntested) {
        // the child list with the records: one round trip less if it opens
        const int4 *kids = reinterpret_cast<const int4 *>(ws.node_kids + (size_t)node * 8);
        k0 = kids[0];
        k1 = kids[1];
        if (meta.z > 0) {
          state = kLeaf;
        } else if (a.w == 0.0) {
          keep = false;  // zero-mass cell (barnes_hut.cu:259-271)
        } else {
          ++tests;
          state = judge_cell(sh, a, c);
          keep = state != kUntested;
          if (state != kAccepted) nc = min(max(meta.w, 0), 8);
        }
      }
    }
    // entries before the first one that grows are finished and leave the
    // frontier; an undecided cell comes right before its children
    const unsigned grow = __ballot_sync(0xffffffffu, nc > 0);
    const int f = grow ? __ffs(grow) - 1 : 32;
    bool emit = keep && lane <= f;
    int first = meta.y, cnt = emit ? 1 : 0, off;
    if (state == kLeaf && emit) {
      const int skip = node == part_node ? part : 0;
      first += skip;
      cnt = meta.z - skip;
    }
    part_node = -1;
    int total;
    const bool single = __all_sync(0xffffffffu, cnt <= 1);
    if (single) {
      const unsigned b = __ballot_sync(0xffffffffu, cnt > 0);
      off = __popc(b & lt);
      total = __popc(b);
    } else {
      // leaves with several particles: the entries that fit; a leaf that
      // does not is listed in parts and stays at the front
      int inc = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc = min(inc + v, 0x3fffffff);
      }
      off = inc - cnt;
      const int room = kListCap - ls;
      const unsigned over = __ballot_sync(0xffffffffu, cnt > 0 && inc > room);
      total = __shfl_sync(0xffffffffu, inc, 31);
      if (over) {
        const int l = __ffs(over) - 1;
        total = room;
        part_node = __shfl_sync(0xffffffffu, node, l);
        part = __shfl_sync(0xffffffffu, room - off + (first - meta.y), l);
        if (lane >= l) {
          emit = false;
          cnt = lane == l ? room - off : 0;
        }
      }
    }
    // what is not listed goes back, first in preorder on top
    const bool again = keep && !emit;
    const int back = (again ? 1 : 0) + nc;
    int inc = back;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const int added = __shfl_sync(0xffffffffu, inc, 31);
    if (sp + added > kFrontier || rounds-- == 0u) {  // only by inconsistent records (see kFrontierReserve, rounds)
      if (lane == 0) record_error(ws.sc, kStageTraversal, 4);
      sp = 0;
      continue;
    }
    int at = sp + added - 1 - (inc - back);  // the lane's first entry
    if (again) sh.stack[at--] = (unsigned)node | (state << 30);
    if (nc > 0) {
      const int kid[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < nc) sh.stack[at - j] = (unsigned)kid[j] & kNodeBits;
    }
    sp += added;
    // the list entries
    const bool leaf = state == kLeaf;
    const int j = ls + off;
    if (cnt > 0) {
      const double4 v = leaf && first != meta.y ? ws.pm4[first] : a;
      list->src[j] = make_double4(v.x, v.y, v.z, __dmul_rn(mscale, v.w));
      list->tag[j] = make_int2(v.w != 0.0 ? node : -1, leaf ? first : (state == kUndecided ? -meta.x : -1));
      if (state == kUndecided) {
        list->band[j] = make_int2(__double2hiint(c.w), __double2hiint(c.y));
      }
    }
    if (!single) {
      unsigned left = __ballot_sync(0xffffffffu, cnt > 1);
      while (left) {
        const int l = __ffs(left) - 1;
        left &= left - 1;
        const int l_cnt = __shfl_sync(0xffffffffu, cnt, l), l_first = __shfl_sync(0xffffffffu, first, l);
        const int l_node = __shfl_sync(0xffffffffu, node, l), l_j = __shfl_sync(0xffffffffu, j, l);
        for (int i = 1 + lane; i < l_cnt; i += 32) {
          const double4 v = ws.pm4[l_first + i];
          list->src[l_j + i] = make_double4(v.x, v.y, v.z, __dmul_rn(mscale, v.w));
          list->tag[l_j + i] = make_int2(v.w != 0.0 ? l_node : -1, l_first + i);
        }
      }
    }
    ls += total;
    __syncwarp();
  }
}

}  // namespace nbb
