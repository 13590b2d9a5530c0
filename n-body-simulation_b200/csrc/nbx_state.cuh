// nbx_state.cuh -- device state of one simulation handle (one or many
// independent instances, "segments", laid out back to back).
#pragma once
#include "nbx_internal.cuh"

#include <cstddef>

#include <float.h>

namespace nbx {

// Flags of a segment: bodies reach beyond the clamp guard's coordinate limit;
// so many of them lie in leaves deeper than walk_depth (SegDev::deep) that the
// default force pass does the segment without the group walk.
constexpr uint32_t kSegWide = 1u, kSegDeep = 2u;

// Per-segment record in device memory.
struct SegDev {
  uint32_t start, count; // body range [start, start+count)
  // written every step (one store resets both)
  uint32_t flags; // kSegWide, kSegDeep
  uint32_t deep;  // bodies in leaves deeper than walk_depth
  float cell, invCell, smallW; // collision grid cell; boxes wider than
                               // smallW go to the large list
  // written every step
  float cx, cy, size; // root square (Quad::newContaining)
  MortonFrame frame;  // quantisation constants (binary64 bit patterns)
  uint32_t nodeBase;  // first node of this segment's tree (breadth-first
                      // arrays, the reference's numbering)
  uint32_t nodeCount; // nodes in this segment's tree
  uint32_t levelCount;
  uint32_t largeStart, largeCount;
  uint32_t travCount; // nodes in the traversal layout (non-empty nodes)
  uint32_t travBase;  // first record of this segment's traversal layout
};

static_assert(offsetof(SegDev, flags) % 8 == 0 && alignof(SegDev) == 8 &&
                  offsetof(SegDev, deep) == offsetof(SegDev, flags) + 4,
              "flags and deep are one 8-byte word");

// A node of the force traversal, in depth-first preorder: a = {comX, comY,
// mass, size*size}, b = {next, open, start, end}: next = the slot after the
// node's subtree (preorder, global; all ones past the instance's last node),
// open = where a walk that opens the node goes (next for a leaf, the next
// slot -- its first child -- for an interior node, so a node is a leaf iff
// open == next), [start, end) = its bodies.  32-byte aligned so that the
// traversal reads a record with one 256-bit load.
struct alignas(32) TravNode {
  float4 a;
  int4 b;
};
static_assert(sizeof(TravNode) == 32, "32-byte traversal records");

// The (up to four) children of a branching node for the default force walk,
// in digit order as arrays of four: centre of mass, mass and squared size;
// per child a link -- kQuadLeaf | body count for a leaf, the
// child's own record otherwise -- and its first body.  An absent child has
// no mass and a link to an empty leaf.
// A chain of nodes with one non-empty child each is one child here: its
// nodes hold the same bodies, so they share centre of mass and mass bit for
// bit, a walk that accepts any of them adds the same term, and it accepts
// one of them iff it accepts the smallest.  So every record branches, and is
// stored at the index of the first body of its node's second child, which
// no other branching node shares: at most one record per body.  An
// instance's root is the only child of a record of its own, n + instance.
struct alignas(32) QuadRec {
  float4 x, y, m, w;
  uint2 child[4]; // {link, first body}
};
static_assert(sizeof(QuadRec) == 96, "three 32-byte loads");
// The same children for the quadrupole term: {Ixx, Iyy, Ixy, squared size of
// the largest node of the child's chain}.
struct alignas(32) QuadMom {
  float4 m[4];
};
constexpr uint32_t kQuadLeaf = 0x80000000u;
// Bodies up to which exact arithmetic and the quadrupole term walk in groups
// (launch_forces).
constexpr uint32_t kOrderedGroupsMax = 65536;

constexpr int kMaxDepth = 32;   // TreeKernels.cuh:29
constexpr int kLevelSlots = 34; // depths 0..32 plus an end slot

// counters[] slot of the force law's clamp guard.  The force pass may
// leave out the law's FLT_MAX clamp only while every distance it forms
// stays finite: the upload stores the largest coordinate allowed here
// (float bits), and each build marks the instances whose bodies reach
// beyond it (kSegWide), for the force pass to keep the clamp there.
constexpr int kCtrCoordLimit = 15;
constexpr int kCtrSpans = 11; // spanning nodes of the build (DevState::spanList)
constexpr int kCtrBoundsDone = 7; // blocks of the bounds pass done (self-resetting)

// Everything a step's kernels touch.  All pointers are device pointers.
struct DevState {
  uint32_t n;     // bodies over all segments
  uint32_t nseg;  // segments
  uint32_t nodeCapacity;
  uint32_t pairCapacity;
  float dt, tSq, eSq;
  int leafCapacity;
  int collisions;
  // force targets [forceBegin, forceEnd) of a force launch; forceEnd 0:
  // every body (the step graphs of nbx_step_io split the pass in ranges)
  uint32_t forceBegin, forceEnd;
  // with recOut, the force pass also writes each target's 9-word body
  // record (the nbx_body layout) there
  uint32_t *recOut;

  SegDev *seg;
  uint16_t *segOf; // segment of each body index (never permuted)

  // body state, current order (double-buffered across the Morton gather)
  float4 *pv;   // {x, y, vx, vy}
  float2 *mr;   // {mass, radius}
  uint32_t *id; // Body::id
  float4 *pv2;
  float2 *mr2;
  uint32_t *id2;
  float2 *acc;  // accelerations from the last force pass
  float4 *xym;  // {x, y, mass, 0} in Morton order (tree + forces)

  // bounds as float order keys: [seg][minX, maxX, minY, maxY]
  uint32_t *bounds;
  uint32_t *status; // error bits

  // collision scratch
  float4 *box;           // {minX, maxX, minY, maxY}
  int2 *cellXY;          // grid cell of small boxes
  uint32_t *slot;        // slot in bucket (small) or in large list (|bit31)
  uint32_t *bucketCount; // [buckets]
  uint32_t *bucketStart; // [buckets+1]
  uint32_t *grid;        // body index per bucket slot
  float4 *gridBox;       // the box of that body (read with the index)
  uint32_t nBuckets;     // power of two
  uint32_t *largeCount;  // [nseg]
  uint32_t *largeStartA; // [nseg]
  uint32_t *largeList;   // [n]
  uint32_t *deg;         // partners per body
  uint32_t *pstart;      // CSR start per body
  uint32_t *plist;       // partner indices
  uint32_t *plistTmp;    // scratch copy used to sort large bodies' lists
  uint32_t *twin;        // per as-later entry: the partner's chain entry
                         // (index | kFirstEntry | kLastEntry)
  float4 *chain;         // per chain entry: the body's state after it
                         // (published entries only; sentinel until then)
  uint32_t *stash;       // first partners of each body found by the count pass
  uint2 *largePairs;     // (large, small) pairs found by the count pass
  uint32_t *fillLarge;   // fill counters of large bodies
  uint32_t *nLater;      // partners that sort before the body
  uint32_t *unitOrder;   // units in before() order (last collide)
  uint32_t *longRuns;    // Morton sort: starts of runs of > 16 equal high keys
  uint32_t *counters;    // [0]=pairs*2 total [1]=units [2]=unit claim
                         // [3]=splitting entries [4]=total nodes
                         // [5]=small-large pairs [6]=traversal records
                         // [8]=id check
                         // [9]=long Morton runs [12]=upload mass bits
                         // [kCtrSpans] (above)
                         // [7]=bounds blocks done [10]=long unit runs
                         // [13]=expiry test flag [kCtrCoordLimit] (above)

  // Morton / sort
  uint64_t *codes; // unsorted codes (kept for the segment passes)
  uint32_t *perm;  // Morton permutation of the last build (sorted -> old)
  uint64_t *sortedCodes;

  // tree build
  uint32_t *splitCount; // per body
  uint32_t *splitStart;
  uint8_t *splitLo;
  uint32_t *groupStart; // [nseg][kLevelSlots]
  uint32_t *groupEnd;
  uint32_t *levelStart; // [nseg][kLevelSlots+1]
  // BFS-numbered node arrays (TreeKernels.cuh NodeArrays layout)
  float *comX, *comY, *mass, *centerX, *centerY, *size;
  int32_t *children, *next, *start, *end;
  int32_t *parent;
  float *sumX, *sumY;   // raw weighted sums (before the CoM divide)
  float4 *moments;      // {Ixx, Iyy, Ixy, spare}
  uint32_t *subtree;    // nodes in subtree
  uint32_t *arrive;     // bottom-up arrival counters
  // nodes of the traversal layout that reach beyond their block of the build
  // (k_trav_tree): their {record, depth, bodies, first body}, and by (block,
  // depth) the parent record and, empty between builds, the bodies of the
  // children summed in blocks and of those summed at the top, and the
  // children's records by digit
  uint4 *spanList;
  uint32_t *spanParent, *spanArrive, *spanArriveTop;
  uint4 *spanKids;
  // traversal layout (preorder)
  TravNode *tN; // preorder traversal records (32 bytes, one load each)
  QuadRec *tQ;  // records of the group walks (n + nseg)
  QuadMom *tQM; // their moments, where the build computes them (null where they
                // are not there to be read, as beyond kOrderedGroupsMax bodies)
  float4 *tUp; // per traversal record, upward pass: {weighted sums x, y,
               // bottom size^2, link bits}; shares the breadth-first arrays'
               // storage (comX ..)
  // target groups of the default force walk: runs of up to 32 consecutive
  // bodies that never cross an instance, so that a body's group, and with it
  // the order of its sums, is the same in an ensemble and on its own
  uint32_t *groupFirst; // first body of each group (nseg > 1; else 32 g)
  uint32_t nGroups;
  uint32_t largest;        // bodies of the largest instance
  uint32_t tgBegin, tgEnd; // groups of [forceBegin, forceEnd)
  float4 *tM; // {Ixx, Iyy, Ixy, size} for the learned correction
  float2 *tC; // square centre, for the learned correction

  // attractor: [0] = {x, y, mass, softening}, [1].x = active (0 or 1);
  // device-resident so it can move between steps of a captured graph
  float4 *attr;
};

// Points of nbx_accel_at that are not sorted first: a warp or two anyway.
constexpr uint32_t kQueryUnsorted = 64;

// Camera and draw settings of the splat renderer (render.cu).
struct RenderParams {
  float camX, camY, scale, halfW, halfH;
  uint32_t width, height, tilesX, tilesY;
  int mode; // 0 speed ramp, over-composited; 1 glow, additive
  float pointScale, minPoint, brightness, speedMax;
};

// The viewer's attractor pull (attractorKernel, src/cuda/CudaSimulation.cu
// :14-31): acc += d * m / (sqrt(|d|^2 + 1e-12) (|d|^2 + soft^2)), d = a - p,
// added after the gravitational sum.  kExact: IEEE reciprocal square root
// and division, no contraction; otherwise the hardware rsqrt, an IEEE
// division and fused multiply-adds, as the reference's kernel compiles.
template <bool kExact>
__device__ __forceinline__ void add_attractor(const float4 *attr, float px, float py,
                                              float &ax, float &ay) {
  if (attr[1].x == 0.0f) return;
  const float4 a = attr[0];
  if (kExact) {
    const float dx = __fsub_rn(a.x, px), dy = __fsub_rn(a.y, py);
    const float dSq = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
    const float f = __fdiv_rn(__fmul_rn(a.z, __frcp_rn(__fsqrt_rn(__fadd_rn(dSq, 1e-12f)))),
                              __fadd_rn(dSq, __fmul_rn(a.w, a.w)));
    ax = __fadd_rn(ax, __fmul_rn(dx, f));
    ay = __fadd_rn(ay, __fmul_rn(dy, f));
  } else {
    const float dx = a.x - px, dy = a.y - py;
    const float dSq = dx * dx + dy * dy;
    const float f = __fdiv_rn(a.z * rsqrtf(dSq + 1e-12f), dSq + a.w * a.w);
    ax = fmaf(dx, f, ax);
    ay = fmaf(dy, f, ay);
  }
}

// quantise() in native FP64 (TreeKernels.cuh:48-57): one IEEE subtract and
// one multiply, each rounded (no contraction), then floor -- the same
// doubles as the reference's, bit for bit, from the frame's binary64 bits.
__device__ __forceinline__ uint32_t quantise_fp64(float v, double lo, double scale) {
  const double q = floor(__dmul_rn(__dsub_rn((double)v, lo), scale));
  if (!(q > 0.0)) return 0u; // also NaN
  if (q >= 4294967295.0) return 0xFFFFFFFFu;
  return (uint32_t)q;
}

// Morton code of a body at {x, y} in its instance's frame.
__device__ __forceinline__ uint64_t body_code(float4 p, const MortonFrame &f) {
  const double sc = __longlong_as_double((long long)f.scale);
  return (spread_bits(quantise_fp64(p.y, __longlong_as_double((long long)f.y0), sc)) << 1) |
         spread_bits(quantise_fp64(p.x, __longlong_as_double((long long)f.x0), sc));
}

// Depth of a leaf beyond which the group walk (force.cu) hardly ever fits its
// scratch: a walk opens about as many records at every level.  Leaf depths at which half
// the groups fit, theta 0.4 / 0.45 / 0.5 / 0.6: a cusp (density as r^-1.6) 11 / 13
// / 16 / 19, Plummer's density 14 / 16 / 17 to 18 / over 20; bodies spread evenly lie
// at depth 9 (2^20) or 10 (2^22).
__device__ __forceinline__ int walk_depth(float tSq) {
  return (int)(36.0f * sqrtf(tSq) - 1.5f);
}

// Adds bodies of a segment in deeper leaves.  kSegDeep from an eighth of its bodies
// on: a cursor takes about twice the time at the group walk's occupancy, and
// groups save a fifth.
__device__ __forceinline__ void add_deep(SegDev &G, uint32_t bodies) {
  const uint32_t limit = G.count / 8u, before = atomicAdd(&G.deep, bodies);
  if (before <= limit && before + bodies > limit) atomicOr(&G.flags, kSegDeep);
}

__device__ __forceinline__ float key_to_float(uint32_t k) {
  return u2f((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Root square of instance sg (Quad::newContaining, QuadTree.cpp:30-51, and
// rootSquare, CudaQuadTree.cu:25-30) and its Morton frame, from the step's
// bound accumulators, which it resets for the next step.
__device__ __forceinline__ void root_frame_seg(const DevState &S, uint32_t sg) {
  uint32_t *b = S.bounds + 4 * sg;
  const uint32_t k0 = __ldcg(b), k1 = __ldcg(b + 1), k2 = __ldcg(b + 2), k3 = __ldcg(b + 3);
  const float minX = k0 == 0xffffffffu ? FLT_MAX : key_to_float(k0);
  const float maxX = k1 == 0u ? -FLT_MAX : key_to_float(k1);
  const float minY = k2 == 0xffffffffu ? FLT_MAX : key_to_float(k2);
  const float maxY = k3 == 0u ? -FLT_MAX : key_to_float(k3);
  const float cx = __fmul_rn(__fadd_rn(minX, maxX), 0.5f);
  const float cy = __fmul_rn(__fadd_rn(minY, maxY), 0.5f);
  const float w = __fsub_rn(maxX, minX), h = __fsub_rn(maxY, minY);
  const float size = (w < h) ? h : w;
  SegDev &G = S.seg[sg];
  G.cx = cx;
  G.cy = cy;
  G.size = size;
  // sd_morton_frame's binary64 steps in native FP64: the same IEEE
  // operations, each correctly rounded, give the same bits
  const double half = __dmul_rn(0.5, (double)size);
  G.frame.x0 = (uint64_t)__double_as_longlong(__dsub_rn((double)cx, half));
  G.frame.y0 = (uint64_t)__double_as_longlong(__dsub_rn((double)cy, half));
  G.frame.scale = size > 0.0f ? (uint64_t)__double_as_longlong(__ddiv_rn(4294967296.0, (double)size))
                              : 0ull;
  // clamp guard: bodies beyond the upload's coordinate limit (NaN-safe)
  const float lim = __uint_as_float(S.counters[kCtrCoordLimit]);
  const float reach = fmaxf(fmaxf(fabsf(minX), fabsf(maxX)), fmaxf(fabsf(minY), fabsf(maxY)));
  *reinterpret_cast<uint2 *>(&G.flags) =
      make_uint2((k0 != 0xffffffffu && !(reach < lim)) ? kSegWide : 0u, 0u);
  b[0] = 0xffffffffu;
  b[1] = 0u;
  b[2] = 0xffffffffu;
  b[3] = 0u;
}

// The step's two sorts for few bodies, one launch each (scan_sort.cu): the
// Morton codes of a single instance of at most kClusterMortonMax bodies, made
// here too (the permutation goes to scratch.vals[0]), and the contact units
// among at most kClusterSortMax bodies, whose keys are in keys32(scratch, 0),
// every other body's key being nonUnit (the units go to the first places of
// scratch.vals[1]).
constexpr uint32_t kClusterMortonMax = 20480, kClusterSortMax = 65536;
void cluster_sort_morton(cudaStream_t s, const DevState &S, SortScratch &scratch);
void cluster_sort_units(cudaStream_t s, const DevState &S, SortScratch &scratch,
                        uint32_t nonUnit);

} // namespace nbx
