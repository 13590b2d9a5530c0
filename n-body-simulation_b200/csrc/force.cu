// force.cu -- warp-cooperative Barnes-Hut traversal.
//
// Every walk here gives each body exactly the terms accelerationAt does
// (src/cuda/TreeKernels.cuh:197-245; QuadTree::acceleration,
// src/QuadTree.cpp:264-389): accept a node when size^2 < d^2*theta^2 and
// add m*d*fastInvSqrt(d^2)/(d^2+eps^2) (clamped to FLT_MAX), otherwise sum
// a leaf's bodies one by one, otherwise descend.
//
// The default force pass walks the tree once per group of 32 bodies over
// records of four children (walk_group), and so do queries, and exact
// arithmetic and the quadrupole term of few bodies.  Many of those, the
// learned correction (walk_learned), the clamped law, counting, short walks of many
// bodies (group_walk_pays), uneven states (k_forces_deep) and whatever does not
// fit a group's scratch keep a cursor per lane (walk_targets, walk_plain_x2): along
// a lane's walk of the depth-first preorder layout (build.cu) the position only
// increases (descend = +1, skip = +subtree size), so the warp always serves the
// smallest position any lane is waiting at.  The node's record is read once
// per warp (one broadcast load through L1; staging 32-node tiles in shared memory
// measured 9-11% slower for the extra per-iteration bookkeeping); a leaf's bodies
// are staged in shared memory with one coalesced load.
//
// kExact = true evaluates every float operation as the reference writes
// it (no FMA contraction, IEEE reciprocal): the result is bit-identical to
// the host-compiled reference traversal on the same tree.  kExact = false
// lets the compiler contract and uses the hardware reciprocal
// approximation (relative difference ~1e-7 per term).
#include "mlp.cuh"
#include "nbx_state.cuh"

#include <algorithm>
#include <float.h>

namespace nbx {
namespace {

constexpr int kForceBlock = 256;
constexpr int kWarps = kForceBlock / 32;
constexpr uint32_t kDone = 0xffffffffu;

// One traversal record with a single 256-bit read-only load (sm_100); the
// records are 32-byte aligned (TravNode).
__device__ __forceinline__ void ld_node(const TravNode *p, float4 &a, int4 &b) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z),
        "=r"(b.w)
      : "l"(p));
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

template <bool kExact>
__device__ __forceinline__ float inv_sqrt_law(float x) {
  if (kExact) {
    const float xhalf = __fmul_rn(0.5f, x);
    const float y = u2f(0x5f3759dfu - (f2u(x) >> 1));
    return __fmul_rn(y, __fsub_rn(1.5f, __fmul_rn(__fmul_rn(xhalf, y), y)));
  } else {
    return fast_inv_sqrt(x);
  }
}

// The tree force law's factor m * fastInvSqrt(d^2) / (d^2 + eps^2), clamped
// to FLT_MAX (the term is d * factor).  kClamp = false leaves the clamp out
// where it cannot act: fastInvSqrt never exceeds ~2e19 (its value at 0), so
// with eps > 0 and every |m| < 1.6e19 * min(1, eps^2) neither m * fastInvSqrt
// nor the factor reaches FLT_MAX (the host checks this before choosing it).
template <bool kExact, bool kClamp = true>
__device__ __forceinline__ float law_factor(float dSq, float m, float eSq) {
  if (kExact)
    return fminf(__fmul_rn(__fmul_rn(m, inv_sqrt_law<true>(dSq)),
                           __frcp_rn(__fadd_rn(dSq, eSq))),
                 FLT_MAX);
  const float f = m * inv_sqrt_law<false>(dSq) * rcp_approx(dSq + eSq);
  return kClamp ? fminf(f, FLT_MAX) : f;
}

// One interaction of the tree force law; accumulates into (ax, ay).
template <bool kExact, bool kClamp = true>
__device__ __forceinline__ void add_term(float dx, float dy, float dSq,
                                         float m, float eSq, float &ax,
                                         float &ay) {
  if (kExact) {
    const float f = fminf(__fmul_rn(__fmul_rn(m, inv_sqrt_law<true>(dSq)),
                                    __frcp_rn(__fadd_rn(dSq, eSq))),
                          FLT_MAX);
    ax = __fadd_rn(ax, __fmul_rn(dx, f));
    ay = __fadd_rn(ay, __fmul_rn(dy, f));
  } else {
    const float f = law_factor<false, kClamp>(dSq, m, eSq);
    ax = fmaf(dx, f, ax);
    ay = fmaf(dy, f, ay);
  }
}

template <bool kExact>
__device__ __forceinline__ float sq_dist(float dx, float dy) {
  if (kExact) return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
  return fmaf(dx, dx, dy * dy);
}

// kCount: instead of writing accelerations, add the walk's far (accepted,
// mass > 0), near (leaf body terms) and visited-node counts to counts[0..2].
// Second-order (quadrupole) term of the softened law for a cell with mass
// M and second moments I about its centre of mass, relative to the kernel
// g(r) = 1/(r (r^2 + eps^2)) of the monopole M g d:
//   delta = 1/2 [ (g'/r)(2 I d + tr(I) d) + (g''/r^2 - g'/r^3) d (d'Id) ],
// returned divided by M g so that the cell term is fac * (d + delta/(M g)).
__device__ __forceinline__ void quad_term(float dx, float dy, float dSq,
                                          float eSq, float mass, float ixx,
                                          float iyy, float ixy, float &qx,
                                          float &qy) {
  const float q = dSq + eSq;
  // a correction term: the hardware reciprocal's ~1 ulp is far below its
  // own truncation error
  const float iq = rcp_approx(q), ir2 = rcp_approx(dSq);
  const float c3 = 3.0f * dSq + eSq;
  const float aOverG = -c3 * ir2 * iq;                        // g'/(r g)
  const float gpp = -6.0f * iq + c3 * (2.0f * ir2 * iq + 4.0f * iq * iq);
  const float bOverG = gpp * ir2 + c3 * ir2 * ir2 * iq;       // B / g
  const float Idx = ixx * dx + ixy * dy, Idy = ixy * dx + iyy * dy;
  const float tr = ixx + iyy;
  const float dId = dx * Idx + dy * Idy;
  const float h = 0.5f * rcp_approx(mass);
  qx = h * (aOverG * (2.0f * Idx + tr * dx) + bOverG * dx * dId);
  qy = h * (aOverG * (2.0f * Idy + tr * dy) + bOverG * dy * dId);
}

// One warp's walk: lane targets (x, y) start at node cur (kDone: none) and
// add their terms to (ax, ay); kCount adds the walk's counts instead.
// kCorr = 2: accepted cells with size^2 >= d^2 * band^2 get the analytic
// quadrupole term (the control of the learned correction, walk_learned).
template <bool kExact, bool kCount, int kCorr, bool kClamp>
__device__ __forceinline__ void walk_targets(
    const DevState &S, float tSq, float eSq, float bandSq, float x, float y, uint32_t cur,
    float4 *sBodyW, float &ax, float &ay, uint32_t &nFar, uint32_t &nNear, uint32_t &nVisit,
    uint32_t &nIter, uint32_t &nChunk) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    const uint32_t k = __reduce_min_sync(0xffffffffu, cur);
    if (k == kDone) break;
    if (kCount) ++nIter;
    // k is the same for the whole warp: one broadcast 256-bit load
    float4 A;
    int4 B;
    ld_node(&S.tN[k], A, B);
    // the node after k's subtree (kDone past the instance's last node)
    const uint32_t nxt = (uint32_t)B.x;
    // every lane evaluates the node; only the lanes waiting at it use it
    const bool at = cur == k;
    const float dx = kExact ? __fsub_rn(A.x, x) : A.x - x;
    const float dy = kExact ? __fsub_rn(A.y, y) : A.y - y;
    const float dSq = sq_dist<kExact>(dx, dy);
    const float far = kExact ? __fmul_rn(dSq, tSq) : dSq * tSq;
    const bool accept = at && A.w < far;
    const bool openLeaf = at && !accept && B.y == B.x; // leaf: open == next
    {
      // the reference adds a cell only if its mass is > 0; in the clamp-free
      // plain walk masses are >= 0 and every term is finite, so a massless
      // cell's term is exactly +-0 and the mass test can go
      constexpr bool kZeroMassAddsNothing = !kExact && !kClamp && kCorr == 0;
      const bool use = accept && (kZeroMassAddsNothing || A.z > 0.0f);
      const float fac = law_factor<kExact, kClamp>(dSq, A.z, eSq);
      float tx, ty;
      if (kExact) {
        tx = __fadd_rn(ax, __fmul_rn(dx, fac));
        ty = __fadd_rn(ay, __fmul_rn(dy, fac));
      } else {
        tx = fmaf(dx, fac, ax);
        ty = fmaf(dy, fac, ay);
      }
      if (kCorr == 2) {
        const bool band = use && A.w >= dSq * bandSq;
        if (__ballot_sync(0xffffffffu, band)) {
          const float4 M = S.tM[k];
          float qx, qy;
          quad_term(dx, dy, dSq, eSq, A.z, M.x, M.y, M.z, qx, qy);
          if (band) {
            tx = ax + fac * (dx + qx);
            ty = ay + fac * (dy + qy);
          }
        }
      }
      ax = use ? tx : ax;
      ay = use ? ty : ay;
      if (kCount) nFar += use ? 1u : 0u;
    }
    if (kCount) nVisit += at ? 1u : 0u;
    // accepted: skip the subtree; opened: the node's open slot (skip a
    // leaf, descend into an interior node)
    cur = at ? (accept ? nxt : (uint32_t)B.y) : cur;
    const uint32_t leafLanes = __ballot_sync(0xffffffffu, openLeaf);
    if (leafLanes) {
      const uint32_t b0 = (uint32_t)B.z, b1 = (uint32_t)B.w;
      const uint32_t bEnd = b1 <= S.n ? b1 : S.n; // defensive bound
      for (uint32_t base = b0; base < bEnd; base += 32) {
        const uint32_t cnt = min(32u, bEnd - base);
        if (kCount) ++nChunk;
        __syncwarp();
        if ((uint32_t)lane < cnt) sBodyW[lane] = S.xym[base + lane];
        __syncwarp();
#pragma unroll 4
        for (uint32_t j = 0; j < cnt; ++j) {
          const float4 q = sBodyW[j];
          const float ex = kExact ? __fsub_rn(q.x, x) : q.x - x;
          const float ey = kExact ? __fsub_rn(q.y, y) : q.y - y;
          float tx = ax, ty = ay;
          add_term<kExact, kClamp>(ex, ey, sq_dist<kExact>(ex, ey), q.z, eSq, tx, ty);
          ax = openLeaf ? tx : ax;
          ay = openLeaf ? ty : ay;
        }
      }
      if (kCount && openLeaf) nNear += bEnd > b0 ? bEnd - b0 : 0u;
    }
  }
}

// One warp's walk with the learned correction (mlp.cuh) of the accepted
// cells with size^2 >= d^2 * band^2, in rounds: the warp walks on (a cursor per
// lane, as walk_targets) and lists the nodes that give some lane a term, and
// the (node, lane) rows that want the network; then evaluates 32 rows at a
// time on the tensor cores; then adds the round's terms in the list's order,
// so every lane's sum is that of evaluating each node's rows on the spot.
// There a call of the network (~400 instructions) holds only the few
// lanes that are at the node: 100,000 bodies of a disc, theta 0.7, band 0.5,
// 412 us; in rounds 221, of which the warps issue for half, with the longest
// walks (one wave of warps) the rest.
constexpr uint32_t kLearnedNodes = 96, kLearnedRows = 224;
struct LearnedStage {
  uint4 node[kLearnedNodes]; // record, lanes that add it, correct it, open it
  float2 term[kLearnedRows]; // a row's corrected direction, to be scaled by the law's factor
  union {
    __nv_bfloat16 feat[32][16]; // while evaluating
    float4 body[32];            // while adding: a leaf's bodies
  };
  uint16_t row[kLearnedRows]; // node << 5 | lane
};
static_assert(kLearnedNodes << 5 <= 65536u, "a row fits 16 bits");

__device__ __forceinline__ void walk_learned(const DevState &S, float tSq, float eSq,
                                             float bandSq, float eps, float x, float y,
                                             uint32_t cur, LearnedStage &st, const MlpDev &sW,
                                             float &ax, float &ay) {
  const int lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
  for (bool more = true; more;) {
    uint32_t nodes = 0, rows = 0;
    while (nodes < kLearnedNodes && rows + 32u <= kLearnedRows) {
      const uint32_t k = __reduce_min_sync(0xffffffffu, cur);
      if (k == kDone) {
        more = false;
        break;
      }
      float4 A;
      int4 B;
      ld_node(&S.tN[k], A, B);
      const bool at = cur == k;
      const float dx = A.x - x, dy = A.y - y;
      const float dSq = sq_dist<false>(dx, dy);
      const bool accept = at && A.w < dSq * tSq;
      const bool use = accept && A.z > 0.0f;
      const bool band = use && A.w >= dSq * bandSq;
      cur = at ? (accept ? (uint32_t)B.x : (uint32_t)B.y) : cur;
      const uint32_t adds = __ballot_sync(0xffffffffu, use);
      const uint32_t opens = __ballot_sync(0xffffffffu, at && !accept && B.y == B.x);
      if ((adds | opens) == 0u) continue;
      const uint32_t corrects = __ballot_sync(0xffffffffu, band);
      if (band) st.row[rows + __popc(corrects & below)] = (uint16_t)(nodes << 5 | lane);
      if (lane == 0) st.node[nodes] = make_uint4(k, adds, corrects, opens);
      rows += __popc(corrects);
      ++nodes;
    }
    __syncwarp();
    for (uint32_t r = 0; r < rows; r += 32) {
      const bool on = r + lane < rows;
      const uint32_t row = st.row[on ? r + lane : r];
      const float px = __shfl_sync(0xffffffffu, x, row & 31u);
      const float py = __shfl_sync(0xffffffffu, y, row & 31u);
      const uint32_t k = st.node[row >> 5].x;
      const float4 A = S.tN[k].a, M = S.tM[k];
      const float2 Q = S.tC[k];
      const float dx = A.x - px, dy = A.y - py;
      const float dSq = sq_dist<false>(dx, dy);
      float f[9], ux = 0.0f, uy = 0.0f;
      const bool ok = on && mlp_features(dx, dy, dSq, A.z, M.w, Q.x, Q.y, A.x, A.y, M.x, M.y,
                                         M.z, 1.0f, eps, f, ux, uy);
      if (!ok)
        for (int q = 0; q < 9; ++q) f[q] = 0.0f;
      float o0, o1;
      mlp_warp(sW, f, st.feat, o0, o1);
      float2 term = make_float2(dx, dy);
      if (ok) {
        // |mono| * ((1 + t0) u + t1 w), w = (-uy, ux)
        const float d = dSq * rsqrtf(dSq);
        term = make_float2(dx * (1.0f + o0) - d * o1 * uy, dy * (1.0f + o0) + d * o1 * ux);
      }
      if (on) st.term[r + lane] = term;
    }
    __syncwarp();
    rows = 0;
    for (uint32_t e = 0; e < nodes; ++e) {
      const uint4 N = st.node[e];
      float4 A;
      int4 B;
      ld_node(&S.tN[N.x], A, B);
      const float dx = A.x - x, dy = A.y - y;
      const float fac = law_factor<false, true>(sq_dist<false>(dx, dy), A.z, eSq);
      float2 term = make_float2(dx, dy);
      if ((N.z >> lane) & 1u) term = st.term[rows + __popc(N.z & below)];
      rows += __popc(N.z);
      const bool use = (N.y >> lane) & 1u, open = (N.w >> lane) & 1u;
      ax = use ? fmaf(term.x, fac, ax) : ax;
      ay = use ? fmaf(term.y, fac, ay) : ay;
      if (N.w == 0u) continue;
      const uint32_t b0 = (uint32_t)B.z, b1 = (uint32_t)B.w;
      const uint32_t bEnd = b1 <= S.n ? b1 : S.n; // defensive bound
      for (uint32_t base = b0; base < bEnd; base += 32) {
        const uint32_t cnt = min(32u, bEnd - base);
        __syncwarp();
        if ((uint32_t)lane < cnt) st.body[lane] = S.xym[base + lane];
        __syncwarp();
#pragma unroll 4
        for (uint32_t j = 0; j < cnt; ++j) {
          const float4 q = st.body[j];
          const float ex = q.x - x, ey = q.y - y;
          float tx = ax, ty = ay;
          add_term<false, true>(ex, ey, sq_dist<false>(ex, ey), q.z, eSq, tx, ty);
          ax = open ? tx : ax;
          ay = open ? ty : ay;
        }
      }
    }
    __syncwarp();
  }
}

// The default plain walk (contracted arithmetic, clamp-free law, no
// correction, no counting) with a cursor per lane and paired FP32 instructions: the cell term's
// {dx, dy} and its accumulation are one pair each, and a leaf's bodies are
// taken two at a time (structure-of-arrays staging, so one 64-bit shared
// load gives two bodies' x, y or mass).  Each body accepts, opens and skips
// exactly the nodes walk_targets does, and every term is the same float
// arithmetic; only the leaf terms' summation order changes (two running
// sums, added to the cell terms at the end).
__device__ __forceinline__ void walk_plain_x2(const DevState &S, float tSq, float eSq,
                                              float x, float y, uint32_t cur,
                                              float *sX, float *sY, float *sM,
                                              float &axOut, float &ayOut) {
  const int lane = threadIdx.x & 31;
  const f2x P = pk2(x, y), XX = pk2(x, x), YY = pk2(y, y), E2 = pk2(eSq, eSq);
  const f2x NHALF = pk2(-0.5f, -0.5f), THREEHALF = pk2(1.5f, 1.5f);
  f2x acc = pk2(0.0f, 0.0f);  // cell terms {ax, ay}
  f2x lx = pk2(0.0f, 0.0f), ly = pk2(0.0f, 0.0f); // leaf terms, two sums each
  for (;;) {
    const uint32_t k = __reduce_min_sync(0xffffffffu, cur);
    if (k == kDone) break;
    float4 A;
    int4 B;
    ld_node(&S.tN[k], A, B);
    const uint32_t nxt = (uint32_t)B.x;
    const bool at = cur == k;
    const f2x D = sub2(pk2(A.x, A.y), P);
    float dx, dy;
    upk2(D, dx, dy);
    const float dSq = fmaf(dx, dx, dy * dy);
    const bool accept = at && A.w < dSq * tSq;
    const bool openLeaf = at && !accept && B.y == B.x; // leaf: open == next
    // a massless cell adds exactly +-0 in the clamp-free law (masses >= 0,
    // finite terms), so no mass test
    float fac = A.z * fast_inv_sqrt(dSq) * rcp_approx(dSq + eSq);
    fac = accept ? fac : 0.0f;
    acc = fma2(D, pk2(fac, fac), acc);
    cur = at ? (accept ? nxt : (uint32_t)B.y) : cur;
    if (__ballot_sync(0xffffffffu, openLeaf)) {
      const uint32_t b0 = (uint32_t)B.z, b1 = (uint32_t)B.w;
      const uint32_t bEnd = b1 <= S.n ? b1 : S.n; // defensive bound
      for (uint32_t base = b0; base < bEnd; base += 32) {
        const uint32_t cnt = min(32u, bEnd - base);
        __syncwarp();
        if ((uint32_t)lane < cnt) {
          const float4 q = S.xym[base + lane];
          sX[lane] = q.x;
          sY[lane] = q.y;
          sM[lane] = q.z;
        } else if ((uint32_t)lane == cnt) { // odd count: a massless partner
          sX[lane] = 0.0f;
          sY[lane] = 0.0f;
          sM[lane] = 0.0f;
        }
        __syncwarp();
        if (openLeaf) {
          const uint32_t pairs = (cnt + 1) >> 1;
          for (uint32_t p = 0; p < pairs; ++p) {
            const f2x X2 = reinterpret_cast<const f2x *>(sX)[p];
            const f2x Y2 = reinterpret_cast<const f2x *>(sY)[p];
            const f2x M2 = reinterpret_cast<const f2x *>(sM)[p];
            const f2x EX = sub2(X2, XX), EY = sub2(Y2, YY);
            const f2x D2 = fma2(EX, EX, mul2(EY, EY));
            float d0, d1;
            upk2(D2, d0, d1);
            // fastInvSqrt of both: magic guess, one Newton step
            const f2x G = pk2(u2f(0x5f3759dfu - (f2u(d0) >> 1)),
                              u2f(0x5f3759dfu - (f2u(d1) >> 1)));
            const f2x T = mul2(mul2(D2, NHALF), G);
            const f2x IS = mul2(G, fma2(T, G, THREEHALF));
            float q0, q1;
            upk2(add2(D2, E2), q0, q1);
            const f2x F = mul2(mul2(M2, IS), pk2(rcp_approx(q0), rcp_approx(q1)));
            lx = fma2(EX, F, lx);
            ly = fma2(EY, F, ly);
          }
        }
      }
    }
  }
  float ax, ay, lx0, lx1, ly0, ly1;
  upk2(acc, ax, ay);
  upk2(lx, lx0, lx1);
  upk2(ly, ly0, ly1);
  axOut = ax + (lx0 + lx1);
  ayOut = ay + (ly0 + ly1);
}

// The law's factor m * fastInvSqrt(d^2) / (d^2 + eps^2) of two terms, from
// half masses.  With g the magic guess, the Newton step g (1.5 - 0.5 d^2 g g)
// is half of gn (d^2 gn gn - 3), gn = -g (the sign bit set in the guess's
// constant); negations and factors of two are exact, so every rounding is
// that of (m * g (1.5 - (0.5 d^2) g g)) * rcp, one operation less.
__device__ __forceinline__ f2x law_pair(f2x d2, f2x halfM, f2x e2, f2x neg3) {
  float d0, d1, q0, q1;
  upk2(d2, d0, d1);
  const f2x gn = pk2(u2f(0xdf3759dfu - (f2u(d0) >> 1)), u2f(0xdf3759dfu - (f2u(d1) >> 1)));
  const f2x is2 = mul2(gn, fma2(mul2(d2, gn), gn, neg3));
  upk2(add2(d2, e2), q0, q1);
  return mul2(mul2(halfM, is2), pk2(rcp_approx(q0), rcp_approx(q1)));
}

// acc += a * b where on != 0.
__device__ __forceinline__ void fma2_if(uint32_t on, f2x a, f2x b, f2x &acc) {
  asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p fma.rn.f32x2 %0, %2, %3, %0;\n\t}"
      : "+l"(acc)
      : "r"(on), "l"(a), "l"(b));
}
__device__ __forceinline__ void fma_if(uint32_t on, float dx, float dy, float f, float &ax,
                                       float &ay) {
  asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p fma.rn.f32 %0, %3, %5, %0;\n\t"
      "@p fma.rn.f32 %1, %4, %5, %1;\n\t}"
      : "+f"(ax), "+f"(ay)
      : "r"(on), "f"(dx), "f"(dy), "f"(f));
}

__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// One warp's scratch of walk_group.
constexpr int kTake = 16;     // records tested at once, four children each
constexpr int kSlots = 192;   // opened records (slots are bytes)
constexpr int kParts = 400;   // children that some lanes accept
constexpr int kCells = 704;   // cell terms
constexpr int kLeaves = 128;  // opened leaves
constexpr int kPairs = 448;   // pairs of their bodies (the plain walk)
constexpr int kTerms = 1408;  // cells and bodies (the walks that keep one order)
constexpr int kChunk = 32;    // terms summed at a time by those
struct alignas(16) WalkStage {
  union {
    struct { // children the lanes disagree on, their lanes, those that accept
      float cx[64], cy[64], cw[64];
      uint32_t cm[64], ca[64];
    };
    uint32_t count[kSlots]; // terms of a record's subtree, later its first
                            // place: cells | leaves << 10 | leaf pairs << 20,
                            // or items | terms << 10
    struct { // terms being summed: place, half mass, lanes (of each / a pair)
      float x[64], y[64], h[64];
      uint32_t m[64];
    };
    struct { // the same of the walks that keep one order: place, mass, lanes,
             // squared size; moments and the chain's largest squared size
      float4 q[kChunk], mom[kChunk];
      uint32_t lanes[kChunk];
    };
  };
  uint32_t rec[kSlots], who[kSlots]; // an opened record and its lanes
  uint32_t part[kParts];             // lanes that accept a child
  uint32_t starts[kTerms / 32];      // bit p: pair (or term) p starts a leaf (an item)
  uint16_t info[kSlots * 4];         // per child: kInfo bits | slot or pairs
  uint16_t partOf[kSlots * 4];       // per child with kInfoPart: index in part
  // in order, as slot << 2 | child: cells, leaves, or both: an item is a cell
  // or (| kItemLeaf) a leaf
  union {
    struct {
      uint16_t cell[kCells], leaf[kLeaves];
    };
    uint16_t item[kCells + kLeaves];
  };
  uint8_t batch[kSlots];             // first slot of each batch
};
static_assert(sizeof(WalkStage) == 9520, "20 warps: 190 KB of an SM's 228");
static_assert(kSlots <= 256 && kSlots * 4 < 1024 && kPairs < 4096 && kPairs <= kTerms,
              "packed fields");
constexpr uint32_t kItemLeaf = 1024u;
// What a group walk sums: the default law; the reference's operations; the
// default law with the quadrupole term.  The last two add a target's cells and
// bodies to one sum in the order of its walk (as walk_targets does).
enum GroupWalk { kPlainWalk, kExactWalk, kQuadWalk };
// a child's low byte: the slot of its opened record, or an opened leaf's pairs
constexpr uint32_t kInfoLeaf = 1u << 8, kInfoInner = 1u << 9;
constexpr uint32_t kInfoTerm = 1u << 10, kInfoPart = 1u << 11; // accepted, by some only

// The default plain walk for a group of targets of instance sg (lanes in
// `valid`; the others hold a copy of a valid target's place), with the
// result of walk_plain_x2 bit for bit: a body's cells are summed in preorder
// into one accumulator, its leaves' bodies in preorder into two.
// Bounded by instruction issue, so the tree is walked once for the group,
// with a node to a lane, instead of by every lane at every node:
//  * records open breadth-first, up to sixteen at a time: lanes 2 r and
//    2 r + 1 test two children each of record r against the group's box.  A target's own test is
//    w < fl(fl(dx^2 + dy^2) theta^2) with every rounding monotone in |dx| and
//    |dy|, so the same expression at the box's nearest (farthest) point is a
//    lower (upper) bound of every lane's: a child all lanes accept is a
//    term, one that none accepts is opened, with no test per lane.  The
//    children in between (a fifth) are tested by every lane, two to a paired
//    instruction;
//  * the batches are then passed in reverse to count each subtree's terms and
//    forwards to place them, which lists the terms in preorder;
//  * all lanes sum the lists, each term with the mask of the lanes it belongs
//    to: the law in pairs, the cells' accumulation one by one in order.
// kExactWalk and kQuadWalk are walk_targets' results bit for bit: cells and
// leaves are listed together, a term a place, and summed in one order, with
// the arithmetic written there.
// Returns false, with nothing summed, if the group's records do not fit.
//
// Two discs of 2^20 bodies, theta 0.5, per group: 95 records in 12 batches, 229
// whole cells, 86 children tested by lane, 34 leaves of 329 bodies; 14.3k
// warp instructions instead of walk_plain_x2's 18.6k.  The force pass takes
// 617 us there (719 before), 99,991 bodies 78 (131), 10,000 at theta 1 20 (36),
// 1000 16 (27): with few warps the walk's latency counts, and a group waits
// for ~12 dependent loads instead of ~400.  Of a group's 87k cycles the opening
// takes 30k, counting and placing 13k, the cells 19k, the leaves 25k.
// Measured and dropped: terms in the order the records open (528 us, no
// counting or placing, but another order of the sums); eight records at a
// time (630); 24 or 28 warps per SM at fewer registers (620, 640); both
// loops over terms unrolled twice more (645); the guess as one mad.hi (+13%).
template <GroupWalk kWalk>
__device__ __forceinline__ bool walk_group(const DevState &S, float tSq, float eSq, float bandSq,
                                           float x, float y, uint32_t sg, uint32_t valid,
                                           WalkStage &st, float &axOut, float &ayOut) {
  constexpr bool kExact = kWalk == kExactWalk, kOneOrder = kWalk != kPlainWalk;
  // (dx^2 + dy^2) theta^2 of two nodes with the roundings of a target's own
  // test.  (Exact: scalar, since a paired multiply and add came out fused and
  // decided one test in 10^7 otherwise.)
  auto far_of = [&](f2x dx, f2x dy, float &f0, float &f1) {
    if (kExact) {
      float x0, x1, y0, y1;
      upk2(dx, x0, x1);
      upk2(dy, y0, y1);
      f0 = __fmul_rn(sq_dist<true>(x0, y0), tSq);
      f1 = __fmul_rn(sq_dist<true>(x1, y1), tSq);
    } else {
      upk2(mul2(fma2(dx, dx, mul2(dy, dy)), pk2(tSq, tSq)), f0, f1);
    }
  };
  const int lane = threadIdx.x & 31;
  const uint32_t laneBit = 1u << lane, below = laneBit - 1u;
  const f2x XX = pk2(x, x), YY = pk2(y, y), E2 = pk2(eSq, eSq), N3 = pk2(-3.0f, -3.0f);
  const QuadRec *__restrict__ tQ = S.tQ;
  const uint32_t lastRec = S.n + S.nseg - 1u;
  uint32_t tail = 1, batches = 0;
  const int half = lane & 1;
  {
    f2x LOX, HIX, LOY, HIY;
    {
      const float loX = warp_min(x), hiX = warp_max(x), loY = warp_min(y), hiY = warp_max(y);
      LOX = pk2(loX, loX);
      HIX = pk2(hiX, hiX);
      LOY = pk2(loY, loY);
      HIY = pk2(hiY, hiY);
    }
    if (lane == 0) { // the root's record
      st.rec[0] = S.n + sg;
      st.who[0] = valid;
    }
    for (int k = lane; k < (kOneOrder ? kTerms : kPairs) / 32; k += 32) st.starts[k] = 0u;
    __syncwarp();
    uint32_t parts = 0, lanePairs = 0, laneItems = 0;
    for (uint32_t head = 0; head < tail;) {
      const uint32_t take = min((uint32_t)kTake, tail - head);
      const uint32_t slot = head + (lane >> 1);
      const bool have = (uint32_t)(lane >> 1) < take;
      f2x X2 = 0, Y2 = 0;
      float w[2] = {0.0f, 0.0f};
      uint32_t link[2] = {kQuadLeaf, kQuadLeaf}, mask = 0;
      if (have) {
        const QuadRec *q = tQ + st.rec[slot];
        mask = st.who[slot];
        X2 = __ldg(reinterpret_cast<const f2x *>(&q->x) + half);
        Y2 = __ldg(reinterpret_cast<const f2x *>(&q->y) + half);
        const float2 ww = __ldg(reinterpret_cast<const float2 *>(&q->w) + half);
        const uint4 cc = __ldg(reinterpret_cast<const uint4 *>(&q->child[0]) + half);
        w[0] = ww.x;
        w[1] = ww.y;
        link[0] = cc.x;
        link[1] = cc.z;
      }
      // per axis: how far the box lies beyond the child on either side
      float ax0[2], ax1[2], ay0[2], ay1[2], near2[2], far2[2];
      upk2(sub2(LOX, X2), ax0[0], ax0[1]);
      upk2(sub2(X2, HIX), ax1[0], ax1[1]);
      upk2(sub2(LOY, Y2), ay0[0], ay0[1]);
      upk2(sub2(Y2, HIY), ay1[0], ay1[1]);
      {
        const f2x NX = pk2(fmaxf(fmaxf(ax0[0], ax1[0]), 0.0f), fmaxf(fmaxf(ax0[1], ax1[1]), 0.0f));
        const f2x NY = pk2(fmaxf(fmaxf(ay0[0], ay1[0]), 0.0f), fmaxf(fmaxf(ay0[1], ay1[1]), 0.0f));
        const f2x FX = pk2(fminf(ax0[0], ax1[0]), fminf(ax0[1], ax1[1]));
        const f2x FY = pk2(fminf(ay0[0], ay1[0]), fminf(ay0[1], ay1[1]));
        far_of(NX, NY, near2[0], near2[1]);
        far_of(FX, FY, far2[0], far2[1]);
      }
      uint32_t accept[2], info[2], lanes[2];
      bool split[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        lanes[j] = link[j] == kQuadLeaf ? 0u : mask; // absent: no lane
        const bool all = w[j] < near2[j], none = !(w[j] < far2[j]);
        accept[j] = all ? lanes[j] : 0u;
        split[j] = lanes[j] != 0 && !all && !none;
        info[j] = split[j] ? kInfoPart : 0u;
      }
      const uint32_t s0 = __ballot_sync(0xffffffffu, split[0]);
      const uint32_t s1 = __ballot_sync(0xffffffffu, split[1]);
      if (s0 | s1) {
        const uint32_t at0 = __popc(s0 & below) + __popc(s1 & below);
        const uint32_t at[2] = {at0, at0 + (split[0] ? 1u : 0u)};
        const uint32_t n = __popc(s0) + __popc(s1);
        float px[2], py[2];
        upk2(X2, px[0], px[1]);
        upk2(Y2, py[0], py[1]);
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (split[j]) {
            st.cx[at[j]] = px[j];
            st.cy[at[j]] = py[j];
            st.cw[at[j]] = w[j];
            st.cm[at[j]] = lanes[j];
          }
        __syncwarp();
        for (uint32_t k = 0; k < n; k += 2) { // an odd last one's partner: unused
          const f2x DX = sub2(*reinterpret_cast<const f2x *>(&st.cx[k]), XX);
          const f2x DY = sub2(*reinterpret_cast<const f2x *>(&st.cy[k]), YY);
          const float2 cw2 = *reinterpret_cast<const float2 *>(&st.cw[k]);
          const uint2 m = *reinterpret_cast<const uint2 *>(&st.cm[k]);
          float r0, r1;
          far_of(DX, DY, r0, r1);
          const uint32_t a0 = m.x & __ballot_sync(0xffffffffu, cw2.x < r0);
          const uint32_t a1 = m.y & __ballot_sync(0xffffffffu, cw2.y < r1);
          if (lane == 0) *reinterpret_cast<uint2 *>(&st.ca[k]) = make_uint2(a0, a1);
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (split[j]) {
            accept[j] = st.ca[at[j]];
            if (parts + at[j] < kParts) {
              st.part[parts + at[j]] = accept[j];
              st.partOf[slot * 4 + 2 * half + j] = (uint16_t)(parts + at[j]);
            }
          }
        parts += n;
      }
      bool inner[2];
      uint32_t open[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        open[j] = lanes[j] & ~accept[j];
        inner[j] = open[j] != 0 && !(link[j] & kQuadLeaf);
        if (accept[j]) {
          info[j] |= kInfoTerm;
          ++laneItems;
        }
        if (open[j] != 0 && !inner[j]) {
          // an odd leaf's last body has a pair of its own
          const uint32_t bodies = link[j] & ~kQuadLeaf;
          const uint32_t pairs = kOneOrder ? bodies : (bodies + 1u) >> 1;
          lanePairs += min(pairs, 65536u);
          ++laneItems;
          info[j] |= (pairs & 255u) | kInfoLeaf;
          if (pairs > 255u) lanePairs = 65536u; // does not fit the byte
        }
      }
      const uint32_t p0 = __ballot_sync(0xffffffffu, inner[0]);
      const uint32_t p1 = __ballot_sync(0xffffffffu, inner[1]);
      uint32_t at = tail + __popc(p0 & below) + __popc(p1 & below);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (inner[j]) {
          if (at < kSlots) {
            st.rec[at] = min(link[j], lastRec); // defensive bound
            st.who[at] = open[j];
          }
          info[j] |= (at & 255u) | kInfoInner;
          ++at;
        }
      if (have) reinterpret_cast<uint32_t *>(st.info)[slot * 2 + half] = info[0] | info[1] << 16;
      if (lane == 0) st.batch[batches] = (uint8_t)head;
      ++batches;
      head += take;
      tail += __popc(p0) + __popc(p1);
      if (tail > kSlots || parts > kParts) return false;
      __syncwarp();
    }
    if (__reduce_add_sync(0xffffffffu, lanePairs) > (kOneOrder ? kTerms : kPairs)) return false;
    if (kOneOrder && __reduce_add_sync(0xffffffffu, laneItems) > kCells + kLeaves) return false;
  }
  // subtree counts, from the last batch to the first
  auto child_terms = [&](uint32_t info) {
    uint32_t v = info & kInfoTerm ? (kOneOrder ? 1u | 1u << 10 : 1u) : 0u;
    if (info & kInfoLeaf)
      v += kOneOrder ? (info & 255u) << 10 | 1u : (info & 255u) << 20 | 1u << 10;
    if (info & kInfoInner) v += st.count[info & 255u];
    return v;
  };
  for (uint32_t b = batches, end = tail; b-- > 0;) {
    const uint32_t head = st.batch[b], slot = head + (lane >> 1);
    const bool have = slot < end;
    const uint32_t info = have ? reinterpret_cast<const uint32_t *>(st.info)[slot * 2 + half] : 0u;
    uint32_t v = child_terms(info & 0xffffu) + child_terms(info >> 16);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if (have && half == 0) st.count[slot] = v;
    end = head;
    __syncwarp();
  }
  const uint32_t total = st.count[0], nCells = total & 1023u, nLeaves = total >> 10 & 1023u;
  const uint32_t nPairs = total >> 20, nTerms = total >> 10;
  if (kOneOrder ? nTerms > kTerms : nCells > kCells || nLeaves > kLeaves) return false;
  __syncwarp();
  if (lane == 0) st.count[0] = 0;
  __syncwarp();
  // places: a child's term, then its subtree's, then the next child's
  for (uint32_t b = 0; b < batches; ++b) {
    const uint32_t head = st.batch[b], end = b + 1 < batches ? st.batch[b + 1] : tail;
    const uint32_t slot = head + (lane >> 1);
    const bool have = slot < end;
    const uint32_t info2 = have ? reinterpret_cast<const uint32_t *>(st.info)[slot * 2 + half] : 0u;
    const uint32_t info[2] = {info2 & 0xffffu, info2 >> 16};
    const uint32_t v[2] = {child_terms(info[0]), child_terms(info[1])};
    const uint32_t before = __shfl_up_sync(0xffffffffu, v[0] + v[1], 1);
    if (have) {
      uint32_t at = st.count[slot] + (half ? before : 0u);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint16_t code = (uint16_t)(slot << 2 | (2 * half + j));
        if (kOneOrder) {
          uint32_t own = at;
          if (info[j] & kInfoTerm) {
            st.item[own & 1023u] = code;
            atomicOr(&st.starts[own >> 15], 1u << (own >> 10 & 31u));
            own += 1u | 1u << 10;
          }
          if (info[j] & kInfoInner) st.count[info[j] & 255u] = own;
          if (info[j] & kInfoLeaf) {
            st.item[own & 1023u] = (uint16_t)(code | kItemLeaf);
            atomicOr(&st.starts[own >> 15], 1u << (own >> 10 & 31u));
          }
        } else {
          if (info[j] & kInfoTerm) st.cell[at & 1023u] = code;
          if (info[j] & kInfoInner)
            st.count[info[j] & 255u] = at + (info[j] & kInfoTerm ? 1u : 0u);
          if (info[j] & kInfoLeaf) {
            st.leaf[at >> 10 & 1023u] = code;
            atomicOr(&st.starts[at >> 25], 1u << (at >> 20 & 31u));
          }
        }
        at += v[j];
      }
    }
    __syncwarp();
  }
  // lanes of a listed child's record that accept it
  auto accepts = [&](uint32_t code, uint32_t lanes) {
    const uint32_t info = st.info[code];
    return info & kInfoTerm ? (info & kInfoPart ? st.part[st.partOf[code]] : lanes) : 0u;
  };
  float ax = 0.0f, ay = 0.0f;
  if (kOneOrder) {
    // the terms in order, 32 at a time (the next ones' loads under way)
    float4 q, mom;
    uint32_t qm;
    uint32_t before = 0, last = 0; // items that start before the terms fetched
                                   // next, and the last one's first term
    auto fetch = [&](uint32_t base) {
      q = mom = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
      qm = 0;
      if (base >= nTerms) return;
      const uint32_t word = st.starts[base >> 5], mine = word & (laneBit | below);
      if (base + lane < nTerms) {
        const uint32_t item = st.item[before + __popc(mine) - 1u], code = item & 1023u;
        const uint32_t slot = code >> 2, c = code & 3u;
        const QuadRec *r = tQ + st.rec[slot];
        const uint32_t lanes = st.who[slot], in = accepts(code, lanes);
        if (item & kItemLeaf) {
          const uint32_t j = base + lane - (mine ? base + 31u - __clz(mine) : last);
          const uint32_t b = __ldg(&r->child[c].y) + j;
          if (b < S.n) { // defensive bound
            const float4 v = S.xym[b];
            q = make_float4(v.x, v.y, v.z, -1.0f);
          }
          qm = lanes & ~in;
        } else {
          q.x = __ldg(reinterpret_cast<const float *>(&r->x) + c);
          q.y = __ldg(reinterpret_cast<const float *>(&r->y) + c);
          q.z = __ldg(reinterpret_cast<const float *>(&r->m) + c);
          qm = q.z > 0.0f ? in : 0u; // the reference adds a cell only with mass
          if (kWalk == kQuadWalk) mom = __ldg(&S.tQM[st.rec[slot]].m[c]);
        }
      }
      before += __popc(word);
      if (word) last = base + 31u - __clz(word);
    };
    fetch(0);
    for (uint32_t base = 0; base < nTerms; base += kChunk) {
      st.q[lane] = q;
      if (kWalk == kQuadWalk) st.mom[lane] = mom;
      st.lanes[lane] = qm;
      __syncwarp();
      fetch(base + kChunk);
      const uint32_t n = min((uint32_t)kChunk, nTerms - base);
#pragma unroll 4
      for (uint32_t k = 0; k < n; ++k) {
        const float4 v = st.q[k];
        const bool on = (st.lanes[k] & laneBit) != 0;
        const float dx = kExact ? __fsub_rn(v.x, x) : v.x - x;
        const float dy = kExact ? __fsub_rn(v.y, y) : v.y - y;
        const float dSq = sq_dist<kExact>(dx, dy);
        const float fac = law_factor<kExact, kExact>(dSq, v.z, eSq);
        float tx, ty;
        if (kExact) {
          tx = __fadd_rn(ax, __fmul_rn(dx, fac));
          ty = __fadd_rn(ay, __fmul_rn(dy, fac));
        } else {
          tx = fmaf(dx, fac, ax);
          ty = fmaf(dy, fac, ay);
        }
        if (kWalk == kQuadWalk) {
          const float4 M = st.mom[k]; // a body's size is -1: never in the band
          // the node of the chain that the target accepts: the largest one that
          // passes (each is exactly a quarter of the last)
          float w = M.w;
          for (int up = 0; up <= kMaxDepth && on && w >= dSq * tSq; ++up) w *= 0.25f;
          const bool band = on && w >= dSq * bandSq;
          if (__ballot_sync(0xffffffffu, band)) {
            float qx, qy;
            quad_term(dx, dy, dSq, eSq, v.z, M.x, M.y, M.z, qx, qy);
            if (band) {
              tx = ax + fac * (dx + qx);
              ty = ay + fac * (dy + qy);
            }
          }
        }
        ax = on ? tx : ax;
        ay = on ? ty : ay;
      }
      __syncwarp();
    }
    if (valid & laneBit) {
      axOut = ax;
      ayOut = ay;
    }
    return true;
  }
  // the cells, 64 at a time, two to a lane (the next ones' loads under way)
  {
    float qx[2], qy[2], qh[2];
    uint32_t qm[2];
    auto fetch = [&](uint32_t k) {
#pragma unroll
      for (uint32_t j = 0; j < 2; ++j) {
        qx[j] = qy[j] = qh[j] = 0.0f;
        qm[j] = 0;
        if (k + j < nCells) {
          const uint32_t code = st.cell[k + j], slot = code >> 2, c = code & 3u;
          const QuadRec *q = tQ + st.rec[slot];
          qx[j] = __ldg(reinterpret_cast<const float *>(&q->x) + c);
          qy[j] = __ldg(reinterpret_cast<const float *>(&q->y) + c);
          qh[j] = 0.5f * __ldg(reinterpret_cast<const float *>(&q->m) + c);
          qm[j] = accepts(code, st.who[slot]);
        }
      }
    };
    fetch(2 * lane);
    for (uint32_t base = 0; base < nCells; base += 64) {
      *reinterpret_cast<float2 *>(&st.x[2 * lane]) = make_float2(qx[0], qx[1]);
      *reinterpret_cast<float2 *>(&st.y[2 * lane]) = make_float2(qy[0], qy[1]);
      *reinterpret_cast<float2 *>(&st.h[2 * lane]) = make_float2(qh[0], qh[1]);
      *reinterpret_cast<uint2 *>(&st.m[2 * lane]) = make_uint2(qm[0], qm[1]);
      __syncwarp();
      fetch(base + 64 + 2 * lane);
      const uint32_t n = min(64u, nCells - base);
      for (uint32_t k = 0; k < n; k += 4) { // past n: no lane
        const ulonglong2 X4 = *reinterpret_cast<const ulonglong2 *>(&st.x[k]);
        const ulonglong2 Y4 = *reinterpret_cast<const ulonglong2 *>(&st.y[k]);
        const ulonglong2 H4 = *reinterpret_cast<const ulonglong2 *>(&st.h[k]);
        const uint4 m = *reinterpret_cast<const uint4 *>(&st.m[k]);
        const f2x DX0 = sub2(X4.x, XX), DY0 = sub2(Y4.x, YY);
        const f2x DX1 = sub2(X4.y, XX), DY1 = sub2(Y4.y, YY);
        const f2x F0 = law_pair(fma2(DX0, DX0, mul2(DY0, DY0)), H4.x, E2, N3);
        const f2x F1 = law_pair(fma2(DX1, DX1, mul2(DY1, DY1)), H4.y, E2, N3);
        float dx0, dx1, dx2, dx3, dy0, dy1, dy2, dy3, f0, f1, f2, f3;
        upk2(DX0, dx0, dx1);
        upk2(DY0, dy0, dy1);
        upk2(F0, f0, f1);
        upk2(DX1, dx2, dx3);
        upk2(DY1, dy2, dy3);
        upk2(F1, f2, f3);
        fma_if(m.x & laneBit, dx0, dy0, f0, ax, ay);
        fma_if(m.y & laneBit, dx1, dy1, f1, ax, ay);
        fma_if(m.z & laneBit, dx2, dy2, f2, ax, ay);
        fma_if(m.w & laneBit, dx3, dy3, f3, ax, ay);
      }
      __syncwarp();
    }
  }
  // the leaves' bodies, 32 pairs at a time (an odd leaf's last body has a
  // massless partner)
  f2x lx = pk2(0.0f, 0.0f), ly = pk2(0.0f, 0.0f);
  {
    float4 q0, q1;
    uint32_t qm;
    uint32_t before = 0, last = 0; // leaves that start before the pairs fetched
                                   // next, and the last one's first pair
    auto fetch = [&](uint32_t base) {
      q0 = q1 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      qm = 0;
      if (base >= nPairs) return;
      const uint32_t word = st.starts[base >> 5], mine = word & (laneBit | below);
      if (base + lane < nPairs) {
        const uint32_t code = st.leaf[before + __popc(mine) - 1u], slot = code >> 2;
        const uint32_t j = 2u * (base + lane - (mine ? base + 31u - __clz(mine) : last));
        const uint2 c = __ldg(&tQ[st.rec[slot]].child[code & 3u]);
        const uint32_t b = c.y + j, lanes = st.who[slot];
        if (b < S.n) q0 = S.xym[b]; // defensive bounds
        if (j + 1u < (c.x & ~kQuadLeaf) && b + 1u < S.n) q1 = S.xym[b + 1u];
        qm = lanes & ~accepts(code, lanes);
      }
      before += __popc(word);
      if (word) last = base + 31u - __clz(word);
    };
    fetch(0);
    for (uint32_t base = 0; base < nPairs; base += 32) {
      *reinterpret_cast<float2 *>(&st.x[2 * lane]) = make_float2(q0.x, q1.x);
      *reinterpret_cast<float2 *>(&st.y[2 * lane]) = make_float2(q0.y, q1.y);
      *reinterpret_cast<float2 *>(&st.h[2 * lane]) = make_float2(0.5f * q0.z, 0.5f * q1.z);
      st.m[lane] = qm;
      __syncwarp();
      fetch(base + 32);
      const uint32_t n = min(32u, nPairs - base);
      for (uint32_t k = 0; k < n; k += 2) { // past n: no lane
        const ulonglong2 X4 = *reinterpret_cast<const ulonglong2 *>(&st.x[2 * k]);
        const ulonglong2 Y4 = *reinterpret_cast<const ulonglong2 *>(&st.y[2 * k]);
        const ulonglong2 H4 = *reinterpret_cast<const ulonglong2 *>(&st.h[2 * k]);
        const uint2 m = *reinterpret_cast<const uint2 *>(&st.m[k]);
        const f2x DX0 = sub2(X4.x, XX), DY0 = sub2(Y4.x, YY);
        const f2x DX1 = sub2(X4.y, XX), DY1 = sub2(Y4.y, YY);
        const f2x F0 = law_pair(fma2(DX0, DX0, mul2(DY0, DY0)), H4.x, E2, N3);
        const f2x F1 = law_pair(fma2(DX1, DX1, mul2(DY1, DY1)), H4.y, E2, N3);
        fma2_if(m.x & laneBit, DX0, F0, lx);
        fma2_if(m.x & laneBit, DY0, F0, ly);
        fma2_if(m.y & laneBit, DX1, F1, lx);
        fma2_if(m.y & laneBit, DY1, F1, ly);
      }
      __syncwarp();
    }
  }
  if (valid & laneBit) {
    float lx0, lx1, ly0, ly1;
    upk2(lx, lx0, lx1);
    upk2(ly, ly0, ly1);
    axOut = ax + (lx0 + lx1);
    ayOut = ay + (ly0 + ly1);
  }
  return true;
}

// Body i's acceleration: the attractor's pull added, and with recOut its
// whole record (nbx_body: pos, vel, acc, mass, radius, id), for a copy to
// the host right after this launch.
template <bool kExact>
__device__ __forceinline__ void store_acc(const DevState &S, uint32_t i, float x, float y,
                                          float ax, float ay) {
  add_attractor<kExact>(S.attr, x, y, ax, ay);
  S.acc[i] = make_float2(ax, ay);
  if (S.recOut) {
    const float4 p = S.pv[i];
    const float2 m = S.mr[i];
    uint32_t *r = S.recOut + (size_t)i * 9;
    r[0] = __float_as_uint(p.x);
    r[1] = __float_as_uint(p.y);
    r[2] = __float_as_uint(p.z);
    r[3] = __float_as_uint(p.w);
    r[4] = __float_as_uint(ax);
    r[5] = __float_as_uint(ay);
    r[6] = __float_as_uint(m.x);
    r[7] = __float_as_uint(m.y);
    r[8] = S.id[i];
  }
}

// Every target of the launch, one warp per 32.  kPairs selects the paired
// leaf loop for the default plain walk.
template <bool kExact, bool kCount, int kCorr, bool kClamp, bool kPairs>
__device__ __forceinline__ void forces_walk(
    const DevState &S, float tSq, float eSq, unsigned long long *counts,
    float bandSq, float2 *query, uint32_t nQuery, float4 (*sBody)[32]) {
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  const uint32_t warpsTotal = (gridDim.x * blockDim.x) >> 5;
  // query points (instance 0's tree) instead of the bodies, if given; for
  // the bodies, the launch's range of targets
  const uint32_t tBegin = query ? 0u : S.forceBegin;
  const uint32_t nTargets = query ? nQuery : (S.forceEnd ? min(S.forceEnd, S.n) : S.n);
  for (uint32_t wb = tBegin + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32;
       wb < nTargets; wb += warpsTotal * 32) {
    const uint32_t i = wb + lane;
    const bool valid = i < nTargets;
    float x = 0.0f, y = 0.0f;
    uint32_t cur = kDone;
    bool wide = false;
    if (valid) {
      if (query) {
        const float2 q = query[i];
        x = q.x;
        y = q.y;
      } else {
        const float4 b = S.xym[i];
        x = b.x;
        y = b.y;
      }
      const SegDev &G = S.seg[query ? 0u : S.segOf[i]];
      if (G.travCount > 0) cur = G.travBase;
      wide = (G.flags & kSegWide) != 0u;
    }
    float ax = 0.0f, ay = 0.0f;
    uint32_t nFar = 0, nNear = 0, nVisit = 0, nIter = 0, nChunk = 0;
    // the clamp-free law only while no lane's instance reaches beyond the
    // coordinate limit (the build's per-instance flag)
    constexpr bool kPlainX2 = kPairs && !kExact && !kCount && kCorr == 0 && !kClamp;
    const bool anyWide = !kClamp && __any_sync(0xffffffffu, wide);
    if (anyWide)
      walk_targets<kExact, kCount, kCorr, true>(S, tSq, eSq, bandSq, x, y, cur, sBody[w], ax,
                                                ay, nFar, nNear, nVisit, nIter, nChunk);
    else if (kPlainX2) {
      float *sX = reinterpret_cast<float *>(sBody[w]);
      walk_plain_x2(S, tSq, eSq, x, y, cur, sX, sX + 32, sX + 64, ax, ay);
    } else
      walk_targets<kExact, kCount, kCorr, kClamp>(S, tSq, eSq, bandSq, x, y, cur, sBody[w], ax,
                                                  ay, nFar, nNear, nVisit, nIter, nChunk);
    if (kCount) {
      unsigned long long f = nFar, nn = nNear, v = nVisit;
      for (int o = 16; o > 0; o >>= 1) {
        f += __shfl_xor_sync(0xffffffffu, f, o);
        nn += __shfl_xor_sync(0xffffffffu, nn, o);
        v += __shfl_xor_sync(0xffffffffu, v, o);
      }
      if (lane == 0) {
        atomicAdd(&counts[0], f);
        atomicAdd(&counts[1], nn);
        atomicAdd(&counts[2], v);
        atomicAdd(&counts[3], (unsigned long long)nIter);
        atomicAdd(&counts[4], (unsigned long long)nChunk);
      }
    } else if (valid) {
      if (query) {
        query[i] = make_float2(ax, ay);
      } else {
        store_acc<kExact>(S, i, x, y, ax, ay);
      }
    }
  }
}

// The force pass.  kClamp = false is the clamp-free law (see law_factor),
// which the host picks only for non-negative masses below its bound; a
// warp holding a target whose instance reaches beyond the coordinate limit
// stored at upload (the build's kSegWide), where distances could
// overflow, takes the clamped walk instead.  Launch bounds: a full SM of
// kBlock-thread blocks (2048 threads: at most 32 registers) for every walk
// but the paired plain walk's: 1536 threads per SM (40 registers),
// 1% faster than 2048 at 32 registers and identical in results.  kBlock
// and kPairs vary only for the default plain walk (the autotuner's block
// shape and leaf width).
template <bool kExact, bool kCount = false, int kCorr = 0, bool kClamp = true,
          int kBlock = kForceBlock, bool kPairs = true>
__global__ void __launch_bounds__(kBlock, kPairs && !kExact && !kCount && kCorr == 0 && !kClamp
                                              ? 1536 / kBlock
                                              : 2048 / kBlock)
    k_forces(DevState S, float tSq, float eSq,
             unsigned long long *counts = nullptr, float bandSq = 0.0f,
             float2 *query = nullptr, uint32_t nQuery = 0) {
  chain_begin();
  __shared__ float4 sBody[kBlock / 32][32];
  forces_walk<kExact, kCount, kCorr, kClamp, kPairs>(S, tSq, eSq, counts, bandSq, query, nQuery,
                                                     sBody);
}

// The force pass with the learned correction, one warp per 32 bodies.  us by
// threads a block at 100,000 bodies (fewer repeat the weights in shared memory,
// more wait for a block's longest walk): 32 264, 64 235, 128 221, 192 226,
// 256 236.
constexpr int kLearnedBlock = 128;
__global__ void __launch_bounds__(kLearnedBlock, 768 / kLearnedBlock)
    k_forces_learned(DevState S, float tSq, float eSq, const MlpDev *__restrict__ mlp,
                     float bandSq, float eps) {
  chain_begin();
  __shared__ LearnedStage sStage[kLearnedBlock / 32];
  __shared__ MlpDev sW;
  for (int q = threadIdx.x; q < (int)(sizeof(MlpDev) / 4); q += blockDim.x)
    reinterpret_cast<uint32_t *>(&sW)[q] = reinterpret_cast<const uint32_t *>(mlp)[q];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint32_t end = S.forceEnd ? min(S.forceEnd, S.n) : S.n;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t wb = S.forceBegin + ((blockIdx.x * blockDim.x + threadIdx.x) & ~31u); wb < end;
       wb += stride) {
    const uint32_t i = wb + lane;
    const bool valid = i < end;
    float x = 0.0f, y = 0.0f, ax = 0.0f, ay = 0.0f;
    uint32_t cur = kDone;
    if (valid) {
      const float4 b = S.xym[i];
      x = b.x;
      y = b.y;
      const SegDev &G = S.seg[S.segOf[i]];
      if (G.travCount > 0) cur = G.travBase;
    }
    walk_learned(S, tSq, eSq, bandSq, eps, x, y, cur, sStage[threadIdx.x >> 5], sW, ax, ay);
    if (valid) store_acc<false>(S, i, x, y, ax, ay);
  }
}

// Sums of a group walk for the targets of `lanes` (places (x, y), a valid
// one on every lane) in instance sg, and, for an instance that reaches beyond the
// coordinate limit, the clamped cursor walk's (exact arithmetic always clamps),
// as in k_forces.  Returns the targets whose walk does not fit (kGated: or is left
// to k_forces_deep): nothing is summed for them, and walk_rest does.
template <GroupWalk kWalk, bool kGated = false>
__device__ __forceinline__ uint32_t group_forces(const DevState &S, float tSq, float eSq,
                                                 float bandSq, float x, float y, uint32_t sg,
                                                 uint32_t lanes, WalkStage &st,
                                                 float &ax, float &ay) {
  constexpr bool kExact = kWalk == kExactWalk;
  constexpr int kCorr = kWalk == kQuadWalk ? 2 : 0;
  const int lane = threadIdx.x & 31;
  const SegDev &G = S.seg[sg];
  if (G.travCount == 0) return 0; // no tree (capacity)
  if (kGated && G.flags == kSegDeep) return lanes;
  if (G.flags & kSegWide) {
    uint32_t c0 = 0, c1 = 0, c2 = 0, c3 = 0, c4 = 0;
    walk_targets<kExact, false, kCorr, true>(S, tSq, eSq, bandSq, x, y,
                                             (lanes >> lane) & 1u ? G.travBase : kDone,
                                             reinterpret_cast<float4 *>(&st), ax, ay, c0, c1, c2,
                                             c3, c4);
    return 0;
  }
  // A group whose walk does not fit goes in two at the widest step along its
  // targets, if that is most of the group's extent (neighbours in Morton
  // order across the gap between two discs, say).  Only once, since each try
  // costs a third of a walk and a cusp has such steps at every scale.
  uint32_t left = lanes, piece = lanes;
  for (bool whole = true;; whole = false) {
    const bool in = (piece >> lane) & 1u;
    const int lead = __ffs(piece) - 1;
    const float leadX = __shfl_sync(0xffffffffu, x, lead);
    const float leadY = __shfl_sync(0xffffffffu, y, lead);
    const float px = in ? x : leadX, py = in ? y : leadY;
    const bool fits = walk_group<kWalk>(S, tSq, eSq, bandSq, px, py, sg, piece, st, ax, ay);
    __syncwarp();
    if (fits) {
      left &= ~piece;
      if (left == 0) return 0;
      piece = left;
      continue;
    }
    if (!whole) return left;
    const float nx = __shfl_down_sync(0xffffffffu, px, 1);
    const float ny = __shfl_down_sync(0xffffffffu, py, 1);
    const bool next = in && lane < 31 && ((piece >> (lane + 1)) & 1u);
    const float step = next ? fabsf(nx - px) + fabsf(ny - py) : 0.0f;
    const float widest = warp_max(step);
    const float extent = warp_max(px) - warp_min(px) + warp_max(py) - warp_min(py);
    const uint32_t at = __ballot_sync(0xffffffffu, step == widest);
    if (!(widest > 0.5f * extent)) return left;
    piece &= (at & (0u - at)) * 2u - 1u; // the lanes up to the step
  }
}

// The targets `left` by group_forces, with a cursor per lane.
template <GroupWalk kWalk>
__device__ __forceinline__ void walk_rest(const DevState &S, float tSq, float eSq, float bandSq,
                                          float x, float y, uint32_t sg, uint32_t left,
                                          WalkStage &st, float &axOut, float &ayOut) {
  constexpr bool kExact = kWalk == kExactWalk;
  constexpr int kCorr = kWalk == kQuadWalk ? 2 : 0;
  static_assert(sizeof(WalkStage) >= 32 * sizeof(float4), "holds a leaf's staged bodies");
  const bool in = (left >> (threadIdx.x & 31)) & 1u;
  const uint32_t root = in ? S.seg[sg].travBase : kDone;
  float ax = 0.0f, ay = 0.0f;
  if (kWalk == kPlainWalk) {
    float *sX = reinterpret_cast<float *>(&st);
    walk_plain_x2(S, tSq, eSq, x, y, root, sX, sX + 32, sX + 64, ax, ay);
  } else {
    uint32_t c0 = 0, c1 = 0, c2 = 0, c3 = 0, c4 = 0;
    walk_targets<kExact, false, kCorr, kExact>(S, tSq, eSq, bandSq, x, y, root,
                                               reinterpret_cast<float4 *>(&st), ax, ay, c0, c1,
                                               c2, c3, c4);
  }
  if (in) {
    axOut = ax;
    ayOut = ay;
  }
}

// A force pass, one group of targets per warp: the default one (leaf_pairs 1),
// exact arithmetic, or the quadrupole term.  Targets that do not fit are walked
// with a cursor per lane.  That takes twice the time here that it takes at
// k_forces' occupancy, so with kGated k_forces_deep does the whole pass where many
// are not likely to fit.
constexpr int kGroupWarpsPerSM = 20;
template <int kBlock, GroupWalk kWalk, bool kGated>
__global__ void __launch_bounds__(kBlock, kGroupWarpsPerSM * 32 / kBlock > 0
                                              ? kGroupWarpsPerSM * 32 / kBlock : 1)
    k_forces_groups(DevState S, float tSq, float eSq, float bandSq) {
  chain_begin();
  extern __shared__ uint4 sDyn[]; // a WalkStage per warp
  const int lane = threadIdx.x & 31;
  WalkStage &st = reinterpret_cast<WalkStage *>(sDyn)[threadIdx.x >> 5];
  const uint32_t warpsTotal = (gridDim.x * blockDim.x) >> 5;
  const uint32_t gEnd = S.tgEnd ? S.tgEnd : S.nGroups;
  for (uint32_t g = S.tgBegin + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); g < gEnd;
       g += warpsTotal) {
    const uint32_t first = S.nseg == 1 ? g * 32u : S.groupFirst[g];
    const uint32_t sg = S.segOf[first];
    const SegDev &G = S.seg[sg];
    const uint32_t count = min(32u, G.start + G.count - first);
    const bool mine = (uint32_t)lane < count;
    const uint32_t i = mine ? first + lane : first;
    const float4 b = S.xym[i];
    float ax = 0.0f, ay = 0.0f;
    const uint32_t left = group_forces<kWalk, kGated>(S, tSq, eSq, bandSq, b.x, b.y, sg,
                                              __ballot_sync(0xffffffffu, mine), st, ax, ay);
    if (left != 0) {
      if (kGated && G.flags == kSegDeep) continue;
      walk_rest<kWalk>(S, tSq, eSq, bandSq, b.x, b.y, sg, left, st, ax, ay);
    }
    if (mine) store_acc<kWalk == kExactWalk>(S, i, b.x, b.y, ax, ay);
    __syncwarp();
  }
}

// The instances that k_forces_groups<.., true> leaves, with a cursor per lane.
constexpr int kDeepBlock = 256;
__global__ void __launch_bounds__(kDeepBlock, 1536 / kDeepBlock)
    k_forces_deep(DevState S, float tSq, float eSq) {
  chain_begin();
  if (S.nseg == 1 && S.seg[0].flags != kSegDeep) return;
  __shared__ float sBody[kDeepBlock / 32][96];
  const uint32_t end = S.forceEnd ? min(S.forceEnd, S.n) : S.n;
  const uint32_t i = S.forceBegin + blockIdx.x * kDeepBlock + threadIdx.x;
  float4 b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  uint32_t root = kDone;
  bool mine = false;
  if (i < end) {
    const SegDev &G = S.seg[S.segOf[i]];
    mine = G.flags == kSegDeep;
    if (mine) {
      b = S.xym[i];
      root = G.travCount > 0 ? G.travBase : kDone;
    }
  }
  if (!__any_sync(0xffffffffu, mine)) return;
  float *sX = sBody[threadIdx.x >> 5];
  float ax = 0.0f, ay = 0.0f;
  walk_plain_x2(S, tSq, eSq, b.x, b.y, root, sX, sX + 32, sX + 64, ax, ay);
  if (mine) store_acc<false>(S, i, b.x, b.y, ax, ay);
}

// The same sums at query points (instance 0's tree), `per` consecutive points
// to a warp.
constexpr int kQueryBlock = 128;
template <GroupWalk kWalk>
__global__ void __launch_bounds__(kQueryBlock, kGroupWarpsPerSM * 32 / kQueryBlock)
    k_query_groups(DevState S, float tSq, float eSq, float2 *query, uint32_t nQuery,
                   uint32_t per) {
  extern __shared__ uint4 sDyn[];
  const int lane = threadIdx.x & 31;
  WalkStage &st = reinterpret_cast<WalkStage *>(sDyn)[threadIdx.x >> 5];
  const uint32_t g = (blockIdx.x * kQueryBlock + threadIdx.x) >> 5;
  const uint64_t first = (uint64_t)g * per;
  if (first >= nQuery) return;
  const uint32_t count = min(per, nQuery - (uint32_t)first);
  const bool mine = (uint32_t)lane < count;
  const uint32_t i = (uint32_t)first + (mine ? lane : 0);
  const float2 q = query[i];
  float ax = 0.0f, ay = 0.0f;
  const uint32_t left = group_forces<kWalk>(S, tSq, eSq, 0.0f, q.x, q.y, 0u,
                                            __ballot_sync(0xffffffffu, mine), st, ax, ay);
  if (left != 0) walk_rest<kWalk>(S, tSq, eSq, 0.0f, q.x, q.y, 0u, left, st, ax, ay);
  if (mine) query[i] = make_float2(ax, ay);
}

// Sort key of a query point: 12 + 12 interleaved bits of its place in the
// points' box, with the digit histograms of its three radix passes.
__global__ void __launch_bounds__(256)
    k_query_keys(const float2 *__restrict__ points, uint32_t n, float x0, float y0, float sx,
                 float sy, uint32_t *__restrict__ keys, uint32_t *hist) {
  __shared__ uint32_t sh[3][256];
  for (int i = threadIdx.x; i < 3 * 256; i += blockDim.x) sh[i >> 8][i & 255] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float2 p = points[i];
    // NaN and anything outside the box (it cannot be) end at an edge
    const uint32_t qx = (uint32_t)fminf(fmaxf((p.x - x0) * sx, 0.0f), 4095.0f);
    const uint32_t qy = (uint32_t)fminf(fmaxf((p.y - y0) * sy, 0.0f), 4095.0f);
    const uint32_t k = (uint32_t)((spread_bits(qy) << 1) | spread_bits(qx));
    keys[i] = k;
#pragma unroll
    for (int q = 0; q < 3; ++q) atomicAdd(&sh[q][(k >> (8 * q)) & 255u], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * 256; i += blockDim.x) {
    const uint32_t v = sh[i >> 8][i & 255];
    if (v) atomicAdd(&hist[i], v);
  }
}

// to[i] = from[order[i]], and back: to[order[i]] = from[i], with the status that
// the sort may have raised behind the last place (one copy takes both to the
// host: a copy of its own 3 us a call).
__global__ void __launch_bounds__(256)
    k_query_gather(const float2 *__restrict__ from, const uint32_t *__restrict__ order,
                   uint32_t n, float2 *__restrict__ to) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) to[i] = from[min(order[i], n - 1u)]; // defensive bound
}
__global__ void __launch_bounds__(256)
    k_query_scatter(const float2 *__restrict__ from, const uint32_t *__restrict__ order,
                    uint32_t n, const uint32_t *status, float2 *__restrict__ to) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) to[n] = make_float2(__uint_as_float(*status), 0.0f);
  if (i < n && order[i] < n) to[order[i]] = from[i]; // defensive bound
}

// FMA throughput probe: 8 independent chains per thread.
__global__ void k_fma_probe(float *out, int iters) {
  float a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = threadIdx.x * 1e-7f + j;
  const float b = 0.999999f, c = 1e-7f;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = fmaf(a[j], b, c);
  }
  float s = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += a[j];
  if (s == 12345.0f) out[0] = s; // keeps the chains live
}

} // namespace

void launch_interaction_count(cudaStream_t s, const DevState &S,
                              unsigned long long *counts) {
  uint32_t warps = (S.n + 31) / 32;
  uint32_t b = (warps + kWarps - 1) / kWarps;
  cudaMemsetAsync(counts, 0, 5 * sizeof(unsigned long long), s);
  k_forces<false, true><<<b ? b : 1, kForceBlock, 0, s>>>(S, S.tSq, S.eSq, counts);
}

// FP32 FMA peak of the device in TFLOP/s (2 flops per FMA), timed with
// CUDA events around one large probe launch.
double fp32_fma_peak_tflops(cudaStream_t s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  float *out = nullptr;
  if (cudaMalloc(&out, 4) != cudaSuccess) return 0.0;
  const int blocks = sms * 8, threads = 256, iters = 1 << 14;
  k_fma_probe<<<blocks, threads, 0, s>>>(out, 64); // warm-up
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, s);
  k_fma_probe<<<blocks, threads, 0, s>>>(out, iters);
  cudaEventRecord(e1, s);
  cudaEventSynchronize(e1);
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  const double flops = 2.0 * 8.0 * (double)iters * blocks * threads;
  return ms > 0 ? flops / (ms * 1e-3) / 1e12 : 0.0;
}

// Bodies a force launch over S covers (its target range, or all).
uint32_t force_targets(const DevState &S) {
  const uint32_t e = S.forceEnd ? (S.forceEnd < S.n ? S.forceEnd : S.n) : S.n;
  return e > S.forceBegin ? e - S.forceBegin : 0u;
}

// Whether groups' walks nearly always fit their scratch, for bodies spread
// evenly (what does not fit is walked with a cursor per lane at few warps per SM; the
// kernels see uneven states themselves, walk_depth): a group opens about
// 3 log4(n / L) / theta^2 records and its leaves hold about 2.3 L (1 + 1 / theta)^2
// bodies, n the largest instance.  Time without groups / with, discs and squares
// of 10,000 to 2^22 bodies, theta 0.28 to 0.45, leaf capacities 4 and 16, by
// log4(n / L) / theta^2: up to 48 from 1.16 to 3.3, at 50 from 0.71 (30,000 bodies, L 4,
// theta 0.36) to 2.5, from 60 on down to 0.44.  L 64 at theta 0.5 (refused), 2^20
// bodies: 874 us / 3700.  An instance of 2^20 bodies and 200 of 1000, theta 0.33: 1411
// us / 2720 (9841 before what does not fit was walked at once).
bool group_walk_fits(const DevState &S) {
  const float L = (float)S.leafCapacity, n = (float)S.largest, t = sqrtf(S.tSq);
  if (!(t > 0.0f)) return false;
  const float near = 1.0f + 1.0f / t;
  return 0.5f * log2f(fmaxf(n / L, 1.0f)) <= 48.0f * S.tSq && L * near * near <= 330.0f;
}

// Whether the default force pass gains by groups where they fit: at a large theta
// the walk is short, and a group's ~12 dependent batches cost more than a cursor's
// steps as soon as warps queue for the GPU.  Force pass of a disc, a square and
// bodies in clumps of clumps, us with a cursor / in groups: 100,000 bodies theta 1
// 51 / 46, 52 / 44, 47 / 48; 200,000 theta 0.85 88 / 85, 86 / 83, 71 / 81, theta 1 76 / 77,
// 72 / 75, 61 / 77, theta 2 of the disc 24 / 36; 400,000 theta 0.7 178 / 163, 174 / 159,
// 145 / 155, theta 1 129 / 132, 125 / 130, 106 / 134; 2^20 theta 0.7 434 / 411, 410 / 411,
// 340 / 388, theta 0.85 360 / 374, 342 / 374, 284 / 359; 2^22 theta 0.7 of the disc
// 1732 / 1663.  Smaller leaves make longer walks: the disc, 200,000, theta 1, leaf
// capacity 1 123 / 100, 4 94 / 82, 8 84 / 78, 32 73 / 79, 64 85 / 98.
// In nbx_step_io (recOut) they are taken all the same: the pass hides behind the
// copies, and the first range ends sooner (2^20 bodies of two discs, theta 1: 2016 /
// 1976 us a call).
bool group_walk_pays(const DevState &S) {
  return S.nGroups <= 148u * kGroupWarpsPerSM || S.recOut ||
         sqrtf(S.tSq) <= 0.715f * powf(fmaxf(1048576.0f / (float)S.n, 1.0f), 0.2f) *
                             powf(16.0f / (float)S.leafCapacity, 0.1f);
}

// Above so many groups the default pass has k_forces_deep behind it, for states in
// which many groups do not fit.  Where none does not it costs 1 us at 60,000
// bodies and 8 at 2^20 (force pass 618 -> 624).  Plummer's density, us without
// groups / with, without k_forces_deep / with it: 60,000 bodies theta 0.4 213 / 274 /
// 216; 2^20 theta 0.5 1239 / 2040 / 1221, 2^22 5242 / 10210 / 5138; a cusp (density as
// r^-1.6): 100,000 theta 0.5 432 / 480 / 433, 2^20 1660 / 1700 / 1652.
constexpr uint32_t kGateGroups = 1024;

template <int kBlock, GroupWalk kWalk, bool kGated = false>
void launch_groups(cudaStream_t s, const DevState &S, int blocks, float band, bool chained) {
  constexpr int smem = kBlock / 32 * (int)sizeof(WalkStage);
  constexpr auto kernel = k_forces_groups<kBlock, kWalk, kGated>;
  if (smem > 48 * 1024) // above what a launch may ask for by default
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (blocks <= 0) {
    const uint32_t warps = (S.tgEnd ? S.tgEnd : S.nGroups) - S.tgBegin, per = kBlock / 32;
    blocks = (int)std::max(1u, (warps + per - 1) / per);
  }
  if (chained) launch_after(s, kernel, blocks, kBlock, smem, S, S.tSq, S.eSq, band * band);
  else kernel<<<blocks, kBlock, smem, s>>>(S, S.tSq, S.eSq, band * band);
}

// The default plain walk with kBlock threads per block and the paired or
// single-body leaf loop.
template <int kBlock>
void launch_plain(cudaStream_t s, const DevState &S, int blocks, bool pairs, bool groups,
                  bool chained) {
  const bool whole = blocks <= 0;
  if (whole) {
    const uint32_t warps = (force_targets(S) + 31) / 32, per = kBlock / 32;
    const uint32_t b = (warps + per - 1) / per;
    blocks = (int)(b ? b : 1);
  }
  if (pairs && groups && S.nGroups > kGateGroups) {
    // Behind the groups in a chain, before them in nbx_step_io's ranges: a
    // range's records leave when its last kernel ends, and behind the groups that
    // one waited for room among the other ranges' blocks (2^20 bodies: 44 us a call).
    const uint32_t deep = std::max(1u, (force_targets(S) + kDeepBlock - 1u) / kDeepBlock);
    if (!chained) k_forces_deep<<<deep, kDeepBlock, 0, s>>>(S, S.tSq, S.eSq);
    launch_groups<kBlock, kPlainWalk, true>(s, S, whole ? 0 : blocks, 0.0f, chained);
    if (chained) launch_after(s, k_forces_deep, deep, kDeepBlock, 0, S, S.tSq, S.eSq);
  } else if (pairs && groups)
    launch_groups<kBlock, kPlainWalk>(s, S, whole ? 0 : blocks, 0.0f, chained);
  else if (pairs)
    k_forces<false, false, 0, false, kBlock, true><<<blocks, kBlock, 0, s>>>(S, S.tSq, S.eSq);
  else
    k_forces<false, false, 0, false, kBlock, false><<<blocks, kBlock, 0, s>>>(S, S.tSq, S.eSq);
}

// Accelerations at nq arbitrary points from instance 0's last tree
// (QuadTree::acceleration, QuadTree.cpp:264-389, for any query position):
// points -> their sums, in place, through the scratch array sorted; beyond
// kQueryUnsorted points the status follows the sums (k_query_scatter).  A target's
// sums do not depend on its warp, so the points are first put in Morton order
// of their box [x0, y0, 1 / cell sizes]: neighbours share a warp and its
// walk.  groups: the clamp-free law may be used (every point within the
// coordinate limit too).  A warp then takes so many points that the warps
// fill the GPU once and a group's box covers about 64 bodies at most, since
// one that covers more does not fit its scratch.  200,003 random points
// over 500,000 bodies, theta 0.5: sorting 55 us and the walk 121 (16 points a
// warp; 356 with 32, 131 with 8) instead of 640 in the callers' order, in
// which a warp's walk is the union of 32 unrelated ones; 100 points 35 and 20
// us instead of 373.
void launch_query_forces(cudaStream_t s, const DevState &S, bool exact, bool groups,
                         SortScratch &sort, float2 *points, uint32_t nq, const float box[4],
                         float2 *sorted) {
  const uint32_t blocks = (nq + 255) / 256;
  const bool order = nq > kQueryUnsorted;
  const uint32_t *vals = nullptr;
  float2 *query = points; // each target's point, then its sums
  if (order) {
    cudaMemsetAsync(sort.hist, 0, 3 * 256 * sizeof(uint32_t), s);
    k_query_keys<<<blocks < 592 ? blocks : 592, 256, 0, s>>>(points, nq, box[0], box[1], box[2],
                                                             box[3], keys32(sort, 0), sort.hist);
    const int buf = radix_sort_u32(s, sort, nq, nullptr, 0, 24, true, true, S.status);
    vals = sort.vals[buf];
    k_query_gather<<<blocks, 256, 0, s>>>(points, vals, nq, sorted);
    query = sorted;
  }
  if ((exact || groups) && group_walk_fits(S)) {
    uint32_t per = 32;
    while (per > 1 && ((nq + per - 1) / per < 148u * kGroupWarpsPerSM ||
                       (uint64_t)per * S.n > 64ull * nq))
      per >>= 1;
    const uint32_t warps = (nq + per - 1) / per;
    auto kernel = exact ? k_query_groups<kExactWalk> : k_query_groups<kPlainWalk>;
    kernel<<<(warps * 32 + kQueryBlock - 1) / kQueryBlock, kQueryBlock,
             kQueryBlock / 32 * sizeof(WalkStage), s>>>(S, S.tSq, S.eSq, query, nq, per);
  } else {
    const uint32_t b = ((nq + 31) / 32 + kWarps - 1) / kWarps;
    if (exact)
      k_forces<true><<<b, kForceBlock, 0, s>>>(S, S.tSq, S.eSq, nullptr, 0.0f, query, nq);
    else
      k_forces<false><<<b, kForceBlock, 0, s>>>(S, S.tSq, S.eSq, nullptr, 0.0f, query, nq);
  }
  if (order) k_query_scatter<<<blocks, 256, 0, s>>>(sorted, vals, nq, S.status, points);
}

// Blocks of launch_forces' kernel that an SM holds, by the kernels' launch bounds.
int force_blocks_per_sm(const DevState &S, bool exact, int corr, bool noClamp, int threads,
                        bool pairs) {
  const bool fits = group_walk_fits(S);
  if (corr == 0 && !exact && noClamp) {
    const bool groups = pairs && fits && group_walk_pays(S);
    if (threads == 0) threads = groups ? 128 : 256;
    return std::max(1, (groups ? kGroupWarpsPerSM * 32 : pairs ? 1536 : 2048) / threads);
  }
  if (S.n <= kOrderedGroupsMax && fits && ((corr == 0 && exact) || (corr == 2 && noClamp)))
    return kGroupWarpsPerSM * 32 / 128;
  return corr == 1 ? 768 / kLearnedBlock : 2048 / kForceBlock;
}

// chained: the launch follows a kernel of the step's chain on s (chain_begin).
void launch_forces(cudaStream_t s, const DevState &S, bool exact, int blocks,
                   const MlpDev *mlp, float band, int corr, bool noClamp, int threads,
                   bool pairs, bool chained) {
  if (corr == 0 && !exact && noClamp) {
    // the group walk where its records nearly always fit, with 128 threads a
    // block by default (see group_walk_fits), else a cursor per lane
    const bool groups = pairs && group_walk_fits(S) && group_walk_pays(S);
    if (threads == 0) threads = groups ? 128 : 256;
    if (threads == 128) launch_plain<128>(s, S, blocks, pairs, groups, chained);
    else if (threads == 512) launch_plain<512>(s, S, blocks, pairs, groups, chained);
    else launch_plain<256>(s, S, blocks, pairs, groups, chained);
    return;
  }
  // The walks that keep one order, in groups too where those fit and a
  // cursor's ~300 dependent loads count: us with a cursor / in groups, exact,
  // theta 0.5: 10,000 bodies 88 / 61, 30,000 119 / 84, 100,000 175 / 164, 262,147
  // 311 / 313, 2^20 1072 / 1142 (theta 1: 100,000 75 / 84); the quadrupole
  // term, theta 0.65, band 0.4: 10,000 66 / 53, 30,000 84 / 66, 100,000 121 / 135,
  // 2^20 746 / 967: scalar sums and terms of every lane's, unlike the plain
  // walk's pairs, are all they have to offer once there are warps enough.
  if (S.n <= kOrderedGroupsMax && group_walk_fits(S)) {
    if (corr == 0 && exact) {
      launch_groups<128, kExactWalk>(s, S, blocks, 0.0f, chained);
      return;
    }
    if (corr == 2 && noClamp && S.tQM) {
      launch_groups<128, kQuadWalk>(s, S, blocks, band, chained);
      return;
    }
  }
  const uint32_t warps = (force_targets(S) + 31) / 32;
  // band >= theta: no accepted cell is corrected, and the plain walk needs no rounds
  // (2^20 bodies, theta 0.7, band 0.7: 997 us in rounds, 476 so)
  if (corr == 1 && mlp && band * band < S.tSq) {
    constexpr uint32_t per = kLearnedBlock / 32;
    const int grid = blocks > 0 ? blocks : (int)std::max(1u, (warps + per - 1) / per);
    if (chained)
      launch_after(s, k_forces_learned, grid, kLearnedBlock, 0, S, S.tSq, S.eSq, mlp,
                   band * band, sqrtf(S.eSq));
    else
      k_forces_learned<<<grid, kLearnedBlock, 0, s>>>(S, S.tSq, S.eSq, mlp, band * band,
                                                      sqrtf(S.eSq));
    return;
  }
  if (blocks <= 0) blocks = (int)std::max(1u, (warps + kWarps - 1) / kWarps);
  if (corr == 2 && noClamp)
    k_forces<false, false, 2, false>
        <<<blocks, kForceBlock, 0, s>>>(S, S.tSq, S.eSq, nullptr, band * band);
  else if (corr == 2)
    k_forces<false, false, 2><<<blocks, kForceBlock, 0, s>>>(S, S.tSq, S.eSq, nullptr, band * band);
  else if (exact)
    k_forces<true><<<blocks, kForceBlock, 0, s>>>(S, S.tSq, S.eSq);
  else
    k_forces<false><<<blocks, kForceBlock, 0, s>>>(S, S.tSq, S.eSq);
}

} // namespace nbx
