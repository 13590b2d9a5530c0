// build.cu -- root square, Morton codes, Morton-order gather and the
// quadtree build, for every instance of a handle in one launch per phase.
//
// The tree is the reference's Morton tree (src/cuda/TreeKernels.cuh:68-177,
// driven as CudaQuadTree.cu:452-498): breadth-first node numbering, the 4
// children of a node consecutive at `children`, `next` skip pointers, body
// ranges [start, end), leaves of <= leafCapacity bodies (or at depth 32).
//
// The reference builds it level by level with grid-wide barriers.  Here
// every level is built at once, straight from the sorted codes:
//  * body i is the first body of the depth-d node containing it iff
//    d > lcp(code[i-1], code[i]); that node splits iff it holds more than
//    L bodies, i.e. code[i+L] shares its d-digit prefix, and d < 32.  So
//    body i starts the splitting nodes of depths [lo_i, hi_i] with
//    lo_i = lcp(i-1, i) + 1 and hi_i = min(lcp(i, i+L), 31);
//  * the (segment, depth, first body) entries are bucketed by depth with a
//    stable radix pass; a splitting node's rank among its level's
//    splitting nodes is its position in its bucket, which fixes the BFS
//    slot of its children (levelStart[d+1] + 4*rank), exactly the
//    numbering of the serial loop;
//  * centres are recomputed along the path from the root with the same
//    float operations as splitNode (bit-identical), and `next` is the slot
//    after the deepest ancestor that is not a last child;
//  * mass / centre-of-mass (and second moments) go up the tree with
//    arrival counters: the fourth child to finish sums its parent in the
//    fixed order c0+c1+c2+c3 of sumNode, so the sums are deterministic.
// Those arrays are made on request only.  A step makes the records of the
// force traversal (force.cu), in depth-first preorder with the group walk's
// records of four children, from the same codes (k_trav_tree, k_trav_top).
#include "nbx_state.cuh"

#include <float.h>

namespace nbx {
namespace {

constexpr int kBlock = 256;

int grid_for(uint32_t n) {
  uint32_t b = (n + kBlock - 1) / kBlock;
  if (b > 148u * 16u) b = 148u * 16u;
  return b ? (int)b : 1;
}

// Morton code of every body; the sort key is its high half (depth-16
// cells), with the digit histograms of its four radix passes fused.
__global__ void __launch_bounds__(kBlock)
    k_morton(DevState S, uint32_t *__restrict__ keys, uint32_t *hist) {
  chain_begin();
  __shared__ uint32_t sh[4][256];
  for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) sh[i >> 8][i & 255] = 0;
  __syncthreads();
  const uint32_t n = S.n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += gridDim.x * blockDim.x) {
    const uint64_t c = body_code(S.pv[i], S.seg[S.segOf[i]].frame);
    const uint32_t k = (uint32_t)(c >> 32);
    keys[i] = k;
    S.codes[i] = c;
#pragma unroll
    for (int q = 0; q < 4; ++q) atomicAdd(&sh[q][(k >> (8 * q)) & 255u], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) {
    const uint32_t v = sh[i >> 8][i & 255];
    if (v) atomicAdd(&hist[i], v);
  }
}

// Sort key for the instance passes: segment of the element's original index.
__global__ void k_seg_keys(DevState S, const uint32_t *__restrict__ vals,
                           uint32_t *__restrict__ keys) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n;
       i += gridDim.x * blockDim.x)
    keys[i] = S.segOf[vals[i]];
}

// ------------------------------------------------------------ tree build

// Splitting nodes that start at body i: depths [lo, hi].
__global__ void __launch_bounds__(kBlock) k_split_counts(DevState S) {
  const uint64_t *c = S.sortedCodes;
  const int L = S.leafCapacity;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n;
       i += gridDim.x * blockDim.x) {
    const SegDev &G = S.seg[S.segOf[i]];
    const uint32_t s0 = G.start, s1 = G.start + G.count;
    const int lo = (i == s0) ? 0 : lcp_digits(c[i - 1], c[i]) + 1;
    int hi = -1;
    if ((uint64_t)i + (uint32_t)L < s1) {
      hi = lcp_digits(c[i], c[i + L]);
      if (hi > kMaxDepth - 1) hi = kMaxDepth - 1;
    }
    const int cnt = hi >= lo ? hi - lo + 1 : 0;
    S.splitCount[i] = (uint32_t)cnt;
    S.splitLo[i] = (uint8_t)(lo > 255 ? 255 : lo);
  }
}

__global__ void __launch_bounds__(kBlock)
    k_split_emit(DevState S, uint64_t *__restrict__ keys,
                 uint32_t *__restrict__ vals) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n;
       i += gridDim.x * blockDim.x) {
    const uint32_t cnt = S.splitCount[i];
    if (!cnt) continue;
    const uint32_t base = S.splitStart[i];
    const uint32_t lo = S.splitLo[i];
    const uint64_t sg = S.segOf[i];
    for (uint32_t k = 0; k < cnt; ++k) {
      keys[base + k] = (sg << 6) | (lo + k);
      vals[base + k] = i;
    }
  }
}

// Bucket boundaries of the depth-sorted entries.
__global__ void __launch_bounds__(kBlock)
    k_groups(DevState S, const uint64_t *__restrict__ keys) {
  const uint32_t total = S.counters[3];
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < total;
       k += gridDim.x * blockDim.x) {
    const uint64_t key = keys[k];
    const uint32_t slot = (uint32_t)(key >> 6) * kLevelSlots + (uint32_t)(key & 63u);
    if (k == 0 || keys[k - 1] != key) S.groupStart[slot] = k;
    if (k + 1 == total || keys[k + 1] != key) S.groupEnd[slot] = k + 1;
  }
}

// Level starts, node counts and node bases per instance; root nodes.
__global__ void k_levels(DevState S) {
  __shared__ uint32_t sRun;
  if (threadIdx.x == 0) sRun = 0;
  __syncthreads();
  for (uint32_t base = 0; base < S.nseg; base += blockDim.x) {
    const uint32_t sg = base + threadIdx.x;
    uint32_t nodes = 0, levels = 0;
    if (sg < S.nseg) {
      SegDev &G = S.seg[sg];
      uint32_t *ls = S.levelStart + sg * (kLevelSlots + 1);
      const uint32_t *gs = S.groupStart + sg * kLevelSlots;
      const uint32_t *ge = S.groupEnd + sg * kLevelSlots;
      if (G.count > 0) {
        ls[0] = 0;
        ls[1] = 1;
        uint32_t maxLevel = 0; // deepest level with nodes
        for (int d = 1; d <= kMaxDepth; ++d) {
          const uint32_t split = ge[d - 1] - gs[d - 1];
          ls[d + 1] = ls[d] + 4u * split;
          if (split) maxLevel = d;
        }
        nodes = ls[maxLevel + 1];
        for (int d = maxLevel + 2; d <= kLevelSlots; ++d) ls[d] = nodes;
        levels = maxLevel + 1;
      } else {
        for (int d = 0; d <= kLevelSlots; ++d) ls[d] = 0;
      }
      G.nodeCount = nodes;
      G.levelCount = levels;
    }
    // block-wide exclusive scan of node counts -> node bases
    __shared__ uint32_t sScan[1024];
    sScan[threadIdx.x] = nodes;
    __syncthreads();
    for (uint32_t o = 1; o < blockDim.x; o <<= 1) {
      const uint32_t v = threadIdx.x >= o ? sScan[threadIdx.x - o] : 0u;
      __syncthreads();
      sScan[threadIdx.x] += v;
      __syncthreads();
    }
    const uint32_t excl = sRun + sScan[threadIdx.x] - nodes;
    if (sg < S.nseg) {
      SegDev &G = S.seg[sg];
      G.nodeBase = excl;
      if (excl + nodes <= S.nodeCapacity && nodes > 0) {
        const uint32_t r = excl;
        S.comX[r] = 0.0f;
        S.comY[r] = 0.0f;
        S.mass[r] = 0.0f;
        S.centerX[r] = G.cx;
        S.centerY[r] = G.cy;
        S.size[r] = G.size;
        S.children[r] = 0;
        S.next[r] = 0;
        S.start[r] = 0;
        S.end[r] = (int32_t)G.count;
        S.parent[r] = -1;
      }
    }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) sRun += sScan[blockDim.x - 1];
    __syncthreads();
  }
  __syncthreads();
  if (sRun > S.nodeCapacity) {
    // all-or-nothing: no instance gets a tree, the step reports the error
    for (uint32_t sg = threadIdx.x; sg < S.nseg; sg += blockDim.x)
      S.seg[sg].nodeCount = 0;
    if (threadIdx.x == 0) {
      atomicOr(S.status, kStatusTreeCapacity);
      S.counters[4] = 0;
    }
  } else if (threadIdx.x == 0) {
    S.counters[4] = sRun;
  }
}

// Index of the depth-t splitting node containing body i, by its rank.
__device__ __forceinline__ uint32_t split_rank(const DevState &S,
                                               const uint32_t *vals,
                                               uint32_t sg, int t, uint32_t i) {
  uint32_t lo = S.groupStart[sg * kLevelSlots + t];
  uint32_t hi = S.groupEnd[sg * kLevelSlots + t];
  const uint32_t g0 = lo;
  // last position with vals[pos] <= i
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (vals[mid] <= i) lo = mid + 1;
    else hi = mid;
  }
  return lo > g0 ? lo - 1 - g0 : 0u; // the parent always exists
}

// firstWithDigit (TreeKernels.cuh:72-85) over global body indices.
__device__ __forceinline__ uint32_t first_with_digit(const uint64_t *codes,
                                                     uint32_t lo, uint32_t hi,
                                                     int depth, int q) {
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (digit_at(codes[mid], depth) < q) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(kBlock)
    k_split_nodes(DevState S, const uint64_t *__restrict__ keys,
                  const uint32_t *__restrict__ vals) {
  const uint32_t total = S.counters[3];
  const uint64_t *codes = S.sortedCodes;
  const uint32_t L = (uint32_t)S.leafCapacity;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < total;
       k += gridDim.x * blockDim.x) {
    const uint64_t key = keys[k];
    const uint32_t sg = (uint32_t)(key >> 6);
    const int d = (int)(key & 63u);
    const uint32_t i = vals[k];
    if (sg >= S.nseg || d >= kMaxDepth) continue;
    const SegDev &G = S.seg[sg];
    if (G.nodeCount == 0) continue; // capacity overflow: instance skipped
    const uint32_t nb = G.nodeBase;
    const uint32_t s0 = G.start, s1 = G.start + G.count;
    const uint32_t *ls = S.levelStart + sg * (kLevelSlots + 1);
    const uint32_t r = k - S.groupStart[sg * kLevelSlots + d];
    const uint64_t ci = codes[i];
    uint32_t own = 0;
    if (d > 0) own = ls[d] + 4u * split_rank(S, vals, sg, d - 1, i) +
                     (uint32_t)digit_at(ci, d - 1);
    const uint32_t childBase = ls[d + 1] + 4u * r;
    if (childBase + 4 > G.nodeCount || own >= G.nodeCount) {
      atomicOr(S.status, kStatusTreeCapacity);
      continue;
    }
    // end of this node's body range
    uint32_t end = s1;
    if (d > 0) {
      const uint64_t pre = ci >> (64 - 2 * d);
      uint32_t lo = i + 1, hi = s1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if ((codes[mid] >> (64 - 2 * d)) == pre) lo = mid + 1;
        else hi = mid;
      }
      end = lo;
    }
    uint32_t bound[5];
    bound[0] = i;
    bound[4] = end;
    for (int q = 1; q < 4; ++q)
      bound[q] = first_with_digit(codes, bound[q - 1], end, d, q);
    // centre and size along the path (splitNode's arithmetic)
    float cx = G.cx, cy = G.cy, size = G.size;
    for (int t = 0; t < d; ++t) {
      size = __fmul_rn(size, 0.5f);
      const int q = digit_at(ci, t);
      cx = __fadd_rn(cx, __fmul_rn((float)(q & 1) - 0.5f, size));
      cy = __fadd_rn(cy, __fmul_rn((float)(q >> 1) - 0.5f, size));
    }
    // own `next`: after the deepest ancestor-or-self that is not a last child
    uint32_t ownNext = 0;
    for (int t = d; t >= 1; --t) {
      const int q = digit_at(ci, t - 1);
      if (q < 3) {
        const uint32_t idx =
            (t == d) ? own
                     : ls[t] + 4u * split_rank(S, vals, sg, t - 1, i) + (uint32_t)q;
        ownNext = idx + 1;
        break;
      }
    }
    const float childSize = __fmul_rn(size, 0.5f);
    S.children[nb + own] = (int32_t)childBase;
    S.arrive[nb + own] = 0;
    for (int q = 0; q < 4; ++q) {
      const uint32_t ch = nb + childBase + q;
      S.comX[ch] = 0.0f;
      S.comY[ch] = 0.0f;
      S.mass[ch] = 0.0f;
      S.centerX[ch] = __fadd_rn(cx, __fmul_rn((float)(q & 1) - 0.5f, childSize));
      S.centerY[ch] = __fadd_rn(cy, __fmul_rn((float)(q >> 1) - 0.5f, childSize));
      S.size[ch] = childSize;
      S.next[ch] = (int32_t)(q < 3 ? childBase + q + 1 : ownNext);
      S.start[ch] = (int32_t)(bound[q] - s0);
      S.end[ch] = (int32_t)(bound[q + 1] - s0);
      S.parent[ch] = (int32_t)own;
      const bool splits = bound[q + 1] - bound[q] > L && d + 1 < kMaxDepth;
      if (!splits) S.children[ch] = 0;
    }
  }
}

__device__ __forceinline__ uint32_t seg_of_node(const DevState &S, uint32_t g) {
  uint32_t lo = 0, hi = S.nseg;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (S.seg[mid].nodeBase <= g) lo = mid;
    else hi = mid;
  }
  // skip empty instances sharing the same base
  while (lo + 1 < S.nseg && S.seg[lo].nodeCount == 0 && S.seg[lo + 1].nodeBase <= g)
    ++lo;
  return lo;
}

// Bottom-up pass: leaves sum their bodies (sumNode order), the last of
// four children to finish sums their parent, then finishNode's divide.
__global__ void __launch_bounds__(kBlock) k_upward(DevState S) {
  const uint32_t total = S.counters[4];
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += gridDim.x * blockDim.x) {
    if (S.children[g] != 0) continue;
    const uint32_t sg = seg_of_node(S, g);
    const SegDev &G = S.seg[sg];
    const uint32_t nb = G.nodeBase, s0 = G.start;
    const uint32_t b0 = s0 + (uint32_t)S.start[g], b1 = s0 + (uint32_t)S.end[g];
    float px = 0.0f, py = 0.0f, mm = 0.0f;
    for (uint32_t b = b0; b < b1; ++b) {
      const float4 q = S.xym[b];
      px = __fadd_rn(px, __fmul_rn(q.x, q.z));
      py = __fadd_rn(py, __fmul_rn(q.y, q.z));
      mm = __fadd_rn(mm, q.z);
    }
    const float div = fmaxf(mm, FLT_MIN);
    const float X = __fdiv_rn(px, div), Y = __fdiv_rn(py, div);
    float ixx = 0.0f, iyy = 0.0f, ixy = 0.0f;
    for (uint32_t b = b0; b < b1; ++b) {
      const float4 q = S.xym[b];
      const float dx = q.x - X, dy = q.y - Y;
      ixx += q.z * dx * dx;
      iyy += q.z * dy * dy;
      ixy += q.z * dx * dy;
    }
    S.sumX[g] = px;
    S.sumY[g] = py;
    S.mass[g] = mm;
    S.comX[g] = X;
    S.comY[g] = Y;
    S.moments[g] = make_float4(ixx, iyy, ixy, 0.0f);
    // empty leaves (no bodies) add nothing whether accepted or opened, so
    // the traversal layout leaves them out
    S.subtree[g] = b1 > b0 ? 1u : 0u;
    // climb (at most kMaxDepth levels; parent indices are range-checked)
    int32_t node = S.parent[g];
    for (int guard = 0; node >= 0 && guard <= kMaxDepth; ++guard) {
      if ((uint32_t)node >= G.nodeCount) {
        atomicOr(S.status, kStatusTreeCapacity);
        break;
      }
      const uint32_t pg = nb + (uint32_t)node;
      // release: this child's sums are visible to the last arriver; acquire:
      // the last arriver sees all four children's sums
      uint32_t old;
      asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;"
                   : "=r"(old)
                   : "l"(&S.arrive[pg])
                   : "memory");
      if (old != 3u) break;
      const uint32_t c = nb + (uint32_t)S.children[pg];
      float sx = __ldcg(&S.sumX[c]), sy = __ldcg(&S.sumY[c]),
            sm = __ldcg(&S.mass[c]);
      uint32_t sub = 1 + __ldcg(&S.subtree[c]);
      for (int q = 1; q < 4; ++q) {
        sx = __fadd_rn(sx, __ldcg(&S.sumX[c + q]));
        sy = __fadd_rn(sy, __ldcg(&S.sumY[c + q]));
        sm = __fadd_rn(sm, __ldcg(&S.mass[c + q]));
        sub += __ldcg(&S.subtree[c + q]);
      }
      const float dv = fmaxf(sm, FLT_MIN);
      const float PX = __fdiv_rn(sx, dv), PY = __fdiv_rn(sy, dv);
      float jxx = 0.0f, jyy = 0.0f, jxy = 0.0f;
      for (int q = 0; q < 4; ++q) {
        const float4 mo = __ldcg(&S.moments[c + q]);
        const float cm = __ldcg(&S.mass[c + q]);
        const float dx = __ldcg(&S.comX[c + q]) - PX;
        const float dy = __ldcg(&S.comY[c + q]) - PY;
        jxx += mo.x + cm * dx * dx;
        jyy += mo.y + cm * dy * dy;
        jxy += mo.z + cm * dx * dy;
      }
      __stcg(&S.sumX[pg], sx);
      __stcg(&S.sumY[pg], sy);
      __stcg(&S.mass[pg], sm);
      __stcg(&S.comX[pg], PX);
      __stcg(&S.comY[pg], PY);
      __stcg(&S.moments[pg], make_float4(jxx, jyy, jxy, 0.0f));
      __stcg(&S.subtree[pg], sub);
      node = S.parent[pg];
    }
  }
}

// ------------------------------------------- traversal layout, built directly
//
// The force traversal needs only the non-empty nodes, in depth-first
// preorder, and those follow straight from the sorted codes:
//  * a node is (first body i, depth d).  The nodes starting at body i have
//    depths lo_i .. leaf_i: lo_i = lcp(i-1, i) + 1 (0 at an instance's
//    first body), and leaf_i is the depth of i's leaf.  A node containing
//    i splits iff it holds more than L bodies, i.e. iff some window
//    [j, j+L] of the instance around i shares its prefix, so
//    leaf_i = min(max over j in [i-L, i] of lcp(j, j+L), 31) + 1 (0 when no
//    window fits);
//  * in preorder, the nodes starting at i follow every node that starts
//    before i, shallowest first: with P = the exclusive scan of the counts,
//    node (i, d) is record P_i + d - lo_i;
//  * its subtree ends at the first body e past its prefix group, and the
//    record after the subtree is the first node starting at e, P_e;
//  * sums go up with arrival counters over the non-empty children in digit
//    order.  An empty child adds exactly +0 to sums that are never -0 (they
//    start at +0 and only add), so mass and centre of mass equal
//    sumNode/finishNode's over all four children (TreeKernels.cuh:150-177)
//    bit for bit.
// This replaces the breadth-first arrays on the step path; those are built
// only when asked for (launch_bfs_tree).

// Permute the state into Morton order (the 7 gathers of
// CudaQuadTree.cu:408-414, fused), write the {x, y, m} traversal array and,
// from the same sorted codes staged in shared memory, the traversal records
// that start at each body: their count (splitCount) and the depth of the
// first (splitLo).  hi_j = min(lcp(j, j+L), 31) (-1 when j+L leaves the
// instance) is formed once per body, then each body takes the maximum over
// its L+1 windows.  Each block takes 256 consecutive bodies and stages the
// codes of bodies [b0 - L, b0 + 256 + L) through the permutation, so the
// counts need no pass after the gather.
constexpr int kMaxLeafCap = 64; // nbx_params leaf_capacity bound
__global__ void __launch_bounds__(kBlock)
    k_gather_counts(DevState S, const uint32_t *__restrict__ perm) {
  chain_begin();
  __shared__ uint64_t sC[kBlock + 2 * kMaxLeafCap];
  __shared__ int8_t sHi[kBlock + kMaxLeafCap];
  const uint32_t n = S.n;
  const uint32_t L = (uint32_t)S.leafCapacity;
  for (uint32_t b0 = blockIdx.x * kBlock; b0 < n; b0 += gridDim.x * kBlock) {
    const uint32_t jBase = b0 >= L ? b0 - L : 0u;
    const uint32_t cEnd = min(n, b0 + kBlock + L); // codes [jBase, cEnd)
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < cEnd - jBase; t += kBlock)
      sC[t] = S.codes[perm[jBase + t]];
    const uint32_t i = b0 + threadIdx.x;
    if (i < n) {
      const uint32_t p = perm[i];
      const float4 v = S.pv[p];
      const float2 m = S.mr[p];
      S.pv2[i] = v;
      S.mr2[i] = m;
      S.id2[i] = S.id[p];
      S.xym[i] = make_float4(v.x, v.y, m.x, 0.0f);
      S.perm[i] = p;
    }
    __syncthreads();
    if (i < n) S.sortedCodes[i] = sC[i - jBase];
    // windows j in [jBase, b0 + kBlock)
    for (uint32_t t = threadIdx.x; t < b0 + kBlock - jBase; t += kBlock) {
      const uint32_t j = jBase + t;
      int hi = -1;
      if (j < n) {
        const SegDev &G = S.seg[S.segOf[j]];
        if ((uint64_t)j + L < (uint64_t)G.start + G.count)
          hi = min(lcp_digits(sC[t], sC[t + L]), kMaxDepth - 1);
      }
      sHi[t] = (int8_t)hi;
    }
    __syncthreads();
    if (i >= n) continue;
    const SegDev &G = S.seg[S.segOf[i]];
    const uint32_t s0 = G.start;
    const int lo = (i == s0) ? 0 : lcp_digits(sC[i - 1 - jBase], sC[i - jBase]) + 1;
    int w = -1;
    for (uint32_t j = i >= s0 + L ? i - L : s0; j <= i; ++j) w = max(w, (int)sHi[j - jBase]);
    const int leaf = w + 1;
    S.splitCount[i] = lo <= leaf ? (uint32_t)(leaf - lo + 1) : 0u;
    S.splitLo[i] = (uint8_t)lo; // <= 33
  }
}

// Record of the node at depth d starting at body b.
__device__ __forceinline__ uint32_t record_of(const DevState &S, uint32_t b, int d) {
  return S.splitStart[b] + (uint32_t)(d - (int)S.splitLo[b]);
}

// Writes record `at` of the default force walk (QuadRec) from the sums, cell
// and first body of the children in `have` (by digit); returns the link to it.
// (px, py): a finite place for absent children.  kFull: their moments too.
template <bool kFull>
__device__ __forceinline__ uint32_t quad_record(const DevState &S, uint32_t at, float px,
                                                float py, uint32_t have, const float4 (&up)[4],
                                                const float4 (&ca)[4], const float4 (&cm)[4],
                                                const uint32_t (&first)[4]) {
  float x[4], y[4], m[4], w[4];
  uint2 c[4];
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    const bool in = (have >> q) & 1u;
    x[q] = in ? ca[q].x : px;
    y[q] = in ? ca[q].y : py;
    m[q] = in ? ca[q].z : 0.0f;
    w[q] = in ? up[q].z : 0.0f;
    c[q] = in ? make_uint2(__float_as_uint(up[q].w), first[q]) : make_uint2(kQuadLeaf, 0u);
  }
  QuadRec &Q = S.tQ[at];
  Q.x = make_float4(x[0], x[1], x[2], x[3]);
  Q.y = make_float4(y[0], y[1], y[2], y[3]);
  Q.m = make_float4(m[0], m[1], m[2], m[3]);
  Q.w = make_float4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<uint4 *>(&Q.child[0]) = make_uint4(c[0].x, c[0].y, c[1].x, c[1].y);
  *reinterpret_cast<uint4 *>(&Q.child[2]) = make_uint4(c[2].x, c[2].y, c[3].x, c[3].y);
  if (kFull && S.tQM) {
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q)
      if ((have >> q) & 1u) S.tQM[at].m[q] = make_float4(cm[q].x, cm[q].y, cm[q].z, ca[q].w);
  }
  return at;
}

// The record that holds only the root (up, a, moments) of instance sg.
template <bool kFull>
__device__ __forceinline__ void quad_root(const DevState &S, uint32_t sg, float4 up, float4 a,
                                          float4 mom) {
  const float4 ups[4] = {up}, as[4] = {a}, ms[4] = {mom};
  const uint32_t first[4] = {S.seg[sg].start};
  quad_record<kFull>(S, S.n + sg, a.x, a.y, 1u, ups, as, ms, first);
}

// Eight lanes narrow [lo, hi] down to the first index of [lo, hi) where
// before(index) is false (hi if none), before being true up to it: eight
// probes a round.  All groups of the warp call it together.
template <class Before>
__device__ __forceinline__ uint32_t search8(uint32_t lo, uint32_t hi, Before before) {
  const uint32_t g = threadIdx.x & 7u, shift = threadIdx.x & 24u;
  while (__any_sync(0xffffffffu, lo < hi)) {
    const uint64_t len = hi - lo;
    auto probe = [&](uint32_t k) { return lo + (uint32_t)(len * (k + 1u) / 9u); };
    const bool t = lo < hi && before(probe(g));
    const uint32_t yes = __popc((__ballot_sync(0xffffffffu, t) >> shift) & 255u);
    if (lo < hi) {
      const uint32_t l = yes > 0 ? probe(yes - 1u) + 1u : lo;
      hi = yes < 8 ? probe(yes) : hi;
      lo = l;
    }
  }
  return lo;
}

// Sums of a node from those of its children in `have`, in digit order
// (sumNode), then finishNode's divide: up = {weighted sums, bottom size^2,
// link}, own = {centre of mass, mass, size^2}, mom = {moments, size}.  One
// child has the same bodies under a smaller square: its link goes up.  With
// more (true) the link is the node's own record, at its second child's first
// body.
template <bool kFull>
__device__ __forceinline__ bool sum_children(uint32_t have, const float4 (&cu)[4],
                                             const float4 (&ca)[4], const float4 (&cm)[4],
                                             const uint32_t (&first)[4], float w, float size,
                                             float4 &up, float4 &own, float4 &mom) {
  float sx = 0.0f, sy = 0.0f, sm = 0.0f, wBot = 0.0f;
  uint32_t count = 0, link = 0, second = 0;
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    if (!((have >> q) & 1u)) continue;
    sx = count == 0 ? cu[q].x : __fadd_rn(sx, cu[q].x);
    sy = count == 0 ? cu[q].y : __fadd_rn(sy, cu[q].y);
    sm = count == 0 ? ca[q].z : __fadd_rn(sm, ca[q].z);
    if (count == 0) {
      wBot = cu[q].z;
      link = __float_as_uint(cu[q].w);
    }
    if (count == 1) second = first[q];
    ++count;
  }
  const float dv = fmaxf(sm, FLT_MIN);
  const float X = __fdiv_rn(sx, dv), Y = __fdiv_rn(sy, dv);
  if (kFull) {
    float jxx = 0.0f, jyy = 0.0f, jxy = 0.0f;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      if (!((have >> q) & 1u)) continue;
      const float dx = ca[q].x - X, dy = ca[q].y - Y;
      jxx += cm[q].x + ca[q].z * dx * dx;
      jyy += cm[q].y + ca[q].z * dy * dy;
      jxy += cm[q].z + ca[q].z * dx * dy;
    }
    mom = make_float4(jxx, jyy, jxy, size);
  }
  if (count > 1) {
    wBot = w;
    link = second;
  }
  up = make_float4(sx, sy, wBot, __uint_as_float(link));
  own = make_float4(X, Y, sm, w);
  return count > 1;
}

// Place of a spanning node (k_trav_tree) in the arrays span*.
__device__ __forceinline__ uint32_t span_slot(uint32_t record, int depth) {
  return record / kBlock * (kMaxDepth + 1) + (uint32_t)depth;
}

// The traversal records and their sums in one pass, a thread to a record, 256
// consecutive records (preorder) to a block.
//
// A record's parent is the last record before it that is less deep, its
// subtree ends at the first one after it that is no deeper: both come from the
// block's depths in shared memory.  Only the ancestors of the block's first
// record that start before the block (a child's parent) and the ends of the
// last record's ancestors are searched for in the codes, one per depth, eight
// probes a round.
//
// Then upwards, as far as subtrees lie in the block (all nodes but the top
// few): a leaf sums its bodies (sumNode's order) and climbs, and the last child
// to arrive at a node sums its children and climbs on.  A child leaves its
// place at its digit of the node and adds its bodies to the node's arrival
// counter, which is complete at the node's body count.  A node that reaches
// beyond the block ("spans") has its children's records and counter in global
// memory, at (block, depth), which no other spanning node of the block shares;
// k_trav_top sums those, from the children found here.
// kFull: also the cell centres and sizes of tC/tM and the second moments
// about each centre of mass (read only by the corrected forms and the
// network's harvest).
// Bound by the latency of dependent loads.  us between events around the
// stage with k_trav_top: as two kernels, with child bounds, parents and ends
// all bisected and every arrival through global memory, 10,000 bodies 43,
// 99,991 53, 2^20 86, 2^22 167 without the quad records; with the spanning nodes
// summed here, whose threads held their blocks, 31, 34, 70, 228; now 28, 34, 65,
// 157.
template <bool kFull>
__global__ void __launch_bounds__(kBlock, kFull ? 2 : 3)
    k_trav_tree(DevState S, const uint32_t *__restrict__ owner) {
  chain_begin();
  __shared__ float4 sUp[kBlock], sA[kBlock], sM[kFull ? kBlock : 1];
  __shared__ uint32_t sKids[kBlock]; // bytes: a node's children by digit, how far
                                     // after it (less one)
  __shared__ uint32_t sNoDeeper[kMaxDepth + 1][kBlock / 32]; // bit t: depth[t] <= row
  __shared__ uint8_t sDepthEnds[2]; // of the block's first and last record
  __shared__ uint32_t sStart[kBlock], sBodies[kBlock], sArrive[kBlock];
  __shared__ uint32_t sParent[kBlock]; // record
  __shared__ uint8_t sSpans[kBlock];
  __shared__ uint32_t sLeft[kMaxDepth + 1], sRight[kMaxDepth + 1];
  const uint64_t *c = S.sortedCodes;
  const uint32_t total = S.counters[6];
  const bool overflow = total > S.nodeCapacity;
  if (blockIdx.x == 0) {
    // instance bases: all-or-nothing on overflow (the step reports it)
    for (uint32_t sg = threadIdx.x; sg < S.nseg; sg += blockDim.x) {
      SegDev &G = S.seg[sg];
      if (G.count == 0) continue;
      const uint32_t s0 = G.start, s1 = G.start + G.count;
      const uint32_t P = S.splitStart[s0];
      G.travBase = overflow ? 0u : P;
      G.travCount = overflow ? 0u : (s1 < S.n ? S.splitStart[s1] : total) - P;
    }
    if (overflow && threadIdx.x == 0) atomicOr(S.status, kStatusTreeCapacity);
  }
  if (overflow) return;
  const uint32_t t = threadIdx.x;
  const uint32_t lane = t & 31u, warp = t >> 5;
  for (uint32_t base = blockIdx.x * kBlock; base < total; base += gridDim.x * kBlock) {
    const uint32_t p = base + t, held = min((uint32_t)kBlock, total - base);
    bool leaf = false, spans = false;
    uint32_t i = 0, sg = 0, s0 = 0, s1 = 0;
    int d = 0;
    uint64_t ci = 0;
    float w = 0.0f, size = 0.0f;
    if (t < held) {
      i = owner[p];
      sg = S.segOf[i];
      const SegDev &G = S.seg[sg];
      s0 = G.start;
      s1 = G.start + G.count;
      const uint32_t k = p - S.splitStart[i];
      d = S.splitLo[i] + (int)k;
      leaf = k + 1 == S.splitCount[i];
      ci = c[i];
      float cx = G.cx, cy = G.cy;
      size = G.size;
      if (kFull || !(fabsf(G.size) >= 0x1p-90f && fabsf(G.size) <= 0x1p+120f)) {
        for (int q = 0; q < d; ++q) {
          size = __fmul_rn(size, 0.5f);
          const int g = digit_at(ci, q);
          cx = __fadd_rn(cx, __fmul_rn((float)(g & 1) - 0.5f, size));
          cy = __fadd_rn(cy, __fmul_rn((float)(g >> 1) - 0.5f, size));
        }
      } else {
        // d <= 32 halvings of a normal size stay normal: each is exact, so
        // the repeated halving is one exponent step
        size = ldexpf(size, -d);
      }
      w = __fmul_rn(size, size);
      if (kFull) S.tC[p] = make_float2(cx, cy);
      sA[t] = make_float4(0.0f, 0.0f, 0.0f, w);
      if (kFull) sM[t] = make_float4(0.0f, 0.0f, 0.0f, size);
    }
    if (t == 0) sDepthEnds[0] = (uint8_t)d;
    if (t == held - 1u) sDepthEnds[1] = (uint8_t)d;
    {
      uint32_t row = 0, last = 0; // lane's row, and row 32 for lane 0
#pragma unroll
      for (int depth = 0; depth <= kMaxDepth; ++depth) {
        const uint32_t m = __ballot_sync(0xffffffffu, t < held && d <= depth);
        if (depth == kMaxDepth) last = m;
        else if (lane == (uint32_t)depth) row = m;
      }
      sNoDeeper[lane][warp] = row;
      if (lane == 0) sNoDeeper[kMaxDepth][warp] = last;
    }
    sStart[t] = i;
    sKids[t] = 0xffffffffu;
    sArrive[t] = 0u;
    __syncthreads();
    {
      // by eight lanes a depth: four warps the record at it that holds the
      // block's first record, four the end of the one that holds the last
      const bool leftHalf = t < kBlock / 2;
      const uint32_t b = sStart[leftHalf ? 0 : held - 1];
      const int dEnd = leftHalf ? (int)sDepthEnds[0] : (int)sDepthEnds[1] + 1;
      const SegDev &G = S.seg[S.segOf[b]];
      const uint32_t g0 = G.start, g1 = G.start + G.count;
      const uint64_t code = c[b];
      for (int depth = (int)((t & (kBlock / 2 - 1)) >> 3); __any_sync(0xffffffffu, depth < dEnd);
           depth += kBlock / 16) {
        // depth 0 is the whole instance
        const bool search = depth > 0 && depth < dEnd;
        const int sh = search ? 64 - 2 * depth : 0;
        uint32_t lo = leftHalf ? g0 : g1, hi = lo;
        if (search && leftHalf) hi = b;
        if (search && !leftHalf) lo = b + 1u;
        const uint32_t j = search8(lo, hi, [&](uint32_t m) {
          return ((c[m] >> sh) != (code >> sh)) == leftHalf;
        });
        if ((t & 7u) == 0 && depth < dEnd) {
          if (leftHalf) sLeft[depth] = record_of(S, j, depth);
          else sRight[depth] = j;
        }
      }
    }
    __syncthreads();
    uint32_t e = 0, after = 0;
    if (t < held) {
      // the first record after this one that is no deeper ends its subtree
      uint32_t q = kBlock;
      {
        uint32_t m = lane < 31 ? sNoDeeper[d][warp] & (0xfffffffeu << lane) : 0u;
        uint32_t word = warp;
        while (m == 0 && ++word < kBlock / 32) m = sNoDeeper[d][word];
        if (m != 0) q = 32u * word + __ffs(m) - 1u;
      }
      if (q < held) {
        after = base + q;
        e = sStart[q];
      } else {
        e = sRight[d];
        after = e < S.n ? S.splitStart[e] : total;
        spans = !leaf && after > base + kBlock;
      }
      // the last record before this one that is less deep is its parent
      uint32_t parent = 0xffffffffu;
      if (d > 0) {
        uint32_t m = sNoDeeper[d - 1][warp] & ((1u << lane) - 1u);
        int word = (int)warp;
        while (m == 0 && --word >= 0) m = sNoDeeper[d - 1][word];
        parent = m != 0 ? base + 32u * word + 31u - __clz(m) : sLeft[d - 1];
      }
      const uint32_t next = e < s1 ? after : 0xffffffffu;
      S.tN[p].b = make_int4((int)next, (int)(leaf ? next : p + 1), (int)i, (int)e);
      sParent[t] = parent;
      sBodies[t] = e - i;
      sSpans[t] = spans ? 1u : 0u;
      if (spans) { // for k_trav_top
        S.tN[p].a = make_float4(0.0f, 0.0f, 0.0f, w);
        if (kFull) S.tM[p] = make_float4(0.0f, 0.0f, 0.0f, size);
        S.spanParent[span_slot(p, d)] = parent;
      }
    }
    // bodies in leaves too deep for the group walk: one addition a warp where it
    // has one instance
    const uint32_t deep = leaf && d > walk_depth(S.tSq) ? e - i : 0u;
    const uint32_t deepLanes = __ballot_sync(0xffffffffu, deep != 0);
    if (deepLanes != 0) {
      const uint32_t one = __shfl_sync(0xffffffffu, sg, __ffs(deepLanes) - 1);
      if (__all_sync(0xffffffffu, deep == 0 || sg == one)) {
        const uint32_t sum = __reduce_add_sync(0xffffffffu, deep);
        if (lane == 0) add_deep(S.seg[one], sum);
      } else if (deep != 0) {
        add_deep(S.seg[sg], deep);
      }
    }
    // the spanning nodes' list
    const uint32_t spanning = __ballot_sync(0xffffffffu, spans);
    if (spanning) {
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&S.counters[kCtrSpans], (uint32_t)__popc(spanning));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(spanning & ((1u << lane) - 1u));
      if (spans) S.spanList[at] = make_uint4(p, (uint32_t)d, e - i, i);
    }
    __syncthreads();
    // the node this thread holds the sums of: its record, depth and bodies
    uint32_t node = p, bodies = e - i;
    float4 up = make_float4(0.0f, 0.0f, 0.0f, 0.0f), own = up, mom = up;
    if (leaf) {
      const uint32_t b1 = min(e, S.n);
      float px = 0.0f, py = 0.0f, mm = 0.0f;
      for (uint32_t b = i; b < b1; b += 4) { // four loads in flight
        float4 q[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) q[k] = S.xym[min(b + k, b1 - 1u)];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          if (b + k >= b1) continue;
          px = __fadd_rn(px, __fmul_rn(q[k].x, q[k].z));
          py = __fadd_rn(py, __fmul_rn(q[k].y, q[k].z));
          mm = __fadd_rn(mm, q[k].z);
        }
      }
      const float div = fmaxf(mm, FLT_MIN);
      const float X = __fdiv_rn(px, div), Y = __fdiv_rn(py, div);
      if (kFull) {
        float ixx = 0.0f, iyy = 0.0f, ixy = 0.0f;
        for (uint32_t b = i; b < b1; ++b) {
          const float4 q = S.xym[b];
          const float dx = q.x - X, dy = q.y - Y;
          ixx += q.z * dx * dx;
          iyy += q.z * dy * dy;
          ixy += q.z * dx * dy;
        }
        mom = make_float4(ixx, iyy, ixy, size);
      }
      up = make_float4(px, py, w, __uint_as_float(kQuadLeaf | (e - i)));
      own = make_float4(X, Y, mm, w);
    }
    // at most kMaxDepth + 1 nodes, all in the block
    for (int guard = 0; leaf && guard <= kMaxDepth; ++guard) {
      // `node` is summed: keep it (its thread stores it below) and arrive at its
      // parent
      const uint32_t in = node - base;
      sUp[in] = up;
      sA[in] = own;
      if (kFull) sM[in] = mom;
      if (d == 0) {
        quad_root<kFull>(S, sg, up, own, mom);
        break;
      }
      const uint32_t parent = sParent[in];
      if (parent >= total) {
        atomicOr(S.status, kStatusTreeCapacity);
        break;
      }
      --d;
      const uint32_t digit = (uint32_t)digit_at(ci, d); // ci lies in the node
      const uint32_t l = parent - base;
      if (l >= kBlock || sSpans[l] != 0) {
        const uint32_t slot = span_slot(parent, d);
        S.tUp[node] = up;
        reinterpret_cast<uint32_t *>(&S.spanKids[slot])[digit] = node;
        atomicAdd(&S.spanArrive[slot], bodies);
        break;
      }
      reinterpret_cast<uint8_t *>(&sKids[l])[digit] = (uint8_t)(in - l - 1u);
      __threadfence_block();
      if (atomicAdd(&sArrive[l], bodies) + bodies != sBodies[l]) break;
      __threadfence_block();
      node = parent;
      const uint32_t kv = sKids[l];
      bodies = sBodies[l];
      uint32_t have = 0, first[4];
      float4 cu[4], ca[4], cm[4];
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) {
        const uint32_t k = l + 1u + ((kv >> (8 * q)) & 255u);
        if (k >= l + 256u) continue; // 255: empty (a child is at most 255 on)
        have |= 1u << q;
        cu[q] = sUp[k];
        ca[q] = sA[k];
        if (kFull) cm[q] = sM[k];
        first[q] = sStart[k];
      }
      sum_children<kFull>(have, cu, ca, cm, first, sA[l].w, kFull ? sM[l].w : 0.0f, up, own, mom);
    }
    __syncthreads();
    if (t < held && !spans) { // the nodes summed in the block, a thread to each
      const float4 a = sA[t];
      S.tN[p].a = a;
      if (kFull) S.tM[p] = sM[t];
      const uint32_t kv = sKids[t];
      float4 cu[4], ca[4], cm[4];
      uint32_t have = 0, count = 0, second = 0, first[4];
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) {
        const uint32_t k = t + 1u + ((kv >> (8 * q)) & 255u);
        if (k >= t + 256u) continue;
        have |= 1u << q;
        cu[q] = sUp[k];
        ca[q] = sA[k];
        if (kFull) cm[q] = sM[k];
        first[q] = sStart[k];
        if (count == 1) second = first[q];
        ++count;
      }
      if (count > 1) quad_record<kFull>(S, second, a.x, a.y, have, cu, ca, cm, first);
    }
    __syncthreads();
  }
}

// Sums the spanning nodes of k_trav_tree, a thread to each whose children all
// lay in blocks, climbing from there: a child brought to its parent here adds
// its bodies to a second counter, and the one that completes the count of the
// first is the last.  Leaves the nodes' slots empty for the next build.
// ~10 nodes a block of records; bound by the chain of arrivals, so what a level
// needs of its parent is loaded beside its children's sums, and the node's
// own record is written after its arrival (with the moments 48 -> 42 us of the
// stage at 262,144 bodies; without, at 2^22, 159 -> 157).  Depth by depth with
// barriers instead, in one block, takes 2 us less at 10,000 to 100,000
// bodies and 20 more at 2^20.
constexpr int kTopBlock = 64;
template <bool kFull>
__global__ void __launch_bounds__(kTopBlock) k_trav_top(DevState S) {
  chain_begin();
  const uint32_t total = S.counters[6];
  if (total > S.nodeCapacity) return;
  const uint32_t n = S.counters[kCtrSpans];
  for (uint32_t k = blockIdx.x * kTopBlock + threadIdx.x; k < n; k += gridDim.x * kTopBlock) {
    const uint4 entry = S.spanList[k];
    uint32_t node = entry.x, bodies = entry.z;
    int d = (int)entry.y;
    uint32_t slot = span_slot(node, d);
    const uint64_t ci = S.sortedCodes[entry.w];
    uint32_t parent = S.spanParent[slot];
    float w = __ldcg(&S.tN[node].a).w, size = kFull ? __ldcg(&S.tM[node]).w : 0.0f;
    // a node with spanning children never shows its full count here
    if (__ldcg(&S.spanArrive[slot]) != bodies) continue;
    for (int guard = 0; guard <= kMaxDepth; ++guard) {
      const uint4 kv = __ldcg(&S.spanKids[slot]);
      __stcg(&S.spanKids[slot], make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu));
      __stcg(&S.spanArrive[slot], 0u);
      __stcg(&S.spanArriveTop[slot], 0u);
      const bool top = d == 0;
      if (!top && parent >= total) {
        atomicOr(S.status, kStatusTreeCapacity);
        break;
      }
      // of the parent (before this node's arrival nobody empties its count)
      uint32_t pSlot = 0, pParent = 0, pBlocks = 0, pBodies = 0;
      float pw = 0.0f, pSize = 0.0f;
      if (!top) {
        pSlot = span_slot(parent, d - 1);
        pParent = S.spanParent[pSlot];
        pBlocks = __ldcg(&S.spanArrive[pSlot]);
        pw = __ldcg(&S.tN[parent].a).w;
        if (kFull) pSize = __ldcg(&S.tM[parent]).w;
        const int4 b = S.tN[parent].b;
        pBodies = (uint32_t)(b.w - b.z);
      }
      const uint32_t r[4] = {kv.x, kv.y, kv.z, kv.w};
      uint32_t have = 0, first[4];
      float4 cu[4], ca[4], cm[4], up, own, mom;
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) {
        if (r[q] >= total) continue; // all ones: no such child
        have |= 1u << q;
        cu[q] = __ldcg(&S.tUp[r[q]]);
        ca[q] = __ldcg(&S.tN[r[q]].a);
        if (kFull) cm[q] = __ldcg(&S.tM[r[q]]);
        first[q] = (uint32_t)S.tN[r[q]].b.z;
      }
      const bool record = sum_children<kFull>(have, cu, ca, cm, first, w, size, up, own, mom);
      const uint32_t link = __float_as_uint(up.w);
      __stcg(&S.tN[node].a, own);
      if (kFull) __stcg(&S.tM[node], mom);
      uint32_t old = 0;
      if (!top) {
        __stcg(&S.tUp[node], up);
        __stcg(reinterpret_cast<uint32_t *>(&S.spanKids[pSlot]) + digit_at(ci, d - 1), node);
        // release: the child's sums are visible to the last arriver; acquire: the
        // last arriver sees every child's
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;"
                     : "=r"(old)
                     : "l"(&S.spanArriveTop[pSlot]), "r"(bodies)
                     : "memory");
      }
      if (record) quad_record<kFull>(S, link, own.x, own.y, have, cu, ca, cm, first);
      if (top) {
        quad_root<kFull>(S, S.segOf[entry.w], up, own, mom);
        break;
      }
      if (old + bodies + pBlocks != pBodies) break;
      node = parent;
      slot = pSlot;
      parent = pParent;
      bodies = pBodies;
      w = pw;
      size = pSize;
      --d;
    }
  }
}

} // namespace

void launch_bounds(cudaStream_t s, const DevState &S);
void launch_trav_tree(cudaStream_t s, const DevState &S, ScanScratch &scan, bool moments);

void launch_build(cudaStream_t s, DevState &S, ScanScratch &scan,
                  SortScratch &sort, bool moments) {
  const uint32_t n = S.n;
  launch_bounds(s, S); // and the root frames (its last block)
  mark(s, "build.bounds");
  // digit rows, tile counters, look-back words and the long-run count were
  // cleared by the step prologue (launch_step_zero)
  int buf = 0;
  if (S.nseg == 1 && n <= kClusterMortonMax) {
    cluster_sort_morton(s, S, sort); // makes the codes too
  } else {
    launch_after(s, k_morton, grid_for(n), kBlock, 0, S, keys32(sort, 0), sort.hist);
    mark(s, "build.morton");
    // radix passes over the codes' high 32 bits (depth-16 cells), then every
    // run of equal high bits is ordered by its low bits: the same stable order
    // as a full 64-bit sort; such runs are rare and short (at most 2 bodies in
    // the headline states), so this replaces four full passes
    buf = radix_sort_u32(s, sort, n, nullptr, 0, 32, true, true, S.status, 0, true);
    sort_fix_low_bits32(s, sort, buf, n, S.codes, S.longRuns, &S.counters[9], n / 16 + 64,
                        S.status, true);
  }
  mark(s, "build.sort");
  if (S.nseg > 1) {
    // stable passes on the instance id keep instances in their ranges
    k_seg_keys<<<grid_for(n), kBlock, 0, s>>>(S, sort.vals[buf], keys32(sort, buf));
    if (buf == 1) {
      cudaMemcpyAsync(keys32(sort, 0), keys32(sort, 1), sizeof(uint32_t) * n,
                      cudaMemcpyDeviceToDevice, s);
      cudaMemcpyAsync(sort.vals[0], sort.vals[1], sizeof(uint32_t) * n,
                      cudaMemcpyDeviceToDevice, s);
    }
    const int segBits = S.nseg <= 256 ? 8 : 16;
    buf = radix_sort_u32(s, sort, n, nullptr, 0, segBits, false, false, S.status);
  }
  launch_after(s, k_gather_counts, grid_for(n), kBlock, 0, S, sort.vals[buf]);
  mark(s, "build.gather");
  // swap the double-buffered state: the host mirrors this swap
  DevState T = S;
  T.pv = S.pv2;
  T.mr = S.mr2;
  T.id = S.id2;
  T.pv2 = S.pv;
  T.mr2 = S.mr;
  T.id2 = S.id;
  S = T;
  launch_trav_tree(s, S, scan, moments);
}

// The traversal layout straight from the sorted codes (the step path).
// moments: the cells' second moments, centres and sizes too (tM, tC: only
// the corrected forms and the network's harvest read them).
void launch_trav_tree(cudaStream_t s, const DevState &S, ScanScratch &scan, bool moments) {
  const uint32_t n = S.n;
  // per-record scratch in arrays only the breadth-first build uses
  uint32_t *owner = reinterpret_cast<uint32_t *>(S.start);
  // the records per body (splitCount, splitLo) came with the gather
  // the scan also writes each record's first body (owner)
  exclusive_scan_u32(s, S.splitCount, S.splitStart, n, nullptr, &S.counters[6],
                     scan, S.status, owner, S.nodeCapacity, 3);
  mark(s, "tree.counts");
  if (moments) {
    launch_after(s, k_trav_tree<true>, grid_for(n / 4 + 64), kBlock, 0, S, owner);
    launch_after(s, k_trav_top<true>, n / 4096 + 2, kTopBlock, 0, S);
  } else {
    launch_after(s, k_trav_tree<false>, grid_for(n / 4 + 64), kBlock, 0, S, owner);
    launch_after(s, k_trav_top<false>, n / 4096 + 2, kTopBlock, 0, S);
  }
  mark(s, "tree.records");
}

// The reference's breadth-first node arrays (TreeKernels.cuh:88-95) of the
// last build, for introspection only: the step path does not need them.
// Uses the per-body split scratch and the sort scratch, and leaves the
// traversal layout as it is.
void launch_bfs_tree(cudaStream_t s, const DevState &S, ScanScratch &scan,
                     SortScratch &sort) {
  const uint32_t n = S.n;
  k_split_counts<<<grid_for(n), kBlock, 0, s>>>(S);
  exclusive_scan_u32(s, S.splitCount, S.splitStart, n, nullptr, &S.counters[3],
                     scan, S.status);
  k_split_emit<<<grid_for(n), kBlock, 0, s>>>(S, sort.keys[0], sort.vals[0]);
  const int depthBits = S.nseg <= 4 ? 8 : (S.nseg <= 1024 ? 16 : 24);
  const int eb = radix_sort_u64(s, sort, 2 * n + 64, &S.counters[3], 0,
                                depthBits, false, false, S.status);
  cudaMemsetAsync(S.groupStart, 0, sizeof(uint32_t) * S.nseg * kLevelSlots, s);
  cudaMemsetAsync(S.groupEnd, 0, sizeof(uint32_t) * S.nseg * kLevelSlots, s);
  k_groups<<<grid_for(2 * n), kBlock, 0, s>>>(S, sort.keys[eb]);
  k_levels<<<1, 1024, 0, s>>>(S);
  k_split_nodes<<<grid_for(n / 4 + 64), kBlock, 0, s>>>(S, sort.keys[eb],
                                                        sort.vals[eb]);
  k_upward<<<grid_for(n), kBlock, 0, s>>>(S);
}

} // namespace nbx
