// naive.cu -- direct all-pairs gravity: the force pass of NaiveSimulation
// (src/naive/NaiveSimulation.cpp:17-57) and CudaNaiveSimulation
// (src/cuda/CudaNaive.cu:17-57), selected by nbx_params.force_law = 1.
//
// Per pair, in the reference's order of operations:
//   d = pos_j - pos_i, s = |d|^2 + eps^2,
//   acc_i += d * (m_j * (1 / sqrt(s)) * (1 / s)),
// summed over every other body j of the same instance in array order.
//
// The step is iterate -> collide -> attract as for the tree, with an
// identity gather in place of the Morton gather so the state alternates
// between the two buffers exactly as a tree step does.
//
// Default arithmetic with a normal eps^2 (k_naive_pairs): one target per
// thread, sources through shared memory as arrays of x, y and mass, the law of
// two sources at a time in paired FP32 instructions and their accumulation
// one after the other, so every sum keeps its order and rounding.
// Bound: the FP32 pipe, 9 instructions' worth of it per 32 interactions
// (paired instructions save issue slots, not pipe time).  65,537 bodies:
// 3468 -> 1832 us, 131,072: 9568 -> 6090 (2.8e12 interactions/s, 69% of the
// pipe), 5000: 279 -> 84; before, two targets per thread left 8 warps per SM, and
// each of the law's 13 instructions (rsqrtf scales subnormal arguments: a
// compare and two multiplies) waited for the last.  One thread per target
// gives 14 warps per SM there, 3.5 per scheduler, so an SM ends with its
// schedulers of 4: 86% of what an even split would give.
//
// Exact arithmetic, eps = 0 and a subnormal eps^2 run a loop that checks each
// source's instance and skips j == i (k_naive), as the reference does, and so
// does a block of k_naive_pairs whose targets straddle instances.  Otherwise the
// body itself adds m / eps^3 times a distance of zero, and a last tile's padding
// a mass of zero at the origin: exactly zero both, unless m / eps^3 (eps^-3)
// overflows -- m 1 below eps 1.4e-13, m 1e6 below 1.4e-11.  Then the sum is NaN;
// where the largest mass allows that, k_naive runs again over the blocks with a
// NaN (a check in k_naive_pairs itself: 44 registers for 40, 1842 -> 1868 us).
#include "nbx_state.cuh"

#include <float.h>

namespace nbx {
namespace {

constexpr int kNaiveThreads = 128; // targets per block
constexpr int kTile = 256;         // sources staged at a time

// Exact: the reference's IEEE operations, no contraction.
__device__ __forceinline__ void naive_term_exact(float4 q, float x, float y,
                                                 float eSq, float &ax, float &ay) {
  const float dx = __fsub_rn(q.x, x), dy = __fsub_rn(q.y, y);
  const float s = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), eSq);
  const float invSoft = __frcp_rn(s);
  const float invDist = __frcp_rn(__fsqrt_rn(s));
  const float f = __fmul_rn(__fmul_rn(q.z, invDist), invSoft);
  ax = __fadd_rn(ax, __fmul_rn(dx, f));
  ay = __fadd_rn(ay, __fmul_rn(dy, f));
}

// Default: contracted, one hardware rsqrt (s^-3/2 = r^3).
__device__ __forceinline__ void naive_term_fast(float4 q, float x, float y,
                                                float eSq, float &ax, float &ay) {
  const float dx = q.x - x, dy = q.y - y;
  const float s = fmaf(dx, dx, fmaf(dy, dy, eSq));
  const float r = rsqrtf(s);
  const float f = q.z * (r * r * r);
  ax = fmaf(dx, f, ax);
  ay = fmaf(dy, f, ay);
}

// The instances of a block's targets: [lo, hi) covers their bodies, and
// j0, j1 are the thread's own instance; mixed if the targets' instances differ.
struct Sources {
  uint32_t lo, hi, j0, j1;
  bool mixed;
};
__device__ __forceinline__ Sources block_sources(const DevState &S, uint32_t i) {
  const uint32_t first = blockIdx.x * kNaiveThreads;
  const uint32_t last = min(first + kNaiveThreads, S.n) - 1u;
  const uint32_t s0 = S.segOf[first], s1 = S.segOf[last];
  const SegDev &G0 = S.seg[s0], &G1 = S.seg[s1], &G = S.seg[S.segOf[min(i, last)]];
  return {G0.start, G1.start + G1.count, G.start, G.start + G.count, s0 != s1};
}

// Sum over [lo, hi) with the checks.
template <bool kExact>
__device__ __forceinline__ void naive_checked(const DevState &S, const Sources &src, uint32_t i,
                                              float x, float y, float eSq, float4 *tile,
                                              float &ax, float &ay) {
  for (uint32_t base = src.lo; base < src.hi; base += kTile) {
    const uint32_t cnt = min((uint32_t)kTile, src.hi - base);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < cnt; k += kNaiveThreads) tile[k] = S.xym[base + k];
    __syncthreads();
    for (uint32_t k = 0; k < cnt; ++k) {
      const float4 q = tile[k];
      const uint32_t j = base + k;
      if (j < src.j0 || j >= src.j1 || j == i) continue;
      if (kExact) naive_term_exact(q, x, y, eSq, ax, ay);
      else naive_term_fast(q, x, y, eSq, ax, ay);
    }
  }
}

// kAgain: only the blocks in which some sum is NaN.
template <bool kExact, bool kAgain = false>
__global__ void __launch_bounds__(kNaiveThreads) k_naive(DevState S, float eSq) {
  __shared__ float4 tile[kTile];
  const uint32_t i = blockIdx.x * kNaiveThreads + threadIdx.x;
  if (kAgain) {
    const float2 a = S.acc[min(i, S.n - 1u)];
    if (!__syncthreads_or(a.x != a.x || a.y != a.y)) return;
  }
  const Sources src = block_sources(S, i);
  const float4 b = S.xym[min(i, S.n - 1u)];
  float ax = 0.0f, ay = 0.0f;
  naive_checked<kExact>(S, src, i, b.x, b.y, eSq, tile, ax, ay);
  if (i >= S.n) return;
  add_attractor<kExact>(S.attr, b.x, b.y, ax, ay);
  S.acc[i] = make_float2(ax, ay);
}

// For eps^2 >= FLT_MIN: every s is normal, so the flushing reciprocal square
// root gives rsqrtf's bits.
__device__ __forceinline__ float rsqrt_normal(float s) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
  return r;
}

__global__ void __launch_bounds__(kNaiveThreads) k_naive_pairs(DevState S, float eSq) {
  __shared__ float4 tile[kTile]; // or the same bytes as x, y and mass arrays
  const uint32_t i = blockIdx.x * kNaiveThreads + threadIdx.x;
  const Sources src = block_sources(S, i);
  const float4 b = S.xym[min(i, S.n - 1u)];
  const float x = b.x, y = b.y;
  float ax = 0.0f, ay = 0.0f;
  if (src.mixed) {
    naive_checked<false>(S, src, i, x, y, eSq, tile, ax, ay);
  } else {
    float *sx = reinterpret_cast<float *>(tile), *sy = sx + kTile, *sm = sy + kTile;
    constexpr int kPer = kTile / kNaiveThreads;
    float4 next[kPer];
    auto fetch = [&](uint32_t base) {
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const uint32_t j = base + k * kNaiveThreads + threadIdx.x;
        next[k] = j < src.hi ? S.xym[j] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    };
    const f2x XX = pk2(x, x), YY = pk2(y, y), E2 = pk2(eSq, eSq);
    fetch(src.lo);
    for (uint32_t base = src.lo; base < src.hi; base += kTile) {
      __syncthreads();
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        sx[k * kNaiveThreads + threadIdx.x] = next[k].x;
        sy[k * kNaiveThreads + threadIdx.x] = next[k].y;
        sm[k * kNaiveThreads + threadIdx.x] = next[k].z;
      }
      __syncthreads();
      fetch(base + kTile);
      // a last partial tile: massless sources to a multiple of four
      const uint32_t cnt = min((uint32_t)kTile, src.hi - base);
#pragma unroll 8
      for (uint32_t k = 0; k < cnt; k += 4) {
        const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&sx[k]);
        const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&sy[k]);
        const ulonglong2 M = *reinterpret_cast<const ulonglong2 *>(&sm[k]);
        const f2x X2[2] = {X.x, X.y}, Y2[2] = {Y.x, Y.y}, M2[2] = {M.x, M.y};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const f2x DX = sub2(X2[h], XX), DY = sub2(Y2[h], YY);
          float s0, s1, dx0, dx1, dy0, dy1, f0, f1;
          upk2(fma2(DX, DX, fma2(DY, DY, E2)), s0, s1);
          const f2x R = pk2(rsqrt_normal(s0), rsqrt_normal(s1));
          upk2(mul2(M2[h], mul2(mul2(R, R), R)), f0, f1);
          upk2(DX, dx0, dx1);
          upk2(DY, dy0, dy1);
          ax = fmaf(dx0, f0, ax);
          ay = fmaf(dy0, f0, ay);
          ax = fmaf(dx1, f1, ax);
          ay = fmaf(dy1, f1, ay);
        }
      }
    }
  }
  if (i >= S.n) return;
  add_attractor<false>(S.attr, x, y, ax, ay);
  S.acc[i] = make_float2(ax, ay);
}

// The naive step's stand-in for the Morton gather: the same buffer swap,
// bodies kept in their order.
__global__ void k_identity_gather(DevState S) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n;
       i += gridDim.x * blockDim.x) {
    const float4 v = S.pv[i];
    const float2 m = S.mr[i];
    S.pv2[i] = v;
    S.mr2[i] = m;
    S.id2[i] = S.id[i];
    S.xym[i] = make_float4(v.x, v.y, m.x, 0.0f);
  }
}

} // namespace

// Identity gather + buffer swap; returns the state after the swap.
DevState launch_naive_gather(cudaStream_t s, const DevState &S) {
  uint32_t b = (S.n + 255) / 256;
  if (b > 148u * 16u) b = 148u * 16u;
  k_identity_gather<<<b ? b : 1, 256, 0, s>>>(S);
  DevState T = S;
  T.pv = S.pv2;
  T.mr = S.mr2;
  T.id = S.id2;
  T.pv2 = S.pv;
  T.mr2 = S.mr;
  T.id2 = S.id;
  return T;
}

// Whether a body's own term (or the padding's) can overflow in k_naive_pairs;
// maxMass: of all bodies, or infinity where it is not known.
bool naive_overflows(float eSq, float maxMass) {
  const double m = maxMass < 1.0f ? 1.0 : maxMass; // NaN: not known
  return !(m / ((double)eSq * sqrt((double)eSq)) < 1e38);
}

// All-pairs accelerations of the bodies in S.xym into S.acc.
void launch_naive_forces(cudaStream_t s, const DevState &S, bool exact, float maxMass) {
  if (S.n == 0) return;
  const uint32_t blocks = (S.n + kNaiveThreads - 1) / kNaiveThreads;
  if (exact) {
    k_naive<true><<<blocks, kNaiveThreads, 0, s>>>(S, S.eSq);
  } else if (S.eSq >= FLT_MIN) {
    k_naive_pairs<<<blocks, kNaiveThreads, 0, s>>>(S, S.eSq);
    if (naive_overflows(S.eSq, maxMass))
      k_naive<false, true><<<blocks, kNaiveThreads, 0, s>>>(S, S.eSq);
  } else {
    k_naive<false><<<blocks, kNaiveThreads, 0, s>>>(S, S.eSq);
  }
}

} // namespace nbx
