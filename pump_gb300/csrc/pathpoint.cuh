// Edge trajectory states (pathPoint, 2pBVP.cu:117-131): shared by the
// waypoint kernels, the dense-path kernels and the search's edge checks.
// Translation units that include this file compile without multiply-add
// contraction, so every rounding is the reference's.
#pragma once

#include "common.cuh"
#include "ffcost.cuh"

namespace pump {
namespace {

// pathPoint, 2pBVP.cu:117-131, in the expression's own evaluation types, by
// kind of state: the x and y positions, their velocities, the z position and
// its velocity each have their own expression, over one axis's end states (p0,
// v0) and (p1, v1).
enum PathKind { kPathXY = 0, kPathVXY, kPathZ, kPathVZ, kPathKinds };
template <int Kind>
__device__ __forceinline__ float path_state64(float t, float tau, float p0, float v0, float p1, float v1) {
  const double t2 = p2f(t), t3 = p3f(t), u2 = p2f(tau), u3 = p3f(tau);
  if (Kind == kPathXY) {
    double r = (double)(t * v0 + p0);
    r = r + (t3 * (double)(2 * p0 - 2 * p1 + (v0 + v1) * tau)) / u3;
    r = r - (t2 * (double)(3 * p0 - 3 * p1 + (2 * v0 + v1) * tau)) / u2;
    return (float)r;
  }
  if (Kind == kPathVXY) {
    float f1 = -(2 * t * (3 * p0 - 3 * p1 + v1 * tau));
    double r = (double)f1 / u2;
    r = r + (3 * t2 * (double)(2 * p0 - 2 * p1 + v1 * tau)) / u3;
    double inner = 3 * t2 - (double)(4 * t * tau) + u2;
    r = r + ((double)v0 * inner) / u2;
    return (float)r;
  }
  if (Kind == kPathZ) {
    double r = (double)(t * v0) * u3 + (double)p0 * u3;
    double q1 = -3. * p0 + 3. * p1 - 2. * v0 * tau - 1. * v1 * tau;
    r = r + (t2 * (double)tau) * q1;
    double q2 = 2. * p0 - 2. * p1 + (double)((v0 + v1) * tau);
    r = r + t3 * q2;
    return (float)(r / u3);
  }
  double r = (double)v0 * u3;
  double q1 = -6. * p0 + 6. * p1 - 4. * v0 * tau - 2. * v1 * tau;
  r = r + (double)(t * tau) * q1;
  double q2 = 6. * p0 - 6. * p1 + 3. * v0 * tau + 3. * v1 * tau;
  r = r + t2 * q2;
  return (float)(r / u3);
}

// State d (0 .. 5), out of line: evaluated in place, the compiler runs the
// binary64 code ahead of the test that asks for it, which took six times the
// rest of the waypoint kernel's time.
__device__ __noinline__ float path_state_now(int d, float t, float tau, float p0, float v0, float p1,
                                             float v1) {
  if (d < 2) return path_state64<kPathXY>(t, tau, p0, v0, p1, v1);
  if (d == 2) return path_state64<kPathZ>(t, tau, p0, v0, p1, v1);
  if (d < 5) return path_state64<kPathVXY>(t, tau, p0, v0, p1, v1);
  return path_state64<kPathVZ>(t, tau, p0, v0, p1, v1);
}

// The binary32 results of path_state64 from float-float arithmetic
// (ffcost.cuh's operations), certified as in cost_ff: with r = t / tau each
// state is the sum of a few terms (a position x0 + ... as A + X r^3 - Y r^2,
// with A, X and Y the binary32 values the expression converts), evaluated
// exactly enough in float-float.  The binary64 value differs from the exact sum
// of those terms by its roundings (at most 16 of them, each within 2^-53 of a
// partial result no larger than M, the sum of the terms' magnitudes, tau^3 and
// t^3 included: 2^-49 M).  The float-float value: 1 / tau from a reciprocal
// estimate and one residual to 7 u^2 (u = 2^-24), products by a binary32 value
// 3 u^2 and by a float-float one 6 u^2, so r, r^2 and r^3 to 10, 26 and 42 u^2,
// the edge's sums to 9 u^2 and the terms to at most 54 u^2; a sum of n terms
// (their high parts by TwoSum, the errors and unnormalised low parts in
// binary32) adds at most 30 u^2: at most 84 u^2 M = 2^-41.6 M.  When the interval
// of half-width 2^-41 M around the float-float value lies inside the binary32
// rounding cell of its high part, that is the expression's (float) conversion;
// otherwise (or for tau outside [2^-20, 2^20], values outside [2^-40, 2^60] and non-finite
// values) path_state64 gives it.  The per-edge terms (path_ff_edge) are shared
// by the edge's waypoints.
//
// A coordinate at rest (both velocities +0, the same position, up to 2^60 in
// magnitude) has a velocity of exactly +0 throughout, and a position of +0 where
// that position is +0: each difference in the expressions is +0, every product
// of it a zero, and a sum that +0 enters is +0 (-0 only arises from two of
// them; the sums' first zeros of either sign meet a +0).  No bound can certify
// a zero, and evaluating them all in binary64 took most of the time of a plan in
// a plane or on a line (100,000 edges of 8 segments, y and z zero: 371 us when a
// point's states were evaluated together, 498 one at a time, 23 so).
struct PathFF {
  bool ok;                        // tau in range: the float-float values apply
  unsigned zero;                  // the states that are +0 whatever t is
  FF rt, ru2;                     // 1 / tau, 1 / tau^2
  float X[2], Y[2], inner[2];     // the expressions' binary32 edge terms
  FF Z[2];                        // 3 Z / tau, Z the binary32 edge term
  FF q1, q2, c1, c2;              // z's edge sums; its velocity's, over tau^3 and tau
  float mq1, mq2, mc1, mc2;       // their terms' magnitudes
};

// Sum of a binary32 value and float-float terms.
__device__ __forceinline__ FF ff_sum(float a, FF x, FF y) {
  const FF s = ff_two_sum(a, x.hi);
  const FF t = ff_two_sum(s.hi, y.hi);
  return ff_fast_two_sum(t.hi, (s.lo + t.lo) + (x.lo + y.lo));
}

__device__ __forceinline__ PathFF path_ff_edge(float tau, const float *x0, const float *x1) {
  PathFF e;
  e.ok = tau >= 0x1p-20f && tau <= 0x1p20f;
  e.zero = 0u;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const unsigned p = __float_as_uint(x0[k]);
    const unsigned moves = __float_as_uint(x0[k + 3]) | __float_as_uint(x1[k + 3]) | (p ^ __float_as_uint(x1[k]));
    if (moves == 0u && fabsf(x0[k]) <= 0x1p60f) e.zero |= (p == 0u ? 9u : 8u) << k;
  }
  const float r = ff_rcp(tau);
  e.rt = ff_fast_two_sum(r, r * fmaf(-tau, r, 1.0f));
  e.ru2 = ff_mul(e.rt, e.rt);
  const FF ru3 = ff_mul(e.ru2, e.rt);
  const FF rt3 = ff_mul_f(e.rt, 3.0f);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int a = k, b = k + 3;
    // the same binary32 expressions as path_state64
    e.X[k] = 2 * x0[a] - 2 * x1[a] + (x0[b] + x1[b]) * tau;
    e.Y[k] = 3 * x0[a] - 3 * x1[a] + (2 * x0[b] + x1[b]) * tau;
    e.inner[k] = 3 * x0[a] - 3 * x1[a] + x1[b] * tau;
    e.Z[k] = ff_mul_f(rt3, 2 * x0[a] - 2 * x1[a] + x1[b] * tau);
  }
  // -3 x0z + 3 x1z - 2 x0vz tau - x1vz tau (each term exact in binary64)
  {
    const FF a = ff_two_prod(x0[2], -3.0f), b = ff_two_prod(x1[2], 3.0f);
    const FF c = ff_two_prod(2.0f * x0[5], -tau), d = ff_two_prod(x1[5], -tau);
    e.q1 = ff_add(ff_add(ff_add(a, b), c), d);
    e.mq1 = fabsf(a.hi) + fabsf(b.hi) + fabsf(c.hi) + fabsf(d.hi);
  }
  // 2 x0z - 2 x1z + (binary32 (x0vz + x1vz) tau)
  {
    const float w = (x0[5] + x1[5]) * tau;
    const FF ab = ff_two_sum(2.0f * x0[2], -2.0f * x1[2]);
    e.q2 = ff_add_f(ab, w);
    e.mq2 = fabsf(2.0f * x0[2]) + fabsf(2.0f * x1[2]) + fabsf(w);
  }
  // -6 x0z + 6 x1z - 4 x0vz tau - 2 x1vz tau
  {
    const FF a = ff_two_prod(x0[2], -6.0f), b = ff_two_prod(x1[2], 6.0f);
    const FF c = ff_two_prod(4.0f * x0[5], -tau), d = ff_two_prod(2.0f * x1[5], -tau);
    e.c1 = ff_mul(ff_add(ff_add(ff_add(a, b), c), d), ru3);
    e.mc1 = (fabsf(a.hi) + fabsf(b.hi) + fabsf(c.hi) + fabsf(d.hi)) * ru3.hi;
  }
  // 6 x0z - 6 x1z + 3 x0vz tau + 3 x1vz tau
  {
    const FF a = ff_two_prod(x0[2], 6.0f), b = ff_two_prod(x1[2], -6.0f);
    const FF c = ff_mul_f(ff_two_prod(x0[5], tau), 3.0f), d = ff_mul_f(ff_two_prod(x1[5], tau), 3.0f);
    e.c2 = ff_mul(ff_add(ff_add(ff_add(a, b), c), d), e.rt);
    e.mc2 = (fabsf(a.hi) + fabsf(b.hi) + fabsf(c.hi) + fabsf(d.hi)) * e.rt.hi;
  }
  return e;
}

// *out = the binary32 rounding of every value within 2^-41 M + 2^-80 of v
// (true), or false when the interval reaches a rounding boundary (or leaves
// range).  The boundary taken on both sides is the nearer one (half a unit in
// the last place; a quarter at a power of two).  The absolute 2^-80 covers
// float-float parts that fall below binary32's normal range (each at most
// 2^-149 off, scaled by at most 2^60 through 1 / tau^3).
__device__ __forceinline__ bool ff_certify(FF v, float M, float *out) {
  const unsigned bits = __float_as_uint(v.hi) & 0x7fffffffu;
  // |v| in [2^-40, 2^60], which also rules out NaN; M up to 2^60 in B
  const bool in = bits - 0x2b800000u <= 0x5d800000u - 0x2b800000u;
  const unsigned low = (bits & 0x7fffffu) ? 24u << 23 : 25u << 23;
  const float room = __uint_as_float((bits & 0x7f800000u) - low);
  const float B = fmaf(M, 0x1p-41f * 1.01f, 0x1p-80f);
  *out = v.hi;
  return in && B <= 0x1p19f && fabsf(v.lo) + B < room;
}

// The certified states of x; returns a bit per state that is not (its x is
// then unspecified).  The sums give +0 for the states of e.zero.
__device__ __forceinline__ unsigned path_point_try(float t, float tau, const float *x0,
                                                   const float *x1, const PathFF &e, float *x) {
  const FF r = ff_mul_f(e.rt, t);
  const FF r2 = ff_mul(r, r);
  const FF r3 = ff_mul(r2, r);
  unsigned bad = 0u;
  // the velocities' 1 - (4 t tau) / tau^2 + 3 r^2, the binary32 product rounded
  const FF r2x3 = ff_term_f(r2, 3.0f);
  const FF F = ff_term_f(e.ru2, -(4 * t * tau));
  const FF in = ff_sum(1.0f, F, r2x3);
  const float min = 1.0f + (fabsf(F.hi) + r2x3.hi);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int a = k, b = k + 3;
    // position: A + X r^3 - Y r^2
    const float A = t * x0[b] + x0[a];
    const FF T1 = ff_term_f(r3, e.X[k]), T2 = ff_term_f(r2, -e.Y[k]);
    if (!ff_certify(ff_sum(A, T1, T2), fabsf(A) + fabsf(T1.hi) + fabsf(T2.hi), &x[k])) bad |= 1u << k;
    // velocity: f1 / tau^2 + r^2 3 Z / tau + x0v (1 - F / tau^2 + 3 r^2)
    const float f1 = -(2 * t * e.inner[k]);
    const FF S1 = ff_term_f(e.ru2, f1);
    const FF S2 = ff_term(r2, e.Z[k]);
    const FF S3 = ff_term_f(in, x0[b]);
    const FF s = ff_two_sum(S1.hi, S2.hi);
    const FF u = ff_two_sum(s.hi, S3.hi);
    const FF W = ff_fast_two_sum(u.hi, (s.lo + u.lo) + ((S1.lo + S2.lo) + S3.lo));
    if (!ff_certify(W, fabsf(S1.hi) + fabsf(S2.hi) + fabsf(x0[b]) * min, &x[3 + k])) bad |= 1u << (3 + k);
  }
  {
    // z: t x0vz + x0z + r^2 q1 + r^3 q2
    const float P = t * x0[5];
    const FF T1 = ff_term(r2, e.q1), T2 = ff_term(r3, e.q2);
    const FF A = ff_two_sum(P, x0[2]);
    const FF s = ff_two_sum(A.hi, T1.hi);
    const FF u = ff_two_sum(s.hi, T2.hi);
    const FF V = ff_fast_two_sum(u.hi, ((A.lo + s.lo) + u.lo) + (T1.lo + T2.lo));
    const float M = fabsf(P) + fabsf(x0[2]) + r2.hi * e.mq1 + fabsf(r3.hi) * e.mq2;
    if (!ff_certify(V, M, &x[2])) bad |= 1u << 2;
  }
  {
    // vz: x0vz + (t tau) c1 + r^2 c2
    const float tt = t * tau;
    const FF T1 = ff_term_f(e.c1, tt), T2 = ff_term(r2, e.c2);
    const float M = fabsf(x0[5]) + fabsf(tt) * e.mc1 + r2.hi * e.mc2;
    if (!ff_certify(ff_sum(x0[5], T1, T2), M, &x[5])) bad |= 1u << 5;
  }
  return e.ok ? bad & ~e.zero : 0x3fu;
}

// pathPoint's values: certified, the remaining states in binary64.
__device__ __forceinline__ void path_point_fast(float t, float tau, const float *x0,
                                                const float *x1, float *x) {
  const unsigned bad = path_point_try(t, tau, x0, x1, path_ff_edge(tau, x0, x1), x);
  if (bad) {
#pragma unroll
    for (int d = 0; d < kDim; ++d) {
      const int a = d < 3 ? d : d - 3;
      if ((bad >> d) & 1u) x[d] = path_state_now(d, t, tau, x0[a], x0[a + 3], x1[a], x1[a + 3]);
    }
  }
}

// The waypoint and dense-path kernels' queue of states left for binary64, shared
// by a block: (thread, waypoint, axis) entries in one list per kind, so that a warp then
// evaluates 32 of one kind at once (binary64 instructions occupy this GPU's
// binary64 pipe for the same time for one lane as for 32; one state in about
// 200 is left, and evaluating each lane's own as they came took most of the
// kernel's time).  A full list returns false: the thread evaluates it itself.
template <int Cap>
struct PathQueue {
  int n[kPathKinds];
  unsigned e[kPathKinds][Cap];
  __device__ __forceinline__ void clear() {
    if (threadIdx.x < kPathKinds) n[threadIdx.x] = 0;
  }
  // state d (0 .. 5) of waypoint i of thread th's edge
  __device__ __forceinline__ bool push(int th, int i, int d) {
    const int axis = d < 3 ? d : d - 3;
    const int kind = (axis == 2 ? kPathZ : kPathXY) + (d < 3 ? 0 : 1);
    const int at = atomicAdd(&n[kind], 1);
    if (at >= Cap) return false;
    e[kind][at] = ((unsigned)th << 20) | ((unsigned)i << 2) | (unsigned)axis;
    return true;
  }
  // state(kind, th, i, axis) for every entry, 32 of a kind per warp; call after
  // a barrier
  template <class State>
  __device__ __forceinline__ void drain(State state) const {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    int task = 0;
    auto run = [&](auto kind) {
      constexpr int Kind = decltype(kind)::value;
      const int cnt = n[Kind] < Cap ? n[Kind] : Cap;
      for (int q0 = 0; q0 < cnt; q0 += 32, ++task) {
        if (task % warps != warp || q0 + lane >= cnt) continue;
        const unsigned ent = e[Kind][q0 + lane];
        state(kind, (int)(ent >> 20), (int)((ent >> 2) & 0x3ffffu), (int)(ent & 3u));
      }
    };
    run(std::integral_constant<int, kPathXY>{});
    run(std::integral_constant<int, kPathVXY>{});
    run(std::integral_constant<int, kPathZ>{});
    run(std::integral_constant<int, kPathVZ>{});
  }
};

// The same trajectory as path_point (cubic position, quadratic velocity,
// no gravity term) in binary32 Hermite form with s = t / tau; used by the
// precision mode, where FP64 is reserved for the optimal-time root.
__device__ __forceinline__ void path_point_f32(float t, float tau, const float *x0, const float *x1,
                                               float *x) {
  const float s = t / tau;
  const float s2 = s * s, s3 = s2 * s;
  const float h00 = fmaf(2.0f, s3, fmaf(-3.0f, s2, 1.0f)), h01 = fmaf(-2.0f, s3, 3.0f * s2);
  const float h10 = tau * (s3 - 2.0f * s2 + s), h11 = tau * (s3 - s2);
  const float g00 = (6.0f * s2 - 6.0f * s) / tau, g10 = fmaf(3.0f, s2, fmaf(-4.0f, s, 1.0f));
  const float g11 = fmaf(3.0f, s2, -2.0f * s);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    x[k] = fmaf(h00, x0[k], fmaf(h01, x1[k], fmaf(h10, x0[k + 3], h11 * x1[k + 3])));
    x[k + 3] = fmaf(g00, x0[k] - x1[k], fmaf(g10, x0[k + 3], g11 * x1[k + 3]));
  }
}

}  // namespace
}  // namespace pump
