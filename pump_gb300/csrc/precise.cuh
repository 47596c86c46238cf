// Closed-form optimal time of the 2pBVP (precision mode), shared by the
// pair kernels and the path-refinement adjoint.  Include only from
// translation units compiled with multiply-add contraction.
//
// The global minimiser of the reference's cost (2pBVP.cu:97-107) in closed
// form.  Written out, the cost is
//   c(t) = A0/t^3 + A1/t^2 + A2/t + A3 + A4 t with
//   A0 = 12|p1-p0|^2, A1 = -12 (p1-p0).(v0+v1), A2 = 4(|v0|^2+v0.v1+|v1|^2),
//   A3 = 2g(v0z-v1z), A4 = 1+g^2,
// so c'(t) = 0 is the quartic Q(t) = A4 t^4 - A2 t^2 - 2 A1 t - 3 A0 = 0.
// The coefficients are assembled in float-float (pairs of binary32, ~46-bit
// significands).  For almost every pair the root, one Newton step and the cost
// follow in binary32 and float-float with a bound on their error, and the
// rounded results are certain (precise_min).  The other pairs take the general
// way: the roots of Q are bracketed in binary32 (pieces split at the
// inflection point and the real roots of Q'); each candidate minimum is
// refined with one Newton step whose residual Q(x) is evaluated in binary64;
// the candidates (and tmax) are compared by their binary64 cost.  Translation
// units including this header are compiled with multiply-add contraction (the
// mode is not bound to the reference's roundings).
#pragma once
#include <math.h>

#include "common.cuh"

namespace pump {
namespace {

// ---------------------------------------------------------------------------
// Float-float arithmetic (Dekker / Knuth error-free transformations): a value
// is h + l with |l| <= ulp(h) / 2.  No multiply-add is left to the compiler:
// products use explicit fmaf, sums have no products to contract.
struct FF {
  float h, l;
};
__device__ __forceinline__ FF two_sum(float a, float b) {
  const float s = a + b, bp = s - a;
  return {s, (a - (s - bp)) + (b - bp)};
}
__device__ __forceinline__ FF fast_two_sum(float a, float b) {  // |a| >= |b|
  const float s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ FF two_prod(float a, float b) {
  const float p = a * b;
  return {p, fmaf(a, b, -p)};
}
__device__ __forceinline__ FF ff_add(FF x, FF y) {
  const FF s = two_sum(x.h, y.h);
  return fast_two_sum(s.h, s.l + (x.l + y.l));
}
__device__ __forceinline__ FF ff_mul(FF x, FF y) {
  const FF p = two_prod(x.h, y.h);
  return fast_two_sum(p.h, p.l + fmaf(x.h, y.l, x.l * y.h));
}
__device__ __forceinline__ FF ff_mulf(FF x, float c) {
  const FF p = two_prod(x.h, c);
  return fast_two_sum(p.h, fmaf(x.l, c, p.l));
}

// Exact binary32 -> binary64 with integer operations (the FP64 pipe is the
// scarce resource): rebias the exponent, widen the significand.  Binary32
// subnormals become zero; infinities and NaNs stay what they are.
__device__ __forceinline__ double f2d_exact(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned e = (u >> 23) & 0xffu;
  const unsigned long long sign = (unsigned long long)(u >> 31) << 63;
  const unsigned long long frac = (unsigned long long)(u & 0x7fffffu) << 29;
  const unsigned long long ex = e == 0xffu ? 0x7ffull : (unsigned long long)(e + 896u);
  const unsigned long long bits = e == 0 ? sign : (sign | (ex << 52) | frac);
  return __longlong_as_double((long long)bits);
}

// Binary64 -> binary32, round to nearest even, with integer operations for
// results in binary32's normal range; anything else takes the conversion
// instruction.
__device__ __forceinline__ float d2f_rn(double d) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(d);
  const int e = (int)((u >> 52) & 0x7ff) - 896;
  if (e <= 0 || e >= 255) return (float)d;
  unsigned mf = (unsigned)((u >> 29) & 0x7fffffu);
  const unsigned rem = (unsigned)(u & 0x1fffffffu);
  mf += (rem > 0x10000000u) | ((rem == 0x10000000u) & (mf & 1u));
  // a carry out of the significand moves into the exponent field (to
  // infinity only if the value rounds past the largest binary32)
  const unsigned bits = ((unsigned)(u >> 32) & 0x80000000u) + (((unsigned)e << 23) + mf);
  return __uint_as_float(bits);
}

// The cost's binary64 polynomials, with every expression written out in
// explicit fma() so that the all-pairs kernel and the explicit-pair kernel
// produce identical bits for the same pair.
struct Quartic {
  double A0, A1, A2, A3, A4;
  double A0x3, A1x2;  // 3 A0 and 2 A1 for Q
  __device__ double Q(double t) const {
    return fma(fma(fma(A4 * t, t, -A2), t, -A1x2), t, -A0x3);
  }
  // 1/t from the hardware reciprocal estimate refined by one binary64 Newton
  // step (relative error ~1e-14, far below the binary32 the cost becomes)
  __device__ double cost(double t) const {
    const double y0 = rcp_approx(t);
    const double r = fma(y0, fma(-t, y0, 1.0), y0);
    return fma(A4, t, fma(fma(fma(A0, r, A1), r, A2), r, A3));
  }
  __device__ static double rcp_approx(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
  }
};

// A sample with |v|^2 in float-float: prepared once per launch for the
// all-pairs kernel, in registers for explicit pairs.
struct __align__(16) SampleF {
  float p[3], v[3];
  FF vv;
};

__device__ __forceinline__ SampleF to_sample_f(const float *x) {
  SampleF s;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    s.p[d] = x[d];
    s.v[d] = x[3 + d];
  }
  s.vv = ff_add(ff_add(two_prod(x[3], x[3]), two_prod(x[4], x[4])), two_prod(x[5], x[5]));
  return s;
}

__device__ __forceinline__ double ff2d(FF x) { return f2d_exact(x.h) + f2d_exact(x.l); }

// The same polynomials in binary32 for the bracketing phase.
struct QuarticF {
  float A0, A1, A2, A4;  // binary32 copies for the bracketing phase
  __device__ float Q(float t) const { return ((A4 * t * t - A2) * t - 2.0f * A1) * t - 3.0f * A0; }
  __device__ float dQ(float t) const { return (4.0f * A4 * t * t - 2.0f * A2) * t - 2.0f * A1; }
  __device__ float d2Q(float t) const { return 12.0f * A4 * t * t - 2.0f * A2; }
};


// Root of a monotone function on [a, b] (sign change given) with fixed
// convexity: Newton started at x0, on the side where the function and its
// curvature have the same sign, converges monotonically.  Binary32.
template <int Deriv>
__device__ float newton_f(const QuarticF &q, float a, float b, float x0) {
  float x = x0;
  for (int it = 0; it < 40; ++it) {
    const float f = Deriv ? q.dQ(x) : q.Q(x);
    const float df = Deriv ? q.d2Q(x) : q.dQ(x);
    if (f == 0.0f || df == 0.0f) break;
    float xn = x - __fdividef(f, df);  // approximate quotient: a Newton step needs no rounding guarantee
    if (!(xn >= a && xn <= b)) xn = 0.5f * (a + b);
    if (fabsf(xn - x) <= 2e-7f * fabsf(xn)) { x = xn; break; }
    x = xn;
  }
  return x;
}

// Binary32 analysis of the stationarity quartic: the local minima of the cost
// inside (0, tmax) (at most two) and whether the cost still decreases at
// tmax.  (0, tmax] is split at the inflection point tc of Q (Q'' = 0) and at
// the real roots of Q', so on every piece Q is monotone with fixed convexity
// and each upward sign change of Q is found by monotone Newton.
__device__ __forceinline__ int minima_f32(const QuarticF &q, float tmax, float *cand0,
                                          float *cand1, bool *tmax_cand) {
  int nc = 0;
  float a = 0.0f, qa = -3.0f * q.A0;  // left end of the current piece and Q there
  const float tc = sqrtf(q.A2 / (6.0f * q.A4));
  // Fujiwara's bound on the roots of the monic Q / A4 and Q' / (4 A4)
  // (2 max |a_k / a_n|^(1 / (n - k)), the constant term halved), with 1 %
  // margin: right-end Newton starts there instead of at tmax when that is
  // closer, on the same side of the root (checked), so it converges from the
  // same side in about half the steps.
  const float rA4 = 1.0f / q.A4;
  const float bq = 2.02f * fmaxf(sqrtf(fabsf(q.A2 * rA4)),
                                 fmaxf(cbrtf(fabsf(2.0f * q.A1 * rA4)),
                                       sqrtf(sqrtf(fabsf(1.5f * q.A0 * rA4)))));
  const float bd = 2.02f * fmaxf(sqrtf(fabsf(0.5f * q.A2 * rA4)), cbrtf(fabsf(0.25f * q.A1 * rA4)));
  auto start_q = [&](float b) {
    const float x = fminf(b, bq);
    return q.Q(x) >= 0.0f ? x : b;
  };
  auto start_d = [&](float b) {
    const float x = fminf(b, bd);
    return q.dQ(x) >= 0.0f ? x : b;
  };
  // close the piece [a, b]: an upward sign change of Q is a minimum of the cost
  auto piece = [&](float b) {
    const float qb = q.Q(b);
    if (qa < 0.0f && qb > 0.0f && nc < 2) {
      const float r = newton_f<0>(q, a, b, a >= tc ? start_q(b) : a);
      if (nc == 0) *cand0 = r; else *cand1 = r;
      ++nc;
    }
    qa = qb;
    a = b;
  };
  const float d0 = -2.0f * q.A1;  // Q'(0)
  if (tc > 0.0f && tc < tmax) {
    const float dc = q.dQ(tc);
    if (d0 > 0.0f && dc < 0.0f) piece(newton_f<1>(q, 0.0f, tc, 0.0f));
    piece(tc);
    if (dc < 0.0f && q.dQ(tmax) > 0.0f) piece(newton_f<1>(q, tc, tmax, start_d(tmax)));
  } else if (tc <= 0.0f) {
    if (d0 < 0.0f && q.dQ(tmax) > 0.0f) piece(newton_f<1>(q, 0.0f, tmax, start_d(tmax)));
  } else if (d0 > 0.0f && q.dQ(tmax) < 0.0f) {
    piece(newton_f<1>(q, 0.0f, tmax, 0.0f));
  }
  piece(tmax);
  *tmax_cand = qa < 0.0f;
  return nc;
}

// Coefficients of one pair: A0 = 12|D|^2, A1 = -12 D.S, A2 = 4(|v0|^2 +
// v0.v1 + |v1|^2), A3 = 2g(v0z - v1z) with D = p1 - p0, S = v0 + v1, in
// float-float (differences and products exact, sums to ~2^-44 of their terms'
// magnitudes), and |D|.|S| summed by magnitude.
struct PairCoefs {
  FF dd, ds, A2s, A3;  // |D|^2, D.S, A2 / 4, A3
  float abs_ds;        // sum of |D_d S_d|
};
// Products and sums whose low part is left unnormalised (up to a few u of the
// operands' magnitudes): what enters further products and sums.
__device__ __forceinline__ FF ff_mul_raw(FF x, FF y) {
  const FF p = two_prod(x.h, y.h);
  return {p.h, fmaf(x.h, y.l, fmaf(x.l, y.h, p.l))};
}
__device__ __forceinline__ FF ff_mulf_raw(FF x, float c) {
  const FF p = two_prod(x.h, c);
  return {p.h, fmaf(x.l, c, p.l)};
}
__device__ __forceinline__ FF ff_add_raw(FF x, FF y) {
  const FF s = two_sum(x.h, y.h);
  return {s.h, s.l + (x.l + y.l)};
}
// x y added to the float-float sum s: the product exact to u^2, its high part
// by TwoSum, the errors in binary32.
__device__ __forceinline__ void ff_accum(FF x, FF y, FF *s) {
  const FF p = two_prod(x.h, y.h);
  const float pl = fmaf(x.h, y.l, fmaf(x.l, y.h, p.l));
  const FF t = two_sum(s->h, p.h);
  s->h = t.h;
  s->l = s->l + (t.l + pl);
}
__device__ __forceinline__ PairCoefs make_pair_coefs(const SampleF &a, const SampleF &b) {
  PairCoefs r;
  FF D[3], S[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    D[d] = two_sum(b.p[d], -a.p[d]);
    S[d] = two_sum(a.v[d], b.v[d]);
  }
  FF dd = ff_mul_raw(D[0], D[0]), ds = ff_mul_raw(D[0], S[0]), vv = a.vv;
  r.abs_ds = fabsf(D[0].h) * fabsf(S[0].h);
#pragma unroll
  for (int d = 1; d < 3; ++d) {
    ff_accum(D[d], D[d], &dd);
    ff_accum(D[d], S[d], &ds);
    r.abs_ds = fmaf(fabsf(D[d].h), fabsf(S[d].h), r.abs_ds);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) vv = ff_add_raw(vv, two_prod(a.v[d], b.v[d]));
  r.dd = fast_two_sum(dd.h, dd.l);
  r.ds = two_sum(ds.h, ds.l);
  r.A2s = ff_add(vv, b.vv);
  r.A3 = ff_mulf(two_sum(a.v[2], -b.v[2]), 2.0f * PUMP_G);
  return r;
}

// The binary32 copies (the high parts) for bracketing and the binary64 values
// (hi + lo, one addition each) for the refinement and the cost.
struct PairQuartic {
  QuarticF f;
  Quartic q;
};

__device__ __forceinline__ PairQuartic make_pair_quartic(const PairCoefs &c) {
  const FF A0 = ff_mulf(c.dd, 12.0f), A0x3 = ff_mulf(c.dd, 36.0f);
  const FF A1 = ff_mulf(c.ds, -12.0f), A1x2 = ff_mulf(c.ds, -24.0f);
  const double g = (double)PUMP_G;
  PairQuartic r;
  r.f.A0 = A0.h;
  r.f.A1 = A1.h;
  r.f.A2 = 4.0f * c.A2s.h;
  r.f.A4 = fmaf(PUMP_G, PUMP_G, 1.0f);
  r.q.A0 = ff2d(A0);
  r.q.A1 = ff2d(A1);
  r.q.A2 = 4.0 * ff2d(c.A2s);
  r.q.A3 = ff2d(c.A3);
  r.q.A4 = 1.0 + g * g;
  r.q.A0x3 = ff2d(A0x3);
  r.q.A1x2 = ff2d(A1x2);
  return r;
}

// One Newton step from a binary32 root estimate x: the residual Q(x) in
// binary64, the slope and the step size test in binary32 (the step is ~1e-6
// of x, so a binary32 slope leaves ~1e-13 relative error).  Keeps x when the
// step is not small (a tiny slope).
__device__ __forceinline__ double refine(const PairQuartic &pq, float x) {
  const double xd = f2d_exact(x);
  const double f = pq.q.Q(xd);
  const float r = __fdividef(1.0f, pq.f.dQ(x));
  const bool ok = fabsf(d2f_rn(f) * r) <= 1e-3f * x;
  return ok ? fma(-f, f2d_exact(r), xd) : xd;
}

// Global minimiser of the cost on (0, tmax] and its cost, any pair: candidates
// from the binary32 analysis, each refined by one Newton step in binary64
// (quadratic convergence takes a ~1e-6 relative root to ~1e-12) and compared
// by their binary64 cost.  Out of line: one pair in thousands needs it
// (precise_min).
struct Minimum64 {
  double t, c;
};
__device__ __noinline__ Minimum64 precise_general(const PairCoefs pc, float tmax) {
  const PairQuartic pq = make_pair_quartic(pc);
  float cand[2] = {0.0f, 0.0f};
  bool tmax_cand = false;
  const int nc = minima_f32(pq.f, tmax, &cand[0], &cand[1], &tmax_cand);
  const bool primary_root = nc > 0;
  const double tm = f2d_exact(tmax);
  const double xr = refine(pq, primary_root ? cand[0] : tmax);
  Minimum64 m;
  m.t = primary_root ? xr : tm;
  m.c = pq.q.cost(m.t);
  if (nc > 1) {
    const double t2 = refine(pq, cand[1]);
    const double c2 = pq.q.cost(t2);
    if (c2 < m.c) { m.c = c2; m.t = t2; }
  }
  if (primary_root && tmax_cand) {
    const double c3 = pq.q.cost(tm);
    if (c3 < m.c) { m.c = c3; m.t = tm; }
  }
  return m;
}

// Whether every value within `bound` of h + l rounds to h in binary32.
__device__ __forceinline__ bool rounds_to(float h, float l, float bound) {
  const float ah = fabsf(h);
  const unsigned u = __float_as_uint(ah), e = u >> 23;
  const float room = 0.5f * fminf(__uint_as_float(u + 1u) - ah, ah - __uint_as_float(u - 1u)) - fabsf(l);
  return e >= 2u && e <= 253u && bound < 0.99f * room;
}
__device__ __forceinline__ float rcp_f32(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_f32(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The optimal time and cost, correctly rounded binary32 values (t, c) with
// the rest of the time in dt (t + dt: about 2^-44 relative).  (Pairs left to
// precise_general: from one binary64 Newton step, and where tmax is within
// binary32's noise of the root, either of the two.)
//
// In almost every pair Q has one positive root, which is then the cost's only
// minimum (c' = Q / t^4).  That is certain
//   - when A1 >= 0 (one sign change);
//   - when A1^2 < 8/3 A0 A2: if Q has a local maximum at some r > 0 (Q' = 0
//     there, 4 A4 r^3 = 2 A2 r + 2 A1), its value is -A2 r^2 / 2 - 3/2 A1 r - 3 A0
//     <= 9/8 A1^2 / A2 - 3 A0 < 0, so Q < 0 until it crosses once, past its local
//     minimum; without one Q only increases;
//   - when Q' has no zero on t > 0: |A1| >= 2/3 A2 tc with tc = sqrt(A2 / (6 A4)),
//     the inflection point of Q
// (margins of 1.5e-3 and 5e-4 in the last two, and an absolute one where the squares
// leave binary32's normal range).  The root comes from two closed-form steps (the
// biquadratic without the linear term, then with that term frozen at its root) and
// three Halley steps in binary32, up to three more while a step is large.  Any
// positive root that the steps converge to is the root; that it lies beyond tmax
// is confirmed by Q(tmax) < 0.  (With Q < 0 up to tc bounded by leaving the t^2 term
// out, and three steps for all, one pair in six went the general way where
// velocities are several times what a segment's length allows: N = 4000, velocities
// up to 3 over a unit cube, 0.815 ms, 0.391 so, 0.765 with every pair in binary64.)
//
// Then one Newton step with the residual Q(x) in float-float gives dx, and the
// cost at the root is c(x) + c'(x) dx / 2 (c' vanishes at the root; third
// order), c(x) in float-float.  Errors, u = 2^-24, as multiples of the terms'
// magnitudes: the coefficients at most 36 u^2, 1/x 6 u^2 a factor, each product
// 6 u^2 and sum 8 u^2, and 6 u^2 more an operation for the low parts left
// unnormalised between them: under 190 u^2 for the cost, 140 u^2 for Q.  The
// bounds take 2^-40 (256 u^2).  Where a bound reaches a rounding boundary (about 1e-4
// of pairs) and wherever a condition fails, precise_general decides.
//
// Why float-float: the binary64 pipe runs at 1/64 of the binary32 rate here,
// so the 18 binary64 instructions a pair that the refinement and the cost used
// to take bounded the pair kernel at 0.54 ms for N = 4000, and their
// conversions and the bracketing filled the rest of the issue slots.
struct PreciseMin {
  float t, dt, c;
};
__device__ __forceinline__ PreciseMin precise_min(const SampleF &sa, const SampleF &sb, float tmax) {
  const PairCoefs pc = make_pair_coefs(sa, sb);
  constexpr double kA4d = 1.0 + (double)PUMP_G * (double)PUMP_G;
  constexpr float kA4 = (float)kA4d, kA4l = (float)(kA4d - (double)kA4), kR4 = (float)(1.0 / kA4d);
  // Q / A4 = t^4 - a t^2 - b t - c
  const float a = pc.A2s.h * (4.0f * kR4), b = pc.ds.h * (-24.0f * kR4), c = pc.dd.h * (36.0f * kR4);
  const bool unique = b >= 0.0f || b * b < fmaf(3.55f * a, c, -1e-36f) ||
                      -b >= 1.334f * a * sqrt_f32(a * (1.0f / 6.0f));
  const float aa = a * a;
  const float t0 = sqrt_f32(0.5f * (a + sqrt_f32(fmaf(4.0f, c, aa))));
  const float t1 = 0.5f * (a + sqrt_f32(fmaxf(fmaf(4.0f, fmaf(b, t0, c), aa), c)));
  float x = sqrt_f32(t1), step = 0.0f;
  auto halley = [&] {
    const float x2 = x * x;
    const float q = fmaf(fmaf(x2 - a, x, -b), x, -c);
    const float dq = fmaf(fmaf(4.0f, x2, -2.0f * a), x, -b);
    const float r = rcp_f32(dq);
    const float s = q * r;
    // Halley: s / (1 - s q'' / (2 q')), the quotient by its own estimate
    step = s * rcp_f32(fmaf(-s * r, fmaf(6.0f, x2, -a), 1.0f));
    x = x - step;
  };
#pragma unroll
  for (int it = 0; it < 3; ++it) halley();
  for (int it = 0; it < 3 && unique && fabsf(step) > 2e-3f * x; ++it) halley();
  bool ok = unique && fabsf(step) <= 2e-3f * x && x >= 1e-6f && x <= 1e6f;
  const bool beyond = x > tmax * 1.00001f;  // the cost still falls at tmax (Q < 0 there, tested below)
  x = fminf(x, tmax);
  // Q(x), the Newton step and its error
  const FF x2 = two_prod(x, x);
  const FF A2 = {4.0f * pc.A2s.h, 4.0f * pc.A2s.l};
  FF q = ff_mul_raw({kA4, kA4l}, x2);
  const float dq = fmaf(fmaf(4.0f, q.h, -2.0f * A2.h), x, 24.0f * pc.ds.h);
  const float ddq = fmaf(12.0f, q.h, 2.0f * A2.h) * 1.01f;  // (over its magnitude)
  const float mq = fmaf(fmaf(q.h + 3.0f * A2.h, x, 24.0f * pc.abs_ds), x, 36.0f * pc.dd.h);
  q = ff_mulf_raw(ff_add_raw(q, {-A2.h, -A2.l}), x);
  q = ff_mulf_raw(ff_add_raw(q, ff_mulf_raw(pc.ds, 24.0f)), x);
  q = ff_add_raw(q, ff_mulf_raw(pc.dd, -36.0f));
  const float qv = q.h + q.l;
  const float r = rcp_f32(x);
  const float rq = rcp_f32(dq);
  float dx = -(qv * rq);
  if (x >= tmax) dx = beyond ? 0.0f : fminf(dx, 0.0f);
  const float bt = beyond ? 0.0f
                          : fabsf(rq) * fmaf(fabsf(dx), fmaf(mq * r, 0x1p-18f, fabsf(dx) * ddq), mq * 0x1p-40f);
  ok = ok && fabsf(dx) <= 0x1p-18f * x && (beyond ? qv < -(mq * 0x1p-40f) : dq > 0.0f);
  // c(x) = A3 + A4 x + r (A2 + r (A1 + r A0)), 1/x in float-float
  const FF rr = {r, r * fmaf(-x, r, 1.0f)};
  FF v = ff_add_raw(ff_mul_raw(ff_mulf_raw(pc.dd, 12.0f), rr), ff_mulf_raw(pc.ds, -12.0f));
  v = ff_add_raw(ff_mul_raw(v, rr), A2);
  v = ff_add_raw(ff_mul_raw(v, rr), pc.A3);
  v = ff_add_raw(v, ff_mulf_raw({kA4, kA4l}, x));
  const float r2 = r * r;
  const float mc = fmaf(r, fmaf(r, fmaf(r, 12.0f * pc.dd.h, 12.0f * pc.abs_ds), 3.0f * A2.h),
                        fmaf(kA4, x, fabsf(pc.A3.h)));
  v = two_sum(v.h, fmaf(qv * r2 * r2, beyond ? 0.0f : 0.5f * dx, v.l));
  PreciseMin m;
  const FF t = fast_two_sum(x, dx);
  m.t = t.h;
  m.dt = t.l;
  m.c = v.h;
  ok = ok && rounds_to(t.h, t.l, bt) && rounds_to(v.h, v.l, mc * 0x1p-40f);
  if (!ok) {
    const Minimum64 g = precise_general(pc, tmax);
    m.t = d2f_rn(g.t);
    m.dt = (float)(g.t - (double)m.t);
    m.c = d2f_rn(g.c);
  }
  return m;
}

}  // namespace
}  // namespace pump
