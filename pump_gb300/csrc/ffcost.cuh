// Binary32 costs of the reference's 2pBVP cost expression from float-float
// arithmetic, certified against the binary64 evaluation (bvp.cu for the
// reference built for the CPU, bvp_refgpu.cu for its GPU kernel).
//
// The same bound holds for the reference's GPU kernel (bvp_refgpu.cu): there
// nvcc may fuse any of its binary64 multiply-adds (a fused operation rounds
// once, within the same 2^-53 of its result), and CUDA's pow, which the
// expression calls for tau^2, tau^3, tau^4 and the coordinates' squares, is
// within 2 ulp (2^-51) of the power, so the terms' magnitudes times 2^-50
// cover it (2^-46.9 with the roundings, inside the 2^-41 below).  Its one
// binary32 multiply-add, b + c tau in the last two terms, is written here as
// the reference writes it, and bvp_refgpu.cu is compiled with contraction as
// the reference is; the GPU tests compare every pair with the reference
// kernel's own results.
#pragma once
#include "common.cuh"

namespace pump {
namespace {

// cost_eval rounds 25 binary64 additions and about 15 binary64 products, and
// the GB300 executes binary64 at 1/64 of its binary32 rate, so the bit-exact
// kernels would be bound by that pipe.  cost_ff gets the same binary32 result
// from binary32 arithmetic in almost every evaluation: it evaluates the
// bracket sum V (the same terms; the t^2, t^3 and t^4 coefficients summed per
// pair) and V / t^3 in float-float arithmetic (Dekker's and Knuth's
// error-free TwoSum and TwoProduct; double-float operations as in Bailey's
// double-double library, with binary32 parts), and bounds the distance of
// cost_eval's binary64 value from it (u = 2^-24):
//   - cost_eval's sum: each of its 31 additions (s7's six included) and ~15
//     products is rounded once (|error| <= 2^-53 of the partial sum or
//     product; t^3 and t^4 are themselves rounded products), so its error is
//     at most 2^-52 x 33 x (the sum of the terms' magnitudes), about
//     2.1 u^2 of that sum (the reference's GPU kernel: as much, see above);
//   - sums of n terms by TwoSum, whose errors (each at most u of the running
//     sum, itself at most the magnitudes' sum) are added in binary32: at most
//     n (n + 1) / 2 u^2 (with the squares' own low parts, each at most u of
//     its square, one rounding more per term).  The six squares of s7 and of
//     the t^2 coefficient (make_pair_ff): 36 u^2, with the product by 12 and
//     the binary32 products' sums 6 u^2 more; s7's high part and the ten
//     rounded terms: 66 u^2, and 11 u^2 for the errors' sum in the closing fast
//     sum: at most 119 u^2;
//   - the t^2, t^3 and t^4 terms by Horner's rule: two products by t (3 u^2
//     each), two fast sums (8 u^2 each), the product by t^2 (6 u^2), and the
//     t^2 coefficient's own 42 u^2: at most 70 u^2; the last fast sum 8 u^2;
//   - together at most 129 u^2 of the magnitudes' sum; the bound takes
//     2^-40 x 1.01 (258 u^2);
//   - the quotient by t^3 (t^3 to 5 u^2; a reciprocal estimate within 2 u;
//     one residual step: 4 + 12 + 24 u^2) and cost_eval's three binary64
//     roundings: at most 46 u^2; the bound takes 2^-42 (64 u^2) of the
//     result.
// When that interval around the float-float value lies inside the binary32
// rounding cell of its high part (it does not reach the midpoint to either
// neighbour), cost_eval's (float) conversion gives that high part, which is
// returned.  Otherwise (and for tau outside [1e-4, 1e4], or a non-finite or
// subnormal result) the binary64 evaluation runs.  The binary32 terms that
// the reference rounds are products written as __fmul_rn, which no compiler
// fuses into the sums that follow (bvp_refgpu.cu is compiled with
// contraction, and a product with a single use would otherwise become a
// multiply-add); every other product calls fmaf explicitly or is only a
// bound.
struct FF {
  float hi, lo;
};
__device__ __forceinline__ FF ff_two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ FF ff_fast_two_sum(float a, float b) {  // |a| >= |b| or a == 0
  const float s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ FF ff_two_prod(float a, float b) {
  const float p = a * b;
  return {p, fmaf(a, b, -p)};
}
__device__ __forceinline__ FF ff_add(FF x, FF y) {
  FF s = ff_two_sum(x.hi, y.hi);
  const FF t = ff_two_sum(x.lo, y.lo);
  s.lo = s.lo + t.hi;
  s = ff_fast_two_sum(s.hi, s.lo);
  s.lo = s.lo + t.lo;
  return ff_fast_two_sum(s.hi, s.lo);
}
// Double-word sum without the second TwoSum ("sloppy" addition): its error
// is at most about 8 u^2 (|x| + |y|), u = 2^-24, also under cancellation,
// which is all cost_ff's bound (taken over the terms' magnitudes) needs.
__device__ __forceinline__ FF ff_add_fast(FF x, FF y) {
  FF s = ff_two_sum(x.hi, y.hi);
  s.lo = s.lo + (x.lo + y.lo);
  return ff_fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ FF ff_add_f(FF x, float b) {
  FF s = ff_two_sum(x.hi, b);
  s.lo = s.lo + x.lo;
  return ff_fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ FF ff_mul(FF x, FF y) {
  FF p = ff_two_prod(x.hi, y.hi);
  p.lo = fmaf(x.hi, y.lo, fmaf(x.lo, y.hi, p.lo));
  return ff_fast_two_sum(p.hi, p.lo);
}
__device__ __forceinline__ FF ff_mul_f(FF x, float b) {
  FF p = ff_two_prod(x.hi, b);
  p.lo = fmaf(x.lo, b, p.lo);
  return ff_fast_two_sum(p.hi, p.lo);
}
// Products that only enter a sum, left unnormalised (the low part up to 4 u
// of the high part).
__device__ __forceinline__ FF ff_term(FF x, FF y) {
  FF p = ff_two_prod(x.hi, y.hi);
  p.lo = fmaf(x.hi, y.lo, fmaf(x.lo, y.hi, p.lo));
  return p;
}
__device__ __forceinline__ FF ff_term_f(FF x, float b) {
  FF p = ff_two_prod(x.hi, b);
  p.lo = fmaf(x.lo, b, p.lo);
  return p;
}
// Reciprocal estimate (one instruction, within 1 ulp).
__device__ __forceinline__ float ff_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Per-pair data of cost_ff, built without binary64 arithmetic (the GB300's
// binary64 conversions and products would cost the pair kernel a quarter of
// its time): the binary32 coefficients of cost_eval's t-linear and last two
// terms; s7 and the t^2 coefficient as float-float sums of exact squares and
// of the binary32 products cost_eval converts, the t^3 coefficient as an exact
// difference; and the sums of their terms' magnitudes.  cost_eval's own s7
// differs from the exact sum by its six binary64 roundings, which cost_ff's
// bound covers.
struct PairFF {
  float k8, k9, k10, k11, k12, k13, k14, k15;
  float a29, b29, c29, a30, b30, c30;
  FF s7, d2, d3;
  float abs_s7, abs_d2, abs_d3;
  float abs_k;  // |k8| + ... + |k15| (times tau: the t-linear terms' magnitudes)
  // magnitudes of the tau-free and the t-linear terms, the two parts of the
  // last two terms counted separately (cost_delta)
  float mag0, mag1;
};
// x^2 added to the running float-float sum (hi, lo): the square exact as a
// TwoProduct, its high part by TwoSum, the errors added in binary32.
__device__ __forceinline__ void ff_add_sq(float x, float *hi, float *lo) {
  const FF p = ff_two_prod(x, x);
  const FF s = ff_two_sum(*hi, p.hi);
  *hi = s.hi;
  *lo = *lo + (s.lo + p.lo);
}
__device__ __forceinline__ PairFF make_pair_ff(const float *x0, const float *x1) {
  const float g = PUMP_G;
  PairFF f;
  // the binary32 terms, as make_coef computes them
  f.k8 = 12 * x0[4] * x0[1];
  f.k9 = 12 * x0[1] * x1[4];
  f.k10 = 12 * x0[3] * x1[0];
  f.k11 = 12 * x1[3] * x1[0];
  f.k12 = 12 * x0[5] * x1[2];
  f.k13 = 12 * x1[5] * x1[2];
  f.k14 = 12 * x0[4] * x1[1];
  f.k15 = 12 * x1[4] * x1[1];
  f.abs_k = ((fabsf(f.k8) + fabsf(f.k9)) + (fabsf(f.k10) + fabsf(f.k11))) +
            ((fabsf(f.k12) + fabsf(f.k13)) + (fabsf(f.k14) + fabsf(f.k15)));
  f.a29 = 12 * x0[0];
  f.b29 = -2 * x1[0];
  f.c29 = x0[3] + x1[3];
  f.a30 = 12 * x0[2];
  f.b30 = -2 * x1[2];
  f.c30 = x0[5] + x1[5];
  f.mag1 = f.abs_k + fabsf(f.a29 * f.c29) + fabsf(f.a30 * f.c30);
  // s7, make_coef's first seven terms: 12 times the sum of six squares, less
  // the binary32 product
  {
    FF s = ff_two_prod(x0[0], x0[0]);
    ff_add_sq(x0[2], &s.hi, &s.lo);
    ff_add_sq(x0[1], &s.hi, &s.lo);
    ff_add_sq(x1[0], &s.hi, &s.lo);
    ff_add_sq(x1[2], &s.hi, &s.lo);
    ff_add_sq(x1[1], &s.hi, &s.lo);
    s = ff_mul_f(ff_fast_two_sum(s.hi, s.lo), 12.0f);
    const float c24 = __fmul_rn(24 * x0[1], x1[1]);
    f.abs_s7 = s.hi + fabsf(c24);
    f.s7 = ff_add_f(s, -c24);
  }
  f.mag0 = f.abs_s7 + fabsf(f.a29 * f.b29) + fabsf(f.a30 * f.b30);
  // the t^2 coefficient: 4 times the sum of six squares (exact as a scaling)
  // and three binary32 products
  {
    FF s = ff_two_prod(x0[4], x0[4]);
    ff_add_sq(x0[3], &s.hi, &s.lo);
    ff_add_sq(x0[5], &s.hi, &s.lo);
    ff_add_sq(x1[4], &s.hi, &s.lo);
    ff_add_sq(x1[3], &s.hi, &s.lo);
    ff_add_sq(x1[5], &s.hi, &s.lo);
    s = ff_fast_two_sum(4.0f * s.hi, 4.0f * s.lo);
    const float fl[3] = {__fmul_rn(4 * x0[4], x1[4]), __fmul_rn(4 * x0[3], x1[3]),
                         __fmul_rn(4 * x0[5], x1[5])};
    f.abs_d2 = s.hi + (fabsf(fl[0]) + fabsf(fl[1]) + fabsf(fl[2]));
#pragma unroll
    for (int q = 0; q < 3; ++q) s = ff_add_f(s, fl[q]);
    f.d2 = s;
  }
  const float f25 = __fmul_rn(2 * g, x0[5]), f26 = __fmul_rn(2 * g, x1[5]);
  f.d3 = ff_two_sum(f25, -f26);
  f.abs_d3 = fabsf(f25) + fabsf(f26);
  return f;
}

// cost(tau) as a float-float value w and a bound on the distance of
// cost_eval's binary64 value from it; false when tau is out of range.
struct CostFF {
  FF w;
  float bound;
};
__device__ __forceinline__ bool cost_ff_value(const PairFF &f, float tau, CostFF *out) {
  // the float terms, as cost_eval rounds them; b + c tau as the reference
  // writes it (contracted where the reference's build contracts it), the
  // outer product rounded (the reference converts it to binary64 before
  // adding it)
  const float a29 = __fmul_rn(f.a29, f.b29 + f.c29 * tau);
  const float a30 = __fmul_rn(f.a30, f.b30 + f.c30 * tau);
  const float k[10] = {__fmul_rn(f.k8, tau),   __fmul_rn(f.k9, tau),   -__fmul_rn(f.k10, tau),
                       -__fmul_rn(f.k11, tau), -__fmul_rn(f.k12, tau), -__fmul_rn(f.k13, tau),
                       -__fmul_rn(f.k14, tau), -__fmul_rn(f.k15, tau), a29, a30};
  float sum = f.s7.hi, err = f.s7.lo;
#pragma unroll
  for (int q = 0; q < 10; ++q) {
    const FF s = ff_two_sum(sum, k[q]);
    sum = s.hi;
    err = err + s.lo;
  }
  const FF t2 = ff_two_prod(tau, tau);
  const FF t3 = ff_mul_f(t2, tau);
  // 1 + g^2, the t^4 coefficient (g^2 exact as a TwoProduct)
  const float g = PUMP_G;
  const FF d4 = ff_add_f(ff_two_prod(g, g), 1.0f);
  FF h = ff_add_fast(ff_term_f(d4, tau), f.d3);
  h = ff_add_fast(ff_term_f(h, tau), f.d2);
  const FF v = ff_add_fast({sum, err}, ff_term(h, t2));
  // |k[q]| = |k_q| tau to within 2^-24 of each, and abs_k is the sum of the
  // |k_q| to within 2^-21: inside the bound's 1 % margin
  const float mag = fmaf(fmaf(fmaf(d4.hi, tau, f.abs_d3), tau, f.abs_d2), t2.hi,
                         fmaf(f.abs_k, tau, f.abs_s7 + fabsf(a29) + fabsf(a30)));
  // v / t3: an estimate q1 and one residual step
  const float rc = ff_rcp(t3.hi);
  const float q1 = v.hi * rc;
  const float res = fmaf(-q1, t3.hi, v.hi) + fmaf(-q1, t3.lo, v.lo);
  out->w = ff_fast_two_sum(q1, res * rc);
  // (margins for the binary32 evaluation of the bound itself)
  out->bound = fmaf(mag * 1.01f * 0x1p-40f, rc, fabsf(out->w.hi) * 0x1p-42f);
  return tau >= 1e-4f && tau <= 1e4f;
}

// The binary32 rounding of every value within `bound` of w (true), or false
// when the interval reaches a rounding boundary or leaves the normal range.
__device__ __forceinline__ bool ff_round(FF w, float bound, float *out) {
  const float aw = fabsf(w.hi);
  const unsigned int u = __float_as_uint(aw);
  const unsigned int e = u >> 23;
  *out = w.hi;
  if (e < 2u || e > 253u) return false;  // zero, subnormal, huge, inf, NaN
  const float ulp_up = __uint_as_float(u + 1u) - aw, ulp_dn = aw - __uint_as_float(u - 1u);
  const float room = 0.5f * fminf(ulp_up, ulp_dn) - fabsf(w.lo);
  return bound < 0.99f * room;
}

// The certified value, or *ok = false (then cost_eval gives the result).
__device__ __forceinline__ float cost_ff(const PairFF &f, float tau, bool *ok) {
  CostFF c;
  float v;
  const bool in = cost_ff_value(f, tau, &c);
  *ok = ff_round(c.w, c.bound, &v) && in;
  return v;
}

// The sign of the finite difference at topt from the cost's derivative, in
// about 45 binary32 instructions.  The cost as a function of tau is F(t) =
// C0/t^3 + C1/t^2 + d2/t + d3 + d4 t, with C0 and C1 gathered from the tau-free
// and t-linear terms.  cost_eval's binary64 value differs from F by the
// roundings of its binary32 terms, at most u (n0 + n1 t) / t^3 (a product k t
// one rounding, the last two terms three: n0, n1), and by its own binary64
// roundings, under 2.1 u^2 of the terms' magnitudes.  Over the d = ta - tb
// (about 1e-6) between the two points F changes by d F'(x), x between them,
// and F' by at most 4.1 d / t of M = (3 mag0 / t + 2 mag1) / t + |d2|) / t^2 + d4,
// the magnitudes' sum of F'; F' itself is evaluated to 20 u M (its
// coefficients are binary32 sums of at most 14 terms).
struct PairSlope {
  float C0, C1, d2, d3;
  float mag0, mag1, abs_d2, abs_d3;
  float n0, n1;
};
__device__ __forceinline__ PairSlope make_slope(const PairFF &f) {
  PairSlope s;
  const float p29 = f.a29 * f.b29, p30 = f.a30 * f.b30, q29 = f.a29 * f.c29, q30 = f.a30 * f.c30;
  s.C0 = f.s7.hi + (p29 + p30);
  s.C1 = ((f.k8 + f.k9) + (q29 + q30)) - (((f.k10 + f.k11) + (f.k12 + f.k13)) + (f.k14 + f.k15));
  s.d2 = f.d2.hi;
  s.d3 = f.d3.hi;
  s.mag0 = f.mag0;
  s.mag1 = f.mag1;
  s.abs_d2 = f.abs_d2;
  s.abs_d3 = f.abs_d3;
  s.n0 = 3.1f * (fabsf(p29) + fabsf(p30));
  s.n1 = 3.1f * (fabsf(q29) + fabsf(q30)) + f.abs_k;
  return s;
}
// True when the finite difference between tb and ta is certain to be nonzero
// with more than `least` between the two binary32 costs; *sign its sign.
__device__ __forceinline__ bool slope_sign(const PairSlope &s, float ta, float tb, float least,
                                           int *sign) {
  const float u = 0x1p-24f;
  const float d4 = (float)(1.0 + (double)PUMP_G * (double)PUMP_G);
  const float d = ta - tb, r = ff_rcp(tb), r2 = r * r;
  const float slope = fmaf(-r2, fmaf(fmaf(3.0f * s.C0, r, 2.0f * s.C1), r, s.d2), d4);
  const float M = fmaf(r2, fmaf(fmaf(3.0f * s.mag0, r, 2.0f * s.mag1), r, s.abs_d2), d4);
  const float c = fmaf(d4, tb, fmaf(fmaf(fmaf(s.C0, r, s.C1), r, s.d2), r, s.d3));
  const float dv = fabsf(slope) * d;
  // binary32's spacing at the larger cost (F to 20 u of M t + |d3|)
  const float top = fabsf(c) + (fmaf(M, tb, s.abs_d3) * 0x1p-18f + dv);
  const float ulp = __uint_as_float(__float_as_uint(top) & 0x7f800000u) * 0x1p-23f;
  const float noise = fmaf(s.n0, r, s.n1) * r2 * (2.04f * u);
  const float err = M * fmaf(d, fmaf(4.3f * d, r, 24.0f * u), tb * 0x1p-45f);
  *sign = slope > 0.0f ? 1 : -1;
  return tb >= 1e-4f && ta <= 1e4f && d > 0.0f && d <= 2e-3f * tb &&
         dv > (ulp + noise + err) * 1.001f + least;
}

// The difference V(ta) - V(tb) of cost_eval's binary64 values at two nearby
// points ta > tb (the two sides of the reference's finite difference,
// 2pBVP.cu:109-115, about 1e-6 apart), from binary32 arithmetic, without
// evaluating either: *dv and a bound *err on its distance from the true
// difference; *ulp: at least the spacing of binary32 at either value.
// False when the points are out of range (*dv unspecified).
//
// With s(t) the bracket and V = s / t^3, V(ta) - V(tb) =
// (s(ta) - s(tb) - V(tb) (ta^3 - tb^3)) / ta^3.  The differences of the
// rounded binary32 terms are taken term by term (neighbouring binary32
// values: exact but for the last two terms' possible sign change, u of the
// difference), the polynomial's in factored form, d = ta - tb exact.  With
// mag the sum of the terms' magnitudes at tb (the last two terms' two parts
// counted separately) and d <= 2e-3 tb, the errors, as multiples of u mag:
//   - the term differences: the ten differences' sum, 10 (d/t + 6 u) (a
//     rounded term moves by its slope and by up to 6 u of its magnitude);
//   - the polynomial: 9 roundings of 4 d/t;  adding the two: 5 d/t;
//   - V(tb) to 26 u of mag / t^3 (a 14-term binary32 sum and the reciprocal),
//     times 3 d/t: 78 d/t;  its product: 18 d/t;  the subtraction: 8 d/t;
//   - 1 / ta^3 to 8 u, of a difference of at most 8 d/t mag: 64 d/t;
//   - the two binary64 evaluations' own errors: 5 u.
// Altogether at most 220 u d/t + 65 u^2 of mag / t^3; *err takes 256 u d/t +
// 128 u^2.
__device__ __forceinline__ bool cost_delta(const PairFF &f, float ta, float tb, float *dv,
                                           float *err, float *ulp) {
  const float d = ta - tb;
  const float a29 = __fmul_rn(f.a29, f.b29 + f.c29 * tb), a30 = __fmul_rn(f.a30, f.b30 + f.c30 * tb);
  const float b29 = __fmul_rn(f.a29, f.b29 + f.c29 * ta), b30 = __fmul_rn(f.a30, f.b30 + f.c30 * ta);
  const float kb[8] = {__fmul_rn(f.k8, tb),  __fmul_rn(f.k9, tb),  __fmul_rn(f.k10, tb),
                       __fmul_rn(f.k11, tb), __fmul_rn(f.k12, tb), __fmul_rn(f.k13, tb),
                       __fmul_rn(f.k14, tb), __fmul_rn(f.k15, tb)};
  const float ka[8] = {__fmul_rn(f.k8, ta),  __fmul_rn(f.k9, ta),  __fmul_rn(f.k10, ta),
                       __fmul_rn(f.k11, ta), __fmul_rn(f.k12, ta), __fmul_rn(f.k13, ta),
                       __fmul_rn(f.k14, ta), __fmul_rn(f.k15, ta)};
  const float dk = (((ka[0] - kb[0]) + (ka[1] - kb[1])) + ((b29 - a29) + (b30 - a30))) -
                   (((ka[2] - kb[2]) + (ka[3] - kb[3])) +
                    (((ka[4] - kb[4]) + (ka[5] - kb[5])) + ((ka[6] - kb[6]) + (ka[7] - kb[7]))));
  const float sk = ((f.s7.hi + (kb[0] + kb[1])) + (a29 + a30)) -
                   ((kb[2] + kb[3]) + ((kb[4] + kb[5]) + (kb[6] + kb[7])));
  const float d4 = (float)(1.0 + (double)PUMP_G * (double)PUMP_G);
  const float rb = ff_rcp(tb), ra = ff_rcp(ta);
  const float tb2 = tb * tb, sum = ta + tb;
  const float q = fmaf(ta, sum, tb2);                 // (ta^3 - tb^3) / d
  const float p4 = sum * fmaf(ta, ta, tb2);           // (ta^4 - tb^4) / d
  const float ds = fmaf(d, fmaf(f.d2.hi, sum, fmaf(f.d3.hi, q, d4 * p4)), dk);
  const float rb3 = rb * rb * rb;
  const float vb = fmaf(tb2, fmaf(tb, fmaf(tb, d4, f.d3.hi), f.d2.hi), sk) * rb3;
  *dv = fmaf(-vb, d * q, ds) * (ra * ra * ra);
  const float mag = fmaf(tb, fmaf(tb, fmaf(tb, fmaf(tb, d4, f.abs_d3), f.abs_d2), f.mag1), f.mag0) * rb3;
  *err = mag * fmaf(0x1p-16f * d, rb, 0x1p-41f) * 1.01f;
  // V(tb) is within 26 u of mag / t^3 of vb, V(ta) a further |dv| + *err away
  const float top = fabsf(vb) + (fabsf(*dv) + mag * 0x1p-18f);
  *ulp = __uint_as_float(__float_as_uint(top) & 0x7f800000u) * 0x1p-23f;
  return tb >= 1e-4f && ta <= 1e4f && d > 0.0f && d <= 2e-3f * tb;
}

}  // namespace
}  // namespace pump
