// Pair BVPs in the arithmetic of the reference's own GPU kernel
// (fillCoptsTopts, 2pBVP.cu:133-150, with toptBisection :71-95, dcost
// :109-115 and cost :97-107, compiled by nvcc as the reference's Makefile
// compiles it).
//
// Two things make that arithmetic differ from the rounded-once parity
// arithmetic of bvp.cu: nvcc contracts multiply-adds by default, at sites of
// its own choosing, and in device code pow(float, int) promotes to CUDA's
// binary64 pow(double, double), which is not correctly rounded (on the
// GB300 pow(double(x), 2) differs from the exact square for about 6 % of
// binary32 x, pow(x, 3) and pow(x, 4) from the correctly rounded power for
// about 25 %).  Neither can be restated operation by operation, so this
// translation unit is compiled with contraction on, as the reference is,
// calls pow where the reference calls it, and writes the cost as the
// reference's expression with the same operands, types and order, so that
// the compiler sees the same expression tree.  The twelve pow(coordinate, 2)
// terms do not depend on tau and are evaluated once per pair; the tree the
// compiler contracts is unchanged (those leaves are pow results either way).
// A GPU test compares all N(N-1) pairs at N = 1000 and 4000 with the
// reference's fillCoptsTopts run on the GB300 (SHA-256 of both arrays).
//
// The kernel walks the pairs as the parity kernel does (bisect.cuh), which
// changes the order of work, not any pair's arithmetic: almost every
// comparison and cost is certified from binary32 arithmetic (ffcost.cuh).
// What is left first tries a binary64 evaluation with its own bound, and only
// then CUDA's pow: one evaluation of the expression with pow takes tens of
// microseconds, as long as a warp's other work on a chunk of pairs.
#include <math.h>

#include "common.cuh"
#include "ctx.h"
#include "bisect.cuh"
#include "ffcost.cuh"

namespace pump {
namespace {

// the reference's `const float g = -9.81;` (2pBVP.cu:3)
const float kGRef = -9.81;

// pow(coordinate, 2) of both states: the tau-independent pow calls of cost
struct CoordPow {
  double a0, a1, a2, a3, a4, a5, b0, b1, b2, b3, b4, b5;
};
__device__ __forceinline__ CoordPow coord_pow(const float *a, const float *b) {
  CoordPow p;
  p.a0 = pow(a[0], 2); p.a1 = pow(a[1], 2); p.a2 = pow(a[2], 2);
  p.a3 = pow(a[3], 2); p.a4 = pow(a[4], 2); p.a5 = pow(a[5], 2);
  p.b0 = pow(b[0], 2); p.b1 = pow(b[1], 2); p.b2 = pow(b[2], 2);
  p.b3 = pow(b[3], 2); p.b4 = pow(b[4], 2); p.b5 = pow(b[5], 2);
  return p;
}

// cost, 2pBVP.cu:97-107: the same expression (a = x0, b = x1, p.aK and p.bK
// for pow(x0[K], 2) and pow(x1[K], 2))
__device__ __forceinline__ float cost_dev(float tau, const float *a, const float *b, const CoordPow &p) {
  const float g = kGRef;
  float c = (1/pow(tau,3))*(12*p.a0 + 12*p.a2 + 12*p.a1 + 12*p.b0 + 12*p.b2 - 24*a[1]*b[1] +
      12*p.b1 + 12*a[4]*a[1]*tau + 12*a[1]*b[4]*tau - 12*a[3]*b[0]*tau - 12*b[3]*b[0]*tau -
      12*a[5]*b[2]*tau - 12*b[5]*b[2]*tau - 12*a[4]*b[1]*tau - 12*b[4]*b[1]*tau + 4*p.a4*pow(tau,2) +
      4*p.a3*pow(tau,2) + 4*p.a5*pow(tau,2) + 4*a[4]*b[4]*pow(tau,2) + 4*p.b4*pow(tau,2) + 4*a[3]*b[3]*pow(tau,2) +
      4*p.b3*pow(tau,2) + 4*a[5]*b[5]*pow(tau,2) + 4*p.b5*pow(tau,2) + 2*g*a[5]*pow(tau,3) - 2*g*b[5]*pow(tau,3) + pow(tau,4) +
      pow(g,2)*pow(tau,4) + 12*a[0]*(-2*b[0] + (a[3] + b[3])*tau) + 12*a[2]*(-2*b[2] + (a[5] + b[5])*tau));
  return c;
}

// The reference kernel's cost of the pair at tau, out of line (the registers
// of the binary64 powers do not count against the pair kernel's occupancy).
//
// Its binary64 value lies within 2^-46.9 of the terms' magnitudes (over t^3)
// of the exact sum of its rounded binary32 terms (ffcost.cuh); the same sum
// with correctly rounded powers, here, within 2^-47 of them.  When every
// value within 2^-45 of them of the latter converts to the same binary32,
// that is the result; otherwise the expression is evaluated with pow, as the
// reference kernel does.
struct RefGpuCost {
  struct States {
    float a[kDim], b[kDim];
  };
  // the bounded evaluation: NaN where it leaves the value open
  static __device__ __noinline__ float bounded(const States st, float tau) {
    if (!(tau >= 1e-4f && tau <= 1e4f)) return NAN;
    const PairFF f = make_pair_ff(st.a, st.b);
    const float a29 = __fmul_rn(f.a29, f.b29 + f.c29 * tau);
    const float a30 = __fmul_rn(f.a30, f.b30 + f.c30 * tau);
    const double t = tau, t2 = t * t, t3 = t2 * t;
    const float *x = st.a, *y = st.b;
    const double s7 = 12 * (p2f(x[0]) + p2f(x[2]) + p2f(x[1]) + p2f(y[0]) + p2f(y[2]) + p2f(y[1])) -
                      (double)(__fmul_rn(24 * x[1], y[1]));
    const double d2 = 4 * (p2f(x[4]) + p2f(x[3]) + p2f(x[5]) + p2f(y[4]) + p2f(y[3]) + p2f(y[5])) +
                      ((double)__fmul_rn(4 * x[4], y[4]) + (double)__fmul_rn(4 * x[3], y[3]) +
                       (double)__fmul_rn(4 * x[5], y[5]));
    const double d3 = (double)f.d3.hi + (double)f.d3.lo;
    const double d4 = 1.0 + (double)kGRef * (double)kGRef;
    const double k = ((double)__fmul_rn(f.k8, tau) + (double)__fmul_rn(f.k9, tau)) -
                     ((double)__fmul_rn(f.k10, tau) + (double)__fmul_rn(f.k11, tau)) -
                     ((double)__fmul_rn(f.k12, tau) + (double)__fmul_rn(f.k13, tau)) -
                     ((double)__fmul_rn(f.k14, tau) + (double)__fmul_rn(f.k15, tau));
    const double v = ((s7 + k) + ((double)a29 + (double)a30) + ((d4 * t + d3) * t + d2) * t2) / t3;
    const float mag = f.abs_s7 + f.abs_k * tau + fabsf(a29) + fabsf(a30) +
                      ((((float)d4) * tau + f.abs_d3) * tau + f.abs_d2) * tau * tau;
    const double B = (double)mag * 0x1p-45 / t3 + fabs(v) * 0x1p-50;
    const float lo = (float)(v - B), hi = (float)(v + B);
    return lo == hi && fabsf(lo) > 1e-30f && fabsf(lo) < 1e30f ? lo : NAN;
  }
  // the expression at ta and tb; the coordinates' powers, 12 of its 15, are shared
  struct Costs {
    float ca, cb;
  };
  static __device__ __noinline__ Costs powers(const States st, float ta, float tb, bool want_a, bool want_b) {
    const CoordPow p = coord_pow(st.a, st.b);
    Costs r{0.0f, 0.0f};
    if (want_a) r.ca = cost_dev(ta, st.a, st.b, p);
    if (want_b) r.cb = cost_dev(tb, st.a, st.b, p);
    return r;
  }
  static __device__ __forceinline__ void costs(const float *x0, const float *x1, float ta, float tb,
                                               bool want_a, bool want_b, float *ca, float *cb) {
    States st;
#pragma unroll
    for (int d = 0; d < kDim; ++d) {
      st.a[d] = x0[d];
      st.b[d] = x1[d];
    }
    if (want_a) {
      const float v = bounded(st, ta);
      if (v == v) *ca = v, want_a = false;
    }
    if (want_b) {
      const float v = bounded(st, tb);
      if (v == v) *cb = v, want_b = false;
    }
    if (want_a || want_b) {
      const Costs r = powers(st, ta, tb, want_a, want_b);
      if (want_a) *ca = r.ca;
      if (want_b) *cb = r.cb;
    }
  }
};

// N = 1000 (1 M pairs): 1.75-2.1 ms with two float-float costs per finite
// difference and pow for what they do not certify (one wave, its warps held by
// the pow evaluations), 0.21 ms now.  Four blocks an SM (116 registers, no
// spills): 1.98 ms at N = 4000, five 2.12, six 2.61.
__global__ void __launch_bounds__(kBisectThreads, 4) bvp_pairs_refgpu_kernel(AllPairs src, int chunk) {
  __shared__ BisectQueue s_queue[kBisectWarps];
  const long long left = (long long)src.N * (src.N - 1);
  const int warp = threadIdx.x >> 5;
  const long long first = (blockIdx.x * (long long)kBisectWarps + warp) * chunk;
  if (first >= left) return;
  bisect_warp<RefGpuCost, kBisectRefill>(src, s_queue[warp], first,
                                        left - first < chunk ? (int)(left - first) : chunk);
}

// Explicit pairs (the BvpJobs layout of ctx.h), `per` per warp.
__global__ void __launch_bounds__(128) bvp_batch_refgpu_kernel(const JobPairs src, int per) {
  const long long total = (long long)src.jb.n * src.jb.jobs;
  __shared__ BisectQueue s_queue[kBisectWarps];
  const int warp = threadIdx.x >> 5;
  const long long first = (blockIdx.x * (long long)(blockDim.x >> 5) + warp) * per;
  if (first >= total) return;
  bisect_warp<RefGpuCost, 32>(src, s_queue[warp], first, total - first < per ? (int)(total - first) : per);
}

}  // namespace

pump_status_t bvp_pairs_refgpu_launch(const float *d_samples, int N, float tmax, float *d_copts,
                                      float *d_topts, cudaStream_t stream) {
  const long long npairs = (long long)N * (N - 1);
  const int chunk = bisect_chunk(npairs);
  const long long per = (long long)kBisectWarps * chunk, nblk = (npairs + per - 1) / per;
  if (nblk > 2147483647LL) return set_error(PUMP_ERR_CAPACITY, "pump_bvp_pairs: N=%d", N);
  bvp_pairs_refgpu_kernel<<<(unsigned)nblk, kBisectThreads, 0, stream>>>(
      AllPairs{d_samples, N, tmax, d_copts, d_topts}, chunk);
  return launch_status("bvp_pairs_refgpu");
}

pump_status_t bvp_jobs_refgpu_launch(const BvpJobs &jb, cudaStream_t stream) {
  if (jb.n <= 0) return PUMP_OK;
  const long long total = (long long)jb.n * jb.jobs;
  const int per = bisect_jobs_per_warp(total);
  const int warps = per < 32 ? 1 : kBisectWarps;
  bvp_batch_refgpu_kernel<<<grid_for(total, warps * per), warps * 32, 0, stream>>>(JobPairs{jb}, per);
  return launch_status("bvp_batch_refgpu");
}

}  // namespace pump
