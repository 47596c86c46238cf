// toptBisection (2pBVP.cu:71-95) for many pairs, in the two bit-exact
// arithmetics (bvp.cu: the reference built for the CPU; bvp_refgpu.cu: its
// GPU kernel).
//
// What the reference does with a finite difference (cost(topt + h) -
// cost(topt - h)) / dtau is to read its sign and to stop once it is within
// 1e-4 of zero.  The two costs are binary32 values about 1e-6 apart in tau.
// Far from the optimum they differ by many units in the last place, so the
// sign follows from the cost's derivative (slope_sign, ffcost.cuh: about 45
// instructions); nearer, from the difference of the two binary64 costs
// (cost_delta: about 95).  Only the last one or two steps need the costs
// themselves: one in float-float (cost_ff_value: about 180), the other from it
// and the difference, each certified to round as the reference's; what is
// not certified falls back to float-float for the second cost, then to the
// reference's own expression (Exact::costs).  Of a random pair's 11 finite
// differences (states as the benchmark's), 6 are settled by the derivative, 3
// by the difference, and 2 need the costs.
//
// A warp works in two stages, so that its lanes stay together although every
// bisection has its own length.  Stage A takes 32 pairs, one per lane, and runs
// the steps the derivative and then the difference settle, which are nearly as
// many for one pair as for another; the pairs' coefficients and brackets then
// go to a queue in shared memory.  Stage B runs the remaining steps: a lane whose
// pair is done stores it and takes the queue's next, once kBisectRefill lanes
// wait for one.  Every pair walks the same sequence of finite differences as
// toptBisection.
//
// Bound by instruction issue (no DRAM traffic but the results).
#pragma once

#include <string.h>

#include "common.cuh"
#include "ctx.h"
#include "ffcost.cuh"

namespace pump {
namespace {

// The bisection's stopping test compares a binary32 |dcval| with the
// binary64 constant 0.0001 (2pBVP.cu:86).  binary32 0.0001f is below 0.0001
// and the next binary32 above it, so (double)x > 0.0001 exactly when
// x > 0.0001f (NaN false either way): the test runs in binary32.
constexpr float kDcvalTol = 0.0001f;
// A difference is taken as certain when it exceeds spacing + error + this:
// then the rounded costs differ by more than it, and |dcval| = difference /
// 1e-6f is above 2e-4, so the bisection does not stop.
constexpr float kDeltaMin = 2e-10f;
// Steps stage A takes at most by the derivative and by the difference: a pair
// with more of them continues in stage B, so that the warp does not wait for
// its longest.  N = 4000, us (limits in this order): none 2855; (0, 9) 1964,
// (2, 7) 1948, (4, 6) 1922, (4, 5) 1902, (5, 5) 1913, (6, 4) 1935, (7, 3) 2007.
constexpr int kSlopeSteps = 4;
constexpr int kDeltaSteps = 5;

__device__ __forceinline__ bool delta_sign(const PairFF &f, float ta, float tb, int *sign) {
  float dv, err, ulp;
  const bool in = cost_delta(f, ta, tb, &dv, &err, &ulp);
  *sign = dv > 0 ? 1 : -1;
  return in && fabsf(dv) > (ulp + err) * 1.0001f + kDeltaMin;
}

// One bisection: phase 0 the tmax test, 1 the halving loop, 2 the bisection
// steps, 3 the final cost.
struct BisectState {
  float tu, tl, topt;
  int phase, count;  // count: halvings (phase 1), bisection steps (phase 2)
  __device__ __forceinline__ void begin(float tmax) {
    tu = tmax;
    tl = 0;
    phase = 0;
    count = 0;
    topt = tmax;
  }
  // the point of the next finite difference
  __device__ __forceinline__ void aim() {
    if (phase == 1) topt = tl;
    if (phase == 2) topt = (tu + tl) / 2;
  }
  // after a finite difference of this sign (0: zero or NaN); stop: it is
  // within the tolerance
  __device__ __forceinline__ void advance(int sign, bool stop) {
    if (phase == 0) {
      if (sign < 0) {
        phase = 3;  // topt is tmax
      } else {
        tl = (float)0.01;
        phase = 1;
      }
    } else if (phase == 1) {
      // the reference's halving loop (:78-80) is unbounded; here it stops
      // after 160 halvings (tl < 1e-50 has underflowed to zero long before),
      // as the oracle does
      if (sign > 0 && count < 160) {
        tl = tl / 2;
        ++count;
      } else {
        count = 0;
        phase = 2;
      }
    } else {
      ++count;
      if (sign > 0) tu = topt; else tl = topt;
      // once the bracket's ends are neighbours the midpoint is the point just
      // taken, and every further step repeats it: the reference's up to 50
      // steps end on this topt
      if (stop || count >= 50 || (tu + tl) / 2 == topt) phase = 3;
    }
  }
};

// A queued pair: its coefficients (PairFF), bracket, phase and item number,
// as words of a structure of arrays in shared memory.
constexpr int kBisectSlots = 64;
struct BisectItem {
  PairFF f;
  float tu, tl;
  int phase, count, item;
};
constexpr int kBisectWords = sizeof(BisectItem) / 4;
static_assert(sizeof(BisectItem) % 4 == 0, "words");
struct BisectQueue {
  unsigned w[kBisectWords][kBisectSlots];
  __device__ __forceinline__ void put(int slot, const BisectItem &it) {
    unsigned v[kBisectWords];
    memcpy(v, &it, sizeof it);
#pragma unroll
    for (int k = 0; k < kBisectWords; ++k) w[k][slot] = v[k];
  }
  __device__ __forceinline__ void get(int slot, BisectItem *it) const {
    unsigned v[kBisectWords];
#pragma unroll
    for (int k = 0; k < kBisectWords; ++k) v[k] = w[k][slot];
    memcpy(it, v, sizeof *it);
  }
};

// Pairs first .. first + n - 1 of src, by one warp.  Src: load(k, x0, x1) the
// two states, tmax(k), store(k, topt, cost), kWantCost.  Exact::costs(x0, x1,
// ta, tb, want_a, want_b, &ca, &cb): the reference's cost expression.
template <class Exact, int kRefillLanes, class Src>
__device__ __forceinline__ void bisect_warp(const Src &src, BisectQueue &queue, long long first, int n) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const float h = (float)0.000001 / 2;  // dtau / 2 of dcost
  const float dtau = (float)0.000001;
  int next = 0, head = 0, tail = 0;  // warp-uniform
  BisectItem it{};
  BisectState st{};
  bool have = false;
  while (true) {
    if (tail - head < 32 && next < n) {
      // stage A: 32 more pairs
      const int item = next + lane;
      const bool mine = item < n;
      if (mine) {
        float x0[kDim], x1[kDim];
        src.load(first + item, x0, x1);
        BisectItem q;
        q.f = make_pair_ff(x0, x1);
        const PairSlope sl = make_slope(q.f);
        BisectState s;
        s.begin(src.tmax(first + item));
#pragma unroll 1
        for (int k = 0; k < kSlopeSteps && s.phase < 3; ++k) {
          s.aim();
          int sign;
          if (!slope_sign(sl, s.topt + h, s.topt - h, kDeltaMin, &sign)) break;
          s.advance(sign, false);
        }
#pragma unroll 1
        for (int k = 0; k < kDeltaSteps && s.phase < 3; ++k) {
          s.aim();
          int sign;
          if (!delta_sign(q.f, s.topt + h, s.topt - h, &sign)) break;
          s.advance(sign, false);
        }
        q.tu = s.phase == 3 ? s.topt : s.tu;
        q.tl = s.tl;
        q.phase = s.phase;
        q.count = s.count;
        q.item = item;
        queue.put((tail + lane) & (kBisectSlots - 1), q);
      }
      const int got = n - next < 32 ? n - next : 32;
      tail += got;
      next += got;
      __syncwarp();
    }
    // stage B: lanes without a pair take the queue's next
    const unsigned need = __ballot_sync(0xffffffffu, !have);
    if (need && head < tail && (__popc(need) >= kRefillLanes || need == 0xffffffffu)) {
      const int rank = __popc(need & lt);
      if (!have && rank < tail - head) {
        queue.get((head + rank) & (kBisectSlots - 1), &it);
        st.tu = it.tu;
        st.tl = it.tl;
        st.topt = it.tu;  // phase 0: tmax; phase 3: the time stage A ended on
        st.phase = it.phase;
        st.count = it.count;
        have = true;
      }
      head += __popc(need) < tail - head ? __popc(need) : tail - head;
      __syncwarp();  // the slots just read are rewritten by stage A
    }
    if (!__any_sync(0xffffffffu, have)) {
      if (head == tail && next >= n) break;
      continue;
    }
    if (!have) continue;
    if (Src::kWantCost || st.phase != 3) {
      st.aim();
      const float ta = st.phase == 3 ? st.topt : st.topt + h;
      const float tb = st.phase == 3 ? st.topt : st.topt - h;
      float dv, err, ulp;
      const bool in = cost_delta(it.f, ta, tb, &dv, &err, &ulp);
      int sign = dv > 0 ? 1 : -1;
      bool stop = false;
      float ca = 0;
      if (!(in && fabsf(dv) > (ulp + err) * 1.0001f + kDeltaMin)) {
        CostFF va;
        bool ok_a = cost_ff_value(it.f, ta, &va);
        const FF wb = ff_add_f(va.w, -dv);
        // (the float-float subtraction's rounding: 2^-44 of the value)
        float cb;
        bool ok_b = ff_round(wb, va.bound + err + fabsf(wb.hi) * 0x1p-44f, &cb) && in && ok_a;
        ok_a = ff_round(va.w, va.bound, &ca) && ok_a;
        if (st.phase == 3) ok_b = true;
        else if (!ok_b) cb = cost_ff(it.f, tb, &ok_b);
        if (!(ok_a && ok_b)) {
          float x0[kDim], x1[kDim];
          src.load(first + it.item, x0, x1);
          Exact::costs(x0, x1, ta, tb, !ok_a, !ok_b, &ca, &cb);
        }
        const float d = (ca - cb) / dtau;
        sign = d > 0 ? 1 : (d < 0 ? -1 : 0);
        stop = !(fabsf(d) > kDcvalTol);
      }
      if (st.phase == 3) {
        src.store(first + it.item, st.topt, ca);
        have = false;
      } else {
        st.advance(sign, stop);
      }
    }
    if (!Src::kWantCost && have && st.phase == 3) {
      src.store(first + it.item, st.topt, 0.0f);
      have = false;
    }
  }
}

// All ordered pairs of N samples in pair order (idx = i (N-1) + j - (i < j)).
struct AllPairs {
  static constexpr bool kWantCost = true;
  const float *__restrict__ samples;
  int N;
  float tm;
  float *__restrict__ copts, *__restrict__ topts;
  __device__ __forceinline__ void load(long long k, float *x0, float *x1) const {
    const int i = (int)(k / (N - 1));
    const int r = (int)(k - (long long)i * (N - 1));
    const int j = r + (r >= i);
#pragma unroll
    for (int d = 0; d < kDim; ++d) {
      x0[d] = __ldg(&samples[i * kDim + d]);
      x1[d] = __ldg(&samples[j * kDim + d]);
    }
  }
  __device__ __forceinline__ float tmax(long long) const { return tm; }
  __device__ __forceinline__ void store(long long k, float t, float c) const {
    topts[k] = t;
    copts[k] = c;
  }
};

// Explicit pairs, one or two jobs (BvpJobs): item k is pair k % n of job k / n.
struct JobPairs {
  static constexpr bool kWantCost = true;
  BvpJobs jb;
  __device__ __forceinline__ void load(long long k, float *x0, float *x1) const {
    const int p = (int)(k >= jb.n ? k - jb.n : k);
#pragma unroll
    for (int d = 0; d < kDim; ++d) {
      x0[d] = __ldg(&jb.x0[p * kDim + d]);
      x1[d] = __ldg(&jb.x1[(jb.x1_same ? 0 : p) * kDim + d]);
    }
  }
  __device__ __forceinline__ float tmax(long long k) const { return jb.tmax[k >= jb.n ? 1 : 0]; }
  __device__ __forceinline__ void store(long long k, float t, float c) const {
    const int j = k >= jb.n ? 1 : 0, p = (int)(j ? k - jb.n : k);
    if (jb.topt[j]) jb.topt[j][p] = t;
    if (jb.cost[j]) jb.cost[j][p] = c;
  }
};

constexpr int kBisectThreads = 128;
constexpr int kBisectWarps = kBisectThreads / 32;
constexpr int kBisectRefill = 4;

// Pairs per warp of the all-pairs kernels: two rounds of the resident warps
// (fewer pairs a warp end in more partly filled last queues, one round ends
// with its slowest warp: N = 1000, reference-GPU arithmetic, 246 us in four
// rounds, 209 in two, 231 in one), at least 64, and at most 768 (24 per lane).
inline int bisect_chunk(long long npairs) {
  const long long warps = (long long)kNumSMs * 24 * 2;
  const long long c = ((npairs + warps - 1) / warps + 31) & ~31LL;
  return c >= 768 ? 768 : (c <= 64 ? 64 : (int)c);
}

// Explicit pairs per warp: a warp takes as many rounds as its longest
// bisection, so a small call (a smoothing batch has about a hundred) spreads
// its pairs over the SMs, up to two warps each, before it fills warps.
inline int bisect_jobs_per_warp(long long total) {
  const long long per = (total + 2 * kNumSMs - 1) / (2 * kNumSMs);
  return per < 1 ? 1 : (per < 32 ? (int)per : 32);
}

}  // namespace
}  // namespace pump
