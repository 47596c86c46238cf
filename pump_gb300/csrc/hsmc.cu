// Particle stream, half-space Monte Carlo (HSMC) propagation and full Monte
// Carlo collision probability (reference: PUMP.cu:613-758,
// collisionProbability.cu:4-92, hardCoded.cuh:12-19).
//
// Particle stream.  The reference reads precomputed closed-loop tracking
// errors (xcomb / xcombTime) from a data file that is not part of its source
// tree.  They are regenerated here from a documented model: per axis a
// double integrator at dt = 0.05 s under the PD tracking law a = w - (16 p +
// 5.6 v), w ~ N(0, 4^2), starting from zero error, simulated in binary64.
// Noise comes from Philox4x32-10 (Salmon et al., SC'11) at counter
// (particle, step, 0, 0), turned into Gaussians by Box-Muller whose log and
// sine/cosine are evaluated by fixed series with +,-,*,/ and sqrt only
// (atanh series for log, Taylor series on a quarter period for sin/cos), so
// the table is bit-identical on any IEEE machine that does not contract
// multiply-adds.
//
// HSMC.  One warp per new path, its lanes over quads of particles.  The
// half-spaces of a waypoint are the same for every particle of the path, so the
// warp tests up to five of them at once on each quad that it loads; offsets are
// read time-major, 128 consecutive particles a step.  Validity is kept as a bit
// per particle, in registers, and the hit count of calculateCP_HSMC is the
// warp's popcount sum, so the CP needs no second pass.
//
// Monte Carlo CP.  A block takes 32 or 128 particles of one path, its 16 warps
// consecutive runs of the path's segments; obstacles staged in shared memory,
// those that no particle of a warp comes near dropped per segment; the same
// segment test as freeEdges.
#include <math.h>

#include <type_traits>

#include "collide.cuh"
#include "search.h"

namespace pump {
namespace {

// ------------------------------------------------------- particle stream
__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                              uint32_t k0, uint32_t k1, uint32_t out[4]) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t lo0 = 0xD2511F53u * c0, hi0 = __umulhi(0xD2511F53u, c0);
    const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = __umulhi(0xCD9E8D57u, c2);
    const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

__device__ double det_log(double x) {
  int e;
  double m = frexp(x, &e);
  if (m < 0.70710678118654752440) { m = m * 2.0; e = e - 1; }
  const double s = (m - 1.0) / (m + 1.0);
  const double z = s * s;
  double t = 1.0 / 25.0;
  t = t * z + 1.0 / 23.0;
  t = t * z + 1.0 / 21.0;
  t = t * z + 1.0 / 19.0;
  t = t * z + 1.0 / 17.0;
  t = t * z + 1.0 / 15.0;
  t = t * z + 1.0 / 13.0;
  t = t * z + 1.0 / 11.0;
  t = t * z + 1.0 / 9.0;
  t = t * z + 1.0 / 7.0;
  t = t * z + 1.0 / 5.0;
  t = t * z + 1.0 / 3.0;
  t = t * z + 1.0;
  return (double)e * 0.69314718055994530942 + 2.0 * s * t;
}

__device__ void det_sincos_2pi(double u, double *s, double *c) {
  const double q = u * 4.0;
  const int k = (int)q;
  const double f = q - (double)k;
  const double th = f * 1.57079632679489661923;
  const double z = th * th;
  double sn = -1.0 / 15511210043330985984000000.0;
  sn = sn * z + 1.0 / 25852016738884976640000.0;
  sn = sn * z - 1.0 / 51090942171709440000.0;
  sn = sn * z + 1.0 / 121645100408832000.0;
  sn = sn * z - 1.0 / 355687428096000.0;
  sn = sn * z + 1.0 / 1307674368000.0;
  sn = sn * z - 1.0 / 6227020800.0;
  sn = sn * z + 1.0 / 39916800.0;
  sn = sn * z - 1.0 / 362880.0;
  sn = sn * z + 1.0 / 5040.0;
  sn = sn * z - 1.0 / 120.0;
  sn = sn * z + 1.0 / 6.0;
  sn = sn * z - 1.0;
  sn = -(sn * th);
  double cs = 1.0 / 620448401733239439360000.0;
  cs = cs * z - 1.0 / 1124000727777607680000.0;
  cs = cs * z + 1.0 / 2432902008176640000.0;
  cs = cs * z - 1.0 / 6402373705728000.0;
  cs = cs * z + 1.0 / 20922789888000.0;
  cs = cs * z - 1.0 / 87178291200.0;
  cs = cs * z + 1.0 / 479001600.0;
  cs = cs * z - 1.0 / 3628800.0;
  cs = cs * z + 1.0 / 40320.0;
  cs = cs * z - 1.0 / 720.0;
  cs = cs * z + 1.0 / 24.0;
  cs = cs * z - 0.5;
  cs = cs * z + 1.0;
  switch (k & 3) {
    case 0: *s = sn; *c = cs; break;
    case 1: *s = cs; *c = -sn; break;
    case 2: *s = -sn; *c = -cs; break;
    default: *s = -cs; *c = sn; break;
  }
}

constexpr double kDT = 0.05, kH2 = 0.00125, kKP = 16.0, kKD = 5.6, kSigmaW = 4.0;

// The table in two launches.  Gaussians of every (particle, step) are
// independent: one thread each (Philox, Box-Muller) into a binary64 buffer
// z[t][p][3].  The closed-loop recurrence is sequential in time only: one
// thread per (particle, axis) runs it over the steps.  (A binary64 warp
// instruction occupies this GPU's FP64 pipe for the same time whether one
// lane or 32 are active, so the recurrence must not run in one lane of a warp
// while the others wait.)  Each value is produced by the same operations in
// the same order as a scalar loop, without contraction.
__global__ void __launch_bounds__(256) particle_gauss_kernel(uint32_t k0, uint32_t k1, int P, int T,
                                                             double *__restrict__ z) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)P * T) return;
  const int t = (int)(i / P), p = (int)(i - (long long)t * P);
  const double sc = 2.3283064365386962890625e-10;  // 2^-32
  uint32_t o[4];
  philox4x32_10((uint32_t)p, (uint32_t)t, 0u, 0u, k0, k1, o);
  const double u0 = ((double)o[0] + 0.5) * sc, u1 = ((double)o[1] + 0.5) * sc;
  const double u2 = ((double)o[2] + 0.5) * sc, u3 = ((double)o[3] + 0.5) * sc;
  const double r0 = sqrt(-2.0 * det_log(u0));
  const double r1 = sqrt(-2.0 * det_log(u2));
  double s0, c0, s1, c1;
  det_sincos_2pi(u1, &s0, &c0);
  det_sincos_2pi(u3, &s1, &c1);
  z[i * 3 + 0] = r0 * c0;
  z[i * 3 + 1] = r0 * s0;
  z[i * 3 + 2] = r1 * c1;
}

__global__ void __launch_bounds__(128) particle_table_kernel(const double *__restrict__ z, int P,
                                                             int T, float *__restrict__ tmajor,
                                                             float *__restrict__ pmajor) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P * 3) return;
  const int p = i / 3, d = i - 3 * (i / 3);
  double pos = 0, vel = 0;
  for (int t = 0; t < T; ++t) {
    const float v = (float)pos;
    if (tmajor) tmajor[((long long)t * P + p) * 3 + d] = v;
    if (pmajor) pmajor[((long long)p * T + t) * 3 + d] = v;
    const double a = kSigmaW * z[((long long)t * P + p) * 3 + d] - (kKP * pos + kKD * vel);
    const double pn = (pos + kDT * vel) + kH2 * a;
    const double vn = vel + kDT * a;
    pos = pn;
    vel = vn;
  }
}

// Per-axis position variance of the same closed loop: S' = A S A^T + g g^T
// with A = [[1 - H2 KP, DT - H2 KD], [-DT KP, 1 - DT KD]] and g = [H2, DT]
// sigma_w, from S = 0 (the particles start on the path).  A sequential
// recurrence of a few hundred steps: one thread, binary64.
__global__ void position_variance_kernel(int T, double *__restrict__ var) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  const double a00 = 1.0 - kH2 * kKP, a01 = kDT - kH2 * kKD;
  const double a10 = -(kDT * kKP), a11 = 1.0 - kDT * kKD;
  const double g0 = kH2 * kSigmaW, g1 = kDT * kSigmaW;
  double spp = 0, spv = 0, svv = 0;
  for (int t = 0; t < T; ++t) {
    var[t] = spp;
    const double m00 = a00 * spp + a01 * spv, m01 = a00 * spv + a01 * svv;
    const double m10 = a10 * spp + a11 * spv, m11 = a10 * spv + a11 * svv;
    const double npp = m00 * a00 + m01 * a01 + g0 * g0;
    const double npv = m00 * a10 + m01 * a11 + g0 * g1;
    const double nvv = m10 * a10 + m11 * a11 + g1 * g1;
    spp = npp;
    spv = npv;
    svv = nvv;
  }
}

// ------------------------------------------------------------------ HSMC
// One warp per new path.  Lane l owns particles 128 c + 4 l + j (j < 4), one
// bit each, so the offsets of a c-step are 128 consecutive particles, three
// 16-byte loads a lane.  (12-byte records of 32 particles, three 4-byte loads
// each: 311 us for 12,000 paths x 1024 particles with about 38 active half-spaces
// a path; 154 us so, with up to five half-spaces of a waypoint tested on each
// loaded particle and the comparison's product folded into its bound.)  A table
// whose rows are not whole 16-byte quads (Pmc not a multiple of four) is read 32
// consecutive records at a time, and a lane's particles are 128 c + 32 j + l.
// The loop over groups of 1024 particles is rolled (the group's bits selected by
// its number): six instantiations of the test, twenty-four with it unrolled at
// 4096 particles, do not stay in the instruction cache (100,000 paths x 4096
// particles, 100 boxes: 4.8 ms with 4-byte loads, 8.5 ms with quads and that
// loop unrolled, 2.9 ms so; 12,000 paths x 1024 particles the same).  Such large
// wavefronts are bound by instruction issue.  The warp first finds the edge's W x H
// half-space slots that are active (the reference skips a half-space when
// b >= 1000, PUMP.cu:642); with none active the new mask is the parent's and
// only the hit count is computed.  Every active half-space is tested for
// every particle exactly as PUMP.cu:645-651 does (binary32, no
// contraction); AND-ing the tests in another order gives the same bits.
//
// Two sources of half-spaces.  Cached: the arrays of pump_cache_halfspaces
// (dense, or sparse with per-waypoint counts).  Boxes: the warp derives
// them itself from the edge's waypoints and the obstacle set staged in
// shared memory, with the same operations (halfspace_of_box), into its own
// shared-memory slots.  It first drops the boxes that no waypoint of the
// edge can bring within the distance gate (gate_keeps_box on the waypoints'
// bounding box; none dropped when a waypoint is not finite or more than
// kHsmcFilterObs boxes are left: 10^6 paths near 200 boxes 6.8 ms where more boxes
// than the list holds were never filtered, 1.9 so), then per waypoint takes the
// remaining boxes 32 at a time, one per lane: the lanes whose box passes the gate
// are ranked by a ballot and the first maxHS - stored of them, in index order,
// fill the next slots, which are the slots cacheHalfspaces fills.  Only the edges
// a wavefront propagates along get half-spaces, and no cache is written.
constexpr int kMaxHsmcWords = 128;   // P <= 4096 particles
constexpr int kMaxHsSlots = 256;     // W * maxHS <= 256
constexpr int kHsmcThreads = 128;
constexpr int kHsmcWarps = kHsmcThreads / 32;
// blocks of a launch that loops over a device-side path count
constexpr int kHsmcPersistBlocks = kNumSMs * 8;
// A wavefront's paths are dealt to the blocks: a block's warps take its paths one
// at a time from a shared-memory counter, so a warp whose paths are cheap (no
// active half-space: the parent's masks copied) takes more of them while another
// tests particles.  One path per warp while that fits the resident blocks (a
// small wavefront spreads over every warp).  Then block k of b takes the paths k,
// k + b, k + 2 b, ...: every block has the same number, whatever n is, and waits
// for its slowest warp once.  (Chunks of 8 consecutive paths took 12,000 paths 1.23
// rounds of the 1,216 blocks; chunks of 16 or 17 taken in turn left one warp of four
// idle for a round in five.)  From 16 paths a block on, if the host knows n, there
// are more blocks than resident ones, of kHsmcRun consecutive paths each, because
// some SMs run them faster (100,000 paths x 1024 particles near 200 boxes: 770 us
// in such blocks, 870 dealt to 1,216, 950 in chunks of 17).
constexpr int kHsmcRun = 8;
constexpr int kHsmcDealt = 16;
// Queries that share a launch take chunks of at most 16 paths, four a warp, so
// that the larger ones' spread over all of its blocks.
__host__ __device__ inline int hsmc_chunks(long long n, long long blocks, bool alone) {
  const long long single = (n + kHsmcWarps - 1) / kHsmcWarps;
  if (single <= blocks) return (int)single;
  return (int)(alone || n <= kHsmcDealt * blocks ? blocks : (n + kHsmcDealt - 1) / kHsmcDealt);
}
inline unsigned hsmc_blocks(long long n, bool device_count) {
  if (!device_count && n > (long long)kHsmcDealt * kHsmcPersistBlocks)
    return (unsigned)((n + kHsmcRun - 1) / kHsmcRun);
  return (unsigned)hsmc_chunks(n, kHsmcPersistBlocks, true);
}
// Half-spaces of one waypoint tested on each loaded quad of particles, 5 being
// the reference's limit (12,000 paths, about 38 active half-spaces each, event
// times of the step that chose it: 230 us with 2, 194 with 3 or 4, 167 with 5; the
// quads' loop is not unrolled: 224 us with two quads in flight, whose code is
// twice as long).
constexpr int kHsmcGroup = 5;
constexpr int kHsmcFilterObs = 128;

// Shared memory of the boxes variant: the staged boxes, then per warp its
// half-space slots (a0, a1, a2, b), stored counts per waypoint and the list
// of boxes that survive the edge's gate bound.
__host__ __device__ inline size_t hsmc_boxes_obs_floats(int numObs) {
  return (size_t)((numObs * 12 + 3) & ~3);
}
// Per warp: W * maxHS half-space slots and W stored counts (rounded to 16
// bytes), sized for the launch's W and maxHS.
__host__ __device__ inline int hsmc_hs_stride(int W, int maxHS) { return W * maxHS; }
__host__ __device__ inline int hsmc_cnt_stride(int W) { return (W + 15) & ~15; }
__host__ __device__ inline size_t hsmc_boxes_smem(int numObs, int W, int maxHS) {
  return sizeof(float) * hsmc_boxes_obs_floats(numObs) +
         (size_t)kHsmcWarps * (sizeof(float4) * hsmc_hs_stride(W, maxHS) + hsmc_cnt_stride(W) +
                               sizeof(int) * kHsmcFilterObs);
}

// The largest LHS with fl(LHS * om) < b (the products grow with LHS, so the
// test is LHS <= *bound): from the quotient, moved to the neighbour that is on
// the boundary.  False (the test needs the product) outside ordinary values or
// if three steps do not reach it.
__device__ __forceinline__ bool hsmc_lhs_bound(float b, float om, float *bound) {
  if (!(b >= 1e-25f && b < 1e25f && om >= 1e-10f && om <= 1e10f)) return false;  // also NaN
  unsigned u = __float_as_uint(b / om);
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (!(__uint_as_float(u) * om < b)) --u;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (__uint_as_float(u + 1u) * om < b) ++u;
  *bound = __uint_as_float(u);
  return __uint_as_float(u) * om < b && !(__uint_as_float(u + 1u) * om < b);
}

// Bit b of lane l <-> bit l of lane b: halves of the 32 x 32 matrix exchanged,
// then halves of those.
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t x) {
  const int lane = threadIdx.x & 31;
  uint32_t m = 0x0000ffffu;  // the bits whose number does not have s
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    x = (lane & s) ? (x & ~m) | ((y >> s) & m) : (x & m) | ((y & m) << s);
    m ^= m << (s >> 1);
  }
  return x;
}

// New path w (the whole warp).  valid_in[prev] is read, valid_out[w] /
// cp_out[w] written (the two may alias one path store with valid_out =
// store + base, as in the reference).  With hs_count (stored half-spaces per
// waypoint), slots at or past a waypoint's count are inactive without
// reading them (they hold the defaults b = 1111 in the dense layout); stored
// slots still need b < 1000.
// Epi: the search's epilogue (HsmcEpilogue) runs for each path.
template <bool Boxes, int Q, bool Epi>
__device__ __forceinline__ void hsmc_path(const HsmcParams &p, int w, int edge, int prev,
                                          const float *s_obs, float4 *hs, uint8_t *hcnt, int *klist) {
  const int lane = threadIdx.x & 31;
  const unsigned int lt = (1u << lane) - 1u;
  if (edge < 0 || edge >= p.num_edges || prev < 0 || prev >= p.num_prev) {
    if (lane == 0 && p.error) atomicExch(p.error, (int)PUMP_ERR_BAD_INPUT);
    return;
  }
  // the edge's waypoints: W records per edge, or its own range (at most p.W)
  int W = p.W;
  long long wp0 = (long long)edge * W;
  if (Boxes && p.disc_off) {
    wp0 = p.disc_off[edge];
    const long long n = p.disc_off[edge + 1] - wp0;
    if (n < 2 || n > p.W) {
      if (lane == 0 && p.error) atomicExch(p.error, (int)PUMP_ERR_BAD_INPUT);
      return;
    }
    W = (int)n;
  }
  // the epilogue's inputs, one per lane, on their way while the path is
  // propagated
  uint32_t epi = 0u;
  if (Epi && lane < 5) {
    const HsmcEpilogue &e = p.epi;
    const void *src = lane == 0   ? (const void *)&e.path_time[prev]
                      : lane == 1 ? (const void *)&e.topt[edge]
                      : lane == 2 ? (const void *)&e.path_cost[prev]
                      : lane == 3 ? (const void *)&e.copt[edge]
                                  : (const void *)&e.wf_node[w];
    epi = *reinterpret_cast<const uint32_t *>(src);
  }
  const int maxHS = p.maxHS, P = p.P;
  const int words = (P + 31) >> 5;
  const int slots = W * maxHS;
  const long long hsHead = (long long)edge * slots;
  // parent's words: lane j holds words j, j+32, ... (issued first: their
  // latency overlaps the half-space work)
  uint32_t mine[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int j = q * 32 + lane;
    mine[q] = (j < words) ? p.valid_in[(long long)prev * words + j] : 0u;
  }
  if (Boxes) {
    // lane i holds waypoint i (W <= 32; otherwise waypoints are read per step)
    const float *ew = p.disc + wp0 * kDim;
    float my[kDim];
    const int mi = lane < W ? lane : 0;
#pragma unroll
    for (int d = 0; d < kDim; ++d) my[d] = __ldg(&ew[mi * kDim + d]);
    // the edge's waypoints bound the boxes worth testing, if they are finite (an
    // infinite one's distance to an infinite box is not a number, which passes
    // the gate)
    float mn[3], mx[3];
    bool odd = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      mn[d] = mx[d] = my[d];
      odd = odd || !(fabsf(my[d]) < INFINITY);
    }
    for (int i = lane + 32; i < W; i += 32)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float x = __ldg(&ew[i * kDim + d]);
        odd = odd || !(fabsf(x) < INFINITY);
        mn[d] = fminf(mn[d], x);
        mx[d] = fmaxf(mx[d], x);
      }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      mn[d] = warp_min_f32(mn[d]);
      mx[d] = warp_max_f32(mx[d]);
    }
    odd = __any_sync(0xffffffffu, odd);
    bool filt = !odd;
    int nk = 0;
    for (int o0 = 0; o0 < p.numObs && filt; o0 += 32) {
      const int o = o0 + lane;
      const bool keep = o < p.numObs && gate_keeps_box(mn, mx, &s_obs[o * 12], p.maxd2);
      const unsigned int bal = __ballot_sync(0xffffffffu, keep);
      filt = nk + __popc(bal) <= kHsmcFilterObs;  // warp-uniform
      if (keep && filt) klist[nk + __popc(bal & lt)] = o;
      nk += __popc(bal);
    }
    if (!filt) nk = p.numObs;
    for (int i = lane; i < W; i += 32) hcnt[i] = 0;
    __syncwarp();
    for (int i = 0; i < W && nk > 0; ++i) {
      float pos[3], vel[3];
      if (i < 32) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          pos[d] = __shfl_sync(0xffffffffu, my[d], i);
          vel[d] = __shfl_sync(0xffffffffu, my[3 + d], i);
        }
      } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          pos[d] = __ldg(&ew[i * kDim + d]);
          vel[d] = __ldg(&ew[i * kDim + 3 + d]);
        }
      }
      int stored = 0;
      for (int c0 = 0; c0 < nk && stored < maxHS; c0 += 32) {
        const int c = c0 + lane;
        float ah[3] = {0.0f, 0.0f, 0.0f}, bh = 0.0f;
        bool pass = false;
        if (c < nk) {
          const int o = filt ? klist[c] : c;
          pass = halfspace_of_box(pos, vel, &s_obs[o * 12], p.maxd2, ah, &bh);
        }
        const unsigned int bal = __ballot_sync(0xffffffffu, pass);
        const int rank = __popc(bal & lt);
        if (pass && stored + rank < maxHS) hs[i * maxHS + stored + rank] = make_float4(ah[0], ah[1], ah[2], bh);
        const int got = __popc(bal);
        stored += got < maxHS - stored ? got : maxHS - stored;
      }
      if (lane == 0) hcnt[i] = (uint8_t)stored;
    }
    __syncwarp();
  }
  // which half-space slots are active (b < 1000 or NaN, as !(b >= 1000)):
  // lane c holds the mask of slots 32 c .. 32 c + 31
  uint32_t act = 0u;
  for (int c = 0; c * 32 < slots; ++c) {
    const int sidx = c * 32 + lane;
    bool a = false;
    if (sidx < slots) {
      const int i = sidx / maxHS, s = sidx - i * maxHS;
      if (Boxes) {
        a = s < (int)hcnt[i] && !(hs[sidx].w >= 1000);
      } else {
        const bool stored = !p.hs_count || s < (int)__ldg(&p.hs_count[(long long)edge * W + i]);
        a = stored && !(__ldg(&p.bs[hsHead + sidx]) >= 1000);
      }
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, a);
    if (lane == c) act = bal;
  }
  int overflow = 0;
  if (__any_sync(0xffffffffu, act != 0u)) {
    // 16-byte loads need whole quads of particles in a table row; other tables
    // are read 32 consecutive 12-byte records at a time, and the lane's four
    // particles are 32 apart instead of consecutive (launch-uniform)
    const bool vec = (p.Pmc & 3) == 0 && (reinterpret_cast<uintptr_t>(p.offsets_t) & 15) == 0;
    // unpack: bit 4 c + j of bits[q] = particle 1024 q + 128 c + 4 lane + j,
    // from word 32 q + 4 c + lane / 8 of the mask (without vec: particle 1024 q
    // + 128 c + 32 j + lane, from word 32 q + 4 c + j)
    uint32_t bits[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      bits[q] = 0u;
      if (q * 1024 >= P) break;
      if (vec) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t wk = __shfl_sync(0xffffffffu, mine[q], 4 * c + (lane >> 3));
          bits[q] |= ((wk >> (4 * (lane & 7))) & 0xFu) << (4 * c);
        }
      } else {
        bits[q] = warp_transpose_bits(mine[q]);
      }
    }
    const float dtLocal = p.topts[edge] / (W - 1);
    const float t0 = p.times[prev];
    // slot sidx: its half-space and its bound on the offset's projection
    auto half_space = [&](int sidx, float (&h)[4]) {
      if (Boxes) {
        const float4 f = hs[sidx];
        h[0] = f.x;
        h[1] = f.y;
        h[2] = f.z;
        h[3] = f.w;
      } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) h[d] = __ldg(&p.as[(hsHead + sidx) * 3 + d]);
        h[3] = __ldg(&p.bs[hsHead + sidx]);
      }
    };
    // The test of N half-spaces of one waypoint (table row `row`) on every
    // particle: dead unless fl(LHS * offset_mult) < b.  Bounded: h[n][3] is the
    // largest LHS that passes (hsmc_lhs_bound), which saves the product.  The
    // tests of a particle already dead are computed and discarded, so the loads
    // do not wait on the bits.  A single half-space leaves registers to load the
    // next quad before this one is tested (200 paths x 4096 particles, 10 boxes:
    // 40 us without, 34 so; with two half-spaces the same and slower for larger
    // wavefronts).
    auto test = [&](const float *row, auto count, auto bounded, const float (&h)[kHsmcGroup][4]) {
      constexpr int N = decltype(count)::value;
      constexpr bool Bounded = decltype(bounded)::value;
      constexpr bool Ahead = Bounded && N == 1;
      // the quad at 128 c of group q (past the last particle: the row's end,
      // whose bits are dropped)
      auto load = [&](int at, float (&o)[4][3]) {
        if (vec) {
          const int p0 = at + 4 * lane < p.Pmc ? at + 4 * lane : p.Pmc - 4;
          const float4 *r4 = reinterpret_cast<const float4 *>(row + p0 * 3);
          const float4 x = __ldg(r4), y = __ldg(r4 + 1), z = __ldg(r4 + 2);
          o[0][0] = x.x; o[0][1] = x.y; o[0][2] = x.z;
          o[1][0] = x.w; o[1][1] = y.x; o[1][2] = y.y;
          o[2][0] = y.z; o[2][1] = y.w; o[2][2] = z.x;
          o[3][0] = z.y; o[3][1] = z.z; o[3][2] = z.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int pp = at + 32 * j + lane < p.Pmc ? at + 32 * j + lane : p.Pmc - 1;
#pragma unroll
            for (int d = 0; d < 3; ++d) o[j][d] = __ldg(&row[pp * 3 + d]);
          }
        }
      };
#pragma unroll 1
      for (int q = 0; q < Q; ++q) {
        if (q * 1024 >= P) break;
        uint32_t bq = bits[0];
#pragma unroll
        for (int k = 1; k < Q; ++k)
          if (q == k) bq = bits[k];
        if (bq == 0u) continue;  // this lane's particles of the group are all dead
        const int end = P - q * 1024 < 1024 ? P - q * 1024 : 1024;
        auto test_quad = [&](int c, const float (&o)[4][3]) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            bool pass = true;
#pragma unroll
            for (int n = 0; n < N; ++n) {
              // (the reference's sum starts from 0, which changes no comparison)
              const float LHS = o[j][0] * h[n][0] + o[j][1] * h[n][1] + o[j][2] * h[n][2];
              pass = pass && (Bounded ? LHS <= h[n][3] : LHS * p.offset_mult < h[n][3]);
            }
            if (!pass) bq &= ~(1u << (4 * c + j));
          }
        };
        float o[4][3];
        if (Ahead && vec) {
          float next[4][3];
          load(q * 1024, o);
#pragma unroll 1
          for (int c = 0; c * 128 < end; ++c) {
            load(q * 1024 + (c + 1) * 128, next);
            test_quad(c, o);
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int d = 0; d < 3; ++d) o[j][d] = next[j][d];
          }
        } else {
#pragma unroll 1
          for (int c = 0; c * 128 < end; ++c) {
            load(q * 1024 + c * 128, o);
            test_quad(c, o);
          }
        }
#pragma unroll
        for (int k = 0; k < Q; ++k)
          if (q == k) bits[k] = bq;
      }
    };
    for (int c = 0; c * 32 < slots; ++c) {
      uint32_t m = __shfl_sync(0xffffffffu, act, c);
      // lane l: the bound of slot 32 c + l
      float lhs_bound = 0.0f;
      bool exact = false;
      if ((m >> lane) & 1u) {
        const int sidx = c * 32 + lane;
        const float b = Boxes ? hs[sidx].w : __ldg(&p.bs[hsHead + sidx]);
        exact = hsmc_lhs_bound(b, p.offset_mult, &lhs_bound);
      }
      const uint32_t exact_mask = __ballot_sync(0xffffffffu, exact);
      while (m) {
        // the waypoint's next active slots, up to kHsmcGroup of them
        const int sidx = c * 32 + __ffs(m) - 1;
        const int i = sidx / maxHS;
        const float time = t0 + i * dtLocal;
        int dtIdx = (int)(time / p.dt);
        if (dtIdx < 0 || dtIdx >= p.T_rows) {
          overflow = 1;
          dtIdx = dtIdx < 0 ? 0 : p.T_rows - 1;
        }
        const float *row = p.offsets_t + (long long)dtIdx * p.Pmc * 3;
        float h[kHsmcGroup][4];
        int group = 0;
        bool bounded = true;
#pragma unroll
        for (int n = 0; n < kHsmcGroup; ++n) {
          const int bit = __ffs(m) - 1;
          if (m == 0u || c * 32 + bit >= (i + 1) * maxHS) break;  // warp-uniform
          m &= m - 1;
          half_space(c * 32 + bit, h[n]);
          if ((exact_mask >> bit) & 1u) h[n][3] = __shfl_sync(0xffffffffu, lhs_bound, bit);
          else bounded = false;
          ++group;
        }
        if (!bounded) {
          // (rare: the bounds of the group's others are dropped again)
          uint32_t back = __shfl_sync(0xffffffffu, act, c) & ~m & ~((1u << (sidx & 31)) - 1u);
          for (; back; back &= back - 1u) {
            half_space(c * 32 + __ffs(back) - 1, h[0]);
            test(row, std::integral_constant<int, 1>{}, std::false_type{}, h);
          }
        } else if (group == 1) {
          test(row, std::integral_constant<int, 1>{}, std::true_type{}, h);
        } else if (group == 2) {
          test(row, std::integral_constant<int, 2>{}, std::true_type{}, h);
        } else if (group == 3) {
          test(row, std::integral_constant<int, 3>{}, std::true_type{}, h);
        } else if (group == 4) {
          test(row, std::integral_constant<int, 4>{}, std::true_type{}, h);
        } else {
          test(row, std::integral_constant<int, 5>{}, std::true_type{}, h);
        }
      }
    }
    // repack: an octet's nibbles form word 4 c + lane / 8 (without vec, the
    // lanes' bits b word b); lane j keeps word j
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (q * 1024 >= P) break;
      uint32_t keep = 0u;
      if (vec) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t v = ((bits[q] >> (4 * c)) & 0xFu) << (4 * (lane & 7));
          v |= __shfl_xor_sync(0xffffffffu, v, 1);
          v |= __shfl_xor_sync(0xffffffffu, v, 2);
          v |= __shfl_xor_sync(0xffffffffu, v, 4);
          v = __shfl_sync(0xffffffffu, v, 8 * (lane & 3));
          if ((lane >> 2) == c) keep = v;
        }
      } else {
        keep = warp_transpose_bits(bits[q]);
      }
      mine[q] = keep;
    }
  }
  int valid_count = 0;
  const uint32_t tail = (P & 31) ? ((1u << (P & 31)) - 1u) : 0xffffffffu;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int j = q * 32 + lane;
    if (j < words) {
      if (j == words - 1) mine[q] &= tail;  // no bits past particle P-1
      p.valid_out[(long long)w * words + j] = mine[q];
      valid_count += __popc(mine[q]);
    }
  }
  valid_count = __reduce_add_sync(0xffffffffu, valid_count);
  const float cp = ((float)(P - valid_count)) / P;
  if (lane == 0) {
    p.cp_out[w] = cp;
    if (overflow && p.error) atomicExch(p.error, (int)PUMP_ERR_CAPACITY);
  }
  if (Epi) {
    // PUMP.cu:164-185: time, cost and the CP cut-off of new path w
    const float time = __uint_as_float(__shfl_sync(0xffffffffu, epi, 0));
    const float topt = __uint_as_float(__shfl_sync(0xffffffffu, epi, 1));
    const float cost = __uint_as_float(__shfl_sync(0xffffffffu, epi, 2));
    const float copt = __uint_as_float(__shfl_sync(0xffffffffu, epi, 3));
    const int node = (int)__shfl_sync(0xffffffffu, epi, 4);
    if (lane == 0) {
      const HsmcEpilogue &e = p.epi;
      e.new_time[w] = time + topt;
      e.new_cost[w] = cost + copt;
      const bool alive = !(cp > e.cp_cutoff);
      e.alive[w] = alive ? 1 : 0;
      if (alive) e.new_next[w] = atomicExch(&e.new_head[node], w);
    }
  }
}

// The chunk's paths, every step-th one below n from the block's counter on, by
// its warps, each taking the next one when it is free.  (Taking the next
// path ahead, to load its edge and parent during the one before, lets a warp
// with a long path hold back another: 12 % more for 12,000 such paths.)
template <bool Boxes, int Q, bool Epi>
__device__ __forceinline__ void hsmc_chunk_paths(const HsmcParams &p, unsigned step, int n, unsigned *s_next,
                                                 const float *s_obs, float4 *hs, uint8_t *hcnt, int *klist) {
  while (true) {
    unsigned w = 0u;
    if ((threadIdx.x & 31) == 0) w = atomicAdd(s_next, step);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= (unsigned)n) break;  // warp-uniform
    hsmc_path<Boxes, Q, Epi>(p, (int)w, p.wf_edge[w], p.wf_prev[w], s_obs, hs, hcnt, klist);
    __syncwarp();  // the warp's half-space slots are rewritten by its next path
  }
}

template <bool Boxes, int Q, bool Epi>
__device__ __forceinline__ void hsmc_run(const HsmcParams &p) {
  extern __shared__ float4 s_dyn4[];
  const int warp = threadIdx.x >> 5;
  int n = p.num_new;
  if (p.num_new_dev) n = (p.skip_dev && *p.skip_dev) ? 0 : (int)*p.num_new_dev;
  // more blocks than resident ones: runs of consecutive paths
  const bool runs = gridDim.x > (unsigned)kHsmcPersistBlocks;
  unsigned step = 1u;
  if (!runs) step = (unsigned)hsmc_chunks(n, gridDim.x, true);
  // a block with no path leaves before staging anything (block-uniform)
  if (!runs && blockIdx.x >= step) return;
  const unsigned first = blockIdx.x * (runs ? (unsigned)kHsmcRun : 1u);
  if (runs) n = (unsigned)n - first < (unsigned)kHsmcRun ? n : (int)(first + kHsmcRun);
  __shared__ unsigned s_next;
  if (threadIdx.x == 0) s_next = first;
  float *s_obs = reinterpret_cast<float *>(s_dyn4);
  float4 *hs = nullptr;
  uint8_t *hcnt = nullptr;
  int *klist = nullptr;
  if (Boxes) {
    stage_obstacles(p.obs, p.numObs, s_obs);  // block-wide, before any warp leaves
    const int hs_stride = hsmc_hs_stride(p.W, p.maxHS), cnt_stride = hsmc_cnt_stride(p.W);
    float4 *s_hs = reinterpret_cast<float4 *>(s_obs + hsmc_boxes_obs_floats(p.numObs));
    hs = s_hs + warp * hs_stride;
    uint8_t *s_cnt = reinterpret_cast<uint8_t *>(s_hs + kHsmcWarps * hs_stride);
    hcnt = s_cnt + warp * cnt_stride;
    int *s_klist = reinterpret_cast<int *>(s_cnt + kHsmcWarps * cnt_stride);
    klist = s_klist + warp * kHsmcFilterObs;
  }
  __syncthreads();
  hsmc_chunk_paths<Boxes, Q, Epi>(p, step, n, &s_next, s_obs, hs, hcnt, klist);
}

// Q = 32-bit particle words per lane: P <= 1024 Q.
template <bool Boxes, int Q, bool Epi>
__global__ void __launch_bounds__(kHsmcThreads, 8) hsmc_kernel(const HsmcParams p) {
  hsmc_run<Boxes, Q, Epi>(p);
}

// Out of line: the loop kernel's own state is saved once per chunk, not spilled
// around the tests (N = 32000, 4096 particles, when every box was tested:
// the whole query 266 ms inlined, 247 so).
template <int Q>
__device__ __noinline__ void hsmc_loop_paths(const HsmcParams &p, unsigned step, int n, unsigned *s_next,
                                             const float *s_obs, float4 *hs, uint8_t *hcnt, int *klist) {
  hsmc_chunk_paths<true, Q, true>(p, step, n, s_next, s_obs, hs, hcnt, klist);
}

// The search loop on the device, for every query of a group: the chunks of
// the active queries' wavefronts in query order are the blocks' work items,
// taken in turn (grid-stride).  A block stages a query's parameters (the
// stored-path count, the bound on parents, from its loop state) and boxes
// when its next chunk belongs to another query.  The shared memory holds the
// layout of the group's largest box count, waypoint count and half-space
// count.
template <int Q>
__global__ void __launch_bounds__(kHsmcThreads, 8) hsmc_loop_kernel(const LoopGroup *g) {
  extern __shared__ float4 s_dyn4[];
  __shared__ int s_first[kLoopGroupMax + 1];  // first chunk of each query
  __shared__ HsmcParams s_p;
  __shared__ unsigned s_next;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = g->nq;
  const int share = (int)gridDim.x > nq ? (int)gridDim.x / nq : 1;  // blocks per query
  if (warp == 0) {
    int c = 0;
    if (lane < nq) {
      const LoopArgs *a = g->args[lane];
      if (*reinterpret_cast<const volatile int *>(&a->L.active)) {
        const HsmcParams &hp = a->hp;
        const int n = (hp.skip_dev && *hp.skip_dev) ? 0 : (int)*hp.num_new_dev;
        c = hsmc_chunks(n, share, nq == 1);
      }
    }
    // inclusive scan over the queries (nq <= 32 lanes)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, c, o);
      if (lane >= o) c += u;
    }
    if (lane == 0) s_first[0] = 0;
    if (lane < kLoopGroupMax) s_first[lane + 1] = c;
  }
  __syncthreads();
  const int total = s_first[nq];
  // a block with no chunk leaves before staging anything (block-uniform)
  if ((int)blockIdx.x >= total) return;
  float *s_obs = reinterpret_cast<float *>(s_dyn4);
  int cur = -1;
  for (int ch = blockIdx.x; ch < total; ch += gridDim.x) {  // block-uniform
    int q = 0;
    while (q + 1 < nq && s_first[q + 1] <= ch) ++q;
    __syncthreads();  // every warp is done with the previous chunk (its counter, its query)
    if (q != cur) {
      if (warp == 0) {  // the query's parameters, word by word
        static_assert(sizeof(HsmcParams) % sizeof(int) == 0, "HsmcParams words");
        const int *src = reinterpret_cast<const int *>(&g->args[q]->hp);
        int *dst = reinterpret_cast<int *>(&s_p);
        for (int i = lane; i < (int)(sizeof(HsmcParams) / sizeof(int)); i += 32) dst[i] = src[i];
        __syncwarp();
        if (lane == 0) s_p.num_prev = g->args[q]->L.num_paths;
      }
      __syncthreads();
      stage_obstacles(s_p.obs, s_p.numObs, s_obs);  // ends with a barrier
      cur = q;
    }
    if (threadIdx.x == 0) s_next = (unsigned)(ch - s_first[q]);
    __syncthreads();
    const HsmcParams &p = s_p;
    // this query's layout of the shared memory
    const int hs_stride = hsmc_hs_stride(p.W, p.maxHS), cnt_stride = hsmc_cnt_stride(p.W);
    float4 *s_hs = reinterpret_cast<float4 *>(s_obs + hsmc_boxes_obs_floats(p.numObs));
    uint8_t *s_cnt = reinterpret_cast<uint8_t *>(s_hs + kHsmcWarps * hs_stride);
    int *s_klist = reinterpret_cast<int *>(s_cnt + kHsmcWarps * cnt_stride);
    const int n = (p.skip_dev && *p.skip_dev) ? 0 : (int)*p.num_new_dev;
    hsmc_loop_paths<Q>(p, (unsigned)hsmc_chunks(n, share, nq == 1), n, &s_next, s_obs, s_hs + warp * hs_stride,
                       s_cnt + warp * cnt_stride, s_klist + warp * kHsmcFilterObs);
  }
}

// The kernel of P particles (Q = ceil(P / 1024), 1, 2 or 4).
inline int hsmc_q(int P) {
  const int q = (P + 1023) / 1024;
  return q <= 1 ? 1 : (q <= 2 ? 2 : 4);
}
template <bool Boxes, bool Epi>
const void *hsmc_kernel_for(int P) {
  switch (hsmc_q(P)) {
    case 1: return (const void *)hsmc_kernel<Boxes, 1, Epi>;
    case 2: return (const void *)hsmc_kernel<Boxes, 2, Epi>;
    default: return (const void *)hsmc_kernel<Boxes, 4, Epi>;
  }
}
inline const void *hsmc_loop_kernel_for(int P) {
  switch (hsmc_q(P)) {
    case 1: return (const void *)hsmc_loop_kernel<1>;
    case 2: return (const void *)hsmc_loop_kernel<2>;
    default: return (const void *)hsmc_loop_kernel<4>;
  }
}

// -------------------------------------------------------------- MC CP
// collisionProbability.cu:39-92.  A particle collides when any of the
// segments t = 0 .. T-3 of its perturbed path hits a box; the reference walks
// the segments in order and stops at the first hit, which gives the same
// answer as testing all of them.
//
// Block = 32 K particles (K per lane) of one path x kMcWarps warps, which
// split the path's segments into consecutive runs (a run carries a segment's
// end over as the next one's start).  Per segment the warp takes the bounding
// box of its particles' segments by warp reductions, tests the boxes against it
// one per lane, and only those that it is not broadphase-disjoint from are
// tested per particle: a box disjoint
// from the common bounding box is disjoint from every particle's, whose
// reference test then passes.  With a NaN coordinate every box is kept.  (One
// particle per lane and every box tested by every particle: 268 us for 64
// paths x 2048 particles and 40 boxes, 45 us so.)  Bound by instruction issue for large
// calls, by one warp's chain of segments for small ones; hence K: particles
// per lane share the reductions and box tests of a large call (K = 4), and a
// small call spreads over the SMs (K = 1).
constexpr int kMcWarps = 16;

// Grid (ceil(Pmc / (32 K)), paths).
template <int K>
__global__ void __launch_bounds__(32 * kMcWarps) mc_cp_kernel(
    const float *__restrict__ paths, const int *__restrict__ offset, const int *__restrict__ len,
    const float *__restrict__ offsets_t, int Pmc, int T_rows, float offset_mult,
    const float *__restrict__ obs, int numObs, int k0, int *__restrict__ hits,
    const int *copy_src, int *copy_dst, int copy_words, unsigned int *done, unsigned int seq) {
  extern __shared__ float4 s_obs4[];
  float *s_obs = reinterpret_cast<float *>(s_obs4);
  __shared__ unsigned int s_hit[K][kMcWarps];
  stage_obstacles(obs, numObs, s_obs);
  const int path_k = k0 + blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p0 = blockIdx.x * (32 * K) + lane;
  const int T = len[path_k];
  const float *path = paths + (long long)offset[path_k] * kDim;
  const int segs = T <= T_rows ? T - 2 : 0;
  const int per = segs > 0 ? (segs + kMcWarps - 1) / kMcWarps : 0;
  const int t0 = warp * per, t1 = t0 + per < segs ? t0 + per : segs;
  unsigned int todo = 0u;  // bit k: particle p0 + 32 k exists and has not collided
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (p0 + 32 * k < Pmc) todo |= 1u << k;
  unsigned int coll = 0u;
  float v[K][3], w[K][3];
  auto load = [&](int t, float (&x)[K][3]) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int p = p0 + 32 * k < Pmc ? p0 + 32 * k : Pmc - 1;
#pragma unroll
      for (int d = 0; d < 3; ++d)
        x[k][d] = path[t * kDim + d] + __ldg(&offsets_t[((long long)t * Pmc + p) * 3 + d]) * offset_mult;
    }
  };
  struct Ends {
    float lo[3], hi[3], sum;
  };
  auto ends = [&](const float (&x)[K][3]) {
    Ends e;
    e.sum = 0.0f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      e.lo[d] = e.hi[d] = x[0][d];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        e.sum += x[k][d];  // (infinities of both signs also keep every box)
        if (k > 0) {
          e.lo[d] = fminf(e.lo[d], x[k][d]);
          e.hi[d] = fmaxf(e.hi[d], x[k][d]);
        }
      }
    }
    return e;
  };
  Ends ve{};
  if (t0 < t1) {
    load(t0, v);
    ve = ends(v);
    if (K == 1) load(t0 + 1, w);
  }
  for (int t = t0; t < t1; ++t) {
    if (!__any_sync(0xffffffffu, todo != 0u)) break;
    // one particle per lane: the next segment's end is on its way during the
    // tests (a small call waits on these loads)
    float next[K][3];
    if (K > 1) load(t + 1, w);
    else if (t + 1 < t1) load(t + 2, next);
    // the lane's particles' bounding box, from those of the segment's two
    // ends (the start's was the end's before); a NaN coordinate shows in the sum
    const Ends we = ends(w);
    const bool nan = __any_sync(0xffffffffu, ve.sum != ve.sum || we.sum != we.sum);
    float lo[3], hi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[d] = warp_min_f32(fminf(ve.lo[d], we.lo[d]));
      hi[d] = warp_max_f32(fmaxf(ve.hi[d], we.hi[d]));
    }
    ve = we;
    for (int c0 = 0; c0 < numObs; c0 += 32) {
      bool keep = false;
      if (c0 + lane < numObs) {
        const float4 *bx = s_obs4 + (c0 + lane) * 3;
        const float4 a = bx[0], b = bx[1], c = bx[2];  // lo = a.xyz, hi = (b.z, b.w, c.x)
        keep = nan || !((hi[0] <= a.x) | (b.z <= lo[0]) | (hi[1] <= a.y) | (b.w <= lo[1]) |
                        (hi[2] <= a.z) | (c.x <= lo[2]));
      }
      unsigned int boxes = __ballot_sync(0xffffffffu, keep);
      while (boxes) {
        const float *ob = &s_obs[(c0 + __ffs(boxes) - 1) * 12];
        boxes &= boxes - 1u;
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (((todo >> k) & 1u) && segment_box_hit(v[k], w[k], ob)) {
            coll |= 1u << k;
            todo &= ~(1u << k);
          }
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int d = 0; d < 3; ++d) v[k][d] = w[k][d];
    if (K == 1 && t + 1 < t1)
#pragma unroll
      for (int d = 0; d < 3; ++d) w[0][d] = next[0][d];
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const unsigned int bal = __ballot_sync(0xffffffffu, (coll >> k) & 1u);
    if (lane == 0) s_hit[k][warp] = bal;
  }
  __syncthreads();
  if (warp == 0) {
    int total = 0;
    if (lane < K) {
      unsigned int any = 0;
      for (int q = 0; q < kMcWarps; ++q) any |= s_hit[lane][q];
      total = __popc(any);
    }
    total = __reduce_add_sync(0xffffffffu, total);
    if (lane == 0 && total) atomicAdd(&hits[path_k], total);
  }
  if (copy_dst) {
    // the last block to finish copies the caller's results (hit counts
    // included) to host memory
    __shared__ bool s_last;
    if (threadIdx.x == 0) {
      __threadfence();
      s_last = atomicAdd(done, 1u) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (s_last) {
      __threadfence();
      const volatile int *src = copy_src;
      for (int i = threadIdx.x; i < copy_words; i += blockDim.x) copy_dst[i] = src[i];
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence_system();
        // then the sequence word after the copy, for a host that waits on it
        *reinterpret_cast<volatile unsigned int *>(copy_dst + copy_words) = seq;
      }
    }
  }
}

__global__ void mc_cp_finish_kernel(const int *__restrict__ hits, const int *__restrict__ len,
                                    int n, int Pmc, int T_rows, float *__restrict__ cp,
                                    int *__restrict__ error) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  cp[k] = ((float)hits[k]) / ((float)Pmc);
  if (len[k] > T_rows && error) atomicExch(error, (int)PUMP_ERR_CAPACITY);
}

}  // namespace

pump_status_t mc_cp_hits_async(const float *d_paths, const int *d_offset, const int *d_len,
                               int n_paths, const float *d_offsets_t, int Pmc, int T_rows,
                               float offset_mult, const float *d_obstacles, int numObs,
                               int *d_hits, cudaStream_t stream, const int *copy_src,
                               int *copy_dst, int copy_words, unsigned int *done,
                               unsigned int seq) {
  if (n_paths <= 0) return PUMP_OK;
  if (copy_dst && n_paths > 65535)
    return set_error(PUMP_ERR_BAD_INPUT, "mc_cp: copy-out with %d paths", n_paths);
  const size_t smem = sizeof(float) * (size_t)((numObs * 12 + 3) & ~3);
  if (smem > 200 * 1024) return set_error(PUMP_ERR_CAPACITY, "mc_cp: %d obstacles", numObs);
  auto go = [&](auto per_lane) -> pump_status_t {
    constexpr int K = decltype(per_lane)::value;
    PUMP_TRY(smem_attr((const void *)mc_cp_kernel<K>, smem));
    for (int k0 = 0; k0 < n_paths; k0 += 65535) {
      const int nk = n_paths - k0 < 65535 ? n_paths - k0 : 65535;
      dim3 grid(grid_for(Pmc, 32 * K), (unsigned)nk);
      mc_cp_kernel<K><<<grid, 32 * kMcWarps, smem, stream>>>(
          d_paths, d_offset, d_len, d_offsets_t, Pmc, T_rows, offset_mult, d_obstacles, numObs, k0,
          d_hits, copy_src, copy_dst, copy_words, done, seq);
      PUMP_TRY(launch_status("mc_cp_kernel"));
    }
    return PUMP_OK;
  };
  // particles per lane: four once one per lane is two rounds of its resident
  // blocks (two an SM) and four still leave every SM a block: 8 paths x 4096
  // particles, 1 and 10 boxes, 23 and 24 us with one, 17 and 19 with four.
  const long long blocks = (long long)n_paths * grid_for(Pmc, 32);
  if (blocks >= 4LL * kNumSMs) return go(std::integral_constant<int, 4>{});
  return go(std::integral_constant<int, 1>{});
}

pump_status_t mc_cp_async(const float *d_paths, const int *d_offset, const int *d_len, int n_paths,
                          const float *d_offsets_t, int Pmc, int T_rows, float offset_mult,
                          const float *d_obstacles, int numObs, int *d_hits, float *d_cp,
                          int *d_error, cudaStream_t stream) {
  if (n_paths <= 0) return PUMP_OK;
  PUMP_CUDA_TRY(cudaMemsetAsync(d_hits, 0, sizeof(int) * n_paths, stream));
  PUMP_TRY(mc_cp_hits_async(d_paths, d_offset, d_len, n_paths, d_offsets_t, Pmc, T_rows,
                            offset_mult, d_obstacles, numObs, d_hits, stream, nullptr, nullptr, 0,
                            nullptr, 0u));
  mc_cp_finish_kernel<<<grid_for(n_paths, 128), 128, 0, stream>>>(d_hits, d_len, n_paths, Pmc,
                                                                  T_rows, d_cp, d_error);
  return launch_status("mc_cp_finish_kernel");
}

pump_status_t hsmc_staged_async(int num_new, int W, const int *d_edge, const int *d_prev,
                                long long num_edges, int num_prev, const float *d_as, const float *d_bs, int maxHS,
                                const float *d_times, const float *d_topt, float dt,
                                const float *d_offsets_t, int Pmc, int T_rows, float offset_mult,
                                const uint32_t *d_valid_in, uint32_t *d_valid_out, int P,
                                float *d_cp_out, int *d_error, const uint8_t *d_hs_count,
                                cudaStream_t stream, const unsigned long long *d_num_new,
                                const int *d_skip) {
  if (num_new <= 0) return PUMP_OK;
  if ((P + 31) / 32 > kMaxHsmcWords)
    return set_error(PUMP_ERR_CAPACITY, "hsmc: %d particles exceed %d", P, 32 * kMaxHsmcWords);
  if (W * maxHS > kMaxHsSlots)
    return set_error(PUMP_ERR_CAPACITY, "hsmc: %d half-space slots per edge exceed %d", W * maxHS,
                     kMaxHsSlots);
  HsmcParams hp{};
  hp.num_new = num_new;
  hp.W = W;
  hp.wf_edge = d_edge;
  hp.wf_prev = d_prev;
  hp.num_edges = num_edges;
  hp.num_prev = num_prev;
  hp.as = d_as;
  hp.bs = d_bs;
  hp.hs_count = d_hs_count;
  hp.maxHS = maxHS;
  hp.times = d_times;
  hp.topts = d_topt;
  hp.dt = dt;
  hp.offsets_t = d_offsets_t;
  hp.Pmc = Pmc;
  hp.T_rows = T_rows;
  hp.offset_mult = offset_mult;
  hp.valid_in = d_valid_in;
  hp.valid_out = d_valid_out;
  hp.P = P;
  hp.cp_out = d_cp_out;
  hp.error = d_error;
  hp.num_new_dev = d_num_new;
  hp.skip_dev = d_skip;
  // (with a device-side count, num_new bounds it)
  const unsigned blocks = hsmc_blocks(num_new, d_num_new != nullptr);
  void *args[] = {(void *)&hp};
  PUMP_CUDA_TRY(cudaLaunchKernel(hsmc_kernel_for<false, false>(P), dim3(blocks), dim3(kHsmcThreads), args,
                                 0, stream));
  return launch_status("hsmc_kernel");
}

bool hsmc_boxes_fits(int numObs, int W, int maxHS) {
  return numObs >= 0 && W <= kMaxHsSlots && W * maxHS <= kMaxHsSlots &&
         hsmc_boxes_smem(numObs, W, maxHS) <= 220 * 1024;
}

pump_status_t hsmc_boxes_fill(int num_new, int W, const int *d_edge, const int *d_prev,
                              long long num_edges, int num_prev, const float *d_obs, int numObs,
                              const float *d_disc, float maxd2, int maxHS, const float *d_times,
                              const float *d_topt, float dt, const float *d_offsets_t, int Pmc,
                              int T_rows, float offset_mult, const uint32_t *d_valid_in,
                              uint32_t *d_valid_out, int P, float *d_cp_out, int *d_error,
                              const unsigned long long *d_num_new, const int *d_skip,
                              const HsmcEpilogue *epi, HsmcParams *out,
                              const long long *d_disc_off) {
  if ((P + 31) / 32 > kMaxHsmcWords)
    return set_error(PUMP_ERR_CAPACITY, "hsmc: %d particles exceed %d", P, 32 * kMaxHsmcWords);
  if (!hsmc_boxes_fits(numObs, W, maxHS))
    return set_error(PUMP_ERR_CAPACITY, "hsmc: %d boxes or %d half-space slots per edge exceed the stage",
                     numObs, W * maxHS);
  HsmcParams hp{};
  hp.num_new = num_new;
  hp.W = W;
  hp.wf_edge = d_edge;
  hp.wf_prev = d_prev;
  hp.num_edges = num_edges;
  hp.num_prev = num_prev;
  hp.obs = d_obs;
  hp.numObs = numObs;
  hp.disc = d_disc;
  hp.disc_off = d_disc_off;
  hp.maxd2 = maxd2;
  hp.maxHS = maxHS;
  hp.times = d_times;
  hp.topts = d_topt;
  hp.dt = dt;
  hp.offsets_t = d_offsets_t;
  hp.Pmc = Pmc;
  hp.T_rows = T_rows;
  hp.offset_mult = offset_mult;
  hp.valid_in = d_valid_in;
  hp.valid_out = d_valid_out;
  hp.P = P;
  hp.cp_out = d_cp_out;
  hp.error = d_error;
  hp.num_new_dev = d_num_new;
  hp.skip_dev = d_skip;
  if (epi) hp.epi = *epi;
  *out = hp;
  return PUMP_OK;
}

pump_status_t hsmc_boxes_async(int num_new, int W, const int *d_edge, const int *d_prev,
                               long long num_edges, int num_prev, const float *d_obs, int numObs,
                               const float *d_disc, float maxd2, int maxHS, const float *d_times,
                               const float *d_topt, float dt, const float *d_offsets_t, int Pmc,
                               int T_rows, float offset_mult, const uint32_t *d_valid_in,
                               uint32_t *d_valid_out, int P, float *d_cp_out, int *d_error,
                               cudaStream_t stream, const unsigned long long *d_num_new,
                               const int *d_skip, const HsmcEpilogue *epi,
                               const long long *d_disc_off) {
  if (num_new <= 0) return PUMP_OK;
  HsmcParams hp{};
  PUMP_TRY(hsmc_boxes_fill(num_new, W, d_edge, d_prev, num_edges, num_prev, d_obs, numObs, d_disc,
                           maxd2, maxHS, d_times, d_topt, dt, d_offsets_t, Pmc, T_rows, offset_mult,
                           d_valid_in, d_valid_out, P, d_cp_out, d_error, d_num_new, d_skip, epi,
                           &hp, d_disc_off));
  const size_t smem = hsmc_boxes_smem(numObs, W, maxHS);
  const void *kern = epi ? hsmc_kernel_for<true, true>(P) : hsmc_kernel_for<true, false>(P);
  PUMP_TRY(smem_attr(kern, smem));
  // (with a device-side count, num_new bounds it)
  const unsigned blocks = hsmc_blocks(num_new, d_num_new != nullptr);
  void *args[] = {(void *)&hp};
  PUMP_CUDA_TRY(cudaLaunchKernel(kern, dim3(blocks), dim3(kHsmcThreads), args, smem, stream));
  return launch_status("hsmc_kernel (boxes)");
}

pump_status_t hsmc_loop_prepare(int numObs, int W, int maxHS, int P) {
  return smem_attr(hsmc_loop_kernel_for(P), hsmc_boxes_smem(numObs, W, maxHS));
}

pump_status_t hsmc_loop_launch(const LoopGroup *d_group, int numObs, int W, int maxHS, int P,
                               int blocks, cudaStream_t stream) {
  void *args[] = {(void *)&d_group};
  PUMP_CUDA_TRY(cudaLaunchKernel(hsmc_loop_kernel_for(P), dim3(blocks), dim3(kHsmcThreads), args,
                                 hsmc_boxes_smem(numObs, W, maxHS), stream));
  return launch_status("hsmc_loop_kernel");
}

// Generates the tables on `stream`; the binary64 noise buffer (24 B per
// particle and step) is allocated and freed in stream order.
pump_status_t particle_tables_async(uint64_t seed, int P, int T, float *d_tmajor, float *d_pmajor,
                                    cudaStream_t stream) {
  double *z = nullptr;
  PUMP_CUDA_TRY(pool_malloc_async((void **)&z, sizeof(double) * 3 * (size_t)P * T, stream));
  particle_gauss_kernel<<<grid_for((long long)P * T, 256), 256, 0, stream>>>(
      (uint32_t)seed, (uint32_t)(seed >> 32), P, T, z);
  pump_status_t st = launch_status("particle_gauss_kernel");
  if (st == PUMP_OK) {
    particle_table_kernel<<<grid_for((long long)P * 3, 128), 128, 0, stream>>>(z, P, T, d_tmajor,
                                                                              d_pmajor);
    st = launch_status("particle_table_kernel");
  }
  cudaFreeAsync(z, stream);
  return st;
}

}  // namespace pump

using namespace pump;

extern "C" pump_status_t pump_particle_tables(uint64_t seed, int P, int T, float *d_tmajor,
                                              float *d_pmajor, pump_stream_t stream) {
  if (P <= 0 || T <= 0 || (!d_tmajor && !d_pmajor))
    return set_error(PUMP_ERR_BAD_INPUT, "pump_particle_tables: bad arguments");
  return particle_tables_async(seed, P, T, d_tmajor, d_pmajor, (cudaStream_t)stream);
}

extern "C" pump_status_t pump_position_variance(int T, double *d_var, pump_stream_t stream) {
  if (T <= 0 || !d_var) return set_error(PUMP_ERR_BAD_INPUT, "pump_position_variance: bad arguments");
  position_variance_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(T, d_var);
  return launch_status("position_variance");
}

extern "C" pump_status_t pump_hsmc_propagate(int num_new, int W, const int *d_edge, const int *d_prev,
                                             long long num_edges, int base, const float *d_as,
                                             const float *d_bs,
                                             int maxHS, const float *d_times, const float *d_topt,
                                             float dt, const float *d_offsets_t, int Pmc,
                                             int T_rows, float offset_mult, uint32_t *d_valid,
                                             int P, float *d_path_cp, int *d_error,
                                             const uint8_t *d_hs_count, pump_stream_t stream) {
  if (num_new < 0 || W < 2 || maxHS < 0 || P <= 0 || P > Pmc || T_rows <= 0 || base < 0 ||
      num_edges < 0 ||
      (num_new > 0 && (!d_edge || !d_prev || !d_times || !d_topt || !d_offsets_t || !d_valid ||
                       !d_path_cp || (maxHS > 0 && (!d_as || !d_bs)))))
    return set_error(PUMP_ERR_BAD_INPUT, "pump_hsmc_propagate: bad arguments");
  const size_t words = (size_t)((P + 31) / 32);
  return hsmc_staged_async(num_new, W, d_edge, d_prev, num_edges, base, d_as, d_bs, maxHS, d_times,
                           d_topt, dt,
                           d_offsets_t, Pmc, T_rows, offset_mult, d_valid,
                           d_valid + (size_t)base * words, P, d_path_cp + base, d_error,
                           d_hs_count, (cudaStream_t)stream, nullptr, nullptr);
}

extern "C" pump_status_t pump_hsmc_propagate_boxes_off(
    int num_new, int max_w, const int *d_edge, const int *d_prev, long long num_edges, int base,
    const float *d_obstacles, int numObs, const float *d_disc, const long long *d_disc_off,
    float maxd2, int maxHS, const float *d_times, const float *d_topt, float dt,
    const float *d_offsets_t, int Pmc, int T_rows, float offset_mult, uint32_t *d_valid, int P,
    float *d_path_cp, int *d_error, pump_stream_t stream) {
  if (num_new < 0 || max_w < 2 || maxHS < 0 || P <= 0 || P > Pmc || T_rows <= 0 || base < 0 ||
      num_edges < 0 || numObs < 0 || (numObs > 0 && !d_obstacles) ||
      (num_new > 0 && (!d_edge || !d_prev || !d_times || !d_topt || !d_offsets_t || !d_valid ||
                       !d_path_cp || !d_disc || !d_disc_off)))
    return set_error(PUMP_ERR_BAD_INPUT, "pump_hsmc_propagate_boxes_off: bad arguments");
  const size_t words = (size_t)((P + 31) / 32);
  return hsmc_boxes_async(num_new, max_w, d_edge, d_prev, num_edges, base, d_obstacles, numObs,
                          d_disc, maxd2, maxHS, d_times, d_topt, dt, d_offsets_t, Pmc, T_rows,
                          offset_mult, d_valid, d_valid + (size_t)base * words, P, d_path_cp + base,
                          d_error, (cudaStream_t)stream, nullptr, nullptr, nullptr, d_disc_off);
}

extern "C" pump_status_t pump_hsmc_propagate_boxes(
    int num_new, int W, const int *d_edge, const int *d_prev, long long num_edges, int base,
    const float *d_obstacles, int numObs, const float *d_disc, float maxd2, int maxHS,
    const float *d_times, const float *d_topt, float dt, const float *d_offsets_t, int Pmc,
    int T_rows, float offset_mult, uint32_t *d_valid, int P, float *d_path_cp, int *d_error,
    pump_stream_t stream) {
  if (num_new < 0 || W < 2 || maxHS < 0 || P <= 0 || P > Pmc || T_rows <= 0 || base < 0 ||
      num_edges < 0 || numObs < 0 || (numObs > 0 && !d_obstacles) ||
      (num_new > 0 && (!d_edge || !d_prev || !d_times || !d_topt || !d_offsets_t || !d_valid ||
                       !d_path_cp || !d_disc)))
    return set_error(PUMP_ERR_BAD_INPUT, "pump_hsmc_propagate_boxes: bad arguments");
  const size_t words = (size_t)((P + 31) / 32);
  return hsmc_boxes_async(num_new, W, d_edge, d_prev, num_edges, base, d_obstacles, numObs, d_disc,
                          maxd2, maxHS, d_times, d_topt, dt, d_offsets_t, Pmc, T_rows, offset_mult,
                          d_valid, d_valid + (size_t)base * words, P, d_path_cp + base, d_error,
                          (cudaStream_t)stream, nullptr, nullptr, nullptr, nullptr);
}

extern "C" pump_status_t pump_mc_cp(const float *d_paths, const int *d_offset, const int *d_len,
                                    int n_paths, const float *d_offsets_t, int Pmc, int T_rows,
                                    float offset_mult, const float *d_obstacles, int numObs,
                                    int *d_hits, float *d_cp, int *d_error, pump_stream_t stream) {
  if (n_paths < 0 || Pmc <= 0 || T_rows <= 0 || numObs < 0 || (numObs > 0 && !d_obstacles) ||
      (n_paths > 0 && (!d_paths || !d_offset || !d_len || !d_offsets_t || !d_hits || !d_cp)))
    return set_error(PUMP_ERR_BAD_INPUT, "pump_mc_cp: bad arguments");
  return mc_cp_async(d_paths, d_offset, d_len, n_paths, d_offsets_t, Pmc, T_rows, offset_mult,
                     d_obstacles, numObs, d_hits, d_cp, d_error, (cudaStream_t)stream);
}
