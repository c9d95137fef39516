// mc_philox.cu - FP32 Philox Monte Carlo: the strike strip and the batched book.
//
// Generator: Philox4x32-10, counter {draw block, sample lo, sample hi, stream},
// key = the 64-bit seed; one call yields 4 draws (4 GBM steps or 2 Heston
// steps).  GBM and Heston Euler turn each draw pair into two normals by
// Box-Muller; Heston QE keeps the inverse CDF, which its variance step
// needs (the same uniform drives the exponential branch and, through
// Phi^-1, the quadratic one).  Paths live in registers (one path per thread at a time), payoff
// sums are compensated FP32 per thread and FP64 from the warp level up.
// Compiled with -use_fast_math: sqrt/exp/log/div map to single MUFU
// operations; the few places that need more accuracy say so.
#include <cuda.h>  // CUcontext / CUresult types only; the driver functions are resolved at run time

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

#include "book_greeks.cuh"
#include "bulk_copy.cuh"
#include "of_internal.h"
#include "path_fp32.cuh"

using of::LegState;
using of::StepConsts;

namespace {

constexpr uint32_t kStripStreamTag = 0x53545250u;  // "STRP"

// FP32 constants of a model (computed in FP64, rounded once).
StepConsts make_consts(const of_model* m) {
  StepConsts c{};
  const double dt = m->maturity / (double)m->steps;
  const double sqdt = std::sqrt(dt);
  c.drift = (float)((m->mu - 0.5 * m->sigma * m->sigma) * dt);
  c.diff = (float)(m->sigma * sqdt);
  c.mudt = (float)(m->mu * dt);
  c.half_dt = (float)(0.5 * dt);
  c.sqdt = (float)sqdt;
  c.kdt = (float)(m->kappa * dt);
  c.kdt_theta = (float)(m->kappa * m->theta * dt);
  c.one_m_kdt = (float)(1.0 - m->kappa * dt);
  c.xi = (float)m->xi;
  c.bm_k2 = (float)(-2.0 * 0.69314718055994531 * dt);
  c.rho = (float)m->rho;
  c.rho_c = (float)std::sqrt(1.0 - m->rho * m->rho);
  c.v0 = (float)m->v0;
  c.y_floor = (float)std::log(1e-12 / m->s0);  // s.max(1e-12), simulation.rs:112
  if (m->kind == OF_MODEL_HESTON_QE) {
    const double e = std::exp(-m->kappa * dt);
    c.qe_e = (float)e;
    c.qe_c1 = (float)(m->xi * m->xi * e * (1.0 - e) / m->kappa);
    c.qe_c2 = (float)(m->theta * m->xi * m->xi * (1.0 - e) * (1.0 - e) / (2.0 * m->kappa));
    c.qe_theta = (float)m->theta;
    const double g1 = 0.5, g2 = 0.5, kr = m->kappa * m->rho / m->xi - 0.5;
    c.qe_k0 = (float)(-m->rho * m->kappa * m->theta * dt / m->xi);
    c.qe_k1 = (float)(g1 * dt * kr - m->rho / m->xi);
    c.qe_k2 = (float)(g2 * dt * kr + m->rho / m->xi);
    c.qe_k3 = (float)(g1 * dt * (1.0 - m->rho * m->rho));
    c.qe_k4 = (float)(g2 * dt * (1.0 - m->rho * m->rho));
  }
  return c;
}

// A GBM sample's sum of normals grows by a counter block's four at a time, two
// Box-Muller pair sums in one product and one fma, and by the last, partial
// block's `rem`.  Every rounding is written out, for the compiler contracts
// packed and scalar products with the sum that follows differently: the same
// bits in every strip shape, one sample (gbm_add_block) or two in packed pairs
// (gbm_add_block2).  The fma takes the first pair, which is ready first: the
// other order cost two samples 1 %.
__device__ __forceinline__ float gbm_add_block(float w, const uint4 r) {
  float2 q, s;
  of::normal_pair_sum_factors2_from_u32(r.x, r.y, r.z, r.w, q, s);
  return __fadd_rn(w, fmaf(q.x, s.x, __fmul_rn(q.y, s.y)));
}

__device__ __forceinline__ float2 gbm_add_block2(float2 w, const uint4 r0, const uint4 r1) {
  float2 q01, s01, q23, s23;
  of::normal_pair_sum_factors2_from_u32(r0.x, r0.y, r1.x, r1.y, q01, s01);
  of::normal_pair_sum_factors2_from_u32(r0.z, r0.w, r1.z, r1.w, q23, s23);
  return of::add2(w, of::fma2(q01, s01, of::mul2(q23, s23)));
}

__device__ __forceinline__ float gbm_add_last(float w, const uint4 r, int32_t rem) {
  if (rem == 1) return __fadd_rn(w, of::normal_pair_from_u32(r.x, r.y).x);
  w = __fadd_rn(w, of::normal_pair_sum_from_u32(r.x, r.y));
  return rem == 3 ? __fadd_rn(w, of::normal_pair_from_u32(r.z, r.w).x) : w;
}

// Simulates the terminal log-returns of ILP samples (and of their antithetic
// twins) in one loop: the Philox rounds of the samples are separate dependency
// chains, so their instructions interleave and fill the gaps of one chain, and
// they share each counter block's q terms.  Two samples run in packed pairs
// (each half the one-sample loop's arithmetic, bit for bit) except Heston's
// antithetic ones, whose four legs fit the register budget without the pair
// alignment, and QE.
// FULL: the q table covers every counter block.
template <int MODEL, bool ANTI, int ILP, bool FULL>
__device__ __forceinline__ void simulate_terminal(const StepConsts& c, int32_t steps, const of::PhiloxLane (&L)[ILP],
                                                  const of::PhiloxTab& T, const of::PhiloxKeys& K, float (&ya)[ILP],
                                                  float (&yb)[ILP]) {
  if constexpr (MODEL == OF_MODEL_GBM) {
    // y_T = steps drift + diff sum z; each Box-Muller pair enters as its sum
    // (normal_pair_sum_from_u32), four steps a counter block
    float sum[ILP];
    const int32_t full = steps >> 2;
    if constexpr (ILP == 1) {
      sum[0] = 0.0f;
      for (int32_t q = 0; q < full; ++q)
        sum[0] = gbm_add_block(sum[0], of::philox_block(of::philox_terms<FULL>(T, (uint32_t)q, K), L[0], K));
    } else {
      float2 w = make_float2(0.0f, 0.0f);
      for (int32_t q = 0; q < full; ++q) {
        const uint4 t = of::philox_terms<FULL>(T, (uint32_t)q, K);
        w = gbm_add_block2(w, of::philox_block(t, L[0], K), of::philox_block(t, L[1], K));
      }
      sum[0] = w.x;
      sum[1] = w.y;
    }
    if (const int32_t rem = steps & 3) {
      const uint4 t = of::philox_terms<FULL>(T, (uint32_t)full, K);
#pragma unroll
      for (int l = 0; l < ILP; ++l) sum[l] = gbm_add_last(sum[l], of::philox_block(t, L[l], K), rem);
    }
    const float base = (float)steps * c.drift;
#pragma unroll
    for (int l = 0; l < ILP; ++l) {
      ya[l] = fmaf(c.diff, sum[l], base);
      yb[l] = fmaf(-c.diff, sum[l], base);
    }
  } else if constexpr (MODEL == OF_MODEL_HESTON_EULER && ILP == 2 && !ANTI) {
    of::LegState2 a{make_float2(0.0f, 0.0f), make_float2(c.v0, c.v0)};
    const int32_t pairs = steps >> 1;  // full Philox calls; an odd last step below
    for (int32_t q = 0; q < pairs; ++q) {
      const uint4 t = of::philox_terms<FULL>(T, (uint32_t)q, K);
      const uint4 r0 = of::philox_block(t, L[0], K), r1 = of::philox_block(t, L[1], K);
      of::heston_euler_step2(a, c, of::polars2_from_u32(r0.x, r0.y, r1.x, r1.y, c.bm_k2));
      of::heston_euler_step2(a, c, of::polars2_from_u32(r0.z, r0.w, r1.z, r1.w, c.bm_k2));
    }
    if (steps & 1) {
      const uint4 t = of::philox_terms<FULL>(T, (uint32_t)pairs, K);
      const uint4 r0 = of::philox_block(t, L[0], K), r1 = of::philox_block(t, L[1], K);
      of::heston_euler_step2(a, c, of::polars2_from_u32(r0.x, r0.y, r1.x, r1.y, c.bm_k2));
    }
    ya[0] = a.y.x;  // yb stays 0: there is no antithetic leg
    ya[1] = a.y.y;
  } else if constexpr (MODEL == OF_MODEL_HESTON_QE && ILP > 1) {  // one after the other: two QE samples spill
    for (int l = 0; l < ILP; ++l) {
      const of::PhiloxLane L1[1] = {L[l]};
      float a1[1], b1[1];
      simulate_terminal<MODEL, ANTI, 1, FULL>(c, steps, L1, T, K, a1, b1);
      ya[l] = a1[0];
      yb[l] = b1[0];
    }
  } else {
    LegState a[ILP], b[ILP];
#pragma unroll
    for (int l = 0; l < ILP; ++l) a[l] = b[l] = LegState{0.0f, c.v0};
    auto step = [&](int l, uint32_t r0, uint32_t r1) {
      if (MODEL == OF_MODEL_HESTON_EULER) {
        const of::Polar z = of::polar_from_u32(r0, r1, c.bm_k2);
        of::heston_euler_step(a[l], c, z.q, z.c, z.s);
        if (ANTI) of::heston_euler_step(b[l], c, z.q, -z.c, -z.s);
      } else {
        const float u = of::uniform_from_u32(r0), zx = of::normal_from_u32(r1);
        of::heston_qe_step(a[l], c, u, 1.0f, zx, r0);
        if (ANTI) of::heston_qe_step(b[l], c, 1.0f - u, -1.0f, -zx, r0);
      }
    };
    const int32_t pairs = steps >> 1;
    for (int32_t q = 0; q < pairs; ++q) {
      const uint4 t = of::philox_terms<FULL>(T, (uint32_t)q, K);
#pragma unroll
      for (int l = 0; l < ILP; ++l) {
        const uint4 r = of::philox_block(t, L[l], K);
        step(l, r.x, r.y);
        step(l, r.z, r.w);
      }
    }
    if (steps & 1) {
      const uint4 t = of::philox_terms<FULL>(T, (uint32_t)pairs, K);
#pragma unroll
      for (int l = 0; l < ILP; ++l) {
        const uint4 r = of::philox_block(t, L[l], K);
        step(l, r.x, r.y);
      }
    }
#pragma unroll
    for (int l = 0; l < ILP; ++l) {
      ya[l] = a[l].y;
      yb[l] = b[l].y;
    }
  }
}

// ---------------------------------------------------------------------------
// Strike strip: one shared path set, KPL strikes per lane.
// ---------------------------------------------------------------------------
struct StripParams {
  StepConsts c;
  int64_t samples;
  int32_t steps, n_strikes, option_type, antithetic;
  float s0;
  of::PhiloxKeys keys;
  uint32_t* status;  // warp-specialised kernel: nonzero when a ring wait gave up
  unsigned* ticket;  // last block adds the rows of partials into `out` (strip_fused), or null
  double* out;       // [2 n_strikes]
  float strikes[128];
};

// Whether the block that finishes last adds the blocks' rows: each of its
// threads then adds rows / strip_row_groups of them, about 0.4 us per 16 (one
// trip to the L2); past 96 a reduction launch with a block per column is
// quicker.
constexpr int kStripThreads = 256;
__host__ __device__ inline int strip_row_groups(int cols) { return kStripThreads / cols < 8 ? kStripThreads / cols : 8; }
inline bool strip_fused(int64_t grid, int cols) { return grid <= 96 * (int64_t)strip_row_groups(cols); }

// The last block's part (called by all threads of every block): `sh` holds
// strip_row_groups(cols) x cols doubles.
__device__ __forceinline__ void strip_finish(const StripParams& P, int cols, const double* __restrict__ partials,
                                             double* sh) {
  __shared__ bool last;
  __threadfence();  // this thread's columns of the block's row
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(P.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int groups = strip_row_groups(cols);
  if ((int)threadIdx.x < groups * cols) {
    const int col = threadIdx.x % cols;
    double acc = 0.0;
    for (unsigned r = threadIdx.x / cols; r < gridDim.x; r += 16 * groups) {
      double v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const unsigned row = r + k * groups;
        v[k] = row < gridDim.x ? __ldcg(partials + (size_t)row * cols + col) : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 16; ++k) acc += v[k];
    }
    sh[threadIdx.x] = acc;
  }
  __syncthreads();
  if ((int)threadIdx.x < cols) {
    double acc = 0.0;
    for (int g = 0; g < groups; ++g) acc += sh[g * cols + threadIdx.x];
    P.out[threadIdx.x] = acc;
    __threadfence_system();
  }
  if (threadIdx.x == 0) *P.ticket = 0;
}

// Counter blocks in the q table of the strip (28 KB, four blocks an SM beside
// the sums of 128 strikes): 7,168 GBM or 3,584 Heston steps.  Past it the terms
// are computed in place behind a range test, which costs more than the table
// saves where the warps are few: Heston, 65,536 x 1,024 steps x 41 strikes, took
// 181 us with 256 entries and 158 with all of its 512 (172 before there was a
// table).  A second loop without the test cost the strips that fit 1 %.
constexpr uint32_t kStripTab = 1792;

// KPL 0: one strike, whose sums each lane keeps for its own samples (no
// shuffles; for one strike these took longer than 16 steps).
//
// What bounds it: the FMA pipe's heavy half, 75-80 % busy, with Philox's 15
// wide products of four cycles per counter block and half of the FP32
// operations.  At 2^20 samples x 256 steps x 41 strikes, four blocks per SM and
// two samples per thread: Heston Euler 475 us (548 before the q tables, the
// shared square root, the funnel shifts and the even rounds; 529 and 573 with
// one sample per thread), GBM 217 (288).
template <int KPL, int MODEL, bool ANTI, int ILP = 1>
__global__ void __launch_bounds__(kStripThreads, 4) strip_kernel(const __grid_constant__ StripParams P,
                                                    double* __restrict__ partials) {
  extern __shared__ double sh_strip[];  // [warps][n_strikes][2]
  __shared__ uint4 qtab[kStripTab];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  constexpr int KA = KPL > 0 ? KPL : 1;
  float K[KA];
  of::KahanSq32 acc[KA];
#pragma unroll
  for (int q = 0; q < KA; ++q) {
    const int k = KPL > 0 ? lane + 32 * q : 0;
    K[q] = k < P.n_strikes ? P.strikes[k] : 0.0f;
  }
  const bool call = P.option_type == OF_CALL;
  constexpr int kSpb = MODEL == OF_MODEL_GBM ? 4 : 2;  // steps per counter block
  const uint32_t nq = ((uint32_t)P.steps + kSpb - 1) / kSpb;
  of::PhiloxTab T{qtab, nq < kStripTab ? nq : kStripTab, 0u, kStripStreamTag};
  of::philox_table_fill(qtab, T.n, T.hi, T.stream, P.keys);
  __syncthreads();
  // a warp round covers 32*ILP consecutive samples: lane + 32*l for l < ILP.
  // They share the high word of their index: 2^32 is a multiple of a round.
  // Rounds go to warp 0 of every block, then warp 1 of every block, ...: a
  // last partial round then loads every SM alike, wherever its blocks run
  // (block by block, the busiest SM had 16 % more rounds than the mean).
  const int64_t nwarps = (int64_t)gridDim.x * nw;
  for (int64_t base = ((int64_t)warp * gridDim.x + blockIdx.x) * 32 * ILP; base < P.samples;
       base += nwarps * 32 * ILP) {
    of::PhiloxLane L[ILP];
    float ya[ILP], yb[ILP], sa[ILP], sb[ILP];
    if (const uint32_t hi = (uint32_t)(base >> 32)) {  // past 2^32 samples: the table's hi is 0
      T.hi = hi;
      T.n = 0;
    }
#pragma unroll
    for (int l = 0; l < ILP; ++l) {
      L[l] = of::philox_lane((uint32_t)(base + lane + 32 * l), T.hi, P.keys);
      ya[l] = yb[l] = 0.0f;
    }
    if (base + lane < P.samples) {  // lanes past the end skip the paths; their shuffled values are unused
      if (T.n == nq) simulate_terminal<MODEL, ANTI, ILP, true>(P.c, P.steps, L, T, P.keys, ya, yb);
      else simulate_terminal<MODEL, ANTI, ILP, false>(P.c, P.steps, L, T, P.keys, ya, yb);
    }
#pragma unroll
    for (int l = 0; l < ILP; ++l) {  // rounded before a strike is taken off, with one strike as with several
      sa[l] = __fmul_rn(P.s0, __expf(ya[l]));
      sb[l] = __fmul_rn(P.s0, __expf(yb[l]));
    }
#pragma unroll
    for (int l = 0; l < ILP; ++l) {
      const int64_t rem = P.samples - (base + 32 * l);
      const int nvalid = rem < 0 ? 0 : (rem < 32 ? (int)rem : 32);
      if constexpr (KPL == 0) {
        float x = fmaxf(call ? sa[l] - K[0] : K[0] - sa[l], 0.0f);
        if (ANTI) x = 0.5f * (x + fmaxf(call ? sb[l] - K[0] : K[0] - sb[l], 0.0f));
        if (lane < nvalid) acc[0].add(x);
        continue;
      }
      for (int j = 0; j < nvalid; ++j) {
        const float st = __shfl_sync(of::kFullMask, sa[l], j);
        const float sta = ANTI ? __shfl_sync(of::kFullMask, sb[l], j) : 0.0f;
#pragma unroll
        for (int q = 0; q < KPL; ++q) {
          float x = fmaxf(call ? st - K[q] : K[q] - st, 0.0f);
          if (ANTI) x = 0.5f * (x + fmaxf(call ? sta - K[q] : K[q] - sta, 0.0f));
          acc[q].add(x);
        }
      }
    }
  }
  const int n = P.n_strikes;
  if constexpr (KPL == 0) {
    double v[2] = {acc[0].value(), acc[0].square()};
    of::block_sum<2>(v, sh_strip);
    if (threadIdx.x == 0) {
      partials[(int64_t)blockIdx.x * 2] = v[0];
      partials[(int64_t)blockIdx.x * 2 + 1] = v[1];
    }
  } else {
#pragma unroll
    for (int q = 0; q < KPL; ++q) {
      const int k = lane + 32 * q;
      if (k < n) {
        sh_strip[(warp * n + k) * 2] = acc[q].value();
        sh_strip[(warp * n + k) * 2 + 1] = acc[q].square();
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 2 * n; t += blockDim.x) {
      double sum = 0.0;
      for (int w = 0; w < nw; ++w) sum += sh_strip[w * 2 * n + t];
      partials[(int64_t)blockIdx.x * 2 * n + t] = sum;
    }
  }
  if (P.ticket) strip_finish(P, 2 * n, partials, sh_strip);
}

// ---------------------------------------------------------------------------
// Warp-specialised strike strip (tile_ilp = 3).
//
// The step loop of strip_kernel alternates two instruction mixes: the Philox
// rounds (32x32->64 integer multiplies on the FMA-heavy pipe, three-input
// XORs on the ALU) and the Box-Muller pair plus the Heston step (lg2, sqrt,
// sin, cos and sqrt on the MUFU pipe, FP32 FMAs).  All warps of an SM run the
// same phase at about the same time, so one pipe waits while the other is
// saturated.  Here half of the warps only generate: producer warp c + 4
// computes the Philox blocks of the 32 samples its consumer warp c simulates
// and writes them to a ring in shared memory; the consumer warps only turn
// draws into normals, steps and payoffs.  The scheduler then always has
// warps of both mixes to issue.  Same draws, same steps and same payoffs per
// sample as strip_kernel<..., ILP = 1>; the per-warp sums group samples
// differently, so results agree to the rounding of the FP32 partial sums.
//
// Ring: per consumer kWsSlots chunks of kWsChunk Philox blocks x 32 lanes
// (uint4), with a full and an empty mbarrier per chunk (32 arrivals each).
// Every wait is bounded (kWsWaitNs of the global timer), suspends the warp in
// the barrier between polls so a waiting warp leaves the issue slots to
// working ones, and its outcome is made warp-uniform; a warp whose wait gives up sets P.status and leaves its
// loops, so its partner's next wait gives up too and the block still reaches
// its final reduction.
// ---------------------------------------------------------------------------
constexpr int kWsPairs = 4;   // consumer warps 0..3, producer warps 4..7
constexpr int kWsChunk = 4;   // Philox blocks per ring chunk
constexpr int kWsSlots = 3;   // chunks in flight per pair
constexpr uint64_t kWsWaitNs = 1000000000ull;
constexpr uint32_t kWsSleepNs = 20000;  // suspend-time hint of a ring barrier poll
constexpr size_t kWsRingBytes = (size_t)kWsPairs * kWsSlots * kWsChunk * 32 * sizeof(uint4);

// The steps of Philox block q of one sample (and its antithetic twin), as
// simulate_terminal consumes them.
template <int MODEL, bool ANTI>
__device__ __forceinline__ void ws_consume(const StepConsts& c, const uint4 r, int32_t q, int32_t steps,
                                           LegState& a, LegState& b, float& w) {
  if (MODEL == OF_MODEL_GBM) {
    const int32_t rem = steps - 4 * q;
    w = rem >= 4 ? gbm_add_block(w, r) : gbm_add_last(w, r, rem);
  } else if (MODEL == OF_MODEL_HESTON_EULER) {
    of::Polar z = of::polar_from_u32(r.x, r.y, c.bm_k2);
    of::heston_euler_step(a, c, z.q, z.c, z.s);
    if (ANTI) of::heston_euler_step(b, c, z.q, -z.c, -z.s);
    if (2 * q + 1 < steps) {
      z = of::polar_from_u32(r.z, r.w, c.bm_k2);
      of::heston_euler_step(a, c, z.q, z.c, z.s);
      if (ANTI) of::heston_euler_step(b, c, z.q, -z.c, -z.s);
    }
  } else {
    float u = of::uniform_from_u32(r.x), zx = of::normal_from_u32(r.y);
    of::heston_qe_step(a, c, u, 1.0f, zx, r.x);
    if (ANTI) of::heston_qe_step(b, c, 1.0f - u, -1.0f, -zx, r.x);
    if (2 * q + 1 < steps) {
      u = of::uniform_from_u32(r.z);
      zx = of::normal_from_u32(r.w);
      of::heston_qe_step(a, c, u, 1.0f, zx, r.z);
      if (ANTI) of::heston_qe_step(b, c, 1.0f - u, -1.0f, -zx, r.z);
    }
  }
}

template <int KPL, int MODEL, bool ANTI>
__global__ void __launch_bounds__(256, 5) strip_kernel_ws(const __grid_constant__ StripParams P,
                                                       double* __restrict__ partials) {
  extern __shared__ __align__(16) unsigned char ws_smem[];
  uint4* ring = reinterpret_cast<uint4*>(ws_smem);                       // [pair][slot][block][lane]
  double* sh_strip = reinterpret_cast<double*>(ws_smem + kWsRingBytes);  // [warps][n_strikes][2]
  __shared__ __align__(8) uint64_t full[kWsPairs * kWsSlots], empty[kWsPairs * kWsSlots];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const bool producer = warp >= kWsPairs;
  const int pair = producer ? warp - kWsPairs : warp;
  if (threadIdx.x == 0) {
    for (int k = 0; k < kWsPairs * kWsSlots; ++k) {
      of::mbar_init(of::smem_u32(full + k), 32);
      of::mbar_init(of::smem_u32(empty + k), 32);
    }
    of::mbar_fence_init();
  }
  __syncthreads();
  float K[KPL];
  of::KahanSq32 acc[KPL];
#pragma unroll
  for (int q = 0; q < KPL; ++q) {
    const int k = lane + 32 * q;
    K[q] = k < P.n_strikes ? P.strikes[k] : 0.0f;
  }
  const bool call = P.option_type == OF_CALL;
  const int32_t spb = MODEL == OF_MODEL_GBM ? 4 : 2;  // steps per Philox block
  const int32_t nq = (P.steps + spb - 1) / spb;       // Philox blocks per sample
  const int64_t stride = (int64_t)gridDim.x * kWsPairs * 32;
  uint4* my_ring = ring + (size_t)pair * kWsSlots * kWsChunk * 32;
  uint32_t g = 0;  // chunks this pair has passed through its ring
  bool ok = true;
  for (int64_t base = ((int64_t)blockIdx.x * kWsPairs + pair) * 32; base < P.samples && ok; base += stride) {
    const uint64_t i = (uint64_t)(base + lane);
    const uint32_t lo = (uint32_t)i, hi = (uint32_t)(i >> 32);
    LegState a{0.0f, P.c.v0}, b{0.0f, P.c.v0};
    float w = 0.0f;
    for (int32_t q0 = 0; q0 < nq; q0 += kWsChunk, ++g) {
      const int slot = (int)(g % kWsSlots);
      const uint32_t use = g / kWsSlots;
      uint4* chunk = my_ring + (size_t)slot * kWsChunk * 32;
      if (producer) {
        const bool free_ok =
            use == 0 || of::mbar_wait_backoff(of::smem_u32(empty + pair * kWsSlots + slot), (use - 1) & 1u,
                                              kWsWaitNs, kWsSleepNs);
        if (!__all_sync(of::kFullMask, free_ok)) {  // the warp leaves together
          ok = false;
          break;
        }
#pragma unroll
        for (int k = 0; k < kWsChunk; ++k)
          if (q0 + k < nq)
            chunk[k * 32 + lane] = of::philox4x32_10(make_uint4((uint32_t)(q0 + k), lo, hi, kStripStreamTag), P.keys);
        of::mbar_arrive(of::smem_u32(full + pair * kWsSlots + slot));
      } else {
        const bool full_ok =
            of::mbar_wait_backoff(of::smem_u32(full + pair * kWsSlots + slot), use & 1u, kWsWaitNs, kWsSleepNs);
        if (!__all_sync(of::kFullMask, full_ok)) {
          ok = false;
          break;
        }
#pragma unroll
        for (int k = 0; k < kWsChunk; ++k)
          if (q0 + k < nq) ws_consume<MODEL, ANTI>(P.c, chunk[k * 32 + lane], q0 + k, P.steps, a, b, w);
        of::mbar_arrive(of::smem_u32(empty + pair * kWsSlots + slot));
      }
    }
    if (producer || !ok) continue;
    float ya, yb;
    if (MODEL == OF_MODEL_GBM) {
      const float basev = (float)P.steps * P.c.drift;
      ya = fmaf(P.c.diff, w, basev);
      yb = fmaf(-P.c.diff, w, basev);
    } else {
      ya = a.y;
      yb = b.y;
    }
    const float sa = P.s0 * __expf(ya), sb = P.s0 * __expf(yb);
    const int64_t rem = P.samples - base;
    const int nvalid = rem < 32 ? (int)rem : 32;
    for (int j = 0; j < nvalid; ++j) {
      const float st = __shfl_sync(of::kFullMask, sa, j);
      const float sta = ANTI ? __shfl_sync(of::kFullMask, sb, j) : 0.0f;
#pragma unroll
      for (int q = 0; q < KPL; ++q) {
        float x = fmaxf(call ? st - K[q] : K[q] - st, 0.0f);
        if (ANTI) x = 0.5f * (x + fmaxf(call ? sta - K[q] : K[q] - sta, 0.0f));
        acc[q].add(x);
      }
    }
  }
  if (!ok && lane == 0) atomicOr(P.status, 1u);
  const int n = P.n_strikes;
#pragma unroll
  for (int q = 0; q < KPL; ++q) {
    const int k = lane + 32 * q;
    if (k < n) {
      sh_strip[(warp * n + k) * 2] = acc[q].value();
      sh_strip[(warp * n + k) * 2 + 1] = acc[q].square();
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 2 * n; t += blockDim.x) {
    double acc = 0.0;
    for (int w2 = 0; w2 < nw; ++w2) acc += sh_strip[w2 * 2 * n + t];
    partials[(int64_t)blockIdx.x * 2 * n + t] = acc;
  }
}

typedef void (*StripKernelFn)(StripParams, double*);

template <int KPL, int ILP = 1>
StripKernelFn pick_strip(int model, bool anti) {
  if (model == OF_MODEL_GBM)
    return anti ? strip_kernel<KPL, OF_MODEL_GBM, true, ILP> : strip_kernel<KPL, OF_MODEL_GBM, false, ILP>;
  if (model == OF_MODEL_HESTON_EULER)
    return anti ? strip_kernel<KPL, OF_MODEL_HESTON_EULER, true, ILP>
                : strip_kernel<KPL, OF_MODEL_HESTON_EULER, false, ILP>;
  return anti ? strip_kernel<KPL, OF_MODEL_HESTON_QE, true, ILP> : strip_kernel<KPL, OF_MODEL_HESTON_QE, false, ILP>;
}

template <int KPL>
StripKernelFn pick_strip_ws_kpl(int model, bool anti) {
  if (model == OF_MODEL_GBM) return anti ? strip_kernel_ws<KPL, OF_MODEL_GBM, true> : strip_kernel_ws<KPL, OF_MODEL_GBM, false>;
  if (model == OF_MODEL_HESTON_EULER)
    return anti ? strip_kernel_ws<KPL, OF_MODEL_HESTON_EULER, true> : strip_kernel_ws<KPL, OF_MODEL_HESTON_EULER, false>;
  return anti ? strip_kernel_ws<KPL, OF_MODEL_HESTON_QE, true> : strip_kernel_ws<KPL, OF_MODEL_HESTON_QE, false>;
}

StripKernelFn pick_strip_ilp(int kpl, int ilp, int model, bool anti);

// The kernel, its dynamic shared memory and the samples one block covers per
// round, for a strip tile shape: tile 1 or 2 = strip_kernel with that many
// samples in flight per thread (0: strip_default_tile), tile 3 = the
// warp-specialised strip_kernel_ws.
struct StripShape {
  StripKernelFn fn;
  size_t smem;
  int64_t samples_per_block;
  bool ws;
};

// tile 0: two samples per thread where the samples fill the resident threads
// (four blocks per SM) twice over, one below that, where more warps matter,
// and for QE, whose two samples run one after the other.  2^20 samples of 256
// steps, one / two: Heston 529 / 475 us, GBM 234 / 217, QE 1160 / 1202; 2^19
// antithetic pairs: Heston 329 / 311, GBM 133 / 125.
int strip_default_tile(int64_t samples, int model, int sms) {
  return model != OF_MODEL_HESTON_QE && samples >= (int64_t)sms * 4 * kStripThreads * 2 ? 2 : 1;
}

StripShape strip_shape(int tile, int64_t samples, int64_t n_strikes, int model, bool anti, int sms) {
  constexpr int block = kStripThreads;
  const int kpl = n_strikes == 1 ? 0 : (int)((n_strikes + 31) / 32);
  const size_t sums = (size_t)(block / 32) * (size_t)n_strikes * 2 * sizeof(double);
  if (tile == 3) {
    const StripKernelFn fn = kpl <= 1 ? pick_strip_ws_kpl<1>(model, anti)
                             : kpl <= 2 ? pick_strip_ws_kpl<2>(model, anti) : pick_strip_ws_kpl<4>(model, anti);
    return {fn, kWsRingBytes + sums, (int64_t)kWsPairs * 32, true};
  }
  const int ilp = tile ? tile : strip_default_tile(samples, model, sms);
  return {pick_strip_ilp(kpl, ilp, model, anti), sums, (int64_t)block * ilp, false};
}

// Blocks: enough for the samples, at most the resident ones; few samples are
// spread over all SMs, some warps of each block idle.
int strip_grid(const StripShape& sh, int64_t samples, int sms, int per_sm) {
  const int64_t want = (samples + sh.samples_per_block - 1) / sh.samples_per_block;
  const int64_t rounds = (samples + 31) / 32;
  const int64_t spread = sh.ws ? want : std::max(want, std::min<int64_t>(sms, rounds));
  return (int)std::max<int64_t>(1, std::min(spread, (int64_t)sms * per_sm));
}

// Kernel for KPL strikes per lane and ILP samples in flight per thread.
StripKernelFn pick_strip_ilp(int kpl, int ilp, int model, bool anti) {
  if (ilp == 2) {
    if (kpl == 0) return pick_strip<0, 2>(model, anti);
    if (kpl <= 1) return pick_strip<1, 2>(model, anti);
    if (kpl <= 2) return pick_strip<2, 2>(model, anti);
    return pick_strip<4, 2>(model, anti);
  }
  if (kpl == 0) return pick_strip<0>(model, anti);
  if (kpl <= 1) return pick_strip<1>(model, anti);
  if (kpl <= 2) return pick_strip<2>(model, anti);
  return pick_strip<4>(model, anti);
}

}  // namespace

of_status of_validate_mc(of_ctx* ctx, const of_model* m, const of_payoff* p, const of_mc_config* c);
void of_observation_weights(const of_payoff* p, int64_t steps, std::vector<double>& w, bool& terminal_only);

static of_status validate_fp32_model(of_ctx* ctx, const of_model* m) {
  if (m->steps > 2147483647LL) return of_fail(ctx, OF_ERR_INVALID_INPUT, "num_steps too large for FP32 mode");
  if (m->kind == OF_MODEL_HESTON_QE && !(m->xi > 0.0 && m->theta > 0.0))
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "the QE scheme needs xi > 0 and theta > 0");
  return OF_OK;
}

struct of_strip_plan {
  of_ctx* ctx = nullptr;
  StripParams P{};
  int n_strikes = 0, grid = 0, block = 256;
  size_t smem = 0;
  StripKernelFn fn = nullptr;
  bool ws = false;  // warp-specialised kernel: clears and reads back the status word after the sums
  double discount = 1.0;
  int64_t samples = 0;
  double* d_partials = nullptr;
  double* d_sums = nullptr;
  double* h_sums = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

// The sums go to h_sums (pinned), from the kernel's last block or from the
// reduction launch; behind the 2n sums follows one more double whose first
// word is the status of the warp-specialised kernel (from d_sums).
static of_status strip_enqueue(of_strip_plan* pl, cudaStream_t s) {
  const int64_t cols = 2 * (int64_t)pl->n_strikes;
  if (pl->ws) cudaMemsetAsync(pl->d_sums + cols, 0, sizeof(double), s);
  pl->fn<<<pl->grid, pl->block, pl->smem, s>>>(pl->P, pl->d_partials);
  if (!pl->P.ticket) of_launch_reduce_rows(pl->d_partials, pl->grid, cols, pl->h_sums, s);
  if (pl->ws)
    cudaMemcpyAsync(pl->h_sums + cols, pl->d_sums + cols, sizeof(double), cudaMemcpyDeviceToHost, s);
  return OF_OK;
}

// OF_ERR_TIMEOUT when the warp-specialised kernel's ring gave up.
static of_status strip_status(of_ctx* ctx, const of_strip_plan* pl) {
  if (pl->ws && *(const uint32_t*)(pl->h_sums + 2 * pl->n_strikes))
    return of_fail(ctx, OF_ERR_TIMEOUT, "strike strip: a producer/consumer ring wait did not complete in time");
  return OF_OK;
}

extern "C" void of_strip_plan_destroy(of_strip_plan* pl) {
  if (!pl) return;
  if (pl->ctx) cudaStreamSynchronize(pl->ctx->stream);
  if (pl->exec) cudaGraphExecDestroy(pl->exec);
  if (pl->graph) cudaGraphDestroy(pl->graph);
  cudaFree(pl->d_partials);
  cudaFree(pl->d_sums);
  if (pl->h_sums) cudaFreeHost(pl->h_sums);
  delete pl;
}

// Checks of a strip request that need no device: every strip entry point
// (of_mc_strip, the plans, of_mc_strip_noalloc) runs exactly these.  `ctx`
// only receives the message; it may be a stack context that owns nothing.
static of_status strip_validate(of_ctx* ctx, const of_model* m, int32_t option_type, const double* strikes,
                                int64_t n_strikes, const of_mc_config* cfg) {
  if (!m || !cfg) return of_fail(ctx, OF_ERR_INVALID_INPUT, "null argument");
  of_payoff dummy{};
  dummy.kind = OF_PAYOFF_VANILLA;
  dummy.option_type = option_type;
  dummy.strike = 1.0;
  OF_TRY(of_validate_mc(ctx, m, &dummy, cfg));
  OF_TRY(validate_fp32_model(ctx, m));
  if (m->n_dividends > 0)  // the strip keeps only the sum of the normals of a GBM path
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "the strike strip takes no discrete dividends (price them as a book)");
  if (n_strikes <= 0 || !strikes) return of_fail(ctx, OF_ERR_INVALID_INPUT, "strip needs at least one strike");
  if (n_strikes > 128) return of_fail(ctx, OF_ERR_UNSUPPORTED, "strip supports at most 128 strikes per call");
  for (int64_t k = 0; k < n_strikes; ++k)
    if (!(strikes[k] > 0.0) || !std::isfinite(strikes[k]))
      return of_fail(ctx, OF_ERR_INVALID_INPUT, "strike %lld must be finite and > 0", (long long)k);
  if (cfg->control_variate != OF_CV_NONE)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "the strike strip has no control variate");
  if (cfg->injected_normals)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "injected normals are a FP64 reference-mode test hook");
  if (cfg->tile_ilp < 0 || cfg->tile_ilp > 3)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "tile_ilp must be 0 (default), 1, 2 or 3");
  return OF_OK;
}

// Validates a strip request and fills the plan's parameters, kernel and
// launch shape (no allocation).
static of_status strip_setup(of_ctx* ctx, const of_model* m, int32_t option_type, const double* strikes,
                             int64_t n_strikes, const of_mc_config* cfg, of_strip_plan* pl) {
  OF_TRY(strip_validate(ctx, m, option_type, strikes, n_strikes, cfg));
  OF_TRY(of_ctx_check(ctx));
  OF_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  pl->ctx = ctx;
  pl->n_strikes = (int)n_strikes;
  pl->discount = cfg->discount_factor;
  pl->samples = cfg->antithetic ? (cfg->num_paths + 1) / 2 : cfg->num_paths;
  StripParams& P = pl->P;
  P.c = make_consts(m);
  P.samples = pl->samples;
  P.steps = (int32_t)m->steps;
  P.n_strikes = (int32_t)n_strikes;
  P.option_type = option_type;
  P.antithetic = cfg->antithetic ? 1 : 0;
  P.s0 = (float)m->s0;
  P.keys = of::philox_keys(cfg->seed);
  for (int64_t k = 0; k < n_strikes; ++k) P.strikes[k] = (float)strikes[k];
  const StripShape sh = strip_shape(cfg->tile_ilp, pl->samples, n_strikes, m->kind, P.antithetic, ctx->sm_count);
  pl->fn = sh.fn;
  pl->smem = sh.smem;
  pl->ws = sh.ws;
  const int per_sm = of_blocks_per_sm((const void*)pl->fn, pl->block, pl->smem);
  pl->grid = strip_grid(sh, pl->samples, ctx->sm_count, per_sm);
  return OF_OK;
}

extern "C" of_status of_strip_plan_create(of_ctx* ctx, const of_model* m, int32_t option_type, const double* strikes,
                                          int64_t n_strikes, const of_mc_config* cfg, of_strip_plan** out) {
  if (!ctx || !out) return OF_ERR_INVALID_INPUT;
  *out = nullptr;
  of_strip_plan* pl = new of_strip_plan();
  {
    const of_status st = strip_setup(ctx, m, option_type, strikes, n_strikes, cfg, pl);
    if (st != OF_OK) {
      delete pl;
      return st;
    }
  }
  auto fail = [&](of_status st) {
    of_strip_plan_destroy(pl);
    return st;
  };
  if (cudaMalloc(&pl->d_partials, (size_t)pl->grid * 2 * n_strikes * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&pl->d_sums, (2 * n_strikes + 2) * sizeof(double)) != cudaSuccess ||
      cudaMallocHost(&pl->h_sums, (2 * n_strikes + 1) * sizeof(double)) != cudaSuccess)
    return fail(of_fail(ctx, OF_ERR_ALLOC, "strip plan allocation failed"));
  pl->P.status = (uint32_t*)(pl->d_sums + 2 * n_strikes);
  if (!pl->ws && strip_fused(pl->grid, 2 * (int)n_strikes)) {
    pl->P.ticket = (unsigned*)(pl->d_sums + 2 * n_strikes + 1);
    pl->P.out = pl->h_sums;
  }
  // Capture kernel + reduction + readback once; launches replay the graph.
  // The first launch finds the ticket zeroed: the memset has finished here,
  // whatever the legacy stream holds and whichever stream replays the graph.
  cudaStream_t cap_stream = nullptr;
  if (cudaStreamCreateWithFlags(&cap_stream, cudaStreamNonBlocking) != cudaSuccess)
    return fail(of_fail(ctx, OF_ERR_CUDA, "capture stream creation failed"));
  cudaError_t e = cudaMemsetAsync(pl->d_sums, 0, (2 * n_strikes + 2) * sizeof(double), cap_stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(cap_stream);
  if (e == cudaSuccess) e = cudaStreamBeginCapture(cap_stream, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    strip_enqueue(pl, cap_stream);
    e = cudaStreamEndCapture(cap_stream, &pl->graph);
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&pl->exec, pl->graph, 0);
  cudaStreamDestroy(cap_stream);
  if (e != cudaSuccess) return fail(of_fail(ctx, OF_ERR_CUDA, "strip graph capture failed: %s", cudaGetErrorString(e)));
  *out = pl;
  return OF_OK;
}

extern "C" of_status of_strip_plan_launch(of_strip_plan* pl) {
  if (!pl) return OF_ERR_INVALID_INPUT;
  OF_TRY(of_ctx_check(pl->ctx));
  OF_CUDA_TRY(pl->ctx, cudaGraphLaunch(pl->exec, pl->ctx->stream));
  return OF_OK;
}

extern "C" of_status of_strip_plan_results(of_strip_plan* pl, of_mc_result* res) {
  if (!pl || !res) return OF_ERR_INVALID_INPUT;
  OF_CUDA_TRY(pl->ctx, cudaStreamSynchronize(pl->ctx->stream));
  OF_TRY(strip_status(pl->ctx, pl));
  for (int k = 0; k < pl->n_strikes; ++k) {
    const double s[5] = {pl->h_sums[2 * k], pl->h_sums[2 * k + 1], 0.0, 0.0, 0.0};
    of_mc_finish(s, pl->samples, OF_CV_NONE, 0.0, pl->discount, &res[k]);
    res[k].kernel_ms = 0.0;
  }
  return OF_OK;
}

// One-shot strip: the context's pooled buffers instead of a plan's own, no
// graph (a single replay would not amortise the capture).
extern "C" of_status of_mc_strip(of_ctx* ctx, const of_model* m, int32_t option_type, const double* strikes,
                                 int64_t n_strikes, const of_mc_config* cfg, of_mc_result* results) {
  if (!ctx || !results) return OF_ERR_INVALID_INPUT;
  of_strip_plan pl;  // setup only; buffers come from the context
  OF_TRY(strip_setup(ctx, m, option_type, strikes, n_strikes, cfg, &pl));
  const int64_t cols = 2 * n_strikes;
  void *d_part = nullptr, *d_sums = nullptr, *h = nullptr;
  OF_TRY(of_scratch(ctx, SLOT_PARTIALS, (size_t)pl.grid * cols * sizeof(double), &d_part));
  OF_TRY(of_scratch(ctx, SLOT_SUMS, (size_t)(cols + 1) * sizeof(double), &d_sums));
  OF_TRY(of_pinned(ctx, (size_t)(cols + 1) * sizeof(double), &h));
  pl.P.status = (uint32_t*)((double*)d_sums + cols);
  pl.d_partials = (double*)d_part;
  pl.d_sums = (double*)d_sums;
  pl.h_sums = (double*)h;
  if (!pl.ws && strip_fused(pl.grid, (int)cols)) {
    OF_TRY(of_ticket(ctx, &pl.P.ticket));
    pl.P.out = pl.h_sums;
  }
  OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_start, ctx->stream));
  strip_enqueue(&pl, ctx->stream);
  OF_CUDA_TRY(ctx, cudaGetLastError());
  OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_stop, ctx->stream));
  OF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  float ms = 0.0f;
  OF_CUDA_TRY(ctx, cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
  const of_status st = strip_status(ctx, &pl);
  for (int64_t k = 0; k < n_strikes && st == OF_OK; ++k) {
    const double s[5] = {pl.h_sums[2 * k], pl.h_sums[2 * k + 1], 0.0, 0.0, 0.0};
    of_mc_finish(s, pl.samples, OF_CV_NONE, 0.0, pl.discount, &results[k]);
    results[k].kernel_ms = ms;
  }
  // The buffers belong to the context: detach them before `pl` goes out of scope.
  pl.d_partials = nullptr;
  pl.d_sums = nullptr;
  pl.h_sums = nullptr;
  return st;
}

// ---------------------------------------------------------------------------
// Batched book: persistent kernel over (option, path-block) tiles.
// ---------------------------------------------------------------------------
namespace {

enum : int32_t {
  BF_ANTI = 1,
  BF_UP = 2,
  BF_IN = 4,
  BF_GEOMETRIC = 8,
  BF_FLOATING = 16,
  BF_TERMINAL_ONLY = 32,
  BF_DAILY = 64,        // every step 1..M observed once (daily fixings)
  BF_NEED_ARITH = 128,
  BF_NEED_GEO = 256,
  BF_CALL = 512
};

struct BookOpt {
  StepConsts c;
  int32_t model, payoff, flags, cv_kind;
  int32_t steps;
  int32_t obs_offset;  // into the shared weight array, -1 when unused
  float s0, strike, barrier_y, rebate, inv_nobs;
  uint32_t stream;
  int32_t div_offset, n_div;  // discrete dividend triggers (GBM), in the shared table
  int32_t kind;               // BK_*: which step loop the option needs
};

// Step loops of the book.  GBM options without dividends and without a
// geometric-average control variate get a loop that carries only what their
// payoff reads: nothing per step (vanilla, terminal-only Asian), the barrier
// test, or the daily-fixing arithmetic sum.  Everything else takes the
// general loop.
// BK_ASIAN_DAILY_GEO: a daily-fixing arithmetic Asian that also carries the
// geometric sum of its control variate.
enum : int32_t { BK_GENERIC = 0, BK_TERMINAL = 1, BK_BARRIER = 2, BK_ASIAN_DAILY = 3, BK_ASIAN_DAILY_GEO = 4 };

// A dividend trigger in log-spot form: after step `step`, a cash dividend
// sets y = log(max(e^y - a, 0)) with a = D/S0; a proportional one adds
// a = log(1 - p).
struct BookDiv {
  int32_t step, kind;
  float a, pad;
};

struct BookTile {
  int32_t opt;
  int32_t count;
  int64_t first;
  int32_t slot;  // position of the tile's partials (option-major order)
  int32_t reserved;
};

struct BookParams {
  const BookOpt* opts;
  const BookTile* tiles;
  const float* obs_w;
  const BookDiv* divs;
  int32_t n_tiles;
  int32_t ppt;  // samples per thread per tile (tile = block * ppt samples)
  uint32_t tab;  // entries of the q table in dynamic shared memory
  of::PhiloxKeys keys;
  int* counter;
  double* partials;  // [slot][5]
};

struct PathObs {
  float arith_sum, arith_comp, geo_sum;
  bool hit;
};

__device__ __forceinline__ void book_observe(const BookOpt& o, PathObs& ob, float y, int32_t idx, const float* obs_w) {
  const int f = o.flags;
  if (o.payoff == OF_PAYOFF_BARRIER) ob.hit |= (f & BF_UP) ? (y >= o.barrier_y) : (y <= o.barrier_y);
  if (f & (BF_NEED_ARITH | BF_NEED_GEO)) {
    const float w = (f & BF_DAILY) ? (idx > 0 ? 1.0f : 0.0f) : __ldg(obs_w + o.obs_offset + idx);
    if (w != 0.0f) {
      if (f & BF_NEED_ARITH) {
        const float add = w * __expf(y);
        const float yk = add - ob.arith_comp;
        const float t = ob.arith_sum + yk;
        ob.arith_comp = (t - ob.arith_sum) - yk;
        ob.arith_sum = t;
      }
      if (f & BF_NEED_GEO) ob.geo_sum = fmaf(w, y, ob.geo_sum);
    }
  }
}

__device__ __forceinline__ float vanilla32(bool call, float s, float k) { return fmaxf(call ? s - k : k - s, 0.0f); }

__device__ __forceinline__ void book_payoff(const BookOpt& o, const PathObs& ob, float y, float& x, float& cv) {
  const int f = o.flags;
  const bool call = f & BF_CALL;
  const float st = o.s0 * __expf(y);
  switch (o.payoff) {
    case OF_PAYOFF_VANILLA:
      x = vanilla32(call, st, o.strike);
      break;
    case OF_PAYOFF_BARRIER: {
      const bool active = (f & BF_IN) ? ob.hit : !ob.hit;
      x = active ? vanilla32(call, st, o.strike) : o.rebate;
      break;
    }
    default: {
      float avg;
      if (f & BF_TERMINAL_ONLY) avg = st;
      else if (f & BF_GEOMETRIC) avg = o.s0 * __expf(ob.geo_sum * o.inv_nobs);
      else avg = o.s0 * ((ob.arith_sum - ob.arith_comp) * o.inv_nobs);
      x = (f & BF_FLOATING) ? vanilla32(call, st, avg) : vanilla32(call, avg, o.strike);
    }
  }
  switch (o.cv_kind) {
    case OF_CV_VANILLA_TERMINAL: cv = vanilla32(call, st, o.strike); break;
    case OF_CV_GEOMETRIC_ASIAN:
      cv = vanilla32(call, (f & BF_TERMINAL_ONLY) ? st : o.s0 * __expf(ob.geo_sum * o.inv_nobs), o.strike);
      break;
    case OF_CV_TERMINAL_SPOT: cv = st; break;
    default: cv = 0.0f;
  }
}

// One sample (and its antithetic twin) of option o; returns (x, y).
// DividendEvent::apply_jump (src/market/dividends.rs:76-83) on the log-spot.
__device__ __forceinline__ float book_dividend(const BookDiv& d, float y) {
  return d.kind == OF_DIV_CASH ? __logf(fmaxf(__expf(y) - d.a, 0.0f)) : y + d.a;
}

// DIVS: the option has discrete dividends (GBM only); without them the step
// loop carries no trigger check.
template <int MODEL, bool DIVS, typename GEN>
__device__ __forceinline__ void book_sample(const BookOpt& o, uint64_t i, GEN G, const float* obs_w,
                                            const BookDiv* divs, float& x, float& cvy) {
  const bool anti = o.flags & BF_ANTI;
  const StepConsts& c = o.c;
  LegState a{0.0f, c.v0}, b{0.0f, c.v0};
  PathObs oa{0.0f, 0.0f, 0.0f, false}, obb{0.0f, 0.0f, 0.0f, false};
  book_observe(o, oa, 0.0f, 0, obs_w);
  if (anti) book_observe(o, obb, 0.0f, 0, obs_w);
  const of::PhiloxLane L = G.lane(i);
  int32_t ev = 0;  // next dividend trigger (GBM)
  const bool observe_each = (o.payoff != OF_PAYOFF_VANILLA) || (o.flags & (BF_NEED_ARITH | BF_NEED_GEO));
  constexpr int SPC = MODEL == OF_MODEL_GBM ? 4 : 2;  // steps per Philox call
  for (int32_t j = 0; j < o.steps; j += SPC) {
    const uint4 r = G.block((uint32_t)(j / SPC), L);
    const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
    // Box-Muller normals of the two draw pairs (GBM), their polar form (Heston Euler)
    float2 p01 = make_float2(0.0f, 0.0f), p23 = make_float2(0.0f, 0.0f);
    of::Polar h01{}, h23{};
    if (MODEL == OF_MODEL_GBM) {
      p01 = of::normal_pair_from_u32(r.x, r.y);
      p23 = of::normal_pair_from_u32(r.z, r.w);
    } else if (MODEL == OF_MODEL_HESTON_EULER) {
      h01 = of::polar_from_u32(r.x, r.y, c.bm_k2);
      h23 = of::polar_from_u32(r.z, r.w, c.bm_k2);
    }
#pragma unroll
    for (int q = 0; q < SPC; ++q) {
      if (j + q >= o.steps) break;
      if (MODEL == OF_MODEL_GBM) {
        const float z = q == 0 ? p01.x : q == 1 ? p01.y : q == 2 ? p23.x : p23.y;
        a.y = fmaf(c.diff, z, a.y + c.drift);
        if (anti) b.y = fmaf(-c.diff, z, b.y + c.drift);
        for (; DIVS && ev < o.n_div && divs[o.div_offset + ev].step == j + q; ++ev) {  // mc_engine.rs:157-167
          const BookDiv d = divs[o.div_offset + ev];
          a.y = book_dividend(d, a.y);
          if (anti) b.y = book_dividend(d, b.y);
        }
      } else if (MODEL == OF_MODEL_HESTON_EULER) {
        const of::Polar z = q == 0 ? h01 : h23;
        of::heston_euler_step(a, c, z.q, z.c, z.s);
        if (anti) of::heston_euler_step(b, c, z.q, -z.c, -z.s);
      } else {
        const float u = of::uniform_from_u32(rr[2 * q]), zx = of::normal_from_u32(rr[2 * q + 1]);
        of::heston_qe_step(a, c, u, 1.0f, zx, rr[2 * q]);
        if (anti) of::heston_qe_step(b, c, 1.0f - u, -1.0f, -zx, rr[2 * q]);
      }
      if (observe_each) {
        book_observe(o, oa, a.y, j + q + 1, obs_w);
        if (anti) book_observe(o, obb, b.y, j + q + 1, obs_w);
      }
    }
  }
  book_payoff(o, oa, a.y, x, cvy);
  if (anti) {
    float xb, yb;
    book_payoff(o, obb, b.y, xb, yb);
    x = 0.5f * (x + xb);
    cvy = 0.5f * (cvy + yb);
  }
}

// The GBM step loop of one sample (and its antithetic twin) for the option
// kinds BK_BARRIER, BK_ASIAN_DAILY and BK_ASIAN_DAILY_GEO: the same draws,
// steps and observations as book_sample<OF_MODEL_GBM, false>, bit for bit,
// with the option's payoff and flags resolved at compile time instead of
// tested every step.  Whole Philox counter blocks (four steps) run without a
// bounds test; the last, partial block follows.  BK_TERMINAL options take the
// sum of their normals instead (book_terminal_sum).
template <int KIND, bool TWIN, typename GEN>
__device__ __forceinline__ void book_gbm_legs2(const BookOpt& o, uint64_t i0, uint64_t i1, GEN G,
                                               float2& y, PathObs& oa, PathObs& ob);

// Terminal-only options (BK_TERMINAL) need y_T alone: y_T = steps drift +
// diff sum z.  The sum of the path's normals takes each Box-Muller pair as
// its sum (normal_pair_sum_from_u32), four steps at a time ((z0 + z1) +
// (z2 + z3)); a last partial block of one or three steps adds its odd normal
// from the plain transform.  The antithetic twin has y_T = steps drift -
// diff sum z.  The drift is added once instead of every step, so y_T differs
// from the stepwise sum of the general loop by FP32 rounding only.  The
// packed-pair form below sums in the same order: each of its halves is this
// scalar sum, up to where the compiler contracts a product with the sum.
template <typename GEN>
__device__ __forceinline__ float book_terminal_sum(const BookOpt& o, uint64_t i, GEN G) {
  const of::PhiloxLane L = G.lane(i);
  float w = 0.0f;
  const int32_t full = o.steps & ~3;
  for (int32_t j = 0; j < full; j += 4) {
    const uint4 r = G.block((uint32_t)(j >> 2), L);
    w += of::normal_pair_sum_from_u32(r.x, r.y) + of::normal_pair_sum_from_u32(r.z, r.w);
  }
  const int32_t rem = o.steps - full;
  if (rem > 0) {
    const uint4 r = G.block((uint32_t)(full >> 2), L);
    if (rem == 1) {
      w += of::normal_pair_from_u32(r.x, r.y).x;
    } else {
      w += of::normal_pair_sum_from_u32(r.x, r.y);
      if (rem == 3) w += of::normal_pair_from_u32(r.z, r.w).x;
    }
  }
  return w;
}

// book_terminal_sum of samples i0 and i1 in packed pairs
template <typename GEN>
__device__ __forceinline__ float2 book_terminal_sums2(const BookOpt& o, uint64_t i0, uint64_t i1,
                                                      GEN G) {
  using of::add2;
  const of::PhiloxLane L0 = G.lane(i0), L1 = G.lane(i1);  // i0 and i1 share their high word
  float2 w = make_float2(0.0f, 0.0f);
  const int32_t full = o.steps & ~3;
  for (int32_t j = 0; j < full; j += 4) {
    const uint4 qt = G.terms((uint32_t)(j >> 2));
    const uint4 r0 = of::philox_block(qt, L0, *G.K), r1 = of::philox_block(qt, L1, *G.K);
    w = add2(w, add2(of::normal_pair_sums2_from_u32(r0.x, r0.y, r1.x, r1.y),
                     of::normal_pair_sums2_from_u32(r0.z, r0.w, r1.z, r1.w)));
  }
  const int32_t rem = o.steps - full;
  if (rem > 0) {
    const uint4 qt = G.terms((uint32_t)(full >> 2));
    const uint4 r0 = of::philox_block(qt, L0, *G.K), r1 = of::philox_block(qt, L1, *G.K);
    float2 a1, a2;
    if (rem == 1) {
      of::normal_pairs_scaled2_from_u32(r0.x, r0.y, r1.x, r1.y, of::kBoxMullerK2, a1, a2);
      w = add2(w, a1);
    } else {
      w = add2(w, of::normal_pair_sums2_from_u32(r0.x, r0.y, r1.x, r1.y));
      if (rem == 3) {
        of::normal_pairs_scaled2_from_u32(r0.z, r0.w, r1.z, r1.w, of::kBoxMullerK2, a1, a2);
        w = add2(w, a1);
      }
    }
  }
  return w;
}

// The payoff of a terminal-only sample from its sum of normals w, averaged
// with its antithetic twin's (-w) when ANTI.
template <bool ANTI>
__device__ __forceinline__ void book_terminal_payoff(const BookOpt& o, float w, float& x, float& cvy) {
  const PathObs none{0.0f, 0.0f, 0.0f, false};
  const float base = (float)o.steps * o.c.drift;
  book_payoff(o, none, fmaf(o.c.diff, w, base), x, cvy);
  if (ANTI) {
    float xb, yb;
    book_payoff(o, none, fmaf(-o.c.diff, w, base), xb, yb);
    x = 0.5f * (x + xb);
    cvy = 0.5f * (cvy + yb);
  }
}

template <int KIND, bool ANTI, typename GEN>
__device__ __forceinline__ void book_sample_gbm(const BookOpt& o, uint64_t i, GEN G, float& x,
                                                float& cvy) {
  if (KIND == BK_TERMINAL) {
    book_terminal_payoff<ANTI>(o, book_terminal_sum(o, i, G), x, cvy);
    return;
  }
  if (ANTI) {  // the sample and its antithetic twin as the two halves of packed pairs
    float2 y;
    PathObs oa, ob;
    book_gbm_legs2<KIND, true>(o, i, i, G, y, oa, ob);
    float xb, yb2;
    book_payoff(o, oa, y.x, x, cvy);
    book_payoff(o, ob, y.y, xb, yb2);
    x = 0.5f * (x + xb);
    cvy = 0.5f * (cvy + yb2);
    return;
  }
  // a barrier path runs with the sign that makes its barrier an upper one:
  // sg y, sg drift, sg diff and sg b (sg = +1 up, -1 down; exact), one
  // comparison per step
  const float sg = KIND == BK_BARRIER && !(o.flags & BF_UP) ? -1.0f : 1.0f;
  const float drift = sg * o.c.drift, diff = sg * o.c.diff, sgb = sg * o.barrier_y;
  float ya = 0.0f;
  PathObs oa{0.0f, 0.0f, 0.0f, false};
  if (KIND == BK_BARRIER) oa.hit = 0.0f >= sgb;  // the scan includes path[0]
  auto step = [&](float z) {
    ya = fmaf(diff, z, ya + drift);
    if (KIND == BK_BARRIER) {
      oa.hit |= ya >= sgb;
    } else {  // Kahan sum of the daily fixings S/S0
      const float yk = __expf(ya) - oa.arith_comp;
      const float t = oa.arith_sum + yk;
      oa.arith_comp = (t - oa.arith_sum) - yk;
      oa.arith_sum = t;
      if (KIND == BK_ASIAN_DAILY_GEO) oa.geo_sum += ya;  // the general loop's fmaf(1, y, sum): one rounding
    }
  };
  const of::PhiloxLane L = G.lane(i);
  for (int32_t j = 0; j < o.steps; j += 4) {
    const uint4 r = G.block((uint32_t)(j >> 2), L);
    const float2 p01 = of::normal_pair_from_u32(r.x, r.y), p23 = of::normal_pair_from_u32(r.z, r.w);
    step(p01.x);
    if (j + 1 < o.steps) step(p01.y);
    if (j + 2 < o.steps) step(p23.x);
    if (j + 3 < o.steps) step(p23.y);
  }
  book_payoff(o, oa, sg * ya, x, cvy);
}

// Two legs of the specialised GBM loop in packed pairs (.x and .y), each half
// the arithmetic of book_sample_gbm bit for bit.  TWIN: the legs are sample
// i0 and its antithetic twin (one Philox stream, normals z and -z); otherwise
// the independent samples i0 and i1 (two streams, Box-Muller of both in packed
// pairs).
template <int KIND, bool TWIN, typename GEN>
__device__ __forceinline__ void book_gbm_legs2(const BookOpt& o, uint64_t i0, uint64_t i1, GEN G,
                                               float2& y, PathObs& oa, PathObs& ob) {
  using of::add2;
  using of::fma2;
  using of::mul2;
  using of::splat2;
  using of::sub2;
  const float sg = KIND == BK_BARRIER && !(o.flags & BF_UP) ? -1.0f : 1.0f;
  const float2 drift = splat2(sg * o.c.drift);
  const float2 diff = TWIN ? make_float2(sg * o.c.diff, -sg * o.c.diff) : splat2(sg * o.c.diff);
  const float sgb = sg * o.barrier_y;
  y = make_float2(0.0f, 0.0f);
  float2 as = make_float2(0.0f, 0.0f), ac = make_float2(0.0f, 0.0f);  // Kahan sums of the daily fixings
  float2 ag = make_float2(0.0f, 0.0f);                                 // geometric sums
  bool ha = false, hb = false;
  if (KIND == BK_BARRIER) ha = hb = 0.0f >= sgb;  // the scan includes path[0]
  auto step = [&](float2 z) {
    y = fma2(diff, z, add2(y, drift));
    if (KIND == BK_BARRIER) {
      ha |= y.x >= sgb;
      hb |= y.y >= sgb;
    } else if (KIND == BK_ASIAN_DAILY || KIND == BK_ASIAN_DAILY_GEO) {
      const float2 yk = sub2(make_float2(__expf(y.x), __expf(y.y)), ac);
      const float2 t = add2(as, yk);
      ac = sub2(sub2(t, as), yk);
      as = t;
      if (KIND == BK_ASIAN_DAILY_GEO) ag = add2(ag, y);
    }
  };
  const of::PhiloxLane L0 = G.lane(i0), L1 = G.lane(i1);  // i0 and i1 share their high word
  for (int32_t j = 0; j < o.steps; j += 4) {
    const uint4 qt = G.terms((uint32_t)(j >> 2));
    const uint4 r0 = of::philox_block(qt, L0, *G.K);
    float2 w1, w2, w3, w4;
    if (TWIN) {  // w1 = (z_j, z_j+2), w2 = (z_j+1, z_j+3)
      of::normal_pairs_scaled2_from_u32(r0.x, r0.y, r0.z, r0.w, of::kBoxMullerK2, w1, w2);
      w3 = splat2(w1.y);
      w4 = splat2(w2.y);
      w1 = splat2(w1.x);
      w2 = splat2(w2.x);
    } else {  // wk = step j+k-1 of (i0, i1)
      const uint4 r1 = of::philox_block(qt, L1, *G.K);
      of::normal_pairs_scaled2_from_u32(r0.x, r0.y, r1.x, r1.y, of::kBoxMullerK2, w1, w2);
      of::normal_pairs_scaled2_from_u32(r0.z, r0.w, r1.z, r1.w, of::kBoxMullerK2, w3, w4);
    }
    if (j + 4 <= o.steps) {
      step(w1);
      step(w2);
      step(w3);
      step(w4);
    } else {
      step(w1);
      if (j + 1 < o.steps) step(w2);
      if (j + 2 < o.steps) step(w3);
    }
  }
  if (KIND == BK_BARRIER) y = mul2(splat2(sg), y);
  oa = PathObs{as.x, ac.x, ag.x, ha};
  ob = PathObs{as.y, ac.y, ag.y, hb};
}

// book_sample_gbm<KIND, false> of two samples in one packed loop.
template <int KIND, typename GEN>
__device__ __forceinline__ void book_sample_gbm_pair(const BookOpt& o, uint64_t i0, uint64_t i1,
                                                     GEN G, float& x0, float& cv0, float& x1,
                                                     float& cv1) {
  float2 y;
  PathObs oa, ob;
  book_gbm_legs2<KIND, false>(o, i0, i1, G, y, oa, ob);
  book_payoff(o, oa, y.x, x0, cv0);
  book_payoff(o, ob, y.y, x1, cv1);
}

// book_sample_gbm<BK_TERMINAL, ANTI> of samples i0 and i1: their sums of
// normals in packed pairs (two Philox streams per thread), then each sample's
// payoff (and its twin's) as the scalar form takes it.
template <bool ANTI, typename GEN>
__device__ __forceinline__ void book_terminal_pair(const BookOpt& o, uint64_t i0, uint64_t i1, GEN G,
                                                   float& x0, float& cv0, float& x1, float& cv1) {
  const float2 w = book_terminal_sums2(o, i0, i1, G);
  book_terminal_payoff<ANTI>(o, w.x, x0, cv0);
  book_terminal_payoff<ANTI>(o, w.y, x1, cv1);
}

// One sample of option o: the specialised GBM loop when the option has one,
// the general loop otherwise.
template <typename GEN>
__device__ __forceinline__ void book_dispatch(const BookOpt& o, uint64_t i, const BookParams& P, const GEN& G,
                                              float& x, float& y) {
  const bool anti = o.flags & BF_ANTI;
  switch (o.kind) {
    case BK_TERMINAL:
      if (anti) book_sample_gbm<BK_TERMINAL, true>(o, i, G, x, y);
      else book_sample_gbm<BK_TERMINAL, false>(o, i, G, x, y);
      return;
    case BK_BARRIER:
      if (anti) book_sample_gbm<BK_BARRIER, true>(o, i, G, x, y);
      else book_sample_gbm<BK_BARRIER, false>(o, i, G, x, y);
      return;
    case BK_ASIAN_DAILY:
      if (anti) book_sample_gbm<BK_ASIAN_DAILY, true>(o, i, G, x, y);
      else book_sample_gbm<BK_ASIAN_DAILY, false>(o, i, G, x, y);
      return;
    case BK_ASIAN_DAILY_GEO:
      if (anti) book_sample_gbm<BK_ASIAN_DAILY_GEO, true>(o, i, G, x, y);
      else book_sample_gbm<BK_ASIAN_DAILY_GEO, false>(o, i, G, x, y);
      return;
    default:
      break;
  }
  if (o.model == OF_MODEL_GBM) {
    if (o.n_div) book_sample<OF_MODEL_GBM, true>(o, i, G, P.obs_w, P.divs, x, y);
    else book_sample<OF_MODEL_GBM, false>(o, i, G, P.obs_w, P.divs, x, y);
  } else if (o.model == OF_MODEL_HESTON_EULER) {
    book_sample<OF_MODEL_HESTON_EULER, false>(o, i, G, P.obs_w, P.divs, x, y);
  } else {
    book_sample<OF_MODEL_HESTON_QE, false>(o, i, G, P.obs_w, P.divs, x, y);
  }
}

// The generator of a tile's option, its table (`cap` entries) filled by the
// block (called by all threads).  FULL launches have a table that covers every
// option's counter blocks and samples below 2^32; the others compute the terms
// past the table, or past the tile's first high word, in place.  The loops run
// at the integer-multiply rate (a wide multiply takes four issue cycles a warp
// on sm_100); the table saves five of a counter block's twenty.  With the
// signed barrier path and the packed sums of squares, 384 options of
// 2^14..2^17 paths by 25..1260 daily steps took 10.60 ms (antithetic 6.36)
// against 11.58 (6.98); with the range test left in the loop, 11.2.
constexpr uint32_t kBookTab = 2048;  // largest table (32 KB, three blocks an SM): 8,192 GBM steps

template <bool FULL>
__device__ __forceinline__ of::PhiloxGen<FULL> book_gen(uint4* qtab, uint32_t cap, int steps_per_block, int32_t steps,
                                                        int64_t first, uint32_t stream, const of::PhiloxKeys& K) {
  const uint32_t nq = ((uint32_t)steps + steps_per_block - 1) / steps_per_block;
  const of::PhiloxTab T{qtab, nq < cap ? nq : cap, (uint32_t)((uint64_t)first >> 32), stream};
  of::philox_table_fill(qtab, T.n, T.hi, T.stream, K);
  __syncthreads();
  return of::PhiloxGen<FULL>{&K, T};
}

// Three 256-thread blocks per SM: ptxas's own choice without the hint is 64
// registers with spills in the step loop.
template <bool FULL>
__global__ void __launch_bounds__(256, 3) book_kernel(const __grid_constant__ BookParams P) {
  __shared__ int tile_sh;
  __shared__ double red_sh[5 * 8];
  extern __shared__ uint4 qtab[];
  for (;;) {
    if (threadIdx.x == 0) tile_sh = atomicAdd(P.counter, 1);
    __syncthreads();
    const int t = tile_sh;
    if (t >= P.n_tiles) break;
    const BookTile tile = P.tiles[t];
    const BookOpt o = P.opts[tile.opt];
    const of::PhiloxGen<FULL> G =
        book_gen<FULL>(qtab, P.tab, o.model == OF_MODEL_GBM ? 4 : 2, o.steps, tile.first, o.stream, P.keys);
    of::KahanSq32 ax, ay;
    of::Kahan32 axy;
    auto add = [&](float x, float y) {
      ax.add(x);
      ay.add(y);
      axy.add(x * y);
    };
    // specialised GBM kinds without antithetic twins, and terminal-only
    // options with them, run two samples at a time in packed pairs; the sums
    // take them in the same order
    const bool pairs = o.kind != BK_GENERIC && (!(o.flags & BF_ANTI) || o.kind == BK_TERMINAL);
    for (int k = 0; k < P.ppt; ++k) {
      const int local = k * blockDim.x + threadIdx.x;
      if (local >= tile.count) break;
      const uint64_t i = (uint64_t)(tile.first + local);
      float x, y;
      if (const uint64_t i1 = i + blockDim.x;
          pairs && k + 1 < P.ppt && local + (int)blockDim.x < tile.count && (FULL || (i >> 32) == (i1 >> 32))) {
        float x1, y1;
        if (o.kind == BK_TERMINAL) {
          if (o.flags & BF_ANTI) book_terminal_pair<true>(o, i, i1, G, x, y, x1, y1);
          else book_terminal_pair<false>(o, i, i1, G, x, y, x1, y1);
        }
        else if (o.kind == BK_BARRIER) book_sample_gbm_pair<BK_BARRIER>(o, i, i1, G, x, y, x1, y1);
        else if (o.kind == BK_ASIAN_DAILY_GEO) book_sample_gbm_pair<BK_ASIAN_DAILY_GEO>(o, i, i1, G, x, y, x1, y1);
        else book_sample_gbm_pair<BK_ASIAN_DAILY>(o, i, i1, G, x, y, x1, y1);
        add(x, y);
        add(x1, y1);
        ++k;
        continue;
      }
      book_dispatch(o, i, P, G, x, y);
      add(x, y);
    }
    double v[5] = {ax.value(), ax.square(), ay.value(), axy.value(), ay.square()};
    of::block_sum<5>(v, red_sh);
    if (threadIdx.x == 0)
      for (int k = 0; k < 5; ++k) P.partials[(int64_t)tile.slot * 5 + k] = v[k];
    __syncthreads();
  }
}

// Running sums of the Greeks modes.  FP32 (with Greeks): the five sums of
// MonteCarloEngine::run compensated, then per Greek its compensated sum and
// plain sum of squares (a few samples per thread per tile; only the standard
// error reads them).  FP64: the five sums.
template <typename R, bool G>
struct GreekAcc;

template <>
struct GreekAcc<float, true> {
  of::Kahan32 s[5], g[4];
  float g2[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  __device__ __forceinline__ void add(const of::GreekSample<float>& v) {
    s[0].add(v.x);
    s[1].add(v.x * v.x);
    s[2].add(v.y);
    s[3].add(v.x * v.y);
    s[4].add(v.y * v.y);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      g[t].add(v.g[t]);
      g2[t] = fmaf(v.g[t], v.g[t], g2[t]);
    }
  }
  __device__ __forceinline__ void values(double (&out)[13]) const {
#pragma unroll
    for (int k = 0; k < 5; ++k) out[k] = s[k].value();
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      out[5 + t] = g[t].value();
      out[9 + t] = (double)g2[t];
    }
  }
};

template <>
struct GreekAcc<double, true> {
  double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, g[4] = {0.0, 0.0, 0.0, 0.0}, g2[4] = {0.0, 0.0, 0.0, 0.0};
  __device__ __forceinline__ void add(const of::GreekSample<double>& v) {
    s[0] += v.x;
    s[1] += v.x * v.x;
    s[2] += v.y;
    s[3] += v.x * v.y;
    s[4] += v.y * v.y;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      g[t] += v.g[t];
      g2[t] = fma(v.g[t], v.g[t], g2[t]);
    }
  }
  __device__ __forceinline__ void values(double (&out)[13]) const {
#pragma unroll
    for (int k = 0; k < 5; ++k) out[k] = s[k];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      out[5 + t] = g[t];
      out[9 + t] = g2[t];
    }
  }
};

template <>
struct GreekAcc<double, false> {
  double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  __device__ __forceinline__ void add(const of::GreekSample<double>& v) {
    s[0] += v.x;
    s[1] += v.x * v.x;
    s[2] += v.y;
    s[3] += v.x * v.y;
    s[4] += v.y * v.y;
  }
  __device__ __forceinline__ void values(double (&out)[5]) const {
#pragma unroll
    for (int k = 0; k < 5; ++k) out[k] = s[k];
  }
};

// The book's Greeks modes: the persistent tile loop of book_kernel over the
// per-sample kernels of book_greeks.cuh, one launch per kind group (the
// group's tiles only).  <float, true>: prices and pathwise Greeks (13 sums
// per tile); <double, false>: FP64 prices on the same draws.  FP32 Greeks:
// the terminal group at four blocks per SM (64 registers), the Asian and
// survival-barrier groups at three (the survival step's 91 registers capped
// at 80 spill 64 bytes: two blocks cost 5 % more); the FP64 modes at two.
template <typename R, bool G, int KG, bool FULL>
__global__ void __launch_bounds__(256, (!G || sizeof(R) == 8) ? 2 : (KG == of::KG_TERMINAL ? 4 : 3))
    book_greeks_kernel(const __grid_constant__ BookParams P, const of::GreekConsts<R>* __restrict__ gc) {
  constexpr int NC = G ? 13 : 5;
  __shared__ int tile_sh;
  __shared__ double red_sh[NC * 8];
  extern __shared__ uint4 qtab[];
  for (;;) {
    if (threadIdx.x == 0) tile_sh = atomicAdd(P.counter, 1);
    __syncthreads();
    const int t = tile_sh;
    if (t >= P.n_tiles) break;
    const BookTile tile = P.tiles[t];
    const of::GreekConsts<R>& c = gc[tile.opt];
    const of::PhiloxGen<FULL> gen = book_gen<FULL>(qtab, P.tab, 4, c.steps, tile.first, c.stream, P.keys);
    GreekAcc<R, G> acc;
    // FP32: two samples at a time in packed pairs (terminal-only options, and
    // Asian and barrier options without antithetic twins, whose twins pair
    // inside one sample); the sums take them in the same order
    constexpr bool kPairs = std::is_same<R, float>::value;
    const bool pairs = kPairs && (KG == of::KG_TERMINAL || !(c.flags & of::GF_ANTI));
    for (int k = 0; k < P.ppt; ++k) {
      const int local = k * blockDim.x + threadIdx.x;
      if (local >= tile.count) break;
      if constexpr (kPairs) {
        const uint64_t i0 = (uint64_t)(tile.first + local), i1 = i0 + blockDim.x;
        if (pairs && k + 1 < P.ppt && local + (int)blockDim.x < tile.count && (FULL || (i0 >> 32) == (i1 >> 32))) {
          of::GreekSample<float> v0, v1;
          if constexpr (KG == of::KG_BARRIER) of::gk_barrier_pair_group<G>(c, i0, i1, gen, v0, v1);
          else if constexpr (KG == of::KG_ASIAN) of::gk_asian_pair_group<G>(c, i0, i1, gen, P.obs_w, v0, v1);
          else of::gk_terminal_pair_group<G>(c, i0, i1, gen, v0, v1);
          acc.add(v0);
          acc.add(v1);
          ++k;
          continue;
        }
      }
      of::GreekSample<R> v;
      of::gk_sample_group<R, G, KG>(c, (uint64_t)(tile.first + local), gen, P.obs_w, v);
      acc.add(v);
    }
    double v[NC];
    acc.values(v);
    of::block_sum<NC>(v, red_sh);
    if (threadIdx.x == 0)
      for (int k = 0; k < NC; ++k) P.partials[(int64_t)tile.slot * NC + k] = v[k];
    __syncthreads();
  }
}

// Per-option sums over its tile slots [begin[o], begin[o+1]) in fixed order;
// NC sums per slot, written to pinned host memory.  It runs after the launch's
// last tile, so it also clears the tile counters for the next one.
template <int NC>
__global__ void book_reduce_kernel(const double* __restrict__ partials, const int32_t* __restrict__ begin, int n_opts,
                                   double* __restrict__ sums, int* __restrict__ counter) {
  const int o = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x < of::KG_COUNT) counter[threadIdx.x] = 0;
  if (o >= n_opts) return;
  double acc[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) acc[k] = 0.0;
  for (int s = begin[o] + lane; s < begin[o + 1]; s += 32)
#pragma unroll
    for (int k = 0; k < NC; ++k) acc[k] += partials[(int64_t)s * NC + k];
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    const double v = of::warp_sum(acc[k]);
    if (lane == 0) sums[(int64_t)o * NC + k] = v;
  }
}

}  // namespace

static_assert(OF_CV_NONE == of::GCV_NONE && OF_CV_VANILLA_TERMINAL == of::GCV_VANILLA_TERMINAL &&
                  OF_CV_GEOMETRIC_ASIAN == of::GCV_GEOMETRIC_ASIAN && OF_CV_TERMINAL_SPOT == of::GCV_TERMINAL_SPOT,
              "the Greeks modes read the control-variate kinds of the ABI");

// Constants of one entry in the Greeks modes (FP64; the FP32 mode rounds
// them once).  `d` is the entry's price-mode record (flags, observation
// weights' offset), `w` its observation weights by step index (empty when it
// has none) and `daily` whether they are the daily fixings 1..steps.
static of_status book_greek_consts(of_ctx* ctx, const of_book_entry& b, int64_t o, const BookOpt& d,
                                   const std::vector<double>& w, bool daily, of::GreekConsts<double>& g) {
  const of_model& m = b.model;
  const of_payoff& p = b.payoff;
  if (m.kind != OF_MODEL_GBM)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "the Greeks modes price GBM options (Heston: of_heston_price_adjoint)");
  if (m.n_dividends > 0) return of_fail(ctx, OF_ERR_UNSUPPORTED, "the Greeks modes take no discrete dividends");
  if (!(b.discount_factor > 0.0) || !std::isfinite(b.discount_factor))
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "the Greeks modes need a discount factor exp(-r T) > 0");
  g = of::GreekConsts<double>{};
  const double T = m.maturity, M = (double)m.steps, dt = T / M, sig = m.sigma;
  g.dt = dt;
  g.T = T;
  g.sigma = sig;
  g.a = m.mu - 0.5 * sig * sig;
  g.alpha = g.a * dt;
  g.beta = sig * std::sqrt(dt);
  g.df = b.discount_factor;
  g.r = -std::log(b.discount_factor) / T;
  g.s0 = m.s0;
  g.strike = p.strike;
  g.sig_dt = sig * dt;
  g.inv_sig = 1.0 / sig;
  g.beta_over_sig = std::sqrt(dt);
  g.alpha_over_T = g.alpha / T;
  g.inv_2T = 0.5 / T;
  g.beta_over_2T = g.beta / (2.0 * T);
  g.steps = (int32_t)m.steps;
  g.obs_offset = d.obs_offset;
  g.cv_kind = b.control_variate;
  g.stream = d.stream;
  int32_t f = 0;
  if (p.option_type == OF_CALL) f |= of::GF_CALL;
  if (b.antithetic) f |= of::GF_ANTI;
  switch (p.kind) {
    case OF_PAYOFF_VANILLA:
      g.kind = of::GK_TERMINAL;
      break;
    case OF_PAYOFF_ASIAN:
      if (p.strike_type == OF_STRIKE_FLOATING) f |= of::GF_FLOATING;
      if (p.averaging == OF_AVG_GEOMETRIC) f |= of::GF_GEOMETRIC;
      if (d.flags & BF_TERMINAL_ONLY) {
        f |= of::GF_TERMINAL_ONLY;
        g.kind = of::GK_TERMINAL;
      } else {
        g.kind = daily ? of::GK_ASIAN_DAILY : of::GK_ASIAN_WEIGHTS;
        g.inv_n = 1.0 / (double)p.n_observations;
        double w1 = 0.0;
        for (size_t i = 1; i < w.size(); ++i) w1 += w[i] * (double)i;
        g.w1 = w1;
      }
      break;
    default:  // barrier
      if (!(p.barrier_level > 0.0) || !std::isfinite(p.barrier_level))
        return of_fail(ctx, OF_ERR_INVALID_INPUT, "barrier level must be > 0");
      if (b.control_variate != OF_CV_NONE)
        return of_fail(ctx, OF_ERR_UNSUPPORTED, "a barrier option takes no control variate in the Greeks modes");
      g.kind = p.barrier_style == OF_BARRIER_IN ? of::GK_BARRIER_IN : of::GK_BARRIER_OUT;
      g.rebate = p.rebate;
      g.bar = std::log(p.barrier_level / m.s0);
      g.sgn = p.barrier_direction == OF_BARRIER_UP ? 1.0 : -1.0;
      g.sib = g.sgn / g.beta;
  }
  g.flags = f;
  (void)o;
  return OF_OK;
}

static of::GreekConsts<float> round_greek_consts(const of::GreekConsts<double>& d) {
  of::GreekConsts<float> f{};
  f.alpha = (float)d.alpha;
  f.beta = (float)d.beta;
  f.a = (float)d.a;
  f.dt = (float)d.dt;
  f.T = (float)d.T;
  f.sigma = (float)d.sigma;
  f.r = (float)d.r;
  f.df = (float)d.df;
  f.s0 = (float)d.s0;
  f.strike = (float)d.strike;
  f.rebate = (float)d.rebate;
  f.inv_n = (float)d.inv_n;
  f.w1 = (float)d.w1;
  f.bar = (float)d.bar;
  f.sgn = (float)d.sgn;
  f.sib = (float)d.sib;
  f.sig_dt = (float)d.sig_dt;
  f.inv_sig = (float)d.inv_sig;
  f.beta_over_sig = (float)d.beta_over_sig;
  f.alpha_over_T = (float)d.alpha_over_T;
  f.inv_2T = (float)d.inv_2T;
  f.beta_over_2T = (float)d.beta_over_2T;
  f.kind = d.kind;
  f.flags = d.flags;
  f.steps = d.steps;
  f.obs_offset = d.obs_offset;
  f.cv_kind = d.cv_kind;
  f.stream = d.stream;
  return f;
}

struct of_book_plan {
  of_ctx* ctx = nullptr;
  bool scratch = false;  // buffers borrowed from the context (a plan that lives inside one call)
  int64_t n = 0;
  int mode = OF_BOOK_PRICE;
  int nc = 5;  // sums per option: 5, or 13 with the Greeks
  int block = 256, ppt = 4, grid = 0;
  int64_t n_tiles = 0;
  double path_steps = 0.0;
  std::vector<int64_t> samples;
  std::vector<int32_t> cv_kind;
  std::vector<double> cv_expected, discount;
  BookParams P{};
  BookParams Pg[of::KG_COUNT]{};  // Greeks modes: one launch per kind group
  int grid_g[of::KG_COUNT] = {0, 0, 0};
  BookOpt* d_opts = nullptr;
  BookTile* d_tiles = nullptr;
  float* d_obs = nullptr;
  BookDiv* d_divs = nullptr;
  void* d_gc = nullptr;  // GreekConsts<float> (Greeks mode) or <double> (FP64 mode)
  int* d_counter = nullptr;
  int32_t* d_begin = nullptr;
  char* d_image = nullptr;  // one allocation and one upload: the six tables above and the counters
  double* d_partials = nullptr;
  double* h_sums = nullptr;  // pinned, written by the reduction
  bool use_graph = true;
  bool full = true;  // the q table covers every option (PhiloxGen<true>)
  size_t smem() const { return (size_t)P.tab * sizeof(uint4); }
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

template <typename R, bool G, bool FULL>
static const void* book_greeks_kernel_for(int kg) {
  return kg == of::KG_TERMINAL ? (const void*)book_greeks_kernel<R, G, of::KG_TERMINAL, FULL>
         : kg == of::KG_ASIAN  ? (const void*)book_greeks_kernel<R, G, of::KG_ASIAN, FULL>
                               : (const void*)book_greeks_kernel<R, G, of::KG_BARRIER, FULL>;
}

template <bool FULL>
static const void* book_kernel_for(int mode, int kg) {
  if (mode == OF_BOOK_GREEKS) return book_greeks_kernel_for<float, true, FULL>(kg);
  if (mode == OF_BOOK_PRICE_FP64) return book_greeks_kernel_for<double, false, FULL>(kg);
  if (mode == OF_BOOK_GREEKS_FP64) return book_greeks_kernel_for<double, true, FULL>(kg);
  return (const void*)book_kernel<FULL>;
}

static const void* book_kernel_for(const of_book_plan* pl, int kg) {
  return pl->full ? book_kernel_for<true>(pl->mode, kg) : book_kernel_for<false>(pl->mode, kg);
}

static void book_greeks_enqueue(of_book_plan* pl, cudaStream_t s) {
  for (int kg = 0; kg < of::KG_COUNT; ++kg) {
    if (pl->Pg[kg].n_tiles == 0) continue;
    void* args[] = {(void*)&pl->Pg[kg], (void*)&pl->d_gc};
    cudaLaunchKernel(book_kernel_for(pl, kg), dim3((unsigned)pl->grid_g[kg]), dim3((unsigned)pl->block), args,
                     pl->smem(), s);
  }
}

static void book_enqueue(of_book_plan* pl, cudaStream_t s) {
  if (pl->mode == OF_BOOK_PRICE) {
    void* args[] = {(void*)&pl->P};
    cudaLaunchKernel(book_kernel_for(pl, 0), dim3((unsigned)pl->grid), dim3((unsigned)pl->block), args, pl->smem(), s);
  } else {
    book_greeks_enqueue(pl, s);
  }
  const unsigned rgrid = (unsigned)((pl->n + 7) / 8);
  if (pl->nc == 13)
    book_reduce_kernel<13><<<rgrid, 256, 0, s>>>(pl->d_partials, pl->d_begin, (int)pl->n, pl->h_sums, pl->d_counter);
  else
    book_reduce_kernel<5><<<rgrid, 256, 0, s>>>(pl->d_partials, pl->d_begin, (int)pl->n, pl->h_sums, pl->d_counter);
}

extern "C" void of_book_plan_destroy(of_book_plan* pl) {
  if (!pl) return;
  if (pl->ctx) cudaStreamSynchronize(pl->ctx->stream);
  if (pl->exec) cudaGraphExecDestroy(pl->exec);
  if (pl->graph) cudaGraphDestroy(pl->graph);
  if (pl->scratch) {  // the context owns the buffers
    delete pl;
    return;
  }
  cudaFree(pl->d_image);
  cudaFree(pl->d_partials);
  if (pl->h_sums) cudaFreeHost(pl->h_sums);
  delete pl;
}

// scratch: the plan lives inside one library call and borrows the context's
// cached buffers (of_scratch / of_pinned) instead of allocating its own.
static of_status book_plan_create(of_ctx* ctx, const of_book_entry* e, int64_t n, const of_book_config* cfg,
                                  bool scratch, of_book_plan** out) {
  if (!ctx || !out || !cfg) return OF_ERR_INVALID_INPUT;
  *out = nullptr;
  if (n <= 0 || !e) return of_fail(ctx, OF_ERR_INVALID_INPUT, "book must hold at least one option");
  if (n > (1 << 24)) return of_fail(ctx, OF_ERR_INVALID_INPUT, "book too large");
  OF_TRY(of_ctx_check(ctx));
  OF_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  of_book_plan* pl = new of_book_plan();
  pl->ctx = ctx;
  pl->scratch = scratch;
  pl->n = n;
  pl->block = cfg->block > 0 ? cfg->block : 256;
  pl->ppt = cfg->paths_per_thread > 0 ? cfg->paths_per_thread : 4;
  pl->use_graph = cfg->use_graph != 0;
  pl->mode = cfg->mode;
  if (pl->mode != OF_BOOK_PRICE && pl->mode != OF_BOOK_GREEKS && pl->mode != OF_BOOK_PRICE_FP64 &&
      pl->mode != OF_BOOK_GREEKS_FP64) {
    const int m = pl->mode;
    of_book_plan_destroy(pl);
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown book mode %d", m);
  }
  pl->nc = (pl->mode == OF_BOOK_GREEKS || pl->mode == OF_BOOK_GREEKS_FP64) ? 13 : 5;
  if (pl->block % 32 != 0 || pl->block > 256) {
    of_book_plan_destroy(pl);
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "block must be a multiple of 32 and <= 256");
  }
  auto fail = [&](of_status st) {
    of_book_plan_destroy(pl);
    return st;
  };
  std::vector<BookOpt> opts((size_t)n);
  std::vector<of::GreekConsts<double>> gcs;  // Greeks modes only
  if (pl->mode != OF_BOOK_PRICE) gcs.resize((size_t)n);
  std::vector<float> obs;
  std::vector<BookDiv> divs;
  std::vector<of_div_trigger> trig;
  pl->samples.resize((size_t)n);
  pl->cv_kind.resize((size_t)n);
  pl->cv_expected.resize((size_t)n);
  pl->discount.resize((size_t)n);
  const int64_t tile_samples = (int64_t)pl->block * pl->ppt;
  for (int64_t o = 0; o < n; ++o) {
    const of_book_entry& b = e[o];
    of_mc_config c{};
    c.num_paths = b.num_paths;
    c.antithetic = b.antithetic;
    c.control_variate = b.control_variate;
    c.discount_factor = b.discount_factor;
    c.precision = OF_PREC_FP32_PHILOX;
    of_status st = of_validate_mc(ctx, &b.model, &b.payoff, &c);
    if (st == OF_OK) st = validate_fp32_model(ctx, &b.model);
    if (st != OF_OK) {
      ctx->last_error = "book entry " + std::to_string(o) + ": " + ctx->last_error;
      return fail(st);
    }
    BookOpt& d = opts[(size_t)o];
    d.c = make_consts(&b.model);
    d.model = b.model.kind;
    d.payoff = b.payoff.kind;
    d.cv_kind = b.control_variate;
    d.steps = (int32_t)b.model.steps;
    d.s0 = (float)b.model.s0;
    d.strike = (float)b.payoff.strike;
    d.rebate = (float)b.payoff.rebate;
    d.barrier_y = (float)std::log(b.payoff.barrier_level / b.model.s0);
    if (!(b.payoff.barrier_level > 0.0)) d.barrier_y = b.payoff.barrier_direction == OF_BARRIER_UP ? INFINITY : -INFINITY;
    d.stream = (uint32_t)o;
    d.obs_offset = -1;
    st = of_dividend_triggers(ctx, &b.model, trig);
    if (st != OF_OK) {
      ctx->last_error = "book entry " + std::to_string(o) + ": " + ctx->last_error;
      return fail(st);
    }
    d.div_offset = (int32_t)divs.size();
    d.n_div = (int32_t)trig.size();
    for (const of_div_trigger& t : trig)
      divs.push_back(BookDiv{t.step, t.kind,
                             (float)(t.kind == OF_DIV_CASH ? t.amount / b.model.s0 : std::log1p(-t.amount)), 0.0f});
    int32_t f = 0;
    if (b.antithetic) f |= BF_ANTI;
    if (b.payoff.barrier_direction == OF_BARRIER_UP) f |= BF_UP;
    if (b.payoff.barrier_style == OF_BARRIER_IN) f |= BF_IN;
    if (b.payoff.averaging == OF_AVG_GEOMETRIC) f |= BF_GEOMETRIC;
    if (b.payoff.strike_type == OF_STRIKE_FLOATING) f |= BF_FLOATING;
    if (b.payoff.option_type == OF_CALL) f |= BF_CALL;
    const bool asian = b.payoff.kind == OF_PAYOFF_ASIAN;
    bool need_arith = asian && b.payoff.averaging == OF_AVG_ARITHMETIC;
    bool need_geo = (asian && b.payoff.averaging == OF_AVG_GEOMETRIC) || b.control_variate == OF_CV_GEOMETRIC_ASIAN;
    std::vector<double> w;
    bool daily_obs = false;
    if (need_arith || need_geo) {
      bool terminal_only = true;
      of_observation_weights(&b.payoff, b.model.steps, w, terminal_only);
      if (terminal_only) {
        f |= BF_TERMINAL_ONLY;
        need_arith = need_geo = false;
      } else {
        bool daily = w[0] == 0.0;
        for (size_t k = 1; k < w.size() && daily; ++k) daily = w[k] == 1.0;
        daily_obs = daily;
        if (daily) {
          f |= BF_DAILY;
        } else {
          d.obs_offset = (int32_t)obs.size();
          for (double x : w) obs.push_back((float)x);
        }
        d.inv_nobs = (float)(1.0 / (double)b.payoff.n_observations);
      }
    }
    if (need_arith) f |= BF_NEED_ARITH;
    if (need_geo) f |= BF_NEED_GEO;
    if (asian && !need_arith && !need_geo) f |= BF_TERMINAL_ONLY;
    d.flags = f;
    d.kind = BK_GENERIC;
    if (d.model == OF_MODEL_GBM && d.n_div == 0) {
      if (!need_geo) {
        if (b.payoff.kind == OF_PAYOFF_VANILLA || (f & BF_TERMINAL_ONLY)) d.kind = BK_TERMINAL;
        else if (b.payoff.kind == OF_PAYOFF_BARRIER) d.kind = BK_BARRIER;
        else if (need_arith && (f & BF_DAILY)) d.kind = BK_ASIAN_DAILY;
      } else if (need_arith && (f & BF_DAILY)) {  // with the geometric control variate
        d.kind = BK_ASIAN_DAILY_GEO;
      }
    }
    if (pl->mode != OF_BOOK_PRICE) {
      st = book_greek_consts(ctx, b, o, d, w, daily_obs, gcs[(size_t)o]);
      if (st != OF_OK) {
        ctx->last_error = "book entry " + std::to_string(o) + ": " + ctx->last_error;
        return fail(st);
      }
    }
    const int64_t samples = b.antithetic ? (b.num_paths + 1) / 2 : b.num_paths;
    pl->samples[(size_t)o] = samples;
    pl->cv_kind[(size_t)o] = b.control_variate;
    pl->cv_expected[(size_t)o] = b.cv_expected;
    pl->discount[(size_t)o] = b.discount_factor;
    pl->path_steps += (double)b.num_paths * (double)b.model.steps;
  }
  // Slots in option-major order, schedule longest tile first: the Greeks
  // modes' kind groups in turn, longest tile first within a group, ties in
  // slot order (a stable sort of the tiles by group, then cost descending).
  // An option's tiles are consecutive slots; all but its last share one cost,
  // and the last may be shorter.  So the schedule is built from runs of
  // equal-cost tiles, at most two per option, sorted stably: the same order as
  // sorting the tiles, at O(n log n + tiles) instead of O(tiles log tiles) (a
  // million tiles for a book of long-dated options at 2^25 paths each).
  struct Run {
    int32_t opt, count;  // samples of each of its tiles
    int64_t slot, tiles, first;
    int group;
    double cost;
  };
  std::vector<Run> runs;
  runs.reserve((size_t)n * 2);
  std::vector<int64_t> begin((size_t)n + 1, 0);
  int64_t group_tiles[of::KG_COUNT] = {0, 0, 0};
  for (int64_t o = 0; o < n; ++o) {
    const int group = pl->mode != OF_BOOK_PRICE ? of::gk_group(gcs[(size_t)o].kind) : 0;
    const double per = (e[o].antithetic ? 2.0 : 1.0) * (double)e[o].model.steps;
    const int64_t samples = pl->samples[(size_t)o], whole = samples / tile_samples, rest = samples % tile_samples;
    int64_t slot = begin[(size_t)o];
    if (whole)
      runs.push_back({(int32_t)o, (int32_t)tile_samples, slot, whole, 0, group, (double)tile_samples * per});
    slot += whole;
    if (rest) runs.push_back({(int32_t)o, (int32_t)rest, slot++, 1, whole * tile_samples, group, (double)rest * per});
    group_tiles[group] += slot - begin[(size_t)o];
    begin[(size_t)o + 1] = slot;
    if (slot > 2147483647) return fail(of_fail(ctx, OF_ERR_INVALID_INPUT, "too many tiles"));
  }
  std::stable_sort(runs.begin(), runs.end(), [](const Run& a, const Run& b) {
    return a.group != b.group ? a.group < b.group : a.cost > b.cost;
  });
  const size_t nt = (size_t)begin[(size_t)n];
  pl->n_tiles = (int64_t)nt;
  // The tables in one image, uploaded once: [options | tiles | weights |
  // dividends | Greek constants | slot ranges | counters].  A plan that lives
  // inside one call borrows the context's cached buffers (no cudaMalloc,
  // cudaFree or cudaMallocHost per call) and stages images of up to 8 MB,
  // some 340,000 tiles of 24 bytes, in its pinned buffer behind the sums; larger
  // ones go from pageable memory, so that the buffer stays small.  A call on
  // 384 options (21,000 tiles) spends 0.6 ms beside its kernels, against 2.0
  // and up with nine allocations, six uploads and their frees.
  size_t bytes = 0;
  auto place = [&](size_t size) {
    const size_t at = bytes;
    bytes += (size + 255) & ~(size_t)255;
    return at;
  };
  const size_t gc_size = pl->mode == OF_BOOK_PRICE    ? 0
                         : pl->mode == OF_BOOK_GREEKS ? sizeof(of::GreekConsts<float>)
                                                      : sizeof(of::GreekConsts<double>);
  const size_t at_opts = place(opts.size() * sizeof(BookOpt)), at_tiles = place(nt * sizeof(BookTile)),
               at_obs = place(obs.size() * sizeof(float)), at_divs = place(divs.size() * sizeof(BookDiv)),
               at_gc = place((size_t)n * gc_size), at_begin = place(begin.size() * sizeof(int32_t)),
               at_counter = place(of::KG_COUNT * sizeof(int));
  const size_t sum_bytes = ((size_t)n * pl->nc * sizeof(double) + 255) & ~(size_t)255;
  const bool staged = pl->scratch && bytes <= ((size_t)8 << 20);
  auto dalloc = [&](void** p, size_t size, int slot) {
    if (pl->scratch) return of_scratch(ctx, slot, size, p) == OF_OK;
    return cudaMalloc(p, size) == cudaSuccess;
  };
  bool ok = dalloc((void**)&pl->d_image, bytes, SLOT_BOOK) &&
            dalloc((void**)&pl->d_partials, nt * pl->nc * sizeof(double), SLOT_BOOK_PARTIALS);
  if (ok) ok = pl->scratch ? of_pinned(ctx, sum_bytes + (staged ? bytes : 0), (void**)&pl->h_sums) == OF_OK
                           : cudaMallocHost(&pl->h_sums, sum_bytes) == cudaSuccess;
  if (!ok) return fail(of_fail(ctx, OF_ERR_ALLOC, "book plan allocation failed"));
  std::vector<char> heap(staged ? 0 : bytes);
  char* const image = staged ? (char*)pl->h_sums + sum_bytes : heap.data();
  std::copy(opts.begin(), opts.end(), (BookOpt*)(image + at_opts));
  std::copy(obs.begin(), obs.end(), (float*)(image + at_obs));
  std::copy(divs.begin(), divs.end(), (BookDiv*)(image + at_divs));
  std::copy(begin.begin(), begin.end(), (int32_t*)(image + at_begin));
  std::fill_n((int*)(image + at_counter), (int)of::KG_COUNT, 0);
  if (pl->mode == OF_BOOK_GREEKS)  // the constants rounded once to FP32
    for (size_t k = 0; k < gcs.size(); ++k) ((of::GreekConsts<float>*)(image + at_gc))[k] = round_greek_consts(gcs[k]);
  else
    std::copy(gcs.begin(), gcs.end(), (of::GreekConsts<double>*)(image + at_gc));
  BookTile* tile = (BookTile*)(image + at_tiles);
  for (const Run& r : runs)
    for (int64_t k = 0; k < r.tiles; ++k)
      *tile++ = {r.opt, r.count, r.first + k * tile_samples, (int32_t)(r.slot + k), 0};
  // (from pageable memory the call returns once the bytes have left it)
  // A plan created while the context's stream is captured uploads on a stream
  // of its own and waits: captured, the copy would become a node of the
  // caller's graph that reads `heap` long after it is gone.  (A call that
  // borrows the context's buffers is refused under capture, as it waits.)
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  cudaStream_t up = ctx->stream;
  cudaError_t up_err = pl->scratch ? cudaSuccess : cudaStreamIsCapturing(up, &capturing);
  if (up_err == cudaSuccess && capturing == cudaStreamCaptureStatusNone) {
    up_err = cudaMemcpyAsync(pl->d_image, image, bytes, cudaMemcpyHostToDevice, up);
  } else if (up_err == cudaSuccess && (up_err = cudaStreamCreateWithFlags(&up, cudaStreamNonBlocking)) == cudaSuccess) {
    up_err = cudaMemcpyAsync(pl->d_image, image, bytes, cudaMemcpyHostToDevice, up);
    if (up_err == cudaSuccess) up_err = cudaStreamSynchronize(up);
    cudaStreamDestroy(up);
  }
  if (up_err != cudaSuccess) return fail(of_fail(ctx, OF_ERR_CUDA, "book upload failed"));
  pl->d_opts = (BookOpt*)(pl->d_image + at_opts);
  pl->d_tiles = (BookTile*)(pl->d_image + at_tiles);
  pl->d_obs = (float*)(pl->d_image + at_obs);
  pl->d_divs = (BookDiv*)(pl->d_image + at_divs);
  pl->d_gc = pl->d_image + at_gc;
  pl->d_begin = (int32_t*)(pl->d_image + at_begin);
  pl->d_counter = (int*)(pl->d_image + at_counter);
  BookParams& P = pl->P;
  P.opts = pl->d_opts;
  P.tiles = pl->d_tiles;
  P.obs_w = pl->d_obs;
  P.divs = pl->d_divs;
  P.n_tiles = (int32_t)nt;
  P.ppt = pl->ppt;
  uint32_t most = 1;  // counter blocks of the longest option
  for (int64_t o = 0; o < n; ++o) {
    const uint32_t spb = opts[(size_t)o].model == OF_MODEL_GBM ? 4 : 2;
    most = std::max(most, ((uint32_t)opts[(size_t)o].steps + spb - 1) / spb);
    if (pl->samples[(size_t)o] >> 32) pl->full = false;
  }
  if (most > kBookTab) pl->full = false;
  P.tab = std::min(most, kBookTab);
  P.keys = of::philox_keys(cfg->seed);
  P.counter = pl->d_counter;
  P.partials = pl->d_partials;
  const int per_sm = of_blocks_per_sm(book_kernel_for(pl, of::KG_TERMINAL), pl->block, pl->smem());
  const int64_t cap = (int64_t)ctx->sm_count * per_sm;
  pl->grid = (int)std::max<int64_t>(1, std::min<int64_t>(cap, (int64_t)nt));
  if (pl->mode != OF_BOOK_PRICE) {
    int64_t start = 0;
    for (int kg = 0; kg < of::KG_COUNT; ++kg) {
      const int64_t end = start + group_tiles[kg];
      BookParams& Q = pl->Pg[kg];
      Q = P;
      Q.tiles = pl->d_tiles + start;
      Q.n_tiles = (int32_t)(end - start);
      Q.counter = pl->d_counter + kg;
      const int per = of_blocks_per_sm(book_kernel_for(pl, kg), pl->block, pl->smem());
      pl->grid_g[kg] = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)ctx->sm_count * per, end - start));
      start = end;
    }
  }
  if (pl->use_graph) {
    cudaStream_t cs = nullptr;
    if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess)
      return fail(of_fail(ctx, OF_ERR_CUDA, "capture stream creation failed"));
    cudaError_t err = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (err == cudaSuccess) {
      book_enqueue(pl, cs);
      err = cudaStreamEndCapture(cs, &pl->graph);
    }
    if (err == cudaSuccess) err = cudaGraphInstantiate(&pl->exec, pl->graph, 0);
    cudaStreamDestroy(cs);
    if (err != cudaSuccess) return fail(of_fail(ctx, OF_ERR_CUDA, "book graph capture failed: %s", cudaGetErrorString(err)));
  }
  *out = pl;
  return OF_OK;
}

extern "C" of_status of_book_plan_launch(of_book_plan* pl) {
  if (!pl) return OF_ERR_INVALID_INPUT;
  OF_TRY(of_ctx_check(pl->ctx));
  if (pl->use_graph) {
    OF_CUDA_TRY(pl->ctx, cudaGraphLaunch(pl->exec, pl->ctx->stream));
  } else {
    book_enqueue(pl, pl->ctx->stream);
    OF_CUDA_TRY(pl->ctx, cudaGetLastError());
  }
  return OF_OK;
}

extern "C" of_status of_book_plan_results(of_book_plan* pl, of_mc_result* res) {
  if (!pl || !res) return OF_ERR_INVALID_INPUT;
  OF_CUDA_TRY(pl->ctx, cudaStreamSynchronize(pl->ctx->stream));
  for (int64_t o = 0; o < pl->n; ++o) {
    of_mc_finish(pl->h_sums + o * pl->nc, pl->samples[(size_t)o], pl->cv_kind[(size_t)o], pl->cv_expected[(size_t)o],
                 pl->discount[(size_t)o], &res[o]);
    res[o].kernel_ms = 0.0;
  }
  return OF_OK;
}

extern "C" of_status of_book_plan_greeks(of_book_plan* pl, of_book_greeks* out) {
  if (!pl || !out) return OF_ERR_INVALID_INPUT;
  if (pl->mode != OF_BOOK_GREEKS && pl->mode != OF_BOOK_GREEKS_FP64)
    return of_fail(pl->ctx, OF_ERR_INVALID_INPUT, "the plan was not created in mode OF_BOOK_GREEKS(_FP64)");
  OF_CUDA_TRY(pl->ctx, cudaStreamSynchronize(pl->ctx->stream));
  for (int64_t o = 0; o < pl->n; ++o) {
    const double* s = pl->h_sums + o * pl->nc;
    const double n = (double)pl->samples[(size_t)o];
    double mean[4], se[4];
    for (int t = 0; t < 4; ++t) {  // the sums are of discounted per-sample derivatives
      mean[t] = s[5 + t] / n;
      const double var = n > 1.0 ? std::fmax(s[9 + t] - s[5 + t] * s[5 + t] / n, 0.0) / (n - 1.0) : 0.0;
      se[t] = std::sqrt(var / n);
    }
    of_book_greeks& g = out[o];
    g.delta = mean[0];
    g.vega = mean[1];
    g.rho = mean[2];
    g.theta = mean[3];
    g.gamma = 0.0;
    g.delta_se = se[0];
    g.vega_se = se[1];
    g.rho_se = se[2];
    g.theta_se = se[3];
    g.gamma_se = 0.0;
  }
  return OF_OK;
}

extern "C" of_status of_book_plan_info(of_book_plan* pl, int32_t* block, int32_t* ppt, int64_t* n_tiles,
                                       double* path_steps) {
  if (!pl) return OF_ERR_INVALID_INPUT;
  if (block) *block = pl->block;
  if (ppt) *ppt = pl->ppt;
  if (n_tiles) *n_tiles = pl->n_tiles;
  if (path_steps) *path_steps = pl->path_steps;
  return OF_OK;
}

// One launch of a book: plan, launch, results (and Greeks when `greeks`).
extern "C" of_status of_book_plan_create(of_ctx* ctx, const of_book_entry* e, int64_t n, const of_book_config* cfg,
                                         of_book_plan** out) {
  return book_plan_create(ctx, e, n, cfg, false, out);
}

static of_status book_run(of_ctx* ctx, const of_book_entry* e, int64_t n, const of_book_config* cfg,
                          of_mc_result* res, of_book_greeks* greeks) {
  of_book_plan* pl = nullptr;
  OF_TRY(book_plan_create(ctx, e, n, cfg, true, &pl));
  cudaEventRecord(ctx->ev_start, ctx->stream);
  of_status st = of_book_plan_launch(pl);
  cudaEventRecord(ctx->ev_stop, ctx->stream);
  if (st == OF_OK) st = of_book_plan_results(pl, res);
  if (st == OF_OK && greeks) st = of_book_plan_greeks(pl, greeks);
  float ms = 0.0f;
  if (st == OF_OK && cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop) == cudaSuccess)
    for (int64_t o = 0; o < n; ++o) res[o].kernel_ms = ms;
  of_book_plan_destroy(pl);
  return st;
}

extern "C" of_status of_mc_price_book(of_ctx* ctx, const of_book_entry* e, int64_t n, const of_book_config* cfg,
                                      of_mc_result* res) {
  if (!ctx || !res || !cfg) return OF_ERR_INVALID_INPUT;
  return book_run(ctx, e, n, cfg, res, nullptr);
}

extern "C" of_status of_mc_price_book_greeks(of_ctx* ctx, const of_book_entry* e, int64_t n, const of_book_config* cfg,
                                             of_mc_result* res, of_book_greeks* greeks) {
  if (!ctx || !res || !cfg || !greeks) return OF_ERR_INVALID_INPUT;
  of_book_config c = *cfg;
  c.mode = OF_BOOK_GREEKS;
  return book_run(ctx, e, n, &c, res, greeks);
}

// FP32 branch of of_mc_run: a one-option book.
of_status of_mc_run_fp32(of_ctx* ctx, const of_model* m, const of_payoff* p, const of_mc_config* c,
                         of_mc_result* out) {
  if (c->injected_normals)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "injected normals are a FP64 reference-mode test hook");
  of_book_entry b{};
  b.model = *m;
  b.payoff = *p;
  b.num_paths = c->num_paths;
  b.antithetic = c->antithetic;
  b.control_variate = c->control_variate;
  b.cv_expected = c->cv_expected;
  b.discount_factor = c->discount_factor;
  of_book_config bc{};
  bc.seed = c->seed;
  bc.use_graph = 0;
  return of_mc_price_book(ctx, &b, 1, &bc, out);
}

// ---------------------------------------------------------------------------
// Strike strip without any allocation (of_mc_strip_noalloc).
//
// For callers that cannot allocate device memory when they price: every
// byte of scratch the strip kernel needs lives in the static array below,
// which each GPU that loads this library holds until the process exits.
// Layout: [sums: 2*MAX_STRIKES doubles][status: one double]
//         [per-block partials: MAX_BLOCKS * 2*MAX_STRIKES doubles].
// In host code `g_strip_noalloc_scratch` names a host-side stand-in, not the
// device array: its device address is looked up with cudaGetSymbolAddress
// with the caller's device current, once per CUDA context (a device's
// primary context, or a context the caller made current), and that address
// is what the kernels get.  The lookups are cached by the context's
// process-unique ID, so a context created after cudaDeviceReset, whose copy
// of the array may sit elsewhere, gets a lookup of its own.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_strip_noalloc_scratch[OF_STRIP_NOALLOC_SCRATCH_BYTES];

namespace {

typedef CUresult (*PfnCtxGetCurrent)(CUcontext*);
typedef CUresult (*PfnCtxGetId)(CUcontext, unsigned long long*);

struct NoallocAddr {
  unsigned long long ctx_id;
  void* addr;
};
constexpr int kNoallocCache = 64;
NoallocAddr g_noalloc_cache[kNoallocCache] = {};
int g_noalloc_used = 0;
std::mutex g_noalloc_mutex;

void noalloc_msg(char* err, size_t len, const char* fmt, ...) {
  if (!err || len == 0) return;
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(err, len, fmt, ap);
  va_end(ap);
}

// The process-unique ID of the calling thread's current CUDA context (0 when
// none is current).  The two driver functions are resolved once through the
// runtime, so the library keeps no link-time dependency on libcuda.
cudaError_t noalloc_ctx_id(unsigned long long* id) {
  static PfnCtxGetCurrent get_current = nullptr;
  static PfnCtxGetId get_id = nullptr;
  static cudaError_t resolved = [] {
    cudaDriverEntryPointQueryResult q1 = cudaDriverEntryPointSymbolNotFound, q2 = cudaDriverEntryPointSymbolNotFound;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", (void**)&get_current, 12000,
                                                     cudaEnableDefault, &q1);
    if (e == cudaSuccess)
      e = cudaGetDriverEntryPointByVersion("cuCtxGetId", (void**)&get_id, 12000, cudaEnableDefault, &q2);
    if (e == cudaSuccess && (q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !get_current ||
                             !get_id))
      e = cudaErrorSymbolNotFound;
    return e;
  }();
  *id = 0;
  if (resolved != cudaSuccess) return resolved;
  CUcontext c = nullptr;
  if (get_current(&c) != CUDA_SUCCESS) return cudaErrorDeviceUninitialized;
  if (!c) return cudaSuccess;
  return get_id(c, id) == CUDA_SUCCESS ? cudaSuccess : cudaErrorDeviceUninitialized;
}

// Device address of the scratch array in the current context.  The first
// call in a context makes the runtime's context current (cudaGetSymbolAddress
// initialises the primary context of the current device if needed).
cudaError_t noalloc_scratch_addr(void** out) {
  unsigned long long id = 0;
  cudaError_t e = noalloc_ctx_id(&id);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> guard(g_noalloc_mutex);
  if (id != 0)
    for (int k = 0; k < g_noalloc_used; ++k)
      if (g_noalloc_cache[k].ctx_id == id) {
        *out = g_noalloc_cache[k].addr;
        return cudaSuccess;
      }
  void* p = nullptr;
  e = cudaGetSymbolAddress(&p, g_strip_noalloc_scratch);
  if (e != cudaSuccess) return e;
  if (!p) return cudaErrorInvalidSymbol;
  if (id == 0 && (e = noalloc_ctx_id(&id)) != cudaSuccess) return e;  // the lookup made a context current
  if (id != 0 && g_noalloc_used < kNoallocCache) g_noalloc_cache[g_noalloc_used++] = {id, p};
  *out = p;
  return cudaSuccess;
}

}  // namespace

extern "C" of_status of_mc_strip_noalloc(void* cuda_stream, const of_model* m, int32_t option_type,
                                         const double* strikes, int64_t n_strikes, const of_mc_config* cfg,
                                         of_mc_result* results, char* err, size_t err_len) {
  if (err && err_len) err[0] = '\0';
  if (!results) {
    noalloc_msg(err, err_len, "null argument");
    return OF_ERR_INVALID_INPUT;
  }
  {
    // The checks of of_mc_strip; the stack context only carries the message.
    of_ctx sink;
    const of_status st = strip_validate(&sink, m, option_type, strikes, n_strikes, cfg);
    if (st != OF_OK) {
      noalloc_msg(err, err_len, "%s", sink.last_error.c_str());
      return st;
    }
  }
  if (n_strikes > OF_STRIP_NOALLOC_MAX_STRIKES) {
    noalloc_msg(err, err_len, "n_strikes must be in [1, %d] (static scratch limit), got %lld",
                OF_STRIP_NOALLOC_MAX_STRIKES, (long long)n_strikes);
    return OF_ERR_INVALID_INPUT;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    noalloc_msg(err, err_len, "cudaGetDevice failed: %s", cudaGetErrorString(e));
    return OF_ERR_CUDA;
  }
  // The call synchronises its stream and copies through host stack buffers,
  // neither of which a stream capture allows: refuse before touching it.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if ((e = cudaStreamIsCapturing((cudaStream_t)cuda_stream, &capture)) != cudaSuccess) {
    noalloc_msg(err, err_len, "cudaStreamIsCapturing failed: %s", cudaGetErrorString(e));
    return OF_ERR_CUDA;
  }
  if (capture != cudaStreamCaptureStatusNone) {
    noalloc_msg(err, err_len, "of_mc_strip_noalloc cannot run on a capturing stream");
    return OF_ERR_UNSUPPORTED;
  }
  void* base = nullptr;
  if ((e = noalloc_scratch_addr(&base)) != cudaSuccess) {
    noalloc_msg(err, err_len, "device address of the static scratch: %s", cudaGetErrorString(e));
    return OF_ERR_CUDA;
  }
  double* d_sums = (double*)base;
  double* d_status = d_sums + OF_STRIP_NOALLOC_MAX_STRIKES * 2;  // the warp-specialised kernel's status word
  double* d_partials = d_status + 1;

  StripParams P{};
  P.c = make_consts(m);
  P.samples = cfg->antithetic ? (cfg->num_paths + 1) / 2 : cfg->num_paths;
  P.steps = (int32_t)m->steps;
  P.n_strikes = (int32_t)n_strikes;
  P.option_type = option_type;
  P.antithetic = cfg->antithetic ? 1 : 0;
  P.s0 = (float)m->s0;
  P.keys = of::philox_keys(cfg->seed);
  for (int64_t k = 0; k < n_strikes; ++k) P.strikes[k] = (float)strikes[k];
  P.status = (uint32_t*)d_status;
  // the kernel of_mc_strip picks for the same request (strikes per lane, tile shape)
  const int block = kStripThreads;
  int sms = 0, per_sm = 0;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) {
    noalloc_msg(err, err_len, "device query failed: %s", cudaGetErrorString(e));
    return OF_ERR_CUDA;
  }
  const StripShape sh = strip_shape(cfg->tile_ilp, P.samples, n_strikes, m->kind, P.antithetic, sms);
  const StripKernelFn fn = sh.fn;
  const size_t smem = sh.smem;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)fn, block, smem)) != cudaSuccess) {
    noalloc_msg(err, err_len, "device query failed: %s", cudaGetErrorString(e));
    return OF_ERR_CUDA;
  }
  const int64_t grid =
      std::min<int64_t>(strip_grid(sh, P.samples, sms, std::max(per_sm, 1)), OF_STRIP_NOALLOC_MAX_BLOCKS);

  cudaStream_t s = (cudaStream_t)cuda_stream;
  const int64_t cols = 2 * n_strikes;
  double hs[2 * OF_STRIP_NOALLOC_MAX_STRIKES];
  uint32_t h_status = 0;
  if (sh.ws && (e = cudaMemsetAsync(d_status, 0, sizeof(double), s)) != cudaSuccess) {
    noalloc_msg(err, err_len, "status reset failed: %s", cudaGetErrorString(e));
    return OF_ERR_CUDA;
  }
  fn<<<(unsigned)grid, block, smem, s>>>(P, d_partials);
  of_launch_reduce_rows(d_partials, grid, cols, d_sums, s);
  if ((e = cudaGetLastError()) != cudaSuccess ||
      (e = cudaMemcpyAsync(hs, d_sums, (size_t)cols * sizeof(double), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
      (sh.ws &&
       (e = cudaMemcpyAsync(&h_status, d_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s)) != cudaSuccess) ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess) {
    noalloc_msg(err, err_len, "strip launch failed: %s", cudaGetErrorString(e));
    return OF_ERR_CUDA;
  }
  if (h_status) {
    noalloc_msg(err, err_len, "strike strip: a producer/consumer ring wait did not complete in time");
    return OF_ERR_TIMEOUT;
  }
  for (int64_t k = 0; k < n_strikes; ++k) {
    const double sums[5] = {hs[2 * k], hs[2 * k + 1], 0.0, 0.0, 0.0};
    of_mc_finish(sums, P.samples, OF_CV_NONE, 0.0, cfg->discount_factor, &results[k]);
    results[k].kernel_ms = 0.0;
  }
  return OF_OK;
}

// ---------------------------------------------------------------------------
// Device peak probes (of_measure_device_peaks)
// ---------------------------------------------------------------------------
namespace {

constexpr int kProbeChains = 8;
constexpr int kProbeBlock = 256;

// kProbeChains independent chains per thread.  One link is five MUFU
// operations (lg2, sqrt, sin, cos, sqrt) and a few FP32 adds that keep the
// value bounded: lg2(x + 1.5) in (0.58, 1.81), sqrt(. + 0.5) in (1.04, 1.52),
// sin in (0.86, 1), cos in (0.54, 0.65), sqrt(. + 0.25) in (0.89, 0.95).
__global__ void __launch_bounds__(kProbeBlock) sfu_probe_kernel(int iters, float* sink) {
  float a[kProbeChains];
#pragma unroll
  for (int k = 0; k < kProbeChains; ++k) a[k] = 0.5f + 0.01f * k + 1e-7f * threadIdx.x;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < kProbeChains; ++k) {
      float x = __log2f(a[k] + 1.5f);
      x = sqrtf(x + 0.5f);
      x = __sinf(x);
      x = __cosf(x);
      a[k] = sqrtf(x + 0.25f);
    }
  }
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < kProbeChains; ++k) s += a[k];
  if (s < 0.0f) sink[blockIdx.x] = s;  // never taken (s > 7); keeps the chains live
}

// kProbeChains independent FMA chains per thread converging to 1.
__global__ void __launch_bounds__(kProbeBlock) fma_probe_kernel(int iters, float* sink) {
  float a[kProbeChains];
#pragma unroll
  for (int k = 0; k < kProbeChains; ++k) a[k] = 0.5f + 0.01f * k + 1e-7f * threadIdx.x;
#pragma unroll 16
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < kProbeChains; ++k) a[k] = fmaf(a[k], 0.99993896484375f, 6.103515625e-5f);
  }
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < kProbeChains; ++k) s += a[k];
  if (s < 0.0f) sink[blockIdx.x] = s;  // never taken; keeps the chains live
}

// kProbeChains independent FP64 FMA chains per thread converging to 1.
__global__ void __launch_bounds__(kProbeBlock) dfma_probe_kernel(int iters, double* sink) {
  double a[kProbeChains];
#pragma unroll
  for (int k = 0; k < kProbeChains; ++k) a[k] = 0.5 + 0.01 * k + 1e-7 * threadIdx.x;
#pragma unroll 16
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < kProbeChains; ++k) a[k] = fma(a[k], 0.99993896484375, 6.103515625e-5);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < kProbeChains; ++k) s += a[k];
  if (s < 0.0) sink[blockIdx.x] = s;  // never taken; keeps the chains live
}

}  // namespace

extern "C" of_status of_measure_device_peaks(of_ctx* ctx, of_device_peaks* out) {
  if (!ctx || !out) return OF_ERR_INVALID_INPUT;
  OF_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int per_sm_s = of_blocks_per_sm((const void*)sfu_probe_kernel, kProbeBlock, 0);
  const int per_sm_f = of_blocks_per_sm((const void*)fma_probe_kernel, kProbeBlock, 0);
  const int per_sm_d = of_blocks_per_sm((const void*)dfma_probe_kernel, kProbeBlock, 0);
  const int grid_s = ctx->sm_count * std::max(per_sm_s, 1), grid_f = ctx->sm_count * std::max(per_sm_f, 1);
  const int grid_d = ctx->sm_count * std::max(per_sm_d, 1);
  void* sink = nullptr;
  OF_TRY(of_scratch(ctx, SLOT_MISC, (size_t)std::max(std::max(grid_s, grid_f), grid_d) * sizeof(double), &sink));
  const int it_s = 2048, it_f = 65536;
  // warm-up (clocks up), then the best of three timed launches of each probe
  sfu_probe_kernel<<<grid_s, kProbeBlock, 0, ctx->stream>>>(it_s / 8, (float*)sink);
  fma_probe_kernel<<<grid_f, kProbeBlock, 0, ctx->stream>>>(it_f / 8, (float*)sink);
  OF_CUDA_TRY(ctx, cudaGetLastError());
  float best_s = 1e30f, best_f = 1e30f;
  for (int rep = 0; rep < 3; ++rep) {
    float ms = 0.0f;
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_start, ctx->stream));
    sfu_probe_kernel<<<grid_s, kProbeBlock, 0, ctx->stream>>>(it_s, (float*)sink);
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_stop, ctx->stream));
    OF_CUDA_TRY(ctx, cudaEventSynchronize(ctx->ev_stop));
    OF_CUDA_TRY(ctx, cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
    best_s = std::min(best_s, ms);
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_start, ctx->stream));
    fma_probe_kernel<<<grid_f, kProbeBlock, 0, ctx->stream>>>(it_f, (float*)sink);
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_stop, ctx->stream));
    OF_CUDA_TRY(ctx, cudaEventSynchronize(ctx->ev_stop));
    OF_CUDA_TRY(ctx, cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
    best_f = std::min(best_f, ms);
  }
  // FP64: warm-up, then the best of three
  const int it_d = 4096;
  float best_d = 1e30f;
  dfma_probe_kernel<<<grid_d, kProbeBlock, 0, ctx->stream>>>(it_d / 8, (double*)sink);
  for (int rep = 0; rep < 3; ++rep) {
    float ms = 0.0f;
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_start, ctx->stream));
    dfma_probe_kernel<<<grid_d, kProbeBlock, 0, ctx->stream>>>(it_d, (double*)sink);
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_stop, ctx->stream));
    OF_CUDA_TRY(ctx, cudaEventSynchronize(ctx->ev_stop));
    OF_CUDA_TRY(ctx, cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
    best_d = std::min(best_d, ms);
  }
  OF_CUDA_TRY(ctx, cudaGetLastError());
  const double threads_s = (double)grid_s * kProbeBlock, threads_f = (double)grid_f * kProbeBlock;
  const double threads_d = (double)grid_d * kProbeBlock;
  out->sfu_ops_per_s = threads_s * it_s * kProbeChains * 5.0 / (best_s * 1e-3);
  out->fp32_flops_per_s = threads_f * (double)it_f * kProbeChains * 2.0 / (best_f * 1e-3);
  out->fp64_flops_per_s = threads_d * (double)it_d * kProbeChains * 2.0 / (best_d * 1e-3);
  out->probe_ms = (double)best_s + (double)best_f + (double)best_d;
  return OF_OK;
}
