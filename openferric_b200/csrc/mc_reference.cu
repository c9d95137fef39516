// mc_reference.cu - FP64 reference-stream Monte Carlo (of_mc_run, FP64 mode).
//
// Reproduces openferric's MonteCarloEngine::run (src/mc/simulation.rs:182-348)
// draw for draw: sample i owns a xoshiro256++ stream seeded with
// seed + i*7919, draws z1[j] (and z2[j] for Heston) per step in the reference's
// interleaved order, builds the path with the reference generators and
// evaluates the payoff and control variate.  One thread owns one sample and
// keeps the path in registers: the running barrier flag and the per-step
// observation sums replace the reference's Vec<f64> path buffer.  An
// antithetic sample advances its negated twin in the same loop.
//
// This file is compiled with --fmad=false: the only fused multiply-adds are
// the explicit fma() calls standing for the reference's mul_add.
#include <cmath>
#include <cstring>
#include <vector>

#include "of_device.cuh"
#include "of_internal.h"
#include "ref_stream.cuh"

namespace {

struct RefParams {
  int32_t model, payoff, option_type, antithetic;
  int32_t cv_kind, barrier_up, barrier_in, averaging;
  int32_t floating, terminal_only, need_arith, need_geo;
  int64_t samples, steps;
  uint64_t seed;
  double s0, strike, barrier, rebate, n_obs;
  double drift, diffusion;  // GBM (simulation.rs:63-66)
  double mu, dt, sqrt_dt, kappa, theta, xi, rho, rho_c, v0;  // Heston (stochastic.rs:56-71)
  const double* obs_w;  // [steps+1] observation counts
  const double* inj;    // injected normals or nullptr
  const of_div_trigger* div;  // GBM discrete dividends by trigger step, or nullptr
  int32_t n_div;
  // the log-space kernels
  int32_t bar_hit0;           // barrier: path[0] is beyond the level
  double bar_sign, bar_thr, bar_step;  // +1 up / -1 down; threshold of sign * sum(z) before step 1, its move per step
  double w0, geo0;            // Asian: observations of path[0]; sum of w_j (ln s0 + j drift)
  double y_floor;             // Heston: ln(1e-12 / s0)
  const double2* obs;         // Asian: (w_j, w_j e^(j drift)) of steps 1..steps
  double* partials;           // [blocks][5]
  unsigned* ticket;
  double* out;                // [5], pinned host memory
};

struct Leg {
  double s, v, arith, geo;
  bool hit;
};

__device__ __forceinline__ double vanilla(int option_type, double spot, double strike) {
  const double v = option_type == OF_CALL ? spot - strike : strike - spot;
  return v > 0.0 ? v : 0.0;
}

__device__ __forceinline__ void observe(Leg& L, const RefParams& P, int64_t idx) {
  if (P.payoff == OF_PAYOFF_BARRIER) L.hit |= P.barrier_up ? (L.s >= P.barrier) : (L.s <= P.barrier);
  if (P.need_arith | P.need_geo) {
    const double w = __ldg(P.obs_w + idx);
    if (w != 0.0) {
      if (P.need_arith) L.arith += w * L.s;
      if (P.need_geo) L.geo += w * log(L.s > 1e-12 ? L.s : 1e-12);
    }
  }
}

__device__ __forceinline__ void leg_init(Leg& L, const RefParams& P) {
  L.s = P.s0;
  L.v = P.v0;
  L.arith = -0.0;
  L.geo = -0.0;
  L.hit = false;
  observe(L, P, 0);
}

// HestonPathGenerator::generate_into + Heston::step_euler
// (simulation.rs:104-115, stochastic.rs:56-71), operation order preserved.
__device__ __forceinline__ void heston_step(Leg& L, const RefParams& P, double z1, double z2) {
  const double v_pos = L.v > 0.0 ? L.v : 0.0;
  const double zs = P.rho * z1 + P.rho_c * z2;
  double v_next = L.v + P.kappa * (P.theta - v_pos) * P.dt + P.xi * sqrt(v_pos) * P.sqrt_dt * z1;
  v_next = v_next > 0.0 ? v_next : 0.0;
  const double s_next = L.s * exp((P.mu - 0.5 * v_pos) * P.dt + sqrt(v_pos) * P.sqrt_dt * zs);
  L.s = s_next > 1e-12 ? s_next : 1e-12;
  L.v = v_next;
}

// payoff_from_path (mc_engine.rs:453-545) on the register-resident path summary.
__device__ __forceinline__ double leg_payoff(const Leg& L, const RefParams& P) {
  switch (P.payoff) {
    case OF_PAYOFF_VANILLA:
      return vanilla(P.option_type, L.s, P.strike);
    case OF_PAYOFF_BARRIER: {
      const bool active = P.barrier_in ? L.hit : !L.hit;
      return active ? vanilla(P.option_type, L.s, P.strike) : P.rebate;
    }
    default: {
      double avg;
      if (P.terminal_only) avg = L.s;
      else if (P.averaging == OF_AVG_ARITHMETIC) avg = L.arith / P.n_obs;
      else avg = exp(L.geo / P.n_obs);
      return P.floating ? vanilla(P.option_type, L.s, avg) : vanilla(P.option_type, avg, P.strike);
    }
  }
}

// Control-variate evaluators (mc_engine.rs:481-483, :570-581; simulation.rs:441-444).
__device__ __forceinline__ double leg_cv(const Leg& L, const RefParams& P) {
  switch (P.cv_kind) {
    case OF_CV_VANILLA_TERMINAL:
      return vanilla(P.option_type, L.s, P.strike);
    case OF_CV_GEOMETRIC_ASIAN:
      return vanilla(P.option_type, P.terminal_only ? L.s : exp(L.geo / P.n_obs), P.strike);
    case OF_CV_TERMINAL_SPOT:
      return L.s;
    default:
      return 0.0;
  }
}

// DividendEvent::apply_jump (src/market/dividends.rs:76-83).
__device__ __forceinline__ double dividend_jump(const of_div_trigger& e, double s) {
  if (e.kind == OF_DIV_CASH) {
    const double x = s - e.amount;
    return x > 0.0 ? x : 0.0;
  }
  return s * (1.0 - e.amount);
}

// RNG: of::Xoshiro256pp or of::Pcg64, the FastRngKind of the engine.
template <typename RNG>
__global__ void __launch_bounds__(128) mc_ref_kernel(RefParams P, double* __restrict__ partials) {
  __shared__ double sh[5 * 4];
  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const bool heston = P.model != OF_MODEL_GBM;
  const int streams = heston ? 2 : 1;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.samples; i += stride) {
    RNG rng;
    const double* inj = P.inj ? P.inj + i * P.steps * streams : nullptr;
    if (!inj) rng.seed(P.seed + (uint64_t)i * 7919ULL);  // stream_seed, fast_rng.rs:203-205
    Leg a, b;
    leg_init(a, P);
    if (P.antithetic) leg_init(b, P);
    int32_t ev = 0;  // next dividend trigger
    for (int64_t j = 0; j < P.steps; ++j) {
      double z1, z2 = 0.0;
      if (inj) {
        z1 = inj[j * streams];
        if (heston) z2 = inj[j * streams + 1];
      } else {
        z1 = of::acklam_inv_cdf(rng.next_f64());
        if (heston) z2 = of::acklam_inv_cdf(rng.next_f64());
      }
      if (!heston) {
        a.s *= exp(fma(P.diffusion, z1, P.drift));  // simulation.rs:67-71
        if (P.antithetic) b.s *= exp(fma(P.diffusion, -z1, P.drift));
        for (; ev < P.n_div && P.div[ev].step == j; ++ev) {  // mc_engine.rs:157-167
          a.s = dividend_jump(P.div[ev], a.s);
          if (P.antithetic) b.s = dividend_jump(P.div[ev], b.s);
        }
      } else {
        heston_step(a, P, z1, z2);
        if (P.antithetic) heston_step(b, P, -z1, -z2);
      }
      observe(a, P, j + 1);
      if (P.antithetic) observe(b, P, j + 1);
    }
    double x = leg_payoff(a, P);
    double y = leg_cv(a, P);
    if (P.antithetic) {  // simulation.rs:235-252
      x = 0.5 * (x + leg_payoff(b, P));
      y = 0.5 * (y + leg_cv(b, P));
    }
    acc[0] += x;
    acc[1] += x * x;
    acc[2] += y;
    acc[3] += x * y;
    acc[4] += y * y;
  }
  of::block_sum<5>(acc, sh);
  if (threadIdx.x == 0)
    for (int k = 0; k < 5; ++k) partials[(int64_t)blockIdx.x * 5 + k] = acc[k];
}

// ---------------------------------------------------------------------------
// The kernels of the reference stream without injected normals and without
// dividends: one lane per sample, the normals of ref_stream.cuh, log-space
// paths.  A step's factor exp(drift + diff z) multiplies the spot in the
// reference (simulation.rs:67-71); here its exponent is added, and the spot is
// formed where a payoff reads it.  The draws are the same and the roundings
// fewer: prices agree with mc_ref_kernel's to about 1e-15 relative.
//
// What bounds them: instruction issue, shared by the FP64 pipe (17 operations
// a draw) and the integer pipe (the xoshiro update, 24), about 100 cycles a
// draw and warp at five warps per scheduler.  mc_ref_kernel spent most of its
// issue slots in the tails' branch and the per-step exp.  Device time before
// and after on one B200 (launch included):
//   European 100,000 x 252              387 -> 90 us
//   Asian 50,000 pairs x 252, both averages  ~660 -> 95 us
//   knock-out 25,001 pairs x 126        144 -> 37 us
//   Heston European 131,072 x 256       940 -> 250 us
// ---------------------------------------------------------------------------
constexpr int kRefThreads = 64;  // small blocks: 100,000 samples fill 148 SMs to 96 %, blocks of 128 to 88 %

__device__ __forceinline__ void ref_account(const RefParams& P, const Leg& a, const Leg& b, double (&acc)[5]) {
  double x = leg_payoff(a, P);
  double y = leg_cv(a, P);
  if (P.antithetic) {  // simulation.rs:235-252
    x = 0.5 * (x + leg_payoff(b, P));
    y = 0.5 * (y + leg_cv(b, P));
  }
  acc[0] += x;
  acc[1] += x * x;
  acc[2] += y;
  acc[3] += x * y;
  acc[4] += y * y;
}

// GBM European (its control variate, if any, reads S_T only): the sum of the
// path's normals, one exp per leg.
template <typename RNG>
__global__ void __launch_bounds__(kRefThreads) mc_ref_gbm_terminal(const __grid_constant__ RefParams P) {
  __shared__ double list[kRefThreads * of::kTailCap];
  __shared__ double sh[kRefThreads];
  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const int64_t stride = (int64_t)gridDim.x * kRefThreads;
  const double base = P.drift * (double)P.steps;
  for (int64_t first = (int64_t)blockIdx.x * kRefThreads; first < P.samples; first += stride) {
    const int64_t i = first + threadIdx.x;
    RNG rng;
    rng.seed(P.seed + (uint64_t)i * 7919ULL);  // stream_seed, fast_rng.rs:203-205
    const double w = of::stream_normal_sum(rng, P.steps, list + threadIdx.x, kRefThreads);
    if (i < P.samples) {
      Leg a{P.s0 * exp(fma(P.diffusion, w, base)), 0.0, 0.0, 0.0, false}, b = a;
      if (P.antithetic) b.s = P.s0 * exp(fma(-P.diffusion, w, base));
      ref_account(P, a, b, acc);
    }
  }
  of::grid_sum<5, kRefThreads>(acc, sh, P.partials, P.ticket, P.out);
}

// GBM barrier or Asian.  With W the running sum of the normals, the log-spot
// of a leg after step j is j drift +- diff W:
//   barrier: the spot is beyond the level when +-W reaches a threshold that
//     moves by -drift/diff a step (no exp, one comparison per leg);
//   Asian: sum_j w_j e^(j drift) E^(+-1), E = exp(diff W), with the
//     weights w_j e^(j drift) from the host: the antithetic leg costs a
//     reciprocal instead of a second exp; the geometric sum is diff sum w_j W_j.
enum : int { RK_BARRIER = 0, RK_ARITH = 1, RK_GEO = 2, RK_BOTH = 3 };

template <typename RNG, int KIND, bool ANTI>
__global__ void __launch_bounds__(kRefThreads) mc_ref_gbm_path(const __grid_constant__ RefParams P) {
  __shared__ of::DrawBuf bufs[kRefThreads / 32];
  __shared__ double tab[64];
  __shared__ double sh[kRefThreads];
  constexpr bool kArith = KIND == RK_ARITH || KIND == RK_BOTH, kGeo = KIND == RK_GEO || KIND == RK_BOTH;
  if (kArith) of::exp_table_load(tab);
  __syncthreads();
  of::DrawBuf& buf = bufs[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const int64_t stride = (int64_t)gridDim.x * kRefThreads;
  const double base = P.drift * (double)P.steps;
  const int32_t steps = (int32_t)P.steps;
  for (int64_t first = (int64_t)blockIdx.x * kRefThreads; first < P.samples; first += stride) {
    const int64_t i = first + threadIdx.x;
    RNG rng;
    rng.seed(P.seed + (uint64_t)i * 7919ULL);
    double w = 0.0, aa = P.w0, ab = P.w0, g = 0.0, thr = P.bar_thr;
    bool ha = P.bar_hit0 != 0, hb = ha;
    for (int32_t j0 = 0; j0 < steps; j0 += of::kDrawBatch) {
      const int n = steps - j0 < of::kDrawBatch ? steps - j0 : of::kDrawBatch;
      of::stream_normals(rng, buf, lane, n);
#pragma unroll 4
      for (int k = 0; k < n; ++k) {
        w += buf.z[k * 32 + lane];
        if (KIND == RK_BARRIER) {
          thr += P.bar_step;
          const double sw = P.bar_sign * w;
          ha |= sw >= thr;
          if (ANTI) hb |= -sw >= thr;
        } else {
          const double2 c = __ldg(P.obs + j0 + k);  // (w_j, w_j e^(j drift)) of step j0 + k + 1
          if (c.x != 0.0) {
            if (kArith) {
              const double e = of::exp64(P.diffusion * w, tab);
              aa = fma(c.y, e, aa);
              if (ANTI) ab = fma(c.y, of::rcp64(e), ab);
            }
            if (kGeo) g = fma(c.x, w, g);
          }
        }
      }
      __syncwarp();
    }
    if (i < P.samples) {
      const double y = P.diffusion * w, gy = P.diffusion * g;
      Leg a{P.s0 * exp(base + y), 0.0, P.s0 * aa, P.geo0 + gy, ha}, b = a;
      if (ANTI) b = Leg{P.s0 * exp(base - y), 0.0, P.s0 * ab, P.geo0 - gy, hb};
      ref_account(P, a, b, acc);
    }
  }
  of::grid_sum<5, kRefThreads>(acc, sh, P.partials, P.ticket, P.out);
}

// Heston European: heston_step with the log-spot in place of the spot.
template <typename RNG, bool ANTI>
__global__ void __launch_bounds__(kRefThreads) mc_ref_heston(const __grid_constant__ RefParams P) {
  __shared__ of::DrawBuf bufs[kRefThreads / 32];
  __shared__ double sh[kRefThreads];
  of::DrawBuf& buf = bufs[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const int64_t stride = (int64_t)gridDim.x * kRefThreads;
  const int32_t steps = (int32_t)P.steps;
  const double mudt = P.mu * P.dt, hdt = 0.5 * P.dt, omk = 1.0 - P.kappa * P.dt, kth = P.kappa * P.theta * P.dt;
  const double xsd = P.xi * P.sqrt_dt, r1 = P.rho * P.sqrt_dt, r2 = P.rho_c * P.sqrt_dt;
  auto step = [&](double& y, double& v, double z1, double zs) {
    const double sq = of::sqrt64_from0(v);
    const double y_next = fma(sq, zs, fma(-hdt, v, y + mudt)), v_next = fma(sq, xsd * z1, fma(omk, v, kth));
    y = y_next > P.y_floor ? y_next : P.y_floor;
    v = v_next > 0.0 ? v_next : 0.0;
  };
  for (int64_t first = (int64_t)blockIdx.x * kRefThreads; first < P.samples; first += stride) {
    const int64_t i = first + threadIdx.x;
    RNG rng;
    rng.seed(P.seed + (uint64_t)i * 7919ULL);
    double ya = 0.0, yb = 0.0, va = P.v0, vb = va;
    for (int32_t j0 = 0; j0 < steps; j0 += of::kDrawBatch / 2) {
      const int n = steps - j0 < of::kDrawBatch / 2 ? steps - j0 : of::kDrawBatch / 2;
      of::stream_normals(rng, buf, lane, 2 * n);
#pragma unroll 2
      for (int k = 0; k < n; ++k) {
        const double z1 = buf.z[2 * k * 32 + lane], z2 = buf.z[(2 * k + 1) * 32 + lane];
        const double zs = fma(r1, z1, r2 * z2);
        step(ya, va, z1, zs);
        if (ANTI) step(yb, vb, -z1, -zs);
      }
      __syncwarp();
    }
    if (i < P.samples) {
      Leg a{P.s0 * exp(ya), 0.0, 0.0, 0.0, false}, b = a;
      if (ANTI) b.s = P.s0 * exp(yb);
      ref_account(P, a, b, acc);
    }
  }
  of::grid_sum<5, kRefThreads>(acc, sh, P.partials, P.ticket, P.out);
}

typedef void (*RefKernel)(RefParams);

template <typename RNG, bool ANTI>
RefKernel ref_path_kernel(int kind) {
  return kind == RK_BARRIER ? mc_ref_gbm_path<RNG, RK_BARRIER, ANTI>
         : kind == RK_ARITH ? mc_ref_gbm_path<RNG, RK_ARITH, ANTI>
         : kind == RK_GEO   ? mc_ref_gbm_path<RNG, RK_GEO, ANTI>
                            : mc_ref_gbm_path<RNG, RK_BOTH, ANTI>;
}

// The log-space kernel for a request, or null where the general one runs:
// injected normals, dividends (they act on the spot), path-dependent payoffs
// under Heston, barriers under a vanishing volatility, Asians with so many
// steps that their weights should not be staged in pinned memory, and Asians
// whose log-spot could leave the range of exp64 or reach the reference's
// 1e-12 floor under the logarithm.  (A sum of normals beyond 40 standard
// deviations has probability below 1e-300.)
template <typename RNG>
RefKernel ref_kernel_for(const RefParams& P) {
  if (P.inj || P.n_div) return nullptr;
  const bool obs = P.need_arith || P.need_geo;
  if (P.model != OF_MODEL_GBM) {
    if (P.payoff != OF_PAYOFF_VANILLA || obs) return nullptr;
    return P.antithetic ? mc_ref_heston<RNG, true> : mc_ref_heston<RNG, false>;
  }
  if (P.payoff == OF_PAYOFF_VANILLA && !obs) return mc_ref_gbm_terminal<RNG>;
  if (P.payoff == OF_PAYOFF_BARRIER && !obs && P.diffusion > 1e-100)
    return P.antithetic ? ref_path_kernel<RNG, true>(RK_BARRIER) : ref_path_kernel<RNG, false>(RK_BARRIER);
  if (P.payoff != OF_PAYOFF_ASIAN || !obs || P.steps > (1 << 16)) return nullptr;
  const double n = (double)P.steps, spread = 40.0 * P.diffusion * std::sqrt(n), drift = P.drift * n;
  if (!(spread + std::fabs(drift) < 600.0)) return nullptr;
  if (P.need_geo && !(std::log(P.s0) + std::fmin(drift, 0.0) - spread > std::log(1e-12))) return nullptr;
  const int kind = P.need_arith ? (P.need_geo ? RK_BOTH : RK_ARITH) : RK_GEO;
  return P.antithetic ? ref_path_kernel<RNG, true>(kind) : ref_path_kernel<RNG, false>(kind);
}

}  // namespace

// Observation index of average_for_observations (mc_engine.rs:100-104):
// round(t / maturity * (len-1)) saturated into [0, len-1].
static int64_t obs_index(double t, double maturity, int64_t len) {
  const double idx = std::round((t / maturity) * (double)(len - 1));
  int64_t i = (std::isnan(idx) || idx <= 0.0) ? 0 : (int64_t)idx;
  return i < len - 1 ? i : len - 1;
}

of_status of_dividend_triggers(of_ctx* ctx, const of_model* m, std::vector<of_div_trigger>& out) {
  out.clear();
  if (m->n_dividends <= 0) return OF_OK;
  if (!m->dividends) return of_fail(ctx, OF_ERR_INVALID_INPUT, "dividends is null");
  if (m->kind != OF_MODEL_GBM)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "discrete dividends apply to GBM paths only");
  double prev = 0.0;
  for (int64_t e = 0; e < m->n_dividends; ++e) {
    const of_dividend_event& d = m->dividends[e];
    if (!std::isfinite(d.time) || d.time <= 0.0)
      return of_fail(ctx, OF_ERR_INVALID_INPUT, "dividend event time must be finite and > 0");
    if (d.kind == OF_DIV_CASH) {
      if (!std::isfinite(d.amount) || d.amount < 0.0)
        return of_fail(ctx, OF_ERR_INVALID_INPUT, "cash dividend amount must be finite and >= 0");
    } else if (d.kind == OF_DIV_PROPORTIONAL) {
      if (!std::isfinite(d.amount) || d.amount < 0.0 || d.amount >= 1.0)
        return of_fail(ctx, OF_ERR_INVALID_INPUT, "proportional dividend ratio must be finite and in [0, 1)");
    } else {
      return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown dividend kind %d", d.kind);
    }
    if (d.time <= prev) return of_fail(ctx, OF_ERR_INVALID_INPUT, "dividend event times must be strictly increasing");
    prev = d.time;
  }
  const double dt = m->maturity / (double)m->steps;
  int64_t ev = 0;
  for (int64_t j = 0; j < m->steps && ev < m->n_dividends; ++j) {
    const double t = (double)(j + 1) * dt;
    while (ev < m->n_dividends && m->dividends[ev].time <= m->maturity + 1.0e-12 &&
           m->dividends[ev].time <= t + 1.0e-12) {
      out.push_back(of_div_trigger{(int32_t)j, m->dividends[ev].kind, m->dividends[ev].amount});
      ++ev;
    }
  }
  return OF_OK;
}

of_status of_validate_mc(of_ctx* ctx, const of_model* m, const of_payoff* p, const of_mc_config* c) {
  if (!m || !p || !c) return of_fail(ctx, OF_ERR_INVALID_INPUT, "null argument");
  if (c->num_paths <= 0) return of_fail(ctx, OF_ERR_INVALID_INPUT, "num_paths must be > 0");
  if (m->steps <= 0) return of_fail(ctx, OF_ERR_INVALID_INPUT, "num_steps must be > 0");
  if (m->steps > (int64_t)1 << 30) return of_fail(ctx, OF_ERR_INVALID_INPUT, "num_steps too large");
  if (!(m->maturity > 0.0) || !std::isfinite(m->maturity))
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "maturity must be finite and > 0");
  if (!(m->s0 > 0.0) || !std::isfinite(m->s0)) return of_fail(ctx, OF_ERR_INVALID_INPUT, "spot must be > 0");
  if (!std::isfinite(m->mu)) return of_fail(ctx, OF_ERR_INVALID_INPUT, "drift must be finite");
  if (m->kind == OF_MODEL_GBM) {
    if (!(m->sigma > 0.0) || !std::isfinite(m->sigma))
      return of_fail(ctx, OF_ERR_INVALID_INPUT, "market volatility must be > 0");
  } else if (m->kind == OF_MODEL_HESTON_EULER || m->kind == OF_MODEL_HESTON_QE) {
    // Heston::validate, src/models/stochastic.rs:47-54
    if (!(m->kappa > 0.0 && m->theta >= 0.0 && m->xi >= 0.0 && m->v0 >= 0.0 && m->rho > -1.0 && m->rho < 1.0))
      return of_fail(ctx, OF_ERR_INVALID_INPUT, "invalid Heston parameters");
  } else {
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown model kind %d", m->kind);
  }
  if (m->n_dividends > 0) {
    std::vector<of_div_trigger> trig;
    OF_TRY(of_dividend_triggers(ctx, m, trig));
  }
  if (p->option_type != OF_CALL && p->option_type != OF_PUT)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown option type %d", p->option_type);
  if (p->kind < OF_PAYOFF_VANILLA || p->kind > OF_PAYOFF_ASIAN)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown payoff kind %d", p->kind);
  if (!std::isfinite(p->strike)) return of_fail(ctx, OF_ERR_INVALID_INPUT, "strike must be finite");
  if (p->kind == OF_PAYOFF_ASIAN && p->n_observations > 0 && !p->observation_times)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "observation_times is null");
  if (c->rng_kind != OF_RNG_XOSHIRO256PP && c->rng_kind != OF_RNG_PCG64)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown rng kind %d", c->rng_kind);
  if (c->rng_kind != OF_RNG_XOSHIRO256PP && c->precision != OF_PREC_FP64_REFERENCE)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "the FP32 Philox mode draws from Philox streams only");
  if (c->control_variate < OF_CV_NONE || c->control_variate > OF_CV_TERMINAL_SPOT)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown control variate %d", c->control_variate);
  if (!std::isfinite(c->discount_factor)) return of_fail(ctx, OF_ERR_INVALID_INPUT, "discount factor must be finite");
  return OF_OK;
}

// Observation counts per step index for the Asian payoff / geometric CV.
// Returns terminal_only = true where average_for_observations falls back to
// the terminal spot (no observations or maturity <= 0, mc_engine.rs:92-94).
void of_observation_weights(const of_payoff* p, int64_t steps, std::vector<double>& w, bool& terminal_only) {
  w.assign((size_t)steps + 1, 0.0);
  terminal_only = !(p->n_observations > 0 && p->expiry > 0.0);
  if (terminal_only) return;
  for (int64_t k = 0; k < p->n_observations; ++k) w[(size_t)obs_index(p->observation_times[k], p->expiry, steps + 1)] += 1.0;
}

of_status of_mc_run_fp32(of_ctx* ctx, const of_model* model, const of_payoff* payoff, const of_mc_config* cfg,
                         of_mc_result* out);

extern "C" of_status of_mc_run(of_ctx* ctx, const of_model* m, const of_payoff* p, const of_mc_config* c,
                               of_mc_result* out) {
  if (!ctx || !out) return OF_ERR_INVALID_INPUT;
  OF_TRY(of_validate_mc(ctx, m, p, c));
  if (c->precision == OF_PREC_FP32_PHILOX) return of_mc_run_fp32(ctx, m, p, c, out);
  if (c->precision != OF_PREC_FP64_REFERENCE)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown precision %d", c->precision);
  if (m->kind == OF_MODEL_HESTON_QE)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "the QE scheme has no FP64 reference-stream mode");
  OF_CUDA_TRY(ctx, cudaSetDevice(ctx->device));

  RefParams P{};
  P.model = m->kind;
  P.payoff = p->kind;
  P.option_type = p->option_type;
  P.antithetic = c->antithetic ? 1 : 0;
  P.cv_kind = c->control_variate;
  P.barrier_up = p->barrier_direction == OF_BARRIER_UP;
  P.barrier_in = p->barrier_style == OF_BARRIER_IN;
  P.averaging = p->averaging;
  P.floating = p->strike_type == OF_STRIKE_FLOATING;
  P.samples = c->antithetic ? (c->num_paths + 1) / 2 : c->num_paths;
  P.steps = m->steps;
  P.seed = c->seed;
  P.s0 = m->s0;
  P.strike = p->strike;
  P.barrier = p->barrier_level;
  P.rebate = p->rebate;
  P.v0 = m->v0;
  const double dt = m->maturity / (double)m->steps;
  const double sqrt_dt = std::sqrt(dt);
  P.drift = (m->mu - 0.5 * m->sigma * m->sigma) * dt;
  P.diffusion = m->sigma * sqrt_dt;
  P.mu = m->mu;
  P.dt = dt;
  P.sqrt_dt = sqrt_dt;
  P.kappa = m->kappa;
  P.theta = m->theta;
  P.xi = m->xi;
  P.rho = m->rho;
  P.rho_c = std::sqrt(1.0 - m->rho * m->rho);

  const bool asian = p->kind == OF_PAYOFF_ASIAN;
  P.need_arith = asian && p->averaging == OF_AVG_ARITHMETIC;
  P.need_geo = (asian && p->averaging == OF_AVG_GEOMETRIC) || c->control_variate == OF_CV_GEOMETRIC_ASIAN;
  std::vector<double> w;
  bool terminal_only = true;
  if (P.need_arith || P.need_geo) {
    of_observation_weights(p, m->steps, w, terminal_only);
    if (terminal_only) P.need_arith = P.need_geo = 0;
  }
  P.terminal_only = terminal_only;
  P.n_obs = (double)p->n_observations;

  std::vector<of_div_trigger> trig;
  OF_TRY(of_dividend_triggers(ctx, m, trig));
  if (!trig.empty()) {
    void* d_div = nullptr;
    OF_TRY(of_scratch(ctx, SLOT_DIVIDENDS, trig.size() * sizeof(of_div_trigger), &d_div));
    OF_CUDA_TRY(ctx, cudaMemcpyAsync(d_div, trig.data(), trig.size() * sizeof(of_div_trigger),
                                     cudaMemcpyHostToDevice, ctx->stream));
    P.div = (const of_div_trigger*)d_div;
    P.n_div = (int32_t)trig.size();
  }

  const int streams = m->kind == OF_MODEL_GBM ? 1 : 2;
  if (c->injected_normals) {
    const int64_t need = P.samples * P.steps * streams;
    if (c->n_injected < need)
      return of_fail(ctx, OF_ERR_INVALID_INPUT, "injected normals: need %lld values, got %lld", (long long)need,
                     (long long)c->n_injected);
    void* d_inj = nullptr;
    OF_TRY(of_scratch(ctx, SLOT_INJECT, (size_t)need * sizeof(double), &d_inj));
    OF_CUDA_TRY(ctx, cudaMemcpyAsync(d_inj, c->injected_normals, (size_t)need * sizeof(double),
                                     cudaMemcpyHostToDevice, ctx->stream));
    P.inj = (const double*)d_inj;
  }

  void *d_part = nullptr, *h = nullptr;
  double sums[5];
  float ms = 0.0f;
  const bool pcg = c->rng_kind == OF_RNG_PCG64;
  if (RefKernel fast = pcg ? ref_kernel_for<of::Pcg64>(P) : ref_kernel_for<of::Xoshiro256pp>(P)) {
    const bool obs = P.need_arith || P.need_geo;
    const size_t table = obs ? (size_t)P.steps * sizeof(double2) : 0;
    OF_TRY(of_pinned(ctx, table + 5 * sizeof(double), &h));
    if (obs) {
      void* d_obs = nullptr;
      OF_TRY(of_scratch(ctx, SLOT_OBS, table, &d_obs));
      double2* t = (double2*)h;
      double geo = 0.0;
      for (int64_t j = 1; j <= P.steps; ++j) {
        const double wj = w[(size_t)j], yj = P.drift * (double)j;
        t[j - 1] = make_double2(wj, wj != 0.0 ? wj * std::exp(yj) : 0.0);
        geo += wj * yj;
      }
      P.w0 = w[0];
      P.geo0 = P.n_obs * std::log(P.s0) + geo;  // every observation maps to a step, so the weights sum to n_obs
      OF_CUDA_TRY(ctx, cudaMemcpyAsync(d_obs, t, table, cudaMemcpyHostToDevice, ctx->stream));
      P.obs = (const double2*)d_obs;
    }
    if (P.payoff == OF_PAYOFF_BARRIER) {
      P.bar_sign = P.barrier_up ? 1.0 : -1.0;
      P.bar_hit0 = P.barrier_up ? P.s0 >= P.barrier : P.s0 <= P.barrier;
      // a level <= 0 is below every spot
      const double by = P.barrier <= 0.0 ? -INFINITY : std::log(P.barrier / P.s0);
      P.bar_thr = P.bar_sign * by / P.diffusion;
      P.bar_step = -P.bar_sign * P.drift / P.diffusion;
    }
    P.y_floor = std::log(1e-12 / P.s0);
    const int64_t want = (P.samples + kRefThreads - 1) / kRefThreads, cap = (int64_t)ctx->sm_count * 16;
    const int grid = (int)(want < cap ? want : cap);
    OF_TRY(of_scratch(ctx, SLOT_PARTIALS, (size_t)grid * 5 * sizeof(double), &d_part));
    OF_TRY(of_ticket(ctx, &P.ticket));
    P.partials = (double*)d_part;
    P.out = (double*)((char*)h + table);
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_start, ctx->stream));
    fast<<<grid, kRefThreads, 0, ctx->stream>>>(P);
    OF_CUDA_TRY(ctx, cudaGetLastError());
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_stop, ctx->stream));
    OF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    OF_CUDA_TRY(ctx, cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
    std::memcpy(sums, P.out, sizeof(sums));
  } else {
    void *d_obs = nullptr, *d_sums = nullptr;
    if (P.need_arith || P.need_geo) {
      OF_TRY(of_scratch(ctx, SLOT_OBS, w.size() * sizeof(double), &d_obs));
      OF_CUDA_TRY(ctx, cudaMemcpyAsync(d_obs, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
    }
    P.obs_w = (const double*)d_obs;
    const int block = 128;
    const void* kern = pcg ? (const void*)mc_ref_kernel<of::Pcg64> : (const void*)mc_ref_kernel<of::Xoshiro256pp>;
    const int64_t want = (P.samples + block - 1) / block;
    const int64_t cap = (int64_t)ctx->sm_count * of_blocks_per_sm(kern, block, 0);
    const int grid = (int)(want < cap ? want : cap);
    OF_TRY(of_scratch(ctx, SLOT_PARTIALS, (size_t)grid * 5 * sizeof(double), &d_part));
    OF_TRY(of_scratch(ctx, SLOT_SUMS, 5 * sizeof(double), &d_sums));
    OF_TRY(of_pinned(ctx, 5 * sizeof(double), &h));
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_start, ctx->stream));
    if (pcg) mc_ref_kernel<of::Pcg64><<<grid, block, 0, ctx->stream>>>(P, (double*)d_part);
    else mc_ref_kernel<of::Xoshiro256pp><<<grid, block, 0, ctx->stream>>>(P, (double*)d_part);
    OF_CUDA_TRY(ctx, cudaGetLastError());
    OF_TRY(of_reduce_rows(ctx, (const double*)d_part, grid, 5, (double*)d_sums));
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_stop, ctx->stream));
    OF_CUDA_TRY(ctx, cudaMemcpyAsync(h, d_sums, 5 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    OF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    OF_CUDA_TRY(ctx, cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
    std::memcpy(sums, h, sizeof(sums));
  }
  of_mc_finish(sums, P.samples, c->control_variate, c->cv_expected, c->discount_factor, out);
  out->kernel_ms = ms;
  return OF_OK;
}
