// adjoint.cu - pathwise reverse-mode Heston Greeks with checkpointing (FP32).
//
// Price and d/d(S0, r, v0, kappa, theta, xi, rho) of a European or arithmetic
// Asian option under Andersen's QE scheme (gamma1 = gamma2 = 1/2, psi_c = 1.5):
//   m = theta + (v - theta) e,  s2 = v c1 + c2,  psi = s2 / m^2,  t = 2 / psi
//   quadratic: v' = a (b + Zv)^2,  b^2 = t - 1 + sqrt(t (t - 1)),  a = m / (1 + b^2)
//   exponential: v' = 0 if U <= p else m ln((1-p)/(1-U)) / (1-p),  p = (psi-1)/(psi+1) = (2-t)/(2+t)
//   y' = y + (r-q) dt + K0 + K1 v + K2 v' + sqrt(K34 (v + v')) Zx,   S = S0 e^y
// The branch is the quadratic one for psi <= psi_c - band, the exponential
// one for psi > psi_c + band, and a smoothstep blend of the two in between.
// band = 0 is Andersen's hard switch; its v' jumps at psi_c, and a pathwise
// derivative cannot see that jump, so the Greeks of kappa/theta/xi then miss
// the jump's contribution.  A band > 0 makes the step continuous and the
// pathwise estimator unbiased for the scheme it differentiates.
//
// Two ways to the same per-path derivatives, chosen by the share of paths that
// end in the money (their pathwise derivatives are the only non-zero ones):
//
// adjoint_paths<AP_TANGENT>: one pass.  The state is two numbers and only v0,
// kappa, theta and xi move the variance, so carrying dv/dp and dy/dp along
// with the path (8 numbers) costs less than storing the path, recomputing it
// and sweeping back: no checkpoints, no second Philox and normal per step, and
// the step's branch, roots and reciprocals serve the path and its Jacobian.
//
// adjoint_paths<AP_CHECKPOINT> + adjoint_backward: the forward pass writes
// (v, y) every 32 steps to HBM, time-major ckpt[segment][path], and each
// path's payoff gradient; then each warp scans 128-path ranges (grid stride),
// queues the in-the-money paths in shared memory (ballot; the queue carries
// over between ranges), and sweeps them 32 at a time: per segment (last first)
// the 32 steps are recomputed from the checkpoint into shared memory (v, e^y),
// each step's Philox draws are regenerated from its counter, and the adjoints
// (y_bar, v_bar) and parameter adjoints are propagated through the analytic
// step Jacobian.  Out-of-the-money paths are never swept: the cheaper way when
// few paths end in the money.
//
// Compiled with --fmad=false: every fused multiply-add is an explicit fmaf, so
// every pass over a path and the recompute produce bit-identical states.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "of_device.cuh"
#include "of_internal.h"
#include "ref_stream.cuh"

namespace {

constexpr uint32_t kAdjStreamTag = 0x41444A31u;  // "ADJ1"
constexpr int kSeg = 32;                          // checkpoint interval
constexpr int kMaxSegments = 64;
constexpr int kBwdThreads = 128;
constexpr int kBwdWarps = kBwdThreads / 32;
constexpr int kRangePerWarp = 32 * 4;  // paths one warp scans for in-the-money paths per grid-stride turn
constexpr float kLn2 = 0.69314718055994531f;

constexpr int kPathThreads = 128;
// The sweep back runs where few paths are expected in the money (sweep_pays).
// Its time over the tangent pass's, by paths an SM and share in the money, at 32
// to 2,048 steps (they agree to 0.03 from 128 steps on):
//              Asian                              European
//    3,540     0.90 (0.1 %)  1.07 (3 %)           0.92  1.11
//    7,080     0.88 (6 %)  0.99 (10 %)  1.03 (12 %)   0.92  1.03  1.08
//   14,170     0.89 (10 %)  0.96 (12 %)  1.03 (14 %)  0.92  0.99  1.06
//   28,340     0.90 (12 %)  0.94 (14 %)  1.03 (17 %)  0.92  1.00  1.09
//   56,680     0.87 (12 %)  0.93 (14 %)  1.02 (17 %)  0.90  0.97  1.06
// They meet at a share of 0.16 - 425 / (paths an SM), the second term a round of
// sweeps, whose time does not fall with their number; below 7,000 paths an SM
// that round is no longer covered but where there are next to no sweeps.
// 8,388,608 Asian paths of 128 steps with 12 % in the money: 8.1 ms for the
// tangents, 7.0 for the sweep; 32,768 paths of 512 steps at the money: 0.22 and
// 2.06.
constexpr double kSweepShare = 0.16, kSweepRound = 425.0, kSweepShareFew = 0.01;
constexpr double kSweepPathsPerSm = 7000.0, kSweepPathsPerSmFew = 3500.0;

bool sweep_pays(double share, double paths_per_sm) {
  if (paths_per_sm >= kSweepPathsPerSm) return share < kSweepShare - kSweepRound / paths_per_sm;
  return paths_per_sm >= kSweepPathsPerSmFew && share < kSweepShareFew;
}

__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct AdjC {
  // step
  float e, one_m_e, c1, c2, theta, c0 /* (r-q) dt + K0 */, K1, K2, k34, half_k34, dt;
  float sw_lo, sw_hi, sw_inv_width;  // smoothed switch band [lo, hi] of psi
  // parameter partials of the step constants
  float de_dk, c1_k, c2_k, c2_t, m2_over_xi;
  float K0_k, K0_t, K0_x, K0_r, K1_k, K1_x, K1_r, K2_k, K2_x, K2_r, k34_r;
  // payoff
  float s0, strike, v0, inv_steps;
  double disc, T;
  // tangent pass: d/dp of the linear part of y_j is lin0 j + linV sum_{i<j} (v_i - v0) + K2_p (v_j - v0)
  double lin0[4], linV[4], linK[4];  // kappa, theta, xi, rho
  double rho_w;                      // d/d rho of the diffusive part: rho_w sum sqrt(K34 (v + v')) Zx
  int32_t steps, n_seg, call, asian;
  int64_t paths;
  of::PhiloxKeys keys;
  // device buffers
  float* ck_v;   // [n_seg][paths]
  float* ck_y;   // [n_seg][paths]
  float* grad;   // [paths] d pv / d underlying (0 out of the money)
  float* und;    // [paths] average (or terminal spot)
};

struct QeDraw {
  float u, zv, zx;
};

__device__ __forceinline__ QeDraw draw_of(uint32_t a, uint32_t b) {
  const float2 z = of::normals2_from_u32(a, b);
  return QeDraw{of::uniform_from_u32(a), z.x, z.y};
}

// Both branches are functions of m and t = 2 / psi alone.  JAC: A1 = dv'/dm at
// fixed t and At = dv'/dt.
//
// quadratic: dv'/db^2 = a bz/b - a bz^2/(1+b^2) = a bz (1 - b Zv) / (b (1+b^2)),
// without the cancellation of the two terms; db^2/dt = 1 + (t - 1/2)/root.
template <bool JAC>
__device__ __forceinline__ float quad_branch(float m, float t, float zv, float& A1, float& At) {
  const float tm = t - 1.0f, x = t * tm;
  const float rs = rsqrt_approx(x), root = sqrt_approx(x);
  const float b2 = tm + root;
  const float rb = rsqrt_approx(b2), b = sqrt_approx(b2);
  const float inv = rcp_approx(1.0f + b2);
  const float a = m * inv, bz = b + zv;
  if (JAC) {
    // 1 / (1 + b^2) of the b in use, refined once: E[(b + Zv)^2] / (1 + b^2)
    // is 1 to a rounding, and an error of one sign would build up over the
    // steps that the variance remembers (1e-5 of a Greek)
    const float g = fmaf(inv, fmaf(-fmaf(b, b, 1.0f), inv, 1.0f), inv);
    A1 = bz * bz * g;
    At = a * g * (rb * bz) * fmaf(-b, zv, 1.0f) * fmaf(t - 0.5f, rs, 1.0f);
  }
  return a * bz * bz;
}

// exponential: with 1/(1-p) = 1/t + 1/2, v' = m L (1/t + 1/2) and
// dv'/dt = m (1 - L) / t^2, 1/t = psi / 2
template <bool JAC>
__device__ __forceinline__ float exp_branch(float m, float psi, float u, float& A1, float& At) {
  const float p = __fdividef(psi - 1.0f, psi + 1.0f);
  if (JAC) A1 = At = 0.0f;
  if (u <= p) return 0.0f;
  const float L = (__log2f(1.0f - p) - __log2f(1.0f - u)) * kLn2;
  if (JAC) {
    const float it = 0.5f * psi;
    A1 = L * (it + 0.5f);
    At = m * (1.0f - L) * (it * it);
  }
  return __fdividef(m * L, 1.0f - p);
}

// The variance step with the (optional) smoothed switch.  JAC: the partial of
// v' by m, and P and r = 1/s2 of that by s2, -P r (dt/dm = 2 t / m,
// dt/ds2 = -t / s2).
template <bool JAC>
__device__ __forceinline__ float qe_vnext(const AdjC& c, float v, const QeDraw& d, float& Bm, float& P, float& r) {
  const float m = fmaf(v - c.theta, c.e, c.theta);
  const float s2 = fmaf(v, c.c1, c.c2);
  const float inv_m = rcp_approx(m);
  const float psi = s2 * inv_m * inv_m;
  const float t = __fdividef(2.0f, psi);
  // each branch inlined once: quadratic below the band's top, exponential
  // above its bottom, blended inside the band
  const bool need_q = psi <= c.sw_hi, need_e = psi > c.sw_lo;
  float vn = 0.0f, A1 = 0.0f, At = 0.0f;
  if (need_q) vn = quad_branch<JAC>(m, t, d.zv, A1, At);
  if (need_e) {
    float e1 = 0.0f, et = 0.0f;
    const float ve = exp_branch<JAC>(m, psi, d.u, e1, et);
    if (need_q) {
      const float s = (psi - c.sw_lo) * c.sw_inv_width;
      const float w = s * s * fmaf(-2.0f, s, 3.0f);
      if (JAC) {  // dw/dt = dw/dpsi dpsi/dt, dpsi/dt = -psi^2 / 2
        const float dw = -3.0f * s * (1.0f - s) * c.sw_inv_width * (psi * psi);
        A1 = fmaf(w, e1 - A1, A1);
        At = fmaf(ve - vn, dw, fmaf(w, et - At, At));
      }
      vn = fmaf(w, ve - vn, vn);
    } else {
      vn = ve;
      A1 = e1;
      At = et;
    }
  }
  if (JAC) {
    P = At * t;
    Bm = fmaf(P, 2.0f * inv_m, A1);
    r = 0.5f * t * inv_m * inv_m;
  }
  return vn;
}

// sqrt(K34 (v + v')) and its reciprocal (both 0 at 0)
__device__ __forceinline__ float vol_of(const AdjC& c, float v, float vn, float& inv) {
  const float var = c.k34 * (v + vn);
  inv = var > 0.0f ? rsqrt_approx(var) : 0.0f;
  return sqrt_approx(var);
}

__device__ __forceinline__ float qe_ynext(const AdjC& c, float y, float v, float vn, float sq, float zx) {
  return fmaf(sq, zx, fmaf(c.K2, vn, fmaf(c.K1, v, y + c.c0)));
}

// ---- the pass over the paths ---------------------------------------------------
enum AdjPass { AP_PRICE, AP_CHECKPOINT, AP_TANGENT };

// One path's running tangents.  Only the part of dy/dp that goes through the
// variance (and the diffusive part for rho) is carried; the part linear in the
// path, lin0 j + linV sum (v - v0) + K2_p (v_j - v0), needs the sums below
// once instead of three terms a parameter and step.  For the Asian the same
// quantities are summed with the weight e^{y_j}.
// The four parameters go through packed pairs.
template <bool ASIAN>
struct Tangents {
  float2 dv[2] = {{1.0f, 0.0f}, {0.0f, 0.0f}};  // dv / d(v0, kappa), d(theta, xi)
  float2 Y[2] = {};                             // dy through the variance
  float W = 0.0f;                               // sum of sqrt(K34 (v + v')) Zx
  float u = 0.0f, V = 0.0f;                     // v - v0, and its sum up to the step
  float j = 0.0f;                               // steps taken
  float2 aY[2] = {};
  float aW = 0.0f, aJ = 0.0f, aV = 0.0f, au = 0.0f;

  __device__ __forceinline__ void step(const AdjC& c, float v, float vn, float Bm, float P, float r, float sq,
                                       float inv, float zx) {
    using of::fma2;
    using of::splat2;
    const float vm = v - c.theta, Bs = -P * r;
    const float2 dvn_v = splat2(fmaf(Bm, c.e, Bs * c.c1));
    // direct parts; s2 is proportional to xi^2, so that of xi needs no s2
    const float2 direct[2] = {{0.0f, fmaf(Bm * c.de_dk, vm, Bs * fmaf(v, c.c1_k, c.c2_k))},
                              {fmaf(Bm, c.one_m_e, Bs * c.c2_t), c.m2_over_xi * P}};
    const float kh = c.half_k34 * (zx * inv);
    const float2 D1 = splat2(c.K1 + kh), D2 = splat2(c.K2 + kh);  // dy/dv and dy/dv'
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float2 n = fma2(dvn_v, dv[p], direct[p]);
      Y[p] = fma2(D2, n, fma2(D1, dv[p], Y[p]));
      dv[p] = n;
    }
    W = fmaf(sq, zx, W);
    V += u;
    u = vn - c.v0;
    if (ASIAN) j += 1.0f;
  }
  __device__ __forceinline__ void observe(float S) {
#pragma unroll
    for (int p = 0; p < 2; ++p) aY[p] = of::fma2(of::splat2(S), Y[p], aY[p]);
    aW = fmaf(S, W, aW);
    aJ = fmaf(S, j, aJ);
    aV = fmaf(S, V, aV);
    au = fmaf(S, u, au);
  }
};

// Warps take 32 paths at a time, warp-major over the grid, so that the last,
// partial round spreads over all SMs.  16 sums (price 2, Greeks 7 + 7); without
// Greeks 14 of them are 0, and the price is added in the same order.
//
// Issue-bound: 183 instructions a warp and step with the tangents (130 for the
// price), two thirds of them on the FMA pipe, issued at 70 % of the peak;
// a step has 12 (9) special functions, 8 cycles of their unit each, and half a
// Philox block from the table of its counter terms.  1,048,576 paths of 512
// steps, Asian: price and Greeks 3.82 ms against 8.43 for the forward pass and
// the sweep before it, price alone 2.58 against 2.84.
template <int PASS, bool ASIAN, bool FULL>
__global__ void __launch_bounds__(kPathThreads, 5) adjoint_paths(const __grid_constant__ AdjC c,
                                                                 double* __restrict__ partials, unsigned* ticket,
                                                                 double* out) {
  constexpr int N = 16;
  extern __shared__ uint4 qtab[];
  __shared__ double sh[kPathThreads];
  __shared__ double acc_sh[PASS == AP_TANGENT ? 14 : 1][kPathThreads];  // touched once a path
  const uint32_t nq = ((uint32_t)c.steps + 1) / 2;
  of::PhiloxGen<FULL> G{&c.keys, of::PhiloxTab{qtab, nq, 0u, kAdjStreamTag}};
  of::philox_table_fill(qtab, nq, 0u, kAdjStreamTag, c.keys);
  if (PASS == AP_TANGENT)
    for (int k = 0; k < 14; ++k) acc_sh[k][threadIdx.x] = 0.0;
  __syncthreads();
  double pv_sum = 0.0, pv_sq = 0.0;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  for (int64_t i = warp * 32 + lane; i < c.paths; i += (int64_t)gridDim.x * kPathThreads) {
    const of::PhiloxLane L = G.lane((uint64_t)i);
    float v = c.v0, y = 0.0f;
    of::Kahan32 sum_s;
    Tangents<ASIAN> T;
    auto step = [&](uint32_t a, uint32_t b) {
      const QeDraw d = draw_of(a, b);
      float Bm = 0.0f, P = 0.0f, r, inv;
      const float vn = qe_vnext<PASS == AP_TANGENT>(c, v, d, Bm, P, r);
      const float sq = vol_of(c, v, vn, inv);
      if (PASS == AP_TANGENT) T.step(c, v, vn, Bm, P, r, sq, inv, d.zx);
      y = qe_ynext(c, y, v, vn, sq, d.zx);
      v = vn;
      if (ASIAN) {
        const float S = __expf(y);
        sum_s.add(S);
        if (PASS == AP_TANGENT) T.observe(S);
      }
    };
    for (int j = 0; j < c.steps; j += 2) {
      if (PASS == AP_CHECKPOINT && j % kSeg == 0) {
        c.ck_v[(size_t)(j / kSeg) * c.paths + i] = v;
        c.ck_y[(size_t)(j / kSeg) * c.paths + i] = y;
      }
      const uint4 r = G.block((uint32_t)j >> 1, L);
      step(r.x, r.y);
      if (j + 1 < c.steps) step(r.z, r.w);
    }
    const float und = ASIAN ? c.s0 * (float)(sum_s.value() * (double)c.inv_steps) : c.s0 * __expf(y);
    const float intr = c.call ? und - c.strike : c.strike - und;
    const double pv = intr > 0.0f ? c.disc * (double)intr : 0.0;
    pv_sum += pv;
    pv_sq += pv * pv;
    const float g = intr > 0.0f ? (float)c.disc * (c.call ? 1.0f : -1.0f) : 0.0f;
    if (PASS == AP_CHECKPOINT) {
      c.und[i] = und;
      c.grad[i] = g;
    }
    if (PASS == AP_TANGENT && intr > 0.0f) {
      // d pv / d p = w (sum of the tangents): the average's weight, or the terminal spot's
      const double w = ASIAN ? (double)(g * c.s0 * c.inv_steps) : (double)(g * und);
      const double J = ASIAN ? (double)T.aJ : (double)c.steps, Vs = ASIAN ? (double)T.aV : (double)T.V,
                   vl = ASIAN ? (double)T.au : (double)T.u, Ws = ASIAN ? (double)T.aW : (double)T.W;
      double gk[7];
      gk[0] = (double)(g * und / c.s0);
      gk[1] = w * J * (double)c.dt - c.T * pv;
      const float2 t0 = ASIAN ? T.aY[0] : T.Y[0], t1 = ASIAN ? T.aY[1] : T.Y[1];
      gk[2] = w * (double)t0.x;
      const double part[4] = {(double)t0.y, (double)t1.x, (double)t1.y, c.rho_w * Ws};
#pragma unroll
      for (int p = 0; p < 4; ++p) gk[3 + p] = w * (part[p] + c.lin0[p] * J + c.linV[p] * Vs + c.linK[p] * vl);
#pragma unroll
      for (int k = 0; k < 7; ++k) {
        acc_sh[k][threadIdx.x] += gk[k];
        acc_sh[7 + k][threadIdx.x] += gk[k] * gk[k];
      }
    }
  }
  double sums[N];
  sums[0] = pv_sum;
  sums[1] = pv_sq;
#pragma unroll
  for (int k = 2; k < N; ++k) sums[k] = PASS == AP_TANGENT ? acc_sh[k - 2][threadIdx.x] : 0.0;
  of::grid_sum<N, kPathThreads>(sums, sh, partials, ticket, out);
}

// One path's backward sweep; sv/ss are this lane's columns of the block's
// shared segment buffers (stride kBwdThreads).
__device__ void sweep_path(const AdjC& c, int64_t i, float* sv, float* ss, double* acc) {
  const uint32_t lo = (uint32_t)i, hi = (uint32_t)(i >> 32);
  const float g = c.grad[i];
  const float und = c.und[i];
  const float direct = c.asian ? g * c.s0 * c.inv_steps : 0.0f;  // d pv / d y_j = direct * e^{y_j}
  float ybar = c.asian ? 0.0f : g * und;                         // European: seed at y_M
  float wbar = 0.0f, kbar = 0.0f, tbar = 0.0f, xbar = 0.0f, rbar = 0.0f, mubar = 0.0f;
  for (int seg = c.n_seg - 1; seg >= 0; --seg) {
    const int j0 = seg * kSeg;
    const int len = (c.steps - j0) < kSeg ? (c.steps - j0) : kSeg;
    float vv = c.ck_v[(size_t)seg * c.paths + i], yy = c.ck_y[(size_t)seg * c.paths + i];
    sv[0] = vv;
    for (int k = 0; k < len; k += 2) {
      const int j = j0 + k;
      const uint4 r = of::philox4x32_10(make_uint4((uint32_t)(j >> 1), lo, hi, kAdjStreamTag), c.keys);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        if (k + o < len) {
          const QeDraw d = o ? draw_of(r.z, r.w) : draw_of(r.x, r.y);
          float Bm, P, r2, inv;
          const float vn = qe_vnext<false>(c, vv, d, Bm, P, r2);
          const float sq = vol_of(c, vv, vn, inv);
          yy = qe_ynext(c, yy, vv, vn, sq, d.zx);
          vv = vn;
          sv[(k + o + 1) * kBwdThreads] = vv;
          ss[(k + o + 1) * kBwdThreads] = __expf(yy);
        }
      }
    }
    for (int k = (len - 1) & ~1; k >= 0; k -= 2) {
      const int j = j0 + k;
      const uint4 r = of::philox4x32_10(make_uint4((uint32_t)(j >> 1), lo, hi, kAdjStreamTag), c.keys);
      // not unrolled: one copy of the step Jacobian keeps the kernel's code
      // within the instruction cache (instruction-fetch stalls were the
      // largest stall with two copies)
#pragma unroll 1
      for (int o = 1; o >= 0; --o) {
        if (k + o < len) {
          ybar = fmaf(direct, ss[(k + o + 1) * kBwdThreads], ybar);  // y_{j+o+1} enters the average
          const QeDraw d = o ? draw_of(r.z, r.w) : draw_of(r.x, r.y);
          const float v = sv[(k + o) * kBwdThreads], vn = sv[(k + o + 1) * kBwdThreads];
          float Bm, P, r2, inv;
          qe_vnext<true>(c, v, d, Bm, P, r2);
          const float vm = v - c.theta, Bs = -P * r2;
          const float dvn_v = fmaf(Bm, c.e, Bs * c.c1);
          const float dvn_k = fmaf(Bm * c.de_dk, vm, Bs * fmaf(v, c.c1_k, c.c2_k));
          const float dvn_t = fmaf(Bm, c.one_m_e, Bs * c.c2_t);
          const float dvn_x = c.m2_over_xi * P;
          vol_of(c, v, vn, inv);
          const float h = 0.5f * (d.zx * inv);
          const float dy_r = fmaf(c.k34_r * (v + vn), h, fmaf(c.K2_r, vn, fmaf(c.K1_r, v, c.K0_r)));
          const float Vbar = fmaf(ybar, fmaf(c.k34, h, c.K2), wbar);
          kbar = fmaf(Vbar, dvn_k, fmaf(ybar, fmaf(c.K2_k, vn, fmaf(c.K1_k, v, c.K0_k)), kbar));
          tbar = fmaf(Vbar, dvn_t, fmaf(ybar, c.K0_t, tbar));
          xbar = fmaf(Vbar, dvn_x, fmaf(ybar, fmaf(c.K2_x, vn, fmaf(c.K1_x, v, c.K0_x)), xbar));
          rbar = fmaf(ybar, dy_r, rbar);
          mubar = fmaf(ybar, c.dt, mubar);
          wbar = fmaf(Vbar, dvn_v, ybar * fmaf(c.k34, h, c.K1));
        }
      }
    }
  }
  const double pv = c.disc * (double)(c.call ? und - c.strike : c.strike - und);
  const double gk[7] = {(double)(g * und / c.s0), (double)mubar - c.T * pv, wbar, kbar, tbar, xbar, rbar};
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    acc[k] += gk[k];
    acc[7 + k] += gk[k] * gk[k];
  }
}

// ---- backward sweeps over the in-the-money paths ----------------------------
// Six 128-thread blocks per SM (the 36 KB of segment buffers allow six): at
// most 80 registers, 1.6 % faster than 93 registers and five blocks.
__global__ void __launch_bounds__(kBwdThreads, 6) adjoint_backward(const __grid_constant__ AdjC c,
                                                               double* __restrict__ partials, unsigned* ticket,
                                                               double* out) {
  __shared__ __align__(16) float seg_v[(kSeg + 1) * kBwdThreads];
  __shared__ float seg_s[(kSeg + 1) * kBwdThreads];
  __shared__ int64_t queue[kBwdWarps][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double acc[14];
#pragma unroll
  for (int k = 0; k < 14; ++k) acc[k] = 0.0;
  const int64_t nranges = (c.paths + kRangePerWarp - 1) / kRangePerWarp;
  const int64_t gwarps = (int64_t)gridDim.x * kBwdWarps;
  int qn = 0;  // queued in-the-money paths; the queue carries over from one range to the next
  for (int64_t rg = (int64_t)warp * gridDim.x + blockIdx.x; rg < nranges; rg += gwarps) {
    const int64_t r0 = rg * kRangePerWarp;
    for (int chunk = 0; chunk < kRangePerWarp; chunk += 32) {
      const int64_t i = r0 + chunk + lane;
      const bool itm = i < c.paths && c.grad[i] != 0.0f;
      const unsigned mask = __ballot_sync(of::kFullMask, itm);
      if (itm) queue[warp][qn + __popc(mask & ((1u << lane) - 1u))] = i;
      qn += __popc(mask);
      __syncwarp();
      if (qn >= 32) {
        sweep_path(c, queue[warp][lane], seg_v + threadIdx.x, seg_s + threadIdx.x, acc);
        __syncwarp();
        if (lane < qn - 32) queue[warp][lane] = queue[warp][32 + lane];
        qn -= 32;
        __syncwarp();
      }
    }
  }
  if (lane < qn) sweep_path(c, queue[warp][lane], seg_v + threadIdx.x, seg_s + threadIdx.x, acc);
  __syncthreads();
  of::grid_sum<14, kBwdThreads>(acc, (double*)seg_v, partials, ticket, out);  // fixed order
}

typedef void (*PathKernel)(const AdjC, double*, unsigned*, double*);

template <int PASS>
PathKernel path_kernel(bool asian, bool full) {
  return asian ? (full ? adjoint_paths<PASS, true, true> : adjoint_paths<PASS, true, false>)
               : (full ? adjoint_paths<PASS, false, true> : adjoint_paths<PASS, false, false>);
}

// The share of paths expected in the money: the underlying taken as lognormal
// with the scheme's mean and expected integrated variance (a third of it for
// the average).  It only picks the cheaper of two ways to the same Greeks.
double itm_share(const of_heston_adjoint_params* p) {
  const double mu = (p->rate - p->dividend_yield) * p->expiry, kT = p->kappa * p->expiry;
  const bool asian = p->payoff == OF_PAYOFF_ASIAN;
  const double iv = p->theta * p->expiry + (p->v0 - p->theta) * -std::expm1(-kT) / p->kappa;
  const double w = asian ? iv / 3.0 : iv;
  const double f = asian ? (std::fabs(mu) > 1e-8 ? std::log(std::expm1(mu) / mu) : 0.5 * mu) : mu;
  const double d = (std::log(p->spot / p->strike) + f - 0.5 * w) / std::sqrt(w);
  const double call = 0.5 * std::erfc(-d / std::sqrt(2.0));
  return p->option_type == OF_CALL ? call : 1.0 - call;
}

// Price-only FP64 pass over the same draws (the bits of each Philox counter
// give the same U, Zv, Zx), for bump-and-revalue with common random numbers:
// a relative bump of 1e-4 moves a step's log-increment by ~1e-8, below the
// FP32 resolution of the path state, so the revaluation runs in FP64.
struct AdjC64 {
  double e, c1, c2, theta, c0, K1, K2, k34, s0, strike, inv_steps, disc, v0;
  double sw_lo, sw_hi, sw_inv_width;
  int32_t steps, call, asian;
  int64_t paths;
  of::PhiloxKeys keys;
};

__device__ __forceinline__ double quad64(double m, double psi, double zv) {
  const double t = 2.0 / psi;
  const double b2 = (t - 1.0) + sqrt(t * (t - 1.0));
  const double a = m / (1.0 + b2);
  const double bz = sqrt(b2) + zv;
  return a * bz * bz;
}

__device__ __forceinline__ double exp64(double m, double psi, double u) {
  const double p = (psi - 1.0) / (psi + 1.0);
  return (u <= p) ? 0.0 : m * log((1.0 - p) / (1.0 - u)) / (1.0 - p);
}

__global__ void __launch_bounds__(128) forward64_kernel(const __grid_constant__ AdjC64 c,
                                                        double* __restrict__ partials) {
  __shared__ double sh[2 * 4];
  double acc[2] = {0.0, 0.0};
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < c.paths; i += stride) {
    const uint32_t lo = (uint32_t)i, hi = (uint32_t)(i >> 32);
    double v = c.v0, y = 0.0, sum_s = 0.0;
    for (int j = 0; j < c.steps; j += 2) {
      const uint4 r = of::philox4x32_10(make_uint4((uint32_t)(j >> 1), lo, hi, kAdjStreamTag), c.keys);
      for (int o = 0; o < 2 && j + o < c.steps; ++o) {
        const uint32_t ub = o ? r.z : r.x;
        const double u = (double)of::uniform_from_u32(ub);
        const double zx = (double)of::normal_from_u32(o ? r.w : r.y);
        const double zv = (double)of::normal_from_u32(ub);
        const double m = c.theta + (v - c.theta) * c.e;
        const double s2 = v * c.c1 + c.c2;
        const double psi = s2 / (m * m);
        double vn;
        if (psi <= c.sw_lo) {
          vn = quad64(m, psi, zv);
        } else if (psi > c.sw_hi) {
          vn = exp64(m, psi, u);
        } else {
          const double vq = quad64(m, psi, zv), ve = exp64(m, psi, u);
          const double s = (psi - c.sw_lo) * c.sw_inv_width;
          vn = vq + s * s * (3.0 - 2.0 * s) * (ve - vq);
        }
        y = y + c.c0 + c.K1 * v + c.K2 * vn + sqrt(c.k34 * (v + vn)) * zx;
        v = vn;
        if (c.asian) sum_s += exp(y);
      }
    }
    const double und = c.asian ? c.s0 * sum_s * c.inv_steps : c.s0 * exp(y);
    const double intr = c.call ? und - c.strike : c.strike - und;
    const double pv = intr > 0.0 ? c.disc * intr : 0.0;
    acc[0] += pv;
    acc[1] += pv * pv;
  }
  of::block_sum<2>(acc, sh);
  if (threadIdx.x == 0) {
    partials[(int64_t)blockIdx.x * 2] = acc[0];
    partials[(int64_t)blockIdx.x * 2 + 1] = acc[1];
  }
}

}  // namespace

extern "C" of_status of_heston_price_adjoint(of_ctx* ctx, const of_heston_adjoint_params* p, of_adjoint_result* out) {
  if (!ctx || !p || !out) return OF_ERR_INVALID_INPUT;
  std::memset(out, 0, sizeof(*out));
  if (p->option_type != OF_CALL && p->option_type != OF_PUT)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "unknown option type %d", p->option_type);
  if (p->payoff != OF_PAYOFF_VANILLA && p->payoff != OF_PAYOFF_ASIAN)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "adjoint payoff must be vanilla or arithmetic Asian");
  if (p->scheme != OF_MODEL_HESTON_QE)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "the adjoint kernel implements the QE scheme");
  if (p->num_paths <= 0) return of_fail(ctx, OF_ERR_INVALID_INPUT, "num_paths must be > 0");
  if (p->num_steps <= 0) return of_fail(ctx, OF_ERR_INVALID_INPUT, "num_steps must be > 0");
  if (p->checkpoint_every != kSeg) return of_fail(ctx, OF_ERR_UNSUPPORTED, "checkpoint interval must be 32");
  if (p->forward_only < 0 || p->forward_only > 2)
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "forward_only must be 0, 1 or 2");
  if (!(p->qe_switch_band >= 0.0 && p->qe_switch_band <= 0.25))
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "qe_switch_band must lie in [0, 0.25]");
  if (p->num_steps > (int64_t)kMaxSegments * kSeg)
    return of_fail(ctx, OF_ERR_UNSUPPORTED, "at most %d steps", kMaxSegments * kSeg);
  if (!(p->spot > 0.0) || !(p->strike > 0.0) || !(p->expiry > 0.0))
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "spot, strike and expiry must be > 0");
  if (!(p->kappa > 0.0 && p->theta > 0.0 && p->xi > 0.0 && p->v0 >= 0.0 && p->rho > -1.0 && p->rho < 1.0))
    return of_fail(ctx, OF_ERR_INVALID_INPUT, "invalid Heston parameters (QE needs kappa, theta, xi > 0)");
  OF_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const double dt = p->expiry / (double)p->num_steps;
  const double k = p->kappa, th = p->theta, x = p->xi, r = p->rho;
  const double e = std::exp(-k * dt);
  const double c1 = x * x * e * (1.0 - e) / k;
  const double c2 = th * x * x * (1.0 - e) * (1.0 - e) / (2.0 * k);
  const double de_dk = -dt * e;
  const double K0 = -r * k * th * dt / x;
  const double K1 = 0.5 * dt * (k * r / x - 0.5) - r / x;
  const double K2 = 0.5 * dt * (k * r / x - 0.5) + r / x;
  const double k34 = 0.5 * dt * (1.0 - r * r);
  const double band = p->qe_switch_band;
  const double sw_lo = 1.5 - band, sw_hi = 1.5 + band;
  const double sw_inv_width = band > 0.0 ? 1.0 / (2.0 * band) : 0.0;
  const int32_t n_seg = (int32_t)((p->num_steps + kSeg - 1) / kSeg);
  const bool call = p->option_type == OF_CALL, asian = p->payoff == OF_PAYOFF_ASIAN;

  void *d_part = nullptr, *d_sums = nullptr, *h = nullptr;
  const int blk = 128;
  const int64_t want = (p->num_paths + blk - 1) / blk;
  float ms = 0.0f;
  double s[16] = {0};
  if (p->forward_only == 2) {
    AdjC64 d{};
    d.e = e;
    d.c1 = c1;
    d.c2 = c2;
    d.theta = th;
    d.c0 = (p->rate - p->dividend_yield) * dt + K0;
    d.K1 = K1;
    d.K2 = K2;
    d.k34 = k34;
    d.s0 = p->spot;
    d.strike = p->strike;
    d.inv_steps = 1.0 / (double)p->num_steps;
    d.disc = std::exp(-p->rate * p->expiry);
    d.v0 = p->v0;
    d.sw_lo = sw_lo;
    d.sw_hi = sw_hi;
    d.sw_inv_width = sw_inv_width;
    d.steps = (int32_t)p->num_steps;
    d.call = call;
    d.asian = asian;
    d.paths = p->num_paths;
    d.keys = of::philox_keys(p->seed);
    const int64_t cap = (int64_t)ctx->sm_count * of_blocks_per_sm((const void*)forward64_kernel, blk, 0);
    const int grid = (int)(want < cap ? want : cap);
    OF_TRY(of_scratch(ctx, SLOT_PARTIALS, (size_t)grid * 2 * sizeof(double), &d_part));
    OF_TRY(of_scratch(ctx, SLOT_SUMS, 16 * sizeof(double), &d_sums));
    OF_TRY(of_pinned(ctx, 16 * sizeof(double), &h));
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_start, ctx->stream));
    forward64_kernel<<<grid, blk, 0, ctx->stream>>>(d, (double*)d_part);
    OF_CUDA_TRY(ctx, cudaGetLastError());
    OF_TRY(of_reduce_rows(ctx, (const double*)d_part, grid, 2, (double*)d_sums));
  } else {
    AdjC c{};
    c.e = (float)e;
    c.one_m_e = 1.0f - c.e;  // of the e the path takes
    c.c1 = (float)c1;
    c.c2 = (float)c2;
    c.theta = (float)th;
    c.c0 = (float)((p->rate - p->dividend_yield) * dt + K0);
    c.K1 = (float)K1;
    c.K2 = (float)K2;
    c.k34 = (float)k34;
    c.half_k34 = (float)(0.5 * k34);
    c.dt = (float)dt;
    c.sw_lo = (float)sw_lo;
    c.sw_hi = (float)sw_hi;
    c.sw_inv_width = (float)sw_inv_width;
    c.de_dk = (float)de_dk;
    c.c1_k = (float)(x * x * de_dk * (1.0 - 2.0 * e) / k - c1 / k);
    c.c2_k = (float)(-th * x * x * (1.0 - e) * de_dk / k - c2 / k);
    c.m2_over_xi = (float)(-2.0 / x);
    c.c2_t = (float)(x * x * (1.0 - e) * (1.0 - e) / (2.0 * k));
    // (K0, K1, K2) by kappa, theta, xi, rho
    const double K_k[3] = {-r * th * dt / x, 0.5 * dt * r / x, 0.5 * dt * r / x};
    const double K_x[3] = {r * k * th * dt / (x * x), -0.5 * dt * k * r / (x * x) + r / (x * x),
                           -0.5 * dt * k * r / (x * x) - r / (x * x)};
    const double K_r[3] = {-k * th * dt / x, 0.5 * dt * k / x - 1.0 / x, 0.5 * dt * k / x + 1.0 / x};
    const double K_t[3] = {-r * k * dt / x, 0.0, 0.0};
    c.K0_k = (float)K_k[0];
    c.K0_t = (float)K_t[0];
    c.K0_x = (float)K_x[0];
    c.K0_r = (float)K_r[0];
    c.K1_k = (float)K_k[1];
    c.K1_x = (float)K_x[1];
    c.K1_r = (float)K_r[1];
    c.K2_k = (float)K_k[2];
    c.K2_x = (float)K_x[2];
    c.K2_r = (float)K_r[2];
    c.k34_r = (float)(-dt * r);
    c.s0 = (float)p->spot;
    c.strike = (float)p->strike;
    c.v0 = (float)p->v0;
    c.inv_steps = (float)(1.0 / (double)p->num_steps);
    c.disc = std::exp(-p->rate * p->expiry);
    c.T = p->expiry;
    c.steps = (int32_t)p->num_steps;
    c.n_seg = n_seg;
    c.call = call;
    c.asian = asian;
    c.paths = p->num_paths;
    c.keys = of::philox_keys(p->seed);
    const double* Ks[4] = {K_k, K_t, K_x, K_r};
    // of the FP32 constants, as the path takes them
    for (int q = 0; q < 4; ++q) {
      const double k0 = (float)Ks[q][0], k1 = (float)Ks[q][1], k2 = (float)Ks[q][2];
      c.linV[q] = k1 + k2;
      c.linK[q] = k2;
      c.lin0[q] = k0 + c.linV[q] * (double)c.v0;
    }
    c.rho_w = -r / (1.0 - r * r);
    const bool greeks = p->forward_only == 0;
    bool tangent = greeks && !sweep_pays(itm_share(p), (double)p->num_paths / ctx->sm_count);
    void* d_ck = nullptr;
    if (greeks && !tangent) {
      // checkpoints (v, y) + per-path gradient and underlying
      const size_t ck_bytes = (size_t)n_seg * p->num_paths * 2 * sizeof(float) + (size_t)p->num_paths * 2 * sizeof(float);
      if (of_scratch(ctx, SLOT_ADJ_CKPT, ck_bytes, &d_ck) == OF_OK) {
        c.ck_v = (float*)d_ck;
        c.ck_y = c.ck_v + (size_t)n_seg * p->num_paths;
        c.grad = c.ck_y + (size_t)n_seg * p->num_paths;
        c.und = c.grad + p->num_paths;
      } else {  // no room for them: the tangent pass needs none
        cudaGetLastError();
        tangent = true;
      }
    }
    // every pass runs on the tangent pass's grid, so that a price is the same
    // sum whichever pass computed it
    const bool full = !(((uint64_t)p->num_paths - 1) >> 32);
    const size_t smem = (size_t)((p->num_steps + 1) / 2) * sizeof(uint4);
    const int64_t capf =
        (int64_t)ctx->sm_count * of_blocks_per_sm((const void*)path_kernel<AP_TANGENT>(asian, full), kPathThreads, smem);
    const int gridf = (int)(want < capf ? want : capf);
    const int64_t nranges = (p->num_paths + kRangePerWarp - 1) / kRangePerWarp;
    const int64_t wantb = (nranges + kBwdWarps - 1) / kBwdWarps;
    const int64_t capb = (int64_t)ctx->sm_count * of_blocks_per_sm((const void*)adjoint_backward, kBwdThreads, 0);
    const int gridb = (int)(wantb < capb ? wantb : capb);
    unsigned* ticket = nullptr;
    OF_TRY(of_scratch(ctx, SLOT_PARTIALS, (size_t)std::max(gridf * 16, gridb * 14) * sizeof(double), &d_part));
    OF_TRY(of_pinned(ctx, 16 * sizeof(double), &h));
    OF_TRY(of_ticket(ctx, &ticket));
    OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_start, ctx->stream));
    const PathKernel fn = tangent  ? path_kernel<AP_TANGENT>(asian, full)
                          : greeks ? path_kernel<AP_CHECKPOINT>(asian, full)
                                   : path_kernel<AP_PRICE>(asian, full);
    fn<<<gridf, kPathThreads, smem, ctx->stream>>>(c, (double*)d_part, ticket, (double*)h);
    OF_CUDA_TRY(ctx, cudaGetLastError());
    if (greeks && !tangent) {
      adjoint_backward<<<gridb, kBwdThreads, 0, ctx->stream>>>(c, (double*)d_part, ticket, (double*)h + 2);
      OF_CUDA_TRY(ctx, cudaGetLastError());
    }
  }
  OF_CUDA_TRY(ctx, cudaEventRecord(ctx->ev_stop, ctx->stream));
  if (d_sums) OF_CUDA_TRY(ctx, cudaMemcpyAsync(h, d_sums, 16 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  OF_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  OF_CUDA_TRY(ctx, cudaEventElapsedTime(&ms, ctx->ev_start, ctx->ev_stop));
  std::memcpy(s, h, sizeof(s));
  const double n = (double)p->num_paths;
  auto se = [&](double sum, double sum2) {
    const double var = n > 1.0 ? (sum2 - sum * sum / n) / (n - 1.0) : 0.0;
    return std::sqrt((var > 0.0 ? var : 0.0) / n);
  };
  out->price = s[0] / n;
  out->stderr_ = se(s[0], s[1]);
  if (p->forward_only == 0) {
    for (int k2 = 0; k2 < OF_ADJ_COUNT; ++k2) {
      out->greeks[k2] = s[2 + k2] / n;
      out->greeks_stderr[k2] = se(s[2 + k2], s[9 + k2]);
    }
  }
  out->samples = p->num_paths;
  out->kernel_ms = ms;
  return OF_OK;
}
