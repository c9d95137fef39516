// ref_stream.cuh - the FP64 reference mode's normals, elementary functions
// and grid reduction, for kernels with one lane per sample.
//
// The reference draws each normal as Acklam's rational approximation of
// Phi^-1(u).  Its tails (u < 0.02425 or u > 0.97575, 4.85 % of the draws) need
// a logarithm and a square root; with one branch per draw, a warp of 32
// samples takes that branch on 80 % of its steps.  Here the central formula
// runs unconditionally and the tail draws are put aside and evaluated later
// with most lanes busy: per lane where only the sum of the normals is wanted
// (stream_normal_sum), across the warp where each step's normal is
// (stream_normals).
//
// Units that include this are compiled with --fmad=false: every fused
// multiply-add is an explicit fma().
#pragma once

#include "of_device.cuh"

namespace of {

// 1/d for a normal d, by the cubically convergent iteration
// y' = y (1 + e + e^2), e = 1 - d y (Householder's method for 1/x), from the
// 20-bit rcp.approx: the error left is of the order of the last rounding.
__device__ __forceinline__ double rcp64(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// sqrt(x) for a normal x > 0: y ~ 1/sqrt(x) from rsqrt.approx, one step of
// the cubically convergent iteration s = x y (1 + e/2 + 3 e^2/8),
// e = 1 - x y^2 (the binomial series of (1 - e)^(-1/2)).
__device__ __forceinline__ double sqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double s = x * y;
  const double e = fma(-s, y, 1.0);
  return fma(s * e, fma(e, 0.375, 0.5), s);
}

// sqrt64 for any x >= 0: y is taken of at least the smallest normal number (one
// integer maximum, of the high words), so that it stays finite and 0 gives
// s = 0 y = 0.  The Heston steps need it: a variance that has reached 0 stays
// there under kappa theta = 0, and a positive stand-in for 0 would grow back,
// for each positive normal takes its root (1e-290, 1e-146, 1e-74, ...).
__device__ __forceinline__ double sqrt64_from0(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;"
      : "=d"(y)
      : "d"(__hiloint2double(max(__double2hiint(x), 0x00100000), __double2loint(x))));
  const double s = x * y;
  const double e = fma(-s, y, 1.0);
  return fma(s * e, fma(e, 0.375, 0.5), s);
}

// exp(x) for |x| < 690 by table lookup (P. T. P. Tang, "Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15, 1989): x = (64 m + j) ln2/64 + r, |r| <= ln2/128,
// exp(x) = 2^m 2^(j/64) (1 + r + r^2/2 + ... + r^5/120); the series' next
// term is below 4e-17.  `tab` holds 2^(j/64), in shared memory: the lanes of
// a warp look up different entries.
__device__ const double kExp2Tab[64] = {
    0x1p+0, 0x1.02c9a3e778061p+0, 0x1.059b0d3158574p+0, 0x1.0874518759bc8p+0,
    0x1.0b5586cf9890fp+0, 0x1.0e3ec32d3d1a2p+0, 0x1.11301d0125b51p+0, 0x1.1429aaea92de0p+0,
    0x1.172b83c7d517bp+0, 0x1.1a35beb6fcb75p+0, 0x1.1d4873168b9aap+0, 0x1.2063b88628cd6p+0,
    0x1.2387a6e756238p+0, 0x1.26b4565e27cddp+0, 0x1.29e9df51fdee1p+0, 0x1.2d285a6e4030bp+0,
    0x1.306fe0a31b715p+0, 0x1.33c08b26416ffp+0, 0x1.371a7373aa9cbp+0, 0x1.3a7db34e59ff7p+0,
    0x1.3dea64c123422p+0, 0x1.4160a21f72e2ap+0, 0x1.44e086061892dp+0, 0x1.486a2b5c13cd0p+0,
    0x1.4bfdad5362a27p+0, 0x1.4f9b2769d2ca7p+0, 0x1.5342b569d4f82p+0, 0x1.56f4736b527dap+0,
    0x1.5ab07dd485429p+0, 0x1.5e76f15ad2148p+0, 0x1.6247eb03a5585p+0, 0x1.6623882552225p+0,
    0x1.6a09e667f3bcdp+0, 0x1.6dfb23c651a2fp+0, 0x1.71f75e8ec5f74p+0, 0x1.75feb564267c9p+0,
    0x1.7a11473eb0187p+0, 0x1.7e2f336cf4e62p+0, 0x1.82589994cce13p+0, 0x1.868d99b4492edp+0,
    0x1.8ace5422aa0dbp+0, 0x1.8f1ae99157736p+0, 0x1.93737b0cdc5e5p+0, 0x1.97d829fde4e50p+0,
    0x1.9c49182a3f090p+0, 0x1.a0c667b5de565p+0, 0x1.a5503b23e255dp+0, 0x1.a9e6b5579fdbfp+0,
    0x1.ae89f995ad3adp+0, 0x1.b33a2b84f15fbp+0, 0x1.b7f76f2fb5e47p+0, 0x1.bcc1e904bc1d2p+0,
    0x1.c199bdd85529cp+0, 0x1.c67f12e57d14bp+0, 0x1.cb720dcef9069p+0, 0x1.d072d4a07897cp+0,
    0x1.d5818dcfba487p+0, 0x1.da9e603db3285p+0, 0x1.dfc97337b9b5fp+0, 0x1.e502ee78b3ff6p+0,
    0x1.ea4afa2a490dap+0, 0x1.efa1bee615a27p+0, 0x1.f50765b6e4540p+0, 0x1.fa7c1819e90d8p+0,
};

// Copies the table into shared memory; a __syncthreads must follow.
__device__ __forceinline__ void exp_table_load(double* tab) {
  for (int i = threadIdx.x; i < 64; i += blockDim.x) tab[i] = kExp2Tab[i];
}

__device__ __forceinline__ double exp64(double x, const double* tab) {
  const double big = 0x1.8p+52;
  const double kd = fma(x, 0x1.71547652b82fep+6, big);  // round(x 64/ln2) in the low word
  const int k = __double2loint(kd);
  const double kf = kd - big;
  const double r = fma(-kf, 0x1.a39ef35793c76p-39, fma(-kf, 0x1.62e42fee00000p-7, x));
  double p = fma(r, 1.0 / 120.0, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p * r, r, r);
  const double t = tab[k & 63];
  const double v = fma(t, p, t);
  return __hiloint2double(__double2hiint(v) + ((k >> 6) << 20), __double2loint(v));
}

// -2 ln(x) for a normal x in (0, 1/4), by table lookup (P. T. P. Tang,
// "Table-driven implementation of the logarithm function in IEEE
// floating-point arithmetic", ACM TOMS 16, 1990): x = 2^e m, m in [1, 2);
// kLogTab holds, for the interval of m's top six bits, c ~ 1/m (ten bits) and
// -ln c; with r = m c - 1, |r| < 0.0083, ln x = e ln2 - ln c + (r - r^2/2 +
// ... + r^7/7), the next term below 3e-18.
__device__ const double2 kLogTab[64] = {
    {0.9921875, 0x1.010157588de71p-7}, {0.9775390625, 0x1.74321d3d006d3p-6},
    {0.962890625, 0x1.35c8bfaa1306bp-5}, {0.9482421875, 0x1.b35dd9b58baadp-5},
    {0.9345703125, 0x1.152b799bb3cc9p-4}, {0.9208984375, 0x1.518874226130ap-4},
    {0.908203125, 0x1.8a6477a91dc29p-4}, {0.8955078125, 0x1.c40d6425a5cb1p-4},
    {0.8828125, 0x1.fe89139dbd566p-4}, {0.87109375, 0x1.1aa2b7e23f72ap-3},
    {0.859375, 0x1.365fcb0159016p-3}, {0.84765625, 0x1.527e5e4a1b58dp-3},
    {0.8369140625, 0x1.6c9d07d203fc7p-3}, {0.826171875, 0x1.871213750e994p-3},
    {0.8154296875, 0x1.a1dfc40f1b7f1p-3}, {0.8046875, 0x1.bd087383bd8adp-3},
    {0.794921875, 0x1.d60a17f903515p-3}, {0.78515625, 0x1.ef5ade4dcffe6p-3},
    {0.775390625, 0x1.047e60cde83b8p-2}, {0.7666015625, 0x1.102ac0a35cc1cp-2},
    {0.7578125, 0x1.1bf99635a6b95p-2}, {0.7490234375, 0x1.27ebaf58d8c9dp-2},
    {0.740234375, 0x1.3401e12aecba1p-2}, {0.7314453125, 0x1.403d086cea79cp-2},
    {0.7236328125, 0x1.4b3c077267e9ap-2}, {0.71484375, 0x1.57bf753c8d1fbp-2},
    {0.70703125, 0x1.630030b3aac49p-2}, {0.69921875, 0x1.6e60ee6af1972p-2},
    {0.69140625, 0x1.79e26687cfb3ep-2}, {0.6845703125, 0x1.840f1e12667f0p-2},
    {0.677734375, 0x1.8e55f9b349b83p-2}, {0.669921875, 0x1.9a355c33bd6bap-2},
    {0.6630859375, 0x1.a4b60a46e5dd3p-2}, {0.65625, 0x1.af5295248cdd0p-2},
    {0.6494140625, 0x1.ba0b922e74f22p-2}, {0.6435546875, 0x1.c35383c8850afp-2},
    {0.63671875, 0x1.ce42f18064743p-2}, {0.630859375, 0x1.d7ba7ad9e7da0p-2},
    {0.6240234375, 0x1.e2e28d3d701ccp-2}, {0.6181640625, 0x1.ec8ba06d15ad9p-2},
    {0.6123046875, 0x1.f64c414b926c5p-2}, {0.6064453125, 0x1.001271e716158p-1},
    {0.6005859375, 0x1.050affa5671a5p-1}, {0.595703125, 0x1.0938fae5d8e9bp-1},
    {0.58984375, 0x1.0e4898611cce1p-1}, {0.5849609375, 0x1.128a24f1d9affp-1},
    {0.5791015625, 0x1.17b1ac17cbd5bp-1}, {0.57421875, 0x1.1c07849ae6007p-1},
    {0.5693359375, 0x1.2066d7740737ep-1}, {0.5634765625, 0x1.25b2c55cd5762p-1},
    {0.55859375, 0x1.2a2786d0ec107p-1}, {0.5537109375, 0x1.2ea64c3f97655p-1},
    {0.5498046875, 0x1.32463ebdd34eap-1}, {0.544921875, 0x1.36d77e9d34fd7p-1},
    {0.5400390625, 0x1.3b7344be40311p-1}, {0.53515625, 0x1.4019c2125ca93p-1},
    {0.53125, 0x1.43d9ff2f923c5p-1}, {0.5263671875, 0x1.489445efffcccp-1},
    {0.5224609375, 0x1.4c649aff0ee16p-1}, {0.5185546875, 0x1.503c43cd8eb68p-1},
    {0.513671875, 0x1.55144fdbcbd62p-1}, {0.509765625, 0x1.58fcddce004c4p-1},
    {0.505859375, 0x1.5ced1e17c35c5p-1}, {0.501953125, 0x1.60e52f45788e3p-1},
};

__device__ __forceinline__ double minus2_log(double x) {
  const int hi = __double2hiint(x);
  const double2 t = __ldg(kLogTab + ((hi >> 14) & 63));
  const double m = __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(x));
  const double r = fma(m, t.x, -1.0);
  double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
  p = fma(p, r, 1.0 / 5.0);
  p = fma(p, r, -1.0 / 4.0);
  p = fma(p, r, 1.0 / 3.0);
  p = fma(p, r, -1.0 / 2.0);
  p = fma(p * r, r, r);
  return -2.0 * (fma((double)((hi >> 20) - 1023), 0x1.62e42fefa39efp-1, t.y) + p);
}

// The draw's uniform u = (r >> 11) 2^-53 (next_f64, fast_rng.rs:70-73) as
// q = u - 1/2; exact: r with its low 11 bits cleared has 53 significant bits
// and q is a multiple of 2^-53 below 1/2 in magnitude.
__device__ __forceinline__ double draw_q(uint64_t r) {
  return fma(__ull2double_rn(r & ~0x7FFULL), 0x1p-64, -0.5);
}

// Whether a draw may lie in a tail: |q| with its low word cleared is at
// least 0.47575 with its low word cleared, compared in the high words, which
// order like floats.  True for every u < 0.02425 or u > 1 - 0.02425 and for a
// sliver of central ones, which tail_normal hands back to the central formula.
__device__ __forceinline__ bool draw_in_tail(double q) {
  return fabsf(__int_as_float(__double2hiint(q))) >= __int_as_float(0x3fde72b0);
}

// The argument central_parts gets in place of a tail draw: below 1e-308, so
// that n / d = n adds nothing (one select, of the high word).
__device__ __forceinline__ double draw_masked(double q, bool tail) {
  return __hiloint2double(tail ? 0 : __double2hiint(q), __double2loint(q));
}

// Numerator and denominator of Acklam's central region (acklam_inv_cdf's
// operations): z = n / d, d in [0.0036, 1].
__device__ __forceinline__ void central_parts(double q, double& n, double& d) {
  const double a0 = -3.969683028665376e1, a1 = 2.209460984245205e2, a2 = -2.759285104469687e2,
               a3 = 1.38357751867269e2, a4 = -3.066479806614716e1, a5 = 2.506628277459239;
  const double b0 = -5.447609879822406e1, b1 = 1.615858368580409e2, b2 = -1.556989798598866e2,
               b3 = 6.680131188771972e1, b4 = -1.328068155288572e1;
  const double r = q * q;
  n = fma(fma(fma(fma(fma(a0, r, a1), r, a2), r, a3), r, a4), r, a5) * q;
  d = fma(fma(fma(fma(fma(b0, r, b1), r, b2), r, b3), r, b4), r, 1.0);
}

// The normal of a draw that draw_in_tail picked: both tails in one path,
// u in the lower one or 1 - u in the upper one (each exact), clamped to
// 2^-52 as acklam_inv_cdf clamps u.
__device__ __forceinline__ double tail_normal(double q) {
  const double c0 = -7.784894002430293e-3, c1 = -3.223964580411365e-1, c2 = -2.400758277161838,
               c3 = -2.549732539343734, c4 = 4.374664141464968, c5 = 2.938163982698783;
  const double d0 = 7.784695709041462e-3, d1 = 3.224671290700398e-1, d2 = 2.445134137142996,
               d3 = 3.754408661907416;
  const double u = q + 0.5;
  double n, d;
  if (u >= 0.02425 && u <= 1.0 - 0.02425) {
    central_parts(q, n, d);
    return n * rcp64(d);
  }
  const double w = sqrt64(minus2_log(fmax(0.5 - fabs(q), 0x1p-52)));
  n = fma(fma(fma(fma(fma(c0, w, c1), w, c2), w, c3), w, c4), w, c5);
  d = fma(fma(fma(fma(d0, w, d1), w, d2), w, d3), w, 1.0);
  return copysign(1.0, -q) * n * rcp64(d);
}

// ---------------------------------------------------------------------------
// The sum of a stream's next `steps` normals.  Called by whole warps; a lane
// keeps its tail draws in its own column of `list` (kTailCap entries, `stride`
// apart) and the warp evaluates them, two entries at a time over the lanes,
// when a column fills and at the end: about 0.08 tail evaluations per step and
// warp instead of 0.8.  Every draw is stored and the column's end moves past
// the tail ones, so a draw costs no branch.  The central draws of two steps
// share one reciprocal, n0/d0 + n1/d1 = (n0 d1 + n1 d0) / (d0 d1).  The next
// four draws of the stream (a serial chain of integer operations) are taken
// while the current four are evaluated.
// ---------------------------------------------------------------------------
constexpr int kTailCap = 24;

// Whole groups of four draws: 64 bits, since the pathwise Greeks take any
// positive step count.
__host__ __device__ constexpr int64_t draw_groups(int64_t steps) { return steps >> 2; }

template <typename RNG>
__device__ __forceinline__ double stream_normal_sum(RNG& rng, int64_t steps, double* list, int stride) {
  double sum = 0.0;
  int end = 0;  // offset of the column's end
  auto draw = [&](uint64_t r, double& n, double& d) {
    const double q = draw_q(r);
    const bool tail = draw_in_tail(q);
    list[end] = q;
    if (tail) end += stride;
    central_parts(draw_masked(q, tail), n, d);
  };
  auto flush = [&]() {
    for (int at = 0; __any_sync(kFullMask, at < end); at += 2 * stride) {
      // entries past the column's end are finite draws or skipped
      const double z0 = at < end ? tail_normal(list[at]) : 0.0;
      const double z1 = at + stride < end ? tail_normal(list[at + stride]) : 0.0;
      sum += z0 + z1;
    }
    end = 0;
  };
  uint64_t r[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) r[k] = rng.next_u64();
  for (int64_t g = draw_groups(steps); g; --g) {
    double n[4], d[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      draw(r[k], n[k], d[k]);
      r[k] = rng.next_u64();
    }
    sum = fma(fma(n[0], d[1], n[1] * d[0]), rcp64(d[0] * d[1]), sum);
    sum = fma(fma(n[2], d[3], n[3] * d[2]), rcp64(d[2] * d[3]), sum);
    if (__any_sync(kFullMask, end > (kTailCap - 4) * stride)) flush();
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (k < (int)(steps & 3)) {  // at most three, and the column has room for four
      double n, d;
      draw(r[k], n, d);
      sum = fma(n, rcp64(d), sum);
    }
  flush();
  return sum;
}

// ---------------------------------------------------------------------------
// The next `n` normals of each lane's stream, at most kDrawBatch, in order, into
// the warp's z[draw][lane] (shared memory); n is the warp's, and taken as the next
// multiple of four or one past it (a path of one step would wait for 15 draws
// that nothing reads).  The tail draws of all lanes are queued (a mask per lane, a prefix sum
// over the warp) and evaluated 32 at a time: with 16 draws per lane about 25 of
// 512, one round.  Called by whole warps.
// ---------------------------------------------------------------------------
constexpr int kDrawBatch = 16;

struct DrawBuf {
  double z[kDrawBatch * 32];
  uint16_t queue[kDrawBatch * 32];
};

template <typename RNG>
__device__ __forceinline__ void stream_normals(RNG& rng, DrawBuf& buf, int lane, int n = kDrawBatch) {
  unsigned tails = 0;
  auto draw = [&](int k) {
    const double q = draw_q(rng.next_u64());
    const bool tail = draw_in_tail(q);
    double num, den;
    central_parts(draw_masked(q, tail), num, den);
    const double z = num * rcp64(den);
    buf.z[k * 32 + lane] = tail ? q : z;
    if (tail) tails |= 1u << k;
  };
#pragma unroll
  for (int g = 0; g < kDrawBatch; g += 4) {
    if (g >= n) break;
    draw(g);
    if (g + 1 == n) break;
#pragma unroll
    for (int k = 1; k < 4; ++k) draw(g + k);
  }
  int at = __popc(tails);  // inclusive prefix sum of the counts
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int below = __shfl_up_sync(kFullMask, at, o);
    if (lane >= o) at += below;
  }
  const int total = __shfl_sync(kFullMask, at, 31);
  for (at -= __popc(tails); tails; tails &= tails - 1u, ++at)
    buf.queue[at] = (uint16_t)((__ffs((int)tails) - 1) * 32 + lane);
  __syncwarp();
  for (int i = lane; i < total; i += 32) {
    const int e = buf.queue[i];
    buf.z[e] = tail_normal(buf.z[e]);
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// Sums v[0..N) over the grid in the kernel that computed them: each block
// writes its row of `partials`, and the block that finishes last (a ticket
// counter, no block waits) adds the rows in a fixed order, writes `out` and
// clears the ticket for the next launch.  `out` may be pinned host memory:
// the host reads it after it has waited for the stream.  This replaces a
// reduction launch and a device-to-host copy.  `sh` holds THREADS doubles.
// Called by all threads of blocks of THREADS threads.
// ---------------------------------------------------------------------------
template <int N, int THREADS>
__device__ __forceinline__ void grid_sum(double (&v)[N], double* sh, double* __restrict__ partials,
                                         unsigned* __restrict__ ticket, double* __restrict__ out) {
  static_assert(N * (THREADS / 32) <= THREADS, "sh is too small");
  __shared__ bool last;
  block_sum<N>(v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) partials[(int64_t)blockIdx.x * N + k] = v[k];
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  constexpr int kRows = THREADS / N;  // thread t adds rows t / N, t / N + kRows, ... of column t % N
  constexpr int kAhead = 16;          // loads in flight per thread: one block's latency is the whole grid's here
  if (threadIdx.x < kRows * N) {
    const unsigned total = gridDim.x * N;
    double acc = 0.0;
    for (unsigned i = threadIdx.x; i < total; i += kAhead * kRows * N) {
      double p[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const unsigned at = i + k * kRows * N;
        p[k] = at < total ? __ldcg(partials + at) : 0.0;
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) acc += p[k];
    }
    sh[threadIdx.x] = acc;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    double acc = 0.0;
    for (int i = 0; i < kRows; ++i) acc += sh[i * N + threadIdx.x];
    out[threadIdx.x] = acc;
    __threadfence_system();
  }
  if (threadIdx.x == 0) *ticket = 0;
}

}  // namespace of
