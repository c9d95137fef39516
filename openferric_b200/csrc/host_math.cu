// host_math.cu - host closed forms whose cost shows beside a pricing call.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <new>
#include <stdexcept>
#include <vector>

#include "of_gpu.h"

// The covariance sum of the geometric-Asian closed form, one rounding per
// addition in the reference's order (i outer, j inner: src/pricing/asian.rs:86-136).
// Added one by one it is a chain of n^2 dependent additions (1.3 ns each: 83 us
// at 252 fixings; numpy's cumsum over the n^2 terms took 300).
//
// While the sum s stays within a binade [2^e, 2^(e+1)), of grid u = 2^(e-52),
// RN(s + a) = s + RN_u(a) for every addend a that is not exactly half a grid
// step off the grid (a tie goes by the parity of s).  So in a binade without
// ties a whole row adds the integer sum_j k(min(t_i, t_j)), k(a) = RN_u(a) / u,
// and since k is monotone that is a prefix sum over the sorted fixings plus the
// rest times k(t_i).  Rows that leave the binade, binades with a tie and
// fixings that are not finite and non-negative are added one by one.  Daily
// fixings tie only in the low binades, the first eighth of the rows: 17 us.
static double min_sum_in_order(const double* times, int64_t n) {
  double s = 0.0;
  std::vector<double> sorted(times, times + n);
  bool plain = false;
  for (double x : sorted) plain = plain || !(x >= 0.0 && x <= 1e100);
  std::vector<int64_t> below, k, prefix;  // below[i]: fixings <= t_i; k and its sums in sorted order
  if (!plain) {
    std::sort(sorted.begin(), sorted.end());
    below.resize((size_t)n);
    k.resize((size_t)n);
    prefix.assign((size_t)n + 1, 0);
    for (int64_t i = 0; i < n; ++i)
      below[(size_t)i] = std::upper_bound(sorted.begin(), sorted.end(), times[i]) - sorted.begin();
  }
  int binade = INT32_MIN;
  bool usable = false;
  for (int64_t i = 0; i < n; ++i) {
    if (!plain && s >= 1e-200) {
      const int e = std::ilogb(s);
      const double u = std::ldexp(1.0, e - 52);
      if (e != binade) {
        binade = e;
        const double magic = std::ldexp(1.5, e), half = 0.5 * u;
        usable = sorted.back() < std::ldexp(1.0, e - 1) && n < (int64_t(1) << 20);
        for (int64_t j = 0; usable && j < n; ++j) {
          const double a = sorted[(size_t)j], r = (a + magic) - magic;
          if (std::fabs(a - r) == half) usable = false;
          k[(size_t)j] = (int64_t)(r / u);
          if (prefix[(size_t)j] > (int64_t(1) << 53)) usable = false;  // no row of this binade could stay in it
          if (usable) prefix[(size_t)j + 1] = prefix[(size_t)j] + k[(size_t)j];
        }
      }
      if (usable) {
        const int64_t p = below[(size_t)i], ki = k[(size_t)p - 1], rest = n - p;
        const int64_t limit = int64_t(1) << 53, at = (int64_t)(s / u);
        if (prefix[(size_t)p] <= limit && (rest == 0 || ki <= limit / rest)) {
          const int64_t sum = at + prefix[(size_t)p] + rest * ki;
          if (sum <= limit) {
            s = (double)sum * u;
            continue;
          }
        }
      }
    }
    const double ti = times[i];
    for (int64_t j = 0; j < n; ++j) s += times[j] < ti ? times[j] : ti;
  }
  return s;
}

// No exception leaves the C entry: its tables (5 n words) are what can fail.
extern "C" of_status of_min_sum_in_order(const double* times, int64_t n, double* out) {
  if (!out || n < 0 || (n > 0 && !times)) return OF_ERR_INVALID_INPUT;
  try {
    *out = min_sum_in_order(times, n);
  } catch (const std::bad_alloc&) {
    return OF_ERR_ALLOC;
  } catch (const std::length_error&) {
    return OF_ERR_ALLOC;
  }
  return OF_OK;
}
