// The nucleus gate's squared modulus (Magnitude, fd_device.cuh) against the reference's product
// (Contraction) on random runs of factors: an answer, wherever Magnitude gives one, is
// Contraction's. TEST INFRASTRUCTURE ONLY.
#include <cmath>
#include <cstdint>
#include <limits>
#include <random>

#include "cuda_host_shim.hpp"

#include "perturb_f64.cuh"

// n runs of 1 to 40 factors, one of each run of `kind`: 0 ordinary sizes, 1 below 2^-1023 (where
// Contraction's rescaling overflows), 2 anywhere in binary64's range, 3 zero, 4 infinite, 5 NaN.
// Returns the wrong answers; answered counts the runs Magnitude decided.
extern "C" int64_t magnitude_check(uint64_t seed, uint64_t n, int kind, uint64_t *answered) {
  std::mt19937_64 g(seed);
  const auto unit = [&]() { return (double)(g() >> 11) * 0x1p-53 * 2.0 - 1.0; };
  int64_t wrong = 0;
  *answered = 0;
  for (uint64_t q = 0; q < n; ++q) {
    fdk::Contraction c;
    c.reset();
    fdk::Magnitude m;
    const int len = 1 + (int)(g() % 40), odd = (int)(g() % len);
    m.reset(len);
    double log2p = 0.0;
    for (int i = 0; i < len; ++i) {
      double r = unit(), im = unit();
      // ordinary factors steer the product to the threshold's neighbourhood
      const int pull = i == len - 1 && kind < 3 ? (int)std::fmax(-1000.0, std::fmin(1000.0, -10.0 - log2p)) : (int)(g() % 5) - 2;
      r = std::ldexp(r, pull);
      im = std::ldexp(im, pull);
      if (i == odd && kind > 0) {
        if (kind == 1) {
          r = std::ldexp(r, -1023 - (int)(g() % 50));
          im = std::ldexp(im, -1023 - (int)(g() % 50));
        } else if (kind == 2) {
          const int e = (int)(g() % 2098) - 1074;
          r = std::ldexp(unit(), e);
          im = g() % 4 ? std::ldexp(unit(), e) : 0.0;
        } else {
          const double v = kind == 3 ? 0.0 : kind == 4 ? std::numeric_limits<double>::infinity() : std::nan("");
          r = v;
          if (kind == 3 || g() % 2) im = v;
        }
      }
      const double a = std::fmax(std::fabs(r), std::fabs(im));
      if (a > 0.0 && std::isfinite(a)) log2p += std::log2(a);
      c.multiply(r, im);
      if (!m.times(r * r + im * im, 0)) m.times_wide(r, im);
    }
    const int s = m.small(len);
    if (s < 0) continue;
    ++*answered;
    wrong += (s != 0) != c.small();
  }
  return wrong;
}
