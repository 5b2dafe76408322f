// The extended tier's near returns (sample.rs:492-570) count four times a sample; afterwards an
// iterate near the save point runs the full sequence no more. That shows in the nucleus
// product's exponent: the full sequence folds every factor into it, the short one only where
// the product leaves its range.
// TEST INFRASTRUCTURE ONLY.
#include <cmath>
#include <cstdint>
#include <vector>

#include "cuda_host_shim.hpp"

#include "perturb_f64.cuh"

// `steps` plain iterations of the sample at c + (ar, ai) over the escaping orbit of c =
// -1.25066 + 0.02012i. Returns the near returns counted, or -1 for a sample that ended. Of the
// iterations near the save point after the fourth return, `near` counts all and `folded` those
// that changed the product's exponent.
extern "C" int near_returns_check(double ar, double ai, uint32_t steps, uint32_t *near, uint32_t *folded) {
  std::vector<double2> z;
  for (double x = 0.0, y = 0.0; x * x + y * y < 1e20;) {
    z.push_back(make_double2(x, y));
    const double t = x * x - y * y - 1.25066;
    y = 2.0 * x * y + 0.02012;
    x = t;
  }
  fdk::Params p{};
  p.orbit = z.data();
  p.last = (uint32_t)z.size() - 1;
  p.max_iter = 1u << 30;
  p.r2 = 1e20;
  p.nucleus = 1 << 28;
  fdk::State<true> s{};
  s.ar = ar;
  s.ai = ai;
  s.offset_exp = 0;
  fdk::start_sample<true, false, false, false>(p, s, false, false);
  fdk::Result res{};
  fdk::ExactProduct product;
  product.reset();
  *near = *folded = 0;
  for (uint32_t k = 0; k < steps; ++k) {
    const bool spent = s.returns >= fdk::MAX_RETURNS;
    const double sr = s.sr, si = s.si, bound = s.near;
    const int32_t e = s.ct.e;
    fdk::plain_update<true, false, false>(p, s);
    if (fdk::post<true, false, false>(p, s, res, product)) return -1;
    if (spent && std::fabs(s.fr - sr) + std::fabs(s.fi - si) < bound) {
      ++*near;
      *folded += s.ct.e != e;
    }
  }
  return s.returns;
}
