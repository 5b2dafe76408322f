// A stripe replay that finds no escape (perturb_f64.cuh, sample.rs:397, 576-579): the blocks'
// outcome once the replay reaches its limit, wherever the next block budget ends.
// TEST INFRASTRUCTURE ONLY.
#include <cmath>
#include <cstdint>
#include <vector>

#include "cuda_host_shim.hpp"

#include "perturb_f64.cuh"

// Plain steps of a sample inside c = -1's disc, replaying up to `limit` with the block budget
// ending at `lim`, up to 1000 of them: the iterate the replay ended at with the recorded
// outcome and window, or 0.
template <bool EXT, bool D>
static uint32_t replay(uint32_t limit, uint32_t lim) {
  const uint32_t points = 4096;
  std::vector<double2> z(points), fused(2 * points);
  for (uint32_t m = 0; m < points; ++m) {
    z[m] = make_double2(m % 2 ? -1.0 : 0.0, 0.0);
    fused[2 * m] = z[m];
    fused[2 * m + 1] = make_double2(-1.0, -1.0);
  }
  fdk::Params p{};
  p.orbit = z.data();
  p.fused = fused.data();
  p.last = points - 1;
  p.max_iter = 100000;
  p.r2 = 1e20;
  p.nucleus = -1;
  fdk::State<EXT> s{};
  s.ar = 0.05;
  s.ai = 0.02;
  s.offset_exp = 0;
  fdk::start_sample<EXT, D, true, false>(p, s, false, false);
  fdk::TraceSlot<true> slot;
  fdk::StripeTrace &tr = *slot.get(p);
  tr.start(0);
  fdk::Result first{};
  first.n = 77;
  first.zr = 3.0;
  first.zi = 4.0;
  tr.keep(first);
  s.replaying = true;
  s.limit = limit;
  s.lim = lim;
  fdk::Result res{};
  fdk::ExactProduct product;
  product.reset();
  for (int k = 0; k < 1000; ++k) {
    fdk::plain_update<EXT, D, true>(p, s);
    if (fdk::post<EXT, D, true, false, true>(p, s, res, product, &tr))
      return res.kind == 0 && res.n == 77 && tr.end_at == 77 && tr.end_r == 3.0 && tr.end_i == 4.0 ? s.n : 0;
  }
  return 0;
}

extern "C" uint32_t stripe_limit_check(int extended, int derivative, uint32_t limit, uint32_t lim) {
  if (extended) return derivative ? replay<true, true>(limit, lim) : replay<true, false>(limit, lim);
  return derivative ? replay<false, true>(limit, lim) : replay<false, false>(limit, lim);
}
