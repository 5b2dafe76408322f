// block_level (perturb_f64.cuh): the search over an ordered table and the wide search against
// the reference's order of tests, level by level (bla.rs:234-249), on random ordered tables.
// TEST INFRASTRUCTURE ONLY.
#include <cmath>
#include <cstdint>
#include <random>
#include <vector>

#include "cuda_host_shim.hpp"

#include "perturb_f64.cuh"

namespace {

// the reference's loop: the last level before the first that does not start at m, does not
// fit the budget or the table, or whose radius the delta exceeds
int reference_level(const fdk::Params &p, double d2, uint32_t m, uint64_t budget) {
  const uint32_t k = m - 1;
  int lv = -1;
  for (uint32_t i = 0; i < p.bla_levels; ++i) {
    if ((k & ((2u << i) - 1u)) != 0 || (2ull << i) > budget) break;
    const uint32_t a = k >> (i + 1);
    if (a >= p.bla_count[i] || !(d2 < p.bla_r2[p.bla_off[i] + a])) break;
    lv = (int)i;
  }
  return lv;
}

}  // namespace

extern "C" int64_t block_level_check(uint64_t seed, uint32_t points, uint64_t n) {
  std::mt19937_64 g(seed);
  fdk::Params p{};
  p.last = points - 1;
  const uint32_t steps = points - 2;
  std::vector<double> r2;
  for (uint32_t i = 0; (steps >> (i + 1)) > 0 && i < 20; ++i) {
    p.bla_off[i] = (uint32_t)r2.size();
    p.bla_count[i] = steps >> (i + 1);
    for (uint32_t t = 0; t < p.bla_count[i]; ++t) {
      const double above = i == 0 ? 1.0 : r2[p.bla_off[i - 1] + 2 * t];
      const uint64_t r = g() % 8;  // equal to its first half's, a little or a lot smaller, zero
      r2.push_back(r < 3 ? above : r < 7 ? above * (double)(g() % 1000) / 1000.0 : (r2.size() % 5 ? above : 0.0));
    }
    p.bla_levels = i + 1;
  }
  p.bla_r2 = r2.data();
  int64_t wrong = 0;
  for (uint64_t q = 0; q < n; ++q) {
    fdk::State<false> s{};
    const uint32_t top = (uint32_t)(g() % (p.bla_levels + 1));
    s.m = 1 + (uint32_t)((g() % steps) >> (top + 1) << (top + 1));
    const uint64_t budget = g() % 3 ? 1 + g() % (2u << (g() % 20)) : 0xffffffffu;
    s.n = 5;
    s.lim = (uint32_t)std::fmin(4294967295.0, 5.0 + (double)budget);
    const uint32_t k = (s.m - 1) >> 1;
    const uint32_t i = (uint32_t)(g() % p.bla_levels), a = (s.m - 1) >> (i + 1);
    double d2 = a < p.bla_count[i] ? r2[p.bla_off[i] + a] : 0.5;  // at a radius exactly, or beside one
    if (g() % 2) d2 = d2 * (double)(900 + g() % 200) / 1000.0;
    s.xr = std::sqrt(d2);
    d2 = fdk::block_d2(s);
    const int want = reference_level(p, d2, s.m, s.lim - s.n);
    if (want < 0 || k >= p.bla_count[0]) continue;  // block_starts admits the first level
    for (int mode = 0; mode < 3; ++mode) {
      uint32_t at = 0;
      p.bla_ordered = mode == 1;
      const int got = mode == 2 ? fdk::block_level<false, true>(p, s, at) : fdk::block_level<false, false>(p, s, at);
      wrong += got != want || at != (s.m - 1) >> (want + 1);
    }
  }
  return wrong;
}
