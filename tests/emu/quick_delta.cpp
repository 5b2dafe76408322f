// The precision form's quick sums and derivative blocks (quick_delta, block_dz_quick,
// perturb_f32.cuh) against the wide-exponent ones (add3 with set_delta, block_dz) on random
// terms. TEST INFRASTRUCTURE ONLY.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>

#include "cuda_host_shim.hpp"

#include "perturb_f32.cuh"

namespace {

template <class T>
bool same(T a, T b) {
  return std::memcmp(&a, &b, sizeof a) == 0;
}

double draw(std::mt19937_64 &g, int centre, int spread) {
  const uint64_t r = g();
  if (r % 61 == 0) return 0.0;
  double m = 1.0 + (double)(g() >> 12) * 0x1p-52;
  if (r % 53 == 1) m = 1.0;
  if (r % 53 == 2) m = 2.0 - 0x1p-52 * (double)(1 + (g() % 4096));
  if (r % 53 == 3) m = 1.0 + 0x1p-24 * (double)(1 + 2 * (g() % 4096));  // halfway between two floats
  const double v = std::scalbn(m, centre + (spread ? (int)(g() % (uint64_t)(2 * spread + 1)) - spread : 0));
  return (r >> 32) & 1 ? -v : v;
}

}  // namespace

// sums: whether quick_delta changed the state otherwise than add3 and set_delta would;
// quick counts the sums it took
extern "C" int64_t quick_delta_check(uint64_t seed, uint64_t n, uint64_t *quick) {
  std::mt19937_64 g(seed);
  int64_t wrong = 0;
  *quick = 0;
  for (uint64_t i = 0; i < n; ++i) {
    fdk::StateF s{};
    const int spread = g() % 3 == 0 ? 2 : g() % 2 ? 60 : 420;
    s.oe = -(int)(g() % 1500);
    s.ar = draw(g, 5, 5);
    s.ai = draw(g, 5, 5);
    const int e1 = -(int)(g() % 1500), e2 = g() % 2 ? e1 + (int)(g() % 200) - 100 : -(int)(g() % 3000);
    const int c1 = (int)(g() % 400) - 200;
    double r1 = draw(g, c1, spread / 4), i1 = draw(g, c1, spread / 4), r2 = draw(g, 3, spread), i2 = draw(g, 3, spread);
    if (g() % 8 == 0) r2 = i2 = 0.0;
    if (g() % 16 == 0 && e2 - e1 > -900 && e2 - e1 < 900) r2 = std::scalbn(-r1 * (1.0 + 0x1p-40), e1 - e2);  // cancels
    fdk::StateF q = s, w = s;
    if (!fdk::quick_delta(q, r1, i1, e1, r2, i2, e2)) {
      wrong += !same(q.wr, s.wr) || q.e != s.e;
      continue;
    }
    ++*quick;
    const fdk::Cx3 t = fdk::add3(fdk::Cx3{r1, i1, e1}, fdk::Cx3{r2, i2, e2});
    fdk::set_delta(w, t.re, t.im, t.e);
    wrong += !(same(q.wr, w.wr) && same(q.wi, w.wi) && q.e == w.e && same(q.s32, w.s32) && same(q.s64, w.s64) &&
               same(q.dcr, w.dcr) && same(q.dci, w.dci));
  }
  return wrong;
}

extern "C" int64_t quick_dz_check(uint64_t seed, uint64_t n, uint64_t *quick) {
  std::mt19937_64 g(seed);
  int64_t wrong = 0;
  *quick = 0;
  for (uint64_t i = 0; i < n; ++i) {
    fdk::StateF s{};
    const int spread = g() % 3 == 0 ? 3 : g() % 2 ? 60 : 1000;
    s.dr = draw(g, 10, spread / 4);
    s.di = draw(g, 10, spread / 4);
    s.dexp = g() % 4 ? (int64_t)(g() % 1300) : (int64_t)(g() % 8000) - 2000;
    s.inverse = fdk::exp2i(-s.dexp);
    const int ac = (int)(g() % 60);
    const double2 A = make_double2(draw(g, ac, spread / 4), draw(g, ac, spread / 4));
    const double2 B = make_double2(draw(g, ac, spread / 4), draw(g, ac, spread / 4));
    const fdk::DzF want = fdk::block_dz(s.dr, s.di, s.dexp, A, B);
    if (!fdk::block_dz_quick(s, A, B)) continue;
    ++*quick;
    wrong += !(same(s.dr, want.dr) && same(s.di, want.di) && s.dexp == want.dexp && same(s.inverse, want.inverse));
  }
  return wrong;
}
