// block_quick (perturb_f64.cuh) against block_full, the extended tier's block application
// with every normalisation, on random states and coefficients of all of binary64's range.
// TEST INFRASTRUCTURE ONLY.
#include <cmath>
#include <cstdint>
#include <random>

#include "cuda_host_shim.hpp"

#include "perturb_f64.cuh"

namespace {

uint64_t bits(double a) { return (uint64_t)__double_as_longlong(a); }

// spread: binades around `centre` the magnitude is drawn from; now and then a zero, a
// power of two or a mantissa just below 2
double draw(std::mt19937_64 &g, int centre, int spread) {
  const uint64_t r = g();
  if (r % 97 == 0) return 0.0;
  double m = 1.0 + (double)(g() >> 12) * 0x1p-52;
  if (r % 89 == 1) m = 1.0;
  if (r % 89 == 2) m = 2.0 - 0x1p-52 * (double)(1 + (g() % 4096));
  const int e = centre + (spread ? (int)(g() % (uint64_t)(2 * spread + 1)) - spread : 0);
  const double v = std::scalbn(m, e);
  return (r >> 32) & 1 ? -v : v;
}

template <bool D>
int64_t run(uint64_t seed, uint64_t n, uint64_t *quick) {
  std::mt19937_64 g(seed);
  int64_t wrong = 0;
  for (uint64_t i = 0; i < n; ++i) {
    fdk::State<true> s{};
    const int wide = (int)(g() % 4);
    const int xs = wide == 0 ? 3 : wide == 1 ? 40 : wide == 2 ? 500 : 1060;
    const int xc = g() % 3 ? 0 : -(int)(g() % 1000);
    s.xr = draw(g, xc, xs / 4);
    s.xi = draw(g, xc, xs / 4);
    const int dcen = g() % 3 ? 10 : -(int)(g() % 1000);
    s.dr = draw(g, dcen, xs / 4);
    s.di = draw(g, dcen, xs / 4);
    s.offset_exp = -(int)(g() % 4000);
    s.delta_exp = g() % 4 ? (int)std::fmin(0.0, s.offset_exp + (double)(g() % 1500)) : -(int)(g() % 4000);
    s.derivative_exp = g() % 4 ? (int64_t)(g() % 1300) : (int64_t)(g() % 8000) - 2000;
    s.ar = draw(g, 5, 6);
    s.ai = draw(g, 5, 6);
    s.inverse = fdk::exp2i(-s.derivative_exp);
    const double f = fdk::exp2i(s.offset_exp - s.delta_exp);
    s.dc_r = s.ar * f;
    s.dc_i = s.ai * f;
    const int ac = g() % 3 ? (int)(g() % 60) : (int)(g() % 2000) - 1000, bc = g() % 3 ? ac + (int)(g() % 20) : (int)(g() % 2000) - 1000;
    double2 A = make_double2(draw(g, ac, xs / 4), draw(g, ac, xs / 4));
    double2 B = make_double2(draw(g, bc, xs / 4), draw(g, bc, xs / 4));
    if (g() % 16 == 0 && s.xi != 0.0) A.y = A.x * s.xr / s.xi;  // the products of one part nearly cancel
    const fdk::BlockTerms want = fdk::block_full<D>(
        fdk::BlockTerms{s.xr, s.xi, s.dr, s.di, s.inverse, s.derivative_exp, s.delta_exp}, A, B, s.ar, s.ai,
        s.offset_exp);
    const fdk::State<true> before = s;
    if (!fdk::block_quick<D>(s, A, B)) {
      wrong += bits(s.xr) != bits(before.xr) || s.delta_exp != before.delta_exp || bits(s.dr) != bits(before.dr);
      continue;
    }
    ++*quick;
    bool same = bits(s.xr) == bits(want.xr) && bits(s.xi) == bits(want.xi) && s.delta_exp == want.delta_exp;
    if (D)
      same = same && bits(s.dr) == bits(want.dr) && bits(s.di) == bits(want.di) &&
             s.derivative_exp == want.derivative_exp && bits(s.inverse) == bits(want.inverse);
    wrong += !same;
  }
  return wrong;
}

}  // namespace

extern "C" int64_t block_quick_check(uint64_t seed, uint64_t n, int derivative, uint64_t *quick) {
  *quick = 0;
  return derivative ? run<true>(seed, n, quick) : run<false>(seed, n, quick);
}
