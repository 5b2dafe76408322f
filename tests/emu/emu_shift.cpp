// The kernel emulation (emu.cpp) with the shift estimate on (FDC_SHIFT): one frame of the
// plain form with a table, from a series start where series_n > 0 (ordinary tiers) or from
// Z_0. TEST INFRASTRUCTURE ONLY.
#include "emu.cpp"

extern "C" int emu_render_shift(const double *re, const double *im, uint64_t len, const double *blocks7,
                                const uint64_t *level_offsets, uint32_t levels, const double *series_b,
                                uint32_t series_order, uint32_t series_n, double series_rho, int32_t tier, uint32_t nx,
                                uint32_t ny, double c_re, double c_im, double h_m, int64_t h_e, uint32_t max_iter,
                                double escape_radius, int64_t nucleus, const uint8_t *mask, const double *offsets,
                                uint8_t *cls, uint32_t *n_out, double *z_out, uint64_t *counters, double *shift) {
  Setup s;
  s.ext = tier == 2;
  s.deriv = true;
  s.bla = true;
  stage_orbit(s, re, im, len, blocks7, level_offsets, levels);
  if (!stage_frame(s, tier, nx, ny, 1, c_re, c_im, h_m, h_e, 1.0, 0.0, max_iter, escape_radius, nucleus, 0, 0, 0, 0, 3,
                   mask, offsets, false))
    return -1;
  fdk::Params &p = s.p;
  p.flags |= fdk::F_SHIFT;
  const size_t n = (size_t)nx * ny;
  std::vector<uint8_t> status(n);
  std::vector<double> dz(2 * n);
  std::vector<int64_t> dexp(n);
  stage_outputs(p, cls, n_out, nullptr, nullptr, nullptr, z_out, dz.data(), dexp.data(), status.data());
  unsigned long long queue = 0;
  fdk::Counters cnt{};
  uint32_t timed_out = 0;
  p.queue = &queue;
  p.counters = &cnt;
  p.timed_out = &timed_out;
  p.series_b = (const double2 *)series_b;
  p.series_order = series_order;
  p.series_n = series_n;
  p.series_inv = 1.0 / series_rho;
  if (s.ext) launch<true, true, true, false, false>(p);
  else if (series_n > 0) launch<false, true, true, true, false>(p);
  else launch<false, true, true, false, false>(p);
  copy_counters(cnt, counters);
  std::memcpy(shift, &cnt.shift_bits, sizeof *shift);
  return 0;
}
