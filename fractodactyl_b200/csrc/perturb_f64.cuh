// The plain (FP64) perturbation kernel: one lane per sample, persistent warps that
// refill finished lanes from an atomic tile queue. The per-sample state machine is
// iterate() of crates/fd-kernel/src/sample.rs:170-581 (Binary64 and Binary64Exponent,
// number.rs:92-124) with the reference's operation order: one loop iteration is apply_block
// or plain_update, then post, which tests for rare events once (settle handles them) and
// chooses the next operation; warp_step runs it for a warp (with BLA deferral), step for
// one lane. Compile with -fmad=false.
#pragma once
#include <cstdint>

#include "fd_device.cuh"

namespace fdk {

constexpr int MAX_LEVELS = 40;

// Resident 128-thread blocks per SM each kernel variant is compiled for (caps registers
// at 65536 / (128 * blocks)): floatexp-tier variants (EXT) and ordinary-tier variants;
// chosen by measurement. Kernel ms at 4 / 5 / 6 floatexp blocks: 1920x1080 at a 1e-100 nucleus
// 20.3 / 19.5 / 20.0, 2880x1620 jittered at 1e-300 50.8 / 48.7 / 49.5; at 3 / 4 / 5 ordinary
// ones: 1280x720 with blocks 9.7 / 10.1 / 11.0, 480x270 without 2.97 / 2.53 / 2.59.
#ifndef FDK_MIN_BLOCKS_EXT
#define FDK_MIN_BLOCKS_EXT 5
#endif
#ifndef FDK_MIN_BLOCKS_FIX
#define FDK_MIN_BLOCKS_FIX 4
#endif
template <bool EXT>
struct Occupancy {
  static constexpr int blocks = EXT ? FDK_MIN_BLOCKS_EXT : FDK_MIN_BLOCKS_FIX;
};

struct Counters {
  unsigned long long samples, iterations, blocks, skipped, fallback, closed;
  unsigned long long shift_bits;  // max of the non-negative shift estimates, as bits
  unsigned long long pad;
};

// Everything one launch needs; passed by value (kernel parameter space).
struct Params {
  const double2 *__restrict__ orbit;  // Z_0..Z_last, interleaved re/im
  // With BLA: Z_m fused with the squared radius of the first-level block (2 steps) starting at m,
  // -1 where none starts there: 32-byte entries (zr, zi, r2a, unused), one load each, so that
  // whether a block starts comes with the orbit point each step loads anyway.
  const double2 *__restrict__ fused;
  const void *orbit32;  // precision-form entries (perturb_f32.cuh), per job in batches
  uint32_t last;
  double z0r, z0i;
  // BLA, level-major: r2[off + t], coef[2 (off + t)] = (a.re, a.im), (b.re, b.im), ab = (alpha, beta)
  const double *__restrict__ bla_r2;
  const double2 *__restrict__ bla_coef;
  const double2 *__restrict__ bla_ab;
  uint32_t bla_levels;
  uint32_t bla_ordered;  // no block's radius exceeds that of its first half: levels pass as a prefix
  uint32_t bla_off[MAX_LEVELS];
  uint32_t bla_count[MAX_LEVELS];
  // frame
  uint32_t nx, ny, first_row, rows, tiles_x;
  uint32_t first_col, cols;        // rendered window: columns [first_col, first_col + cols) of those rows
  uint32_t in_pitch, out_pitch;    // row pitch (samples) of the mask/offsets inputs and of the outputs,
                                   // whose pointers address the window's first sample
  uint32_t tile_shift;  // tiles are 2^tile_shift samples wide and 32 / 2^tile_shift rows high
  const uint32_t *tile_order;  // order the queue hands tiles out in (row-major tile indices), or null
  int32_t tier;
  uint32_t flags;
  double c_re, c_im, h, h_m;
  int64_t h_e;
  double cosr, sinr, half_x, half_y;
  uint32_t max_iter;  // < 2^32 (checked by the route)
  double r2;
  int64_t nucleus;
  double px_m;  // DE output pixel h_m * ss (store.rs:57-63)
  int64_t px_e;
  const uint8_t *__restrict__ mask;
  const double2 *__restrict__ offsets;
  // outputs (device)
  uint8_t *cls;
  uint32_t *n_out;
  double *nu;
  float *de;
  uint16_t *normal;
  double2 *z_out, *dz_out;
  int64_t *dexp_out;
  uint8_t *status;
  // scratch: work queue and counters
  unsigned long long *queue;
  Counters *counters;
  uint64_t total;        // queue slots (tiles * 32)
  uint64_t deadline_ns;  // 0 = none
  uint32_t *timed_out;
  uint32_t idle_lanes;  // lanes of each warp that take no sample (small launches)
  uint32_t tail;        // slots left from which a warp takes only what its idle lanes need
  uint32_t defer;     // BLA lanes a warp gathers before it applies their blocks (warp_step)
  // Parameter-series start (series.rs:57-84, ordinary tiers): every sample starts at
  // iterate series_n from delta = sum_k b_k x^k, x = dc / rho; series_n = 0: none.
  const double2 *__restrict__ series_b;  // b_1..b_order as (re, im)
  uint32_t series_order, series_n;
  double series_inv;  // 1 / rho
  // Bounded variant (B, ordinary tiers): the orbit's error radii q[m] >= |A_m - Z_m|
  // (reference.rs:122-148) and the outputs it adds: the Bound column and the raw radii
  const double *__restrict__ q;
  float *bound_out;
  double *ez_out, *ed_out;
  // Stripe variant (T): the column (stripe.rs) and its settings (window 1..64, frequency)
  float *stripe_out;
  uint32_t stripe_window;
  double stripe_freq;
  double2 *stripe_traces;  // StripeTrace::UNITS for every thread of the grid
};

constexpr double SAFE = 1.0 + 8.0 * U;  // sample.rs:56
constexpr uint32_t NO_GATE = 0xffffffffu;
constexpr int MAX_RETURNS = 4;  // near returns the extended tier counts a sample (sample.rs:494)

enum : uint32_t { F_DERIV = 1u, F_BLA = 2u, F_SHIFT = 4u };

// Per-lane sample state (sample.rs:187-236).
template <bool EXT>
struct State {
  double xr, xi, dr, di;
  double fr, fi;  // z = Z[m] + delta (carried between steps on the ordinary tier)
  double Zr, Zi;  // Z[m]
  double Yr, Yi;  // Z[m + 1], loaded an iteration ahead (kernels without BLA, with the derivative)
  double r2a;     // radius^2 of the block of 2 steps starting at m, -1 where none starts (BLA kernels)
  double ar, ai;  // sample offset (mantissa on the extended tier)
  double dc_r, dc_i, scale, inverse;
  double sr, si, qr, qi, qstep;
  double near;  // save_point(): the near-return bound of the save point; infinite while a save is pending
  Multiplier mu;
  Magnitude ct;
  double adc, shift;
  double e, ed, rc;  // B: error radii on z and dz/dc, the offset's own error (sample.rs:221-225)
  int32_t offset_exp, delta_exp;  // |h_e| <= 2^30 (checked by the route): deltas stay within 32 bits
  int64_t derivative_exp;
  uint32_t gate;  // the nucleus gate's iterate, nucleus + 1 < 2^31, or NO_GATE
  uint32_t n, chk, sn, hold, blocks, skipped;  // n < max_iter < 2^32; chk saturates at 2^32 - 1
  uint32_t lim;  // relimit()
  uint32_t m, idx;
  int returns;
  bool on;  // the next operation is a BLA block (set by post)
  bool pending, predicted;
  bool replaying;  // T: re-walking a stripe window plainly (sample.rs:231-236) ...
  uint32_t limit;  // ... up to this iterate
};

// Result of a finished sample (sample.rs:21-40): kind 0 escaped, 1 interior, 2 unresolved.
struct Result {
  int kind;
  uint64_t n;
  double zr, zi, dr, di;
  int64_t dexp;
  double ez, ed;  // B: error radii of an escaped sample (sample.rs:373-377)
};

// The loop state at the start of a BLA block, from which a stripe replay restarts
// (stripe.rs:39-52).
struct StripeSnap {
  uint32_t m, n;
  double xr, xi;
  int32_t delta_exp;
  double scale, dc_r, dc_i;
};

// The Stripe column's recorder for one lane (stripe.rs:12-241): the last 128 iterates, the
// last 8 block starts, and the escape the blocks found while a replay re-walks its window.
// Only the stripe variants (T) hold one. Its 164 units of 16 bytes (2.6 KB) lie in global memory
// in groups of 4, a warp's lanes side by side group by group: a lane that steps alone fills
// whole sectors, lanes that step together whole lines, and a frame of short samples touches
// few lines of what does not fit into L2. Kernel ms by units a group, 1 2 4 8 and a lane's units
// in one piece: 1531x429 at 5e-326, 197 iterations, 0.28 0.36 0.45 0.62 1.23 (0.53 in local
// memory, whose words are interleaved); 640x360 at 1e-100, Fixed tier, 11.6 10.7 10.4 10.5 10.5
// (22.2); 1600x900 of the same 38.9 31.9 30.3 29.5 29.0 (99).
struct StripeTrace {
  static constexpr uint32_t RING = 128, SNAPS = 8, SNAP_UNITS = 4, FIRST = RING + SNAPS * SNAP_UNITS, UNITS = FIRST + 4,
                            GROUP = 4;
#if defined(__CUDA_ARCH__)
  static constexpr uint32_t LANES = 32;
#else
  static constexpr uint32_t LANES = 1;  // host builds run a warp of one lane
#endif
  double2 *at;  // unit 0; the lanes' groups of unit 0 to 3 follow one another
  uint64_t valid;
  uint32_t count;
  uint32_t starts[SNAPS];  // the block starts' iterates
  uint64_t end_at;         // the iterate the outcome's window ends at (end), and z there
  double end_r, end_i;

  static __device__ __forceinline__ uint32_t place(uint32_t u) { return u / GROUP * (GROUP * LANES) + u % GROUP; }
  __device__ __forceinline__ double2 &unit(uint32_t u) const { return at[place(u)]; }
  static __device__ __forceinline__ double bits(uint64_t v) { return __longlong_as_double((long long)v); }
  static __device__ __forceinline__ uint64_t bits(double v) { return (uint64_t)__double_as_longlong(v); }

  __device__ __forceinline__ void begin() {  // stripe.rs:164-168
    valid = ~0ull;
    count = 0;
  }
  __device__ __forceinline__ void start(uint64_t n) { valid = n + 1; }
  __device__ __forceinline__ void record(uint32_t n, double zr, double zi) { unit(n % RING) = make_double2(zr, zi); }
  __device__ __forceinline__ void snap(const StripeSnap &s, uint64_t landed) {  // stripe.rs:180-187
    const uint32_t k = count % SNAPS, u = RING + k * SNAP_UNITS;
    unit(u) = make_double2(bits((uint64_t)s.n << 32 | s.m), s.xr);
    unit(u + 1) = make_double2(s.xi, bits((uint64_t)(uint32_t)s.delta_exp));
    unit(u + 2) = make_double2(s.scale, s.dc_r);
    unit(u + 3) = make_double2(s.dc_i, bits(valid));
    starts[k] = s.n;
    count += 1;
    valid = landed;
  }
  // stripe.rs:157-160 and 189-204: a kept block start to replay from when the windows
  // ending at z_n miss iterates (the latest at or before n - window, else the oldest)
  __device__ bool rewind(uint64_t n, uint32_t window, StripeSnap &out) {
    const uint64_t need = n > window ? n - window : 0;
    if (count == 0 || valid <= (need > 1 ? need : 1)) return false;
    const uint32_t kept = count < SNAPS ? count : SNAPS;
    int pick = -1;
    for (uint32_t j = 0; j < kept && pick < 0; ++j) {
      const uint32_t k = (count - 1 - j) % SNAPS;
      if (starts[k] <= need) pick = (int)k;
    }
    if (pick < 0) {
      for (uint32_t j = 0; j < kept; ++j) {
        const uint32_t k = (count - 1 - j) % SNAPS;
        if (pick < 0 || starts[k] < starts[pick]) pick = (int)k;
      }
    }
    const uint32_t u = RING + (uint32_t)pick * SNAP_UNITS;
    const double2 a = unit(u), b = unit(u + 1), c = unit(u + 2), d = unit(u + 3);
    out.m = (uint32_t)bits(a.x);
    out.n = (uint32_t)(bits(a.x) >> 32);
    out.xr = a.y;
    out.xi = b.x;
    out.delta_exp = (int32_t)(uint32_t)bits(b.y);
    out.scale = c.x;
    out.dc_r = c.y;
    out.dc_i = d.x;
    valid = bits(d.y);
    return true;
  }
  // the escape the blocks found, kept while a replay re-walks its window
  __device__ __forceinline__ void keep(const Result &r) {
    unit(FIRST) = make_double2(bits(r.n), bits((uint64_t)r.dexp));
    unit(FIRST + 1) = make_double2(r.zr, r.zi);
    unit(FIRST + 2) = make_double2(r.dr, r.di);
  }
  __device__ __forceinline__ Result kept() const {
    const double2 a = unit(FIRST), z = unit(FIRST + 1), d = unit(FIRST + 2);
    Result r;
    r.kind = 0;
    r.n = bits(a.x);
    r.dexp = (int64_t)bits(a.y);
    r.zr = z.x;
    r.zi = z.y;
    r.dr = d.x;
    r.di = d.y;
    return r;
  }
  // stripe.rs:132-152: 0.5 + 0.5 sin(k arg z); a whole k up to 16 as the sign of k times
  // Im (z / |z|)^|k|
  __device__ static double term(double zr, double zi, double k) {
    double s;
    if (k == trunc(k) && fabs(k) <= 16.0) {
      const double h = hypot(zr, zi);
      const double ur = zr / h, ui = zi / h;
      double pr = 1.0, pi = 0.0;
      const int reps = (int)fabs(k);
      for (int q = 0; q < reps; ++q) {
        const double nr = pr * ur - pi * ui, ni = pr * ui + pi * ur;
        pr = nr;
        pi = ni;
      }
      s = k < 0.0 ? -pi : pi;
    } else {
      s = sin(k * atan2(zi, zr));
    }
    return 0.5 + 0.5 * s;
  }
  __device__ __forceinline__ void end(uint64_t n, double zr, double zi) {
    end_at = n;
    end_r = zr;
    end_i = zi;
  }
  // stripe.rs:206-240: the windows ending at z_n and z_{n-1}, interpolated by how far past the
  // escape radius z_n landed, of lane l's sample by the whole warp: each lane takes the term of one
  // iterate, and all add them in the reference's order. One lane after the other for every
  // finished sample, the terms (a hypot, two divisions or a sine each) were most of the kernel's
  // work. The value is lane l's; the others' is of no use.
  __device__ float average(unsigned lane, unsigned l, double r2, uint32_t window, double k) const {
    const uint64_t n = __shfl_sync(0xffffffffu, end_at, (int)l), from = __shfl_sync(0xffffffffu, valid, (int)l);
    const double2 *ring = at + ((int)l - (int)lane) * (int)GROUP;
    const uint64_t lo = n > window ? n - window : 0;
    const uint64_t first_i = lo > 1 ? lo : 1;
    double now = 0.0, before = 0.0;
    uint32_t cn = 0, cb = 0;
    for (uint64_t base = first_i; base <= n; base += LANES) {
      const uint64_t mine = base + lane;
      double own = 0.0;
      if (mine <= n && mine >= from) {
        const double2 z = ring[place((uint32_t)(mine % RING))];
        own = term(z.x, z.y, k);
      }
      for (uint64_t i = base; i < base + LANES && i <= n; ++i) {
        const double t = __shfl_sync(0xffffffffu, own, (int)(i - base));
        if (i < from) continue;
        if (i > first_i || (first_i == 1 && n <= window)) {
          now += t;
          cn += 1;
        }
        if (i < n) {
          before += t;
          cb += 1;
        }
      }
    }
    if (cn == 0) return 0.0f;
    now /= (double)cn;
    before = cb > 0 ? before / (double)cb : now;
    double frac = 1.0 - log2(log(end_r * end_r + end_i * end_i) / log(r2));
    if (frac < 0.0) frac = 0.0;  // f64::clamp keeps NaN
    if (frac > 1.0) frac = 1.0;
    return (float)(before * (1.0 - frac) + now * frac);
  }
};

// A periodicity save point (sample.rs:488-491, 522-575): the point and the bound that a
// later z's distance from it is compared with, fabs(sr) + fabs(si) scaled as each tier's
// near-return test scales it. The reference evaluates the bound every iteration from the
// same two values, so evaluating it once here gives the same double. While a save is
// pending every judged z is an event: the bound is infinite (sequence() takes near_bound).
template <bool EXT>
__device__ __forceinline__ double near_bound(const State<EXT> &s) {
  const double size = fabs(s.sr) + fabs(s.si);
  return EXT ? 1e-13 * size + 1e-300 : 1e-3 * size;
}

template <bool EXT>
__device__ __forceinline__ void save_point(State<EXT> &s, double r, double i) {
  s.sr = r;
  s.si = i;
  s.near = near_bound(s);
}

template <bool EXT>
__device__ __forceinline__ void await_save(State<EXT> &s) {  // the next judged iterate is saved
  s.pending = true;
  s.near = __longlong_as_double(0x7ff0000000000000ll);
}

// The iteration limit behind Bla::find's budget (sample.rs:246-263) with n left out:
// min(max_iter, the next periodicity save point, nucleus + 1), kept in the state and
// recomputed whenever one of its inputs (hold, sn, pending, chk, gate) changes, so an
// iteration only subtracts n. The reference's n == 0 case (a budget of 1) never reaches
// the search: with a nucleus gate, m == 0 skips the BLA. lim <= max_iter < 2^32.
template <bool EXT>
__device__ __forceinline__ void relimit(const Params &p, State<EXT> &s) {
  uint32_t cap = s.chk;
  if (!EXT) {
    const uint32_t back = s.sn + s.hold;
    cap = s.hold > 0 ? (back < s.sn ? 0xffffffffu : back) : (s.pending ? 0xffffffffu : s.chk);
  }
  s.lim = min(min(p.max_iter, cap), s.gate);
}

// Bla::find (bla.rs:234-249): the longest valid block starting at m that fits the budget.
// The radius of the first level comes with the orbit entry (r2a); block_starts tests it, and
// block_level searches the others once the lane's turn to apply a block has come.
template <bool EXT>
__device__ __forceinline__ double block_d2(const State<EXT> &s) {
  return EXT ? (s.xr * s.xr + s.xi * s.xi) * s.scale * s.scale : s.xr * s.xr + s.xi * s.xi;
}

// Whether Bla::find finds any block at m: one test for the nucleus gate, the budget and
// the level-1 block (r2a is -1 unless a block starts at m); every operand is evaluated,
// which costs fewer branches than returning at the first that fails.
template <bool EXT>
__device__ __forceinline__ bool block_starts(const State<EXT> &s) {
  const uint32_t budget = s.lim > s.n ? s.lim - s.n : 0u;
  return (s.gate == NO_GATE || s.m != 0) & (budget >= 2) & (block_d2(s) < s.r2a);
}

// The rest of Bla::find once a block starts at m: the level of the longest valid block, with
// its index in that level in `at`. Levels 1 .. top - 1 can start at m and fit: k = m - 1 is a
// multiple of their 2^(i+1) steps, which neither the budget nor the table's last - 1 steps
// cut short. The reference tests them in order and stops at the first that fails. A merged
// block's radius is at most its first half's (bla.rs:99-117; checked for every table when it
// is uploaded or built), so the levels that pass are the first ones, and a search finds how
// many with 6 radii in two rounds of loads instead of 8 and more: every third level, then the
// two between (kernel ms: 2880x1620 jittered 1e-300 51.7 -> 48.7, 1920x1080 1e-100 20.0 -> 19.5,
// tiles batch 16.7 -> 16.0). Blocks of the 1e-100 nucleus view are 2^7 steps long in the
// median. WIDE: levels 1-8 in one round of loads, for the stripe variants:
// a frame that ends with its longest samples gains a round's latency, a large one pays the loads
// (Fixed tier at 1e-100, 640x360 10.4 against 10.9 ms, 1600x900 30.3 against 29.2; Scaled tier 640x360
// 8.35 against 8.30).
template <bool EXT, bool WIDE>
__device__ __forceinline__ int block_level(const Params &p, const State<EXT> &s, uint32_t &at) {
  const double d2 = block_d2(s);
  const uint32_t k = s.m - 1u;
  const uint32_t fit = min(s.lim - s.n, p.last - 1u - k);  // >= 2: a block starts here
  const uint32_t top = min(min((uint32_t)__ffs((int)k) - 1u, p.bla_levels), 31u - (uint32_t)__clz((int)fit));
  const auto valid = [&](uint32_t i) {
    return i < top && d2 < __ldg(p.bla_r2 + (p.bla_off[i] + (k >> (i + 1))));
  };
  uint32_t lv = 0;
  if (WIDE) {
    double r[8];
    bool run = true;
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q)
      r[q] = q + 1 < top ? __ldg(p.bla_r2 + (p.bla_off[q + 1] + (k >> (q + 2)))) : -1.0;
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      run = run & (d2 < r[q]);
      lv += run;
    }
    for (uint32_t i = 9; i < top && run; i += 4) {
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q)
        r[q] = i + q < top ? __ldg(p.bla_r2 + (p.bla_off[i + q] + (k >> (i + q + 1)))) : -1.0;
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) {
        run = run & (d2 < r[q]);
        lv += run;
      }
    }
  } else if (p.bla_ordered) {
    double r[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q)
      r[q] = 3 * q + 3 < top ? __ldg(p.bla_r2 + (p.bla_off[3 * q + 3] + (k >> (3 * q + 4)))) : -1.0;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) lv += d2 < r[q] ? 3u : 0u;
    const bool one = valid(lv + 1), two = valid(lv + 2);
    lv += (uint32_t)one + (uint32_t)two;
    while (lv >= 14 && valid(lv + 1)) ++lv;
  } else {
    while (valid(lv + 1)) ++lv;
  }
  at = k >> (lv + 1);
  return (int)lv;
}

// Contraction's own product of a lane's sample, kept in memory: only a sample iterated again
// for it (Magnitude) reads or writes it.
struct ExactProduct {
  volatile double re, im;
  volatile int64_t exp;
  volatile bool started;
  __device__ __forceinline__ void reset() {
    re = 0.0;
    im = 0.0;
    exp = 0;
    started = false;
  }
  __device__ __forceinline__ Contraction get() const { return Contraction{re, im, exp, started}; }
  __device__ __forceinline__ void multiply(double r, double i) {
    Contraction c = get();
    c.multiply(r, i);
    re = c.re;
    im = c.im;
    exp = c.exp;
    started = c.started;
  }
};

// A factor (r, i) that Magnitude::times did not take: of any size, or for Contraction itself
// where the sample is iterated again for it.
template <bool EXT>
__device__ __forceinline__ void contraction_wide(State<EXT> &s, ExactProduct &product, double r, double i) {
  if (s.ct.exact())
    product.multiply(r, i);
  else
    s.ct.times_wide(r, i);
}

// A block's (a, b), one 32-byte load.
struct Block4 {
  double2 a, b;
};

__device__ __forceinline__ Block4 load_block(const double2 *at) {
  Block4 c;
#if defined(__CUDA_ARCH__)
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(c.a.x), "=d"(c.a.y), "=d"(c.b.x), "=d"(c.b.y) : "l"(at));
#else
  c.a = at[0];
  c.b = at[1];
#endif
  return c;
}

// The orbit entry at m: Z_m, and with BLA the squared radius of the first-level block there,
// in one 32-byte load, whose fourth value is unused.
struct Entry {
  double zr, zi, r2a;
};

template <bool L>
__device__ __forceinline__ Entry load_entry(const Params &p, uint32_t m) {
  if (L) {
#if defined(__CUDA_ARCH__)
    Entry e;
    double unused;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(e.zr), "=d"(e.zi), "=d"(e.r2a), "=d"(unused)
        : "l"(p.fused + 2 * m));
    return e;
#else
    const double2 Z = __ldg(p.fused + 2 * m), R = __ldg(p.fused + 2 * m + 1);
    return Entry{Z.x, Z.y, R.x};
#endif
  }
  const double2 Z = __ldg(p.orbit + m);
  return Entry{Z.x, Z.y, -1.0};
}

// The kernels without BLA but with the derivative load the entry after m's an iteration ahead
// (401x227 at 1e-28 0.92 -> 0.81 ms, bounded 320x180 1.98 -> 1.93; without the derivative the
// 480x270 1e-12 frame ran 2.55 -> 2.65, so those load the entry at m behind the delta's update).
template <bool EXT, bool D, bool L>
__device__ __forceinline__ void ahead(const Params &p, State<EXT> &s) {
  if (L || !D) return;
  const Entry at = load_entry<L>(p, min(s.m + 1u, p.last));
  s.Yr = at.zr;
  s.Yi = at.zi;
}

template <bool EXT, bool D, bool L>
__device__ __forceinline__ void enter(const Params &p, State<EXT> &s) {
  if (!L && D) {
    s.Zr = s.Yr;
    s.Zi = s.Yi;
    ahead<EXT, D, L>(p, s);
    return;
  }
  const Entry at = load_entry<L>(p, s.m);
  s.Zr = at.zr;
  s.Zi = at.zi;
  if (L) s.r2a = at.r2a;
}

// A BLA block application (sample.rs:264-315): delta' = A delta + B dc, dz' = A dz + B.
//
// block_quick: the extended tier's application with its four normalisations (before and after,
// of delta and derivative) folded into one of each result. Scaling by a power of two is
// exact and a normalised value does not depend on how it was scaled before, so the steps
// around the block can be left out wherever nothing that counts leaves binary64's normal
// range in this scaling or in the normalised one. block_fits asks that of each result (high
// words, 2^20 a binade): the input normal; the result's parts in [2^-951, 2^950), within
// 2^900 of each other and of the input (its normalised value then lies within 2^900 of 1), so
// that a product too small for binary64 vanishes in the sum and one too large shows in a
// part; dc and the derivative's 1 less than 2^900 times the input, so that neither scaling
// overflows; and b times an error of 2^-1055 in them, whose scaling may underflow, 80
// binades below the result in both scalings. False, with nothing changed, for
// any other block (a zero part among them) and for a mantissa so close to 2 that
// floor(log2) rounds up; apply_block then runs the full steps.
// Before, the normalisations were half of a block's instructions: with the level search's
// conditions folded into one limit, 15.1 -> 13.1 warp instructions per executed operation and
// 28.3 -> 25.4 ms a call on the 1920x1080 frame at a 1e-100 nucleus.
__device__ __forceinline__ uint32_t magnitude_hi(double a) { return (uint32_t)__double2hiint(a) & 0x7fffffffu; }
__device__ __forceinline__ double pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }  // -1022 <= k <= 1023

__device__ __forceinline__ bool block_fits(uint32_t in, uint32_t top, uint32_t low, uint32_t b) {
  constexpr uint32_t ONE = 1023u << 20, FAR = 900u << 20;
  return (in - (40u << 20) < (2000u << 20)) & (low >= (72u << 20)) & (top < (1973u << 20)) & (top - low <= FAR) &
         ((int)(top - in) <= (int)FAR) & ((int)(in - low) <= (int)FAR) & (b + max(in, ONE) <= low + (1998u << 20)) &
         ((top & 0xfffffu) != 0xfffffu);
}

template <bool D>
__device__ __forceinline__ bool block_quick(State<true> &s, double2 A, double2 B) {
  const uint32_t bh = max(magnitude_hi(B.x), magnitude_hi(B.y));
  const double xr = A.x * s.xr - A.y * s.xi + B.x * s.dc_r - B.y * s.dc_i;
  const double xi = A.x * s.xi + A.y * s.xr + B.x * s.dc_i + B.y * s.dc_r;
  const uint32_t xrh = magnitude_hi(xr), xih = magnitude_hi(xi), top = max(xrh, xih);
  const uint32_t xh = max(magnitude_hi(s.xr), magnitude_hi(s.xi));
  bool ok = block_fits(xh, top, min(xrh, xih), bh) & (s.offset_exp - s.delta_exp + 1043 - (int)(xh >> 20) <= 900);
  if (D) {
    const double dr = A.x * s.dr - A.y * s.di + B.x * s.inverse;
    const double di = A.x * s.di + A.y * s.dr + B.y * s.inverse;
    const uint32_t drh = magnitude_hi(dr), dih = magnitude_hi(di), dtop = max(drh, dih);
    const uint32_t dh = max(magnitude_hi(s.dr), magnitude_hi(s.di));
    ok &= block_fits(dh, dtop, min(drh, dih), bh) & (__double2hiint(s.inverse) - (int)dh <= (int)(900u << 20));
    if (!ok) return false;
    const int k = (int)(dtop >> 20) - 1023;
    const double f = pow2(-k);
    s.dr = dr * f;
    s.di = di * f;
    s.derivative_exp += k;
    s.inverse = exp2i(-s.derivative_exp);
  } else if (!ok) {
    return false;
  }
  const int k = min((int)(top >> 20) - 1023, -s.delta_exp);  // the exponent stays at or below 0
  const double f = pow2(-k);
  s.xr = xr * f;
  s.xi = xi * f;
  s.delta_exp += k;
  return true;
}

// The extended tier's application in full, out of line: no block of ordinary views takes it,
// and inlined its four normalisations stretched the loop's code.
struct BlockTerms {
  double xr, xi, dr, di, inverse;
  int64_t derivative_exp;
  int32_t delta_exp;
};

template <bool D>
static __device__ __noinline__ BlockTerms block_full(BlockTerms s, double2 A, double2 B, double ar, double ai,
                                                     int32_t offset_exp) {
  normalise(s.xr, s.xi, s.delta_exp, 0);
  if (D) {
    normalise(s.dr, s.di, s.derivative_exp, INT64_MAX / 4);
    s.inverse = exp2i(-s.derivative_exp);
    const double t = A.x * s.dr - A.y * s.di + B.x * s.inverse;
    s.di = A.x * s.di + A.y * s.dr + B.y * s.inverse;
    s.dr = t;
  }
  const double factor = exp2i(offset_exp - s.delta_exp);
  const double dc_r = ar * factor, dc_i = ai * factor;
  const double t = A.x * s.xr - A.y * s.xi + B.x * dc_r - B.y * dc_i;
  s.xi = A.x * s.xi + A.y * s.xr + B.x * dc_i + B.y * dc_r;
  s.xr = t;
  normalise(s.xr, s.xi, s.delta_exp, 0);
  if (D) {
    normalise(s.dr, s.di, s.derivative_exp, INT64_MAX / 4);
    s.inverse = exp2i(-s.derivative_exp);
  }
  return s;
}

template <bool EXT, bool D>
struct BlockQuick {
  static __device__ __forceinline__ bool run(State<EXT> &, double2, double2) { return false; }
};
template <bool D>
struct BlockQuick<true, D> {
  static __device__ __forceinline__ bool run(State<true> &s, double2 A, double2 B) { return block_quick<D>(s, A, B); }
};

template <bool EXT, bool D>
__device__ __forceinline__ void apply_block(const Params &p, State<EXT> &s, int lv, uint32_t at,
                                            ExactProduct &product) {
  const uint32_t b = p.bla_off[lv] + at;
  const Block4 c = load_block(p.bla_coef + 2 * b);
  const double2 A = c.a, B = c.b;
  const uint32_t len = 2u << lv;
  // the entry where the block ends, in flight together with its coefficients (a third of the
  // chain of loads that a block waits for where few warps hide it)
  s.m += len;
  s.n += len;
  enter<EXT, D, true>(p, s);
  if (__builtin_expect(!s.ct.times(A.x * A.x + A.y * A.y, 0) && s.gate != NO_GATE, 0))
    contraction_wide(s, product, A.x, A.y);
  if (!EXT && s.hold > 0) s.mu.multiply(A.x, A.y);
  if (EXT) {
    if (!BlockQuick<EXT, D>::run(s, A, B)) {
      const BlockTerms t = block_full<D>(BlockTerms{s.xr, s.xi, s.dr, s.di, s.inverse, s.derivative_exp, s.delta_exp}, A,
                                         B, s.ar, s.ai, s.offset_exp);
      s.xr = t.xr;
      s.xi = t.xi;
      s.dr = t.dr;
      s.di = t.di;
      s.inverse = t.inverse;
      s.derivative_exp = t.derivative_exp;
      s.delta_exp = t.delta_exp;
    }
  } else {
    if (D) {
      double t = A.x * s.dr - A.y * s.di + B.x * s.inverse;
      s.di = A.x * s.di + A.y * s.dr + B.y * s.inverse;
      s.dr = t;
      if (p.flags & F_SHIFT) {
        double2 ab = __ldg(p.bla_ab + b);
        s.shift += (ab.x * sqrt(s.xr * s.xr + s.xi * s.xi) + ab.y * s.adc) / sqrt(s.dr * s.dr + s.di * s.di);
      }
    }
    double t = A.x * s.xr - A.y * s.xi + B.x * s.dc_r - B.y * s.dc_i;
    s.xi = A.x * s.xi + A.y * s.xr + B.x * s.dc_i + B.y * s.dc_r;
    s.xr = t;
  }
  if (EXT) {
    s.scale = exp2i(s.delta_exp);
    const double factor = exp2i(s.offset_exp - s.delta_exp);
    s.dc_r = s.ar * factor;
    s.dc_i = s.ai * factor;
  }
  s.blocks += 1;
  s.skipped += len;
}

// One ordinary step (sample.rs:331-380; number.rs:92-124): z = Z[m] + delta is carried
// from the end of the previous iteration in (fr, fi).
// The entry at the new m is loaded into the state between the delta's update, which uses the
// old one, and the derivative's, which covers the load's latency.
template <bool EXT, bool D, bool L, bool B = false>
__device__ __forceinline__ void plain_update(const Params &p, State<EXT> &s) {
  const double *__restrict__ q = p.q;
  const double fr = s.fr, fi = s.fi;
  if (!EXT && s.hold > 0) s.mu.multiply(2.0 * fr, 2.0 * fi);
  if (B) {  // sample.rs:338-350: the radii through this step, from the state before it
    const double qm = __ldg(q + s.m);
    const double af = sqrt(fr * fr + fi * fi) * (1.0 + 4.0 * U) + 1e-150;  // >= |f|
    const double ef = s.e + qm + 2.0 * U * af;                              // >= |z_exact - f|
    const double ad = fabs(s.dr) + fabs(s.di);
    s.ed = (2.0 * (af + ef) * s.ed + 2.0 * ef * ad + 8.0 * U * (2.0 * af * ad + 1.0)) * SAFE;
    const double aw = fabs(s.Zr) + fabs(s.Zi), ax = fabs(s.xr) + fabs(s.xi);
    // the delta step's defect against 2 A delta + delta^2 + dc_exact
    const double rho = 8.0 * U * (2.0 * aw * ax + ax * ax + fabs(s.ar) + fabs(s.ai)) + 2.0 * qm * ax + s.rc;
    const double w = af + qm + 2.0 * U * af;  // >= |A_m + delta|
    s.e = (s.e * (2.0 * w + s.e) + rho) * SAFE;
  }
  const double wr = s.xr, wi = s.xi, zr = s.Zr, zi = s.Zi;
  if (EXT) {  // number.rs:109-124
    s.xr = 2.0 * (zr * wr - zi * wi) + s.scale * (wr * wr - wi * wi) + s.dc_r;
    s.xi = 2.0 * (zr * wi + zi * wr) + s.scale * (2.0 * wr * wi) + s.dc_i;
  } else {  // number.rs:92-107
    s.xr = 2.0 * (zr * wr - zi * wi) + wr * wr - wi * wi + s.dc_r;
    s.xi = 2.0 * (zr * wi + zi * wr + wr * wi) + s.dc_i;
  }
  s.m += 1;
  s.n += 1;
  enter<EXT, D, L>(p, s);
  if (D) {
    double t = 2.0 * (fr * s.dr - fi * s.di) + s.inverse;
    s.di = 2.0 * (fr * s.di + fi * s.dr);
    s.dr = t;
  }
}

// The full sequence after an update (sample.rs:381-575) for iterations in which some event
// may have happened: bailout, nucleus gate, rebase, rescaling, periodicity. z = (fr, fi) with
// |z|^2 = f2 at the entry Z of the new m, the physical delta (pr, pi). Returns true when the
// sample has an outcome (kind 3: none yet, to be iterated again for Contraction's product).
template <bool EXT, bool D, bool L, bool B, bool T>
__device__ __forceinline__ bool sequence(const Params &p, State<EXT> &s, Result &res, double2 Z, double pr, double pi,
                                         double fr, double fi, double f2, ExactProduct &product,
                                         StripeTrace *tr) {
  const bool replaying = T && s.replaying;  // no nucleus gate or periodicity while replaying
  if (__builtin_expect(f2 > p.r2, 0)) {
    res.kind = 0;
    res.n = s.n;
    res.zr = fr;
    res.zi = fi;
    res.dr = s.dr;
    res.di = s.di;
    res.dexp = s.derivative_exp;
    if (B) {  // sample.rs:373-377
      res.ez = s.e + __ldg(p.q + s.m) + 4.0 * U * sqrt(f2);
      res.ed = s.ed;
    }
    if (T) {  // sample.rs:387-403
      if (replaying) {  // the replay reached an escape: the blocks' outcome, this window
        tr->end(s.n, fr, fi);
        res = tr->kept();
        return true;
      }
      StripeSnap sn;
      if (tr->rewind(s.n, p.stripe_window, sn)) {
        tr->keep(res);
        s.replaying = true;
        const uint64_t give_up = (uint64_t)s.n + 64;  // sample.rs:397
        s.limit = (uint32_t)(give_up < p.max_iter ? give_up : p.max_iter);
        s.m = sn.m;
        s.n = sn.n;
        s.xr = sn.xr;
        s.xi = sn.xi;
        s.delta_exp = sn.delta_exp;
        s.scale = sn.scale;
        s.dc_r = sn.dc_r;
        s.dc_i = sn.dc_i;
        const double2 Zm = __ldg(p.orbit + s.m);  // z of the replay's first step
        s.Zr = Zm.x;
        s.Zi = Zm.y;
        ahead<EXT, D, L>(p, s);
        s.fr = EXT ? s.Zr + s.scale * s.xr : s.Zr + s.xr;
        s.fi = EXT ? s.Zi + s.scale * s.xi : s.Zi + s.xi;
        return false;
      }
      tr->end(s.n, fr, fi);
    }
    return true;
  }
  if (!replaying && s.gate != NO_GATE && s.n == s.gate) {
    const int small = s.ct.exact() ? (int)product.get().small() : s.ct.small((int32_t)s.gate - 1);
    if (small < 0) {
      res.kind = 3;
      return true;
    }
    if (small) {
      res.kind = 1;
      res.n = s.n;
      return true;
    }
    s.gate = NO_GATE;
    relimit(p, s);
  }
  double delta2 = pr * pr + pi * pi;
  bool rebase = EXT ? f2 <= delta2 : f2 < delta2;
  // z of the next iteration, Z[m] + delta with the final m and delta: (fr, fi) unless the
  // delta or its scale changes below
  bool moved = false;
  if (__builtin_expect(rebase || s.m == p.last, 0)) {
    moved = true;
    if (B) s.e += __ldg(p.q + s.m) + 4.0 * U * sqrt(f2) + 1e-300;  // sample.rs:419-421: delta := f
    if (EXT) {
      if (f2 > SQUARE_OK) {
        s.xr = fr;
        s.xi = fi;
        s.delta_exp = 0;
      } else {
        Cx3 t = sum2(Cx3{Z.x, Z.y, 0}, Cx3{s.xr, s.xi, s.delta_exp}, s.delta_exp);
        s.xr = t.re;
        s.xi = t.im;
        s.delta_exp = (int32_t)t.e;
      }
      s.scale = exp2i(s.delta_exp);
      s.m = 0;
      s.Zr = p.z0r;
      s.Zi = p.z0i;
      s.r2a = -1.0;  // no block starts at Z_0 (bla.rs:235-236)
      ahead<EXT, D, L>(p, s);
      if (s.scale < 1.0 / 1e270) {  // TINY, sample.rs:17
        s.gate = NO_GATE;
        relimit(p, s);
        if (D) {
          Cx3 v = zero_step_dz(Cx3{s.xr, s.xi, s.delta_exp}, Cx3{s.dr, s.di, s.derivative_exp});
          s.dr = v.re;
          s.di = v.im;
          s.derivative_exp = v.e;
          s.inverse = exp2i(-s.derivative_exp);
        }
        Cx3 w = zero_step(Cx3{s.xr, s.xi, s.delta_exp}, Cx3{s.ar, s.ai, s.offset_exp});
        s.xr = w.re;
        s.xi = w.im;
        s.delta_exp = (int32_t)w.e;
        s.scale = exp2i(s.delta_exp);
        s.m = 1;
        s.n = s.n + 1;
        if (T) tr->start(s.n);  // this step's iterate is not recorded (sample.rs:444-446)
        double2 Z1 = __ldg(p.orbit + 1);
        s.Zr = Z1.x;
        s.Zi = Z1.y;
        if (L) s.r2a = __ldg(p.fused + 3).x;
        ahead<EXT, D, L>(p, s);
      }
      double factor = exp2i(s.offset_exp - s.delta_exp);
      s.dc_r = s.ar * factor;
      s.dc_i = s.ai * factor;
    } else {
      s.xr = fr;
      s.xi = fi;
      s.m = 0;
      s.Zr = p.z0r;
      s.Zi = p.z0i;
      s.r2a = -1.0;
      ahead<EXT, D, L>(p, s);
    }
  } else if (EXT) {
    double magnitude = rmax(fabs(s.xr), fabs(s.xi));
    int32_t k = 0;
    if (magnitude > HI && s.delta_exp < 0)
      k = -s.delta_exp < 32 ? -s.delta_exp : 32;
    else if (magnitude < LO && magnitude != 0.0)
      k = -32;
    if (__builtin_expect(k != 0, 0)) {
      moved = true;
      double factor = exp2i(-k);
      s.xr = s.xr * factor;
      s.xi = s.xi * factor;
      s.delta_exp = s.delta_exp + k;
      s.scale = exp2i(s.delta_exp);
      double f = exp2i(s.offset_exp - s.delta_exp);
      s.dc_r = s.ar * f;
      s.dc_i = s.ai * f;
    }
  }
  if (moved) {  // the next iteration's z (sample.rs:331; number.rs:113 on the extended tier)
    s.fr = EXT ? s.Zr + s.scale * s.xr : s.Zr + s.xr;
    s.fi = EXT ? s.Zi + s.scale * s.xi : s.Zi + s.xi;
  } else {  // the same expressions on the same values
    s.fr = fr;
    s.fi = fi;
  }
  if (replaying) return false;  // sample.rs:470-472: the replay only re-walks iterates
  double check_r = EXT ? pr : s.xr, check_i = EXT ? pi : s.xi;
  bool judge = check_r * check_r + check_i * check_i > RES2 * f2;
  if (EXT) judge = judge && s.returns < MAX_RETURNS;
  if (!judge) {
    if (EXT) {
      if (s.n >= s.chk) {
        save_point(s, fr, fi);
        s.sn = s.n;
        s.chk = s.chk >= 0x80000000u ? 0xffffffffu : s.chk * 2;
        relimit(p, s);
      }
    } else if (s.hold > 0) {
      if (s.n - s.sn >= s.hold) {  // sn <= n while hold > 0
        s.hold = 0;
        s.predicted = false;
        await_save(s);
        relimit(p, s);
      }
    } else if (s.n >= s.chk) {
      await_save(s);
      relimit(p, s);
    }
    return false;
  }
  const double dist = fabs(fr - s.sr) + fabs(fi - s.si), near = near_bound(s);
  if (EXT) {
    if (s.returns < MAX_RETURNS && dist < near) {
      if (contracting(p.orbit, p.last, s.m, check_r, check_i, s.ar * exp2i(s.offset_exp),
                      s.ai * exp2i(s.offset_exp), (uint64_t)(s.n - s.sn))) {
        res.kind = 2;
        return true;
      }
      s.returns += 1;
    }
    if (s.n >= s.chk) {
      save_point(s, fr, fi);
      s.sn = s.n;
      s.chk = s.chk >= 0x80000000u ? 0xffffffffu : s.chk * 2;
      relimit(p, s);
    }
    return false;
  }
  if (dist < near) {
    uint32_t period = s.n - s.sn;
    if (s.hold == period && s.mu.below_one()) {
      double mr, mi;
      s.mu.value(mr, mi);
      double gr = fr - s.sr, gi = fi - s.si;
      double er = mr - 1.0, ei = mi;
      double den = er * er + ei * ei;
      double qpr = s.sr - (gr * er + gi * ei) / den;
      double qpi = s.si - (gi * er - gr * ei) / den;
      double tol = rmin(0.1 * sqrt(den), 1e-2) * s.qstep + 16.0 * U * (fabs(s.sr) + fabs(s.si));
      if (s.predicted && fabs(qpr - s.qr) + fabs(qpi - s.qi) <= tol) {
        res.kind = 1;
        res.n = s.n;
        return true;
      }
      s.qr = qpr;
      s.qi = qpi;
      s.qstep = (fabs(gr) + fabs(gi)) / sqrt(den);
      s.predicted = true;
    } else {
      s.predicted = false;
    }
    s.hold = period;
    save_point(s, fr, fi);
    s.sn = s.n;
    s.pending = false;
    s.mu.reset();
    relimit(p, s);
    return false;
  }
  if (s.hold > 0) {
    if (s.n - s.sn < s.hold) return false;
    s.hold = 0;
    s.predicted = false;
    await_save(s);
  }
  if (s.pending || s.n >= s.chk) {
    uint64_t np = next_pow2((uint64_t)s.n + 1);
    uint32_t np32 = np > 0xffffffffull ? 0xffffffffu : (uint32_t)np;
    s.chk = s.chk > np32 ? s.chk : np32;
    save_point(s, fr, fi);
    s.sn = s.n;
    s.pending = false;
  }
  relimit(p, s);
  return false;
}

// The end of an iteration in which something may have happened: the derivative's rescaling,
// an event of the full sequence (wild: |z|^2 out of the quiet range), a rebase (reb), a
// rescaling of the delta, a due periodicity check, a near return, a block radius below
// binary64's squares, or a contraction product leaving its range. Each part tests its own
// condition exactly. Rebases and checks keep short forms of their own here: run through the
// full sequence they took the 1920x1080 1e-100 frame from 20.4 to 22.7 ms.
template <bool EXT, bool D, bool L, bool B, bool T>
__device__ __forceinline__ bool settle(const Params &p, State<EXT> &s, Result &res, double pr, double pi,
                                       double fr, double fi, double f2, double delta2, bool reb, bool wild,
                                       ExactProduct &product, StripeTrace *tr) {
  if (EXT && D && ((fabs(s.dr) > HI) | (fabs(s.di) > HI))) {  // sample.rs:355-360
    s.dr = s.dr * LO;
    s.di = s.di * LO;
    s.derivative_exp += 32;
    s.inverse = exp2i(-s.derivative_exp);
  }
  const uint32_t end = T ? s.limit : p.max_iter;
  const bool limit = s.n >= s.lim;
  bool event = wild | (B && reb);
  event |= limit && (s.n == s.gate || s.n >= end || (!EXT && s.hold > 0) || (T && s.replaying));
  event |= T && s.n >= end;  // a replay's limit may lie before lim, the block budget's
  // (a sample that has settled on a cycle stays near its save point after the last return that
  // counts: without the test of returns 69% of the iterations of a 2.5-wide scaled-tier view
  // without a table ran the full sequence for nothing, a batch of its frames 286 against 195 ms)
  event |= (reb && !EXT ? f2 : delta2) > RES2 * f2 && (!EXT || s.returns < MAX_RETURNS) &&
           fabs(fr - s.sr) + fabs(fi - s.si) < s.near;
  if (event) {
    if (sequence<EXT, D, L, B, T>(p, s, res, make_double2(s.Zr, s.Zi), pr, pi, fr, fi, f2, product, tr)) return true;
    if (s.n >= end) {  // the loop's end (sample.rs:237)
      if (T && s.replaying) {  // sample.rs:576-579: the replay gave up; from what was recorded
        res = tr->kept();
        tr->end(res.n, res.zr, res.zi);
      } else {
        res.kind = 2;
      }
      return true;
    }
  } else {
    if (reb) {  // sample.rs:418-452 without sum2 or TINY (scale is 1)
      s.xr = fr;
      s.xi = fi;
      s.m = 0;
      s.Zr = p.z0r;
      s.Zi = p.z0i;
      s.r2a = -1.0;  // no block starts at Z_0 (bla.rs:235-236)
      ahead<EXT, D, L>(p, s);
      if (EXT) {
        s.delta_exp = 0;
        s.scale = 1.0;
        const double factor = exp2i(s.offset_exp);
        s.dc_r = s.ar * factor;
        s.dc_i = s.ai * factor;
      }
      s.fr = EXT ? s.Zr + s.scale * s.xr : s.Zr + s.xr;  // sample.rs:331; number.rs:113
      s.fi = EXT ? s.Zi + s.scale * s.xi : s.Zi + s.xi;
    } else if (EXT) {  // sample.rs:453-467
      const double magnitude = rmax(fabs(s.xr), fabs(s.xi));
      int32_t k = 0;
      if (magnitude > HI && s.delta_exp < 0)
        k = -s.delta_exp < 32 ? -s.delta_exp : 32;
      else if (magnitude < LO && magnitude != 0.0)
        k = -32;
      if (k != 0) {
        double factor = exp2i(-k);
        s.xr = s.xr * factor;
        s.xi = s.xi * factor;
        s.delta_exp = s.delta_exp + k;
        s.scale = exp2i(s.delta_exp);
        double f = exp2i(s.offset_exp - s.delta_exp);
        s.dc_r = s.ar * f;
        s.dc_i = s.ai * f;
        s.fr = s.Zr + s.scale * s.xr;
        s.fi = s.Zi + s.scale * s.xi;
      }
    }
    if (limit) {
      if (EXT) {  // sample.rs:488-491 / :571-574
        save_point(s, fr, fi);
        s.sn = s.n;
        s.chk = s.chk >= 0x80000000u ? 0xffffffffu : s.chk * 2;
      } else if ((reb ? f2 : delta2) > RES2 * f2) {  // judged, no near return and hold = 0: sample.rs:560-570
        const uint64_t np = next_pow2((uint64_t)s.n + 1);
        const uint32_t np32 = np > 0xffffffffull ? 0xffffffffu : (uint32_t)np;
        s.chk = s.chk > np32 ? s.chk : np32;
        save_point(s, fr, fi);
        s.sn = s.n;
      } else {
        await_save(s);
      }
      relimit(p, s);
    }
  }
  s.on = L && !(T && s.replaying) && block_starts(s);
  if (!B && !s.on && s.gate != NO_GATE && (event || !s.ct.times(f2, 2))) contraction_wide(s, product, 2.0 * s.fr, 2.0 * s.fi);
  return false;
}

// The rest of the iteration after the update (sample.rs:381-575), and the choice of the next
// operation (s.on: a BLA block), with the entry at the new m in the state. Returns true when the sample has an outcome. T: the Stripe recorder tr records
// the iterate, and an escape whose window misses iterates replays them (sample.rs:369-403).
//
// A common iteration carries z and chooses the next operation; one test sends every other
// to settle(). The test may be true without cause, never false with one. Its parts are
// integer tests on high words where that is enough: binary64 operations issue at half
// rate, and the iteration holds ~45 of them. Issue slots bound the kernel, and before this
// form a warp step spent them on a region per condition (a branch and a reconvergence
// each) and on the contraction's complex product: 21.3 -> 15.1 warp instructions per
// executed operation and 39.2 -> 28.3 ms a call on the 1920x1080 frame at a 1e-100 nucleus
// (extended tier, blocks), 4.4 -> 3.1 ms on the 480x270 1e-12 frame without a table. One lane
// in 8 warp steps is at a rebase, one in 8 at a save point: settle() runs in a third of
// the warp steps for two or three lanes.
template <bool EXT, bool D, bool L, bool B = false, bool T = false>
__device__ __forceinline__ bool post(const Params &p, State<EXT> &s, Result &res, ExactProduct &product,
                                     StripeTrace *tr = nullptr) {
  const double pr = EXT ? s.scale * s.xr : s.xr, pi = EXT ? s.scale * s.xi : s.xi;
  const double fr = s.Zr + pr, fi = s.Zi + pi;
  const double f2 = fr * fr + fi * fi;
  const double delta2 = pr * pr + pi * pi;
  if (T) tr->record(s.n, fr, fi);
  s.fr = fr;  // the next iteration's z, Z[m] + delta with the final m and delta
  s.fi = fi;
  const uint32_t f2_hi = (uint32_t)__double2hiint(f2);
  // |z|^2 outside (1e-290, R^2) on the extended tier (a rebase below takes wide exponents),
  // not below R^2 on the others, NaN included
  constexpr uint32_t floor_hi = EXT ? 0x03b8f2b1u : 0u;  // the first high word above 1e-290's
  const uint32_t top_hi = max((uint32_t)__double2hiint(p.r2), floor_hi);
  const bool wild = f2_hi - floor_hi >= top_hi - floor_hi;
  const bool reb = (EXT ? f2 <= delta2 : f2 < delta2) | (s.m == p.last);
  bool rare = wild | reb | (s.n >= s.lim);
  // a near return counts where |delta|^2 > 1e-24 |z|^2 (1e-24 > 2^-80), which holds for no
  // high words further than 80 binades apart (and after a rebase of the ordinary tiers)
  rare |= (fabs(fr - s.sr) + fabs(fi - s.si) < s.near) & ((uint32_t)__double2hiint(delta2) + (80u << 20) > f2_hi);
  if (EXT) {
    // the delta's mantissa outside [2^-32, 2^32), the derivative's above
    const uint32_t hr = (uint32_t)__double2hiint(s.xr) & 0x7fffffffu, hi = (uint32_t)__double2hiint(s.xi) & 0x7fffffffu;
    rare |= max(hr, hi) - 0x3df00000u >= 0x04000000u;
    if (D) rare |= (fabs(s.dr) > HI) | (fabs(s.di) > HI);
  }
  if (L) {
    // block_starts on |delta|^2: its own (x^2) scale^2 rounds alike unless a product falls
    // below binary64's range, where both lie below any radius^2 of 2^-880 and more
    s.on = (delta2 < s.r2a) & (s.n + 1u < s.lim);
    if (EXT) rare |= (uint32_t)__double2hiint(s.r2a) < ((1023u - 880u) << 20);
    if (T) rare |= s.replaying;
  }
  // the contraction's factor of a plain step from here (a block's: apply_block)
  Magnitude ct = s.ct;
  if (!B) rare |= !ct.times(f2, 2) & !s.on & (s.gate != NO_GATE);
  if (__builtin_expect(rare, 0))
    return settle<EXT, D, L, B, T>(p, s, res, pr, pi, fr, fi, f2, delta2, reb, wild, product, tr);
  if (!B && !s.on) s.ct = ct;
  return false;
}

// One iteration of the while loop of sample.rs:237-575 for one lane without BLA (the
// allocation-free kernel's form). Returns true when the sample has an outcome (written to res).
template <bool EXT, bool D>
__device__ __forceinline__ bool step(const Params &p, State<EXT> &s, Result &res, ExactProduct &product) {
  if (s.n >= p.max_iter) {
    res.kind = 2;
    return true;
  }
  plain_update<EXT, D, false>(p, s);  // m < last here: a sample that reaches the last point rebases to Z_0
  return post<EXT, D, false>(p, s, res, product);
}

// A warp's reserved queue slots [base, end): one atomic on the queue head takes 32
// consecutive slots (one tile), which the warp then hands to its idle lanes in order, so
// one round trip to the head serves a tile instead of each lane as it finishes, and
// neighbouring samples share a warp. Held slots start only as the warp's own lanes finish,
// so over the last slots of the queue (`last`) a warp takes just the slots its idle lanes
// need: there a long sample left waiting behind busy lanes would lengthen the launch's tail.
// Every lane holds the same copy.
struct Reservation {
  unsigned long long base = 0, end = 0;
  bool tail = false;  // within the last slots of the queue
  // Slots for the `need` idle lanes (warp-uniform): false when the queue is spent;
  // otherwise the lanes of need with rank < count take first + rank.
  __device__ __forceinline__ bool take(unsigned long long *queue, unsigned long long total, unsigned long long last,
                                       unsigned need, unsigned lane, unsigned long long &first, unsigned &count) {
    if (base >= end) {
      const unsigned long long grab = tail ? (unsigned long long)__popc(need) : 32ull;
      unsigned long long b = 0;
      if (lane == 0) b = atomicAdd(queue, grab);
      b = __shfl_sync(0xffffffffu, b, 0);
      if (b >= total) return false;
      base = b;
      end = b + grab < total ? b + grab : total;
      tail = total - b <= last;
    }
    const unsigned long long left = end - base, want = (unsigned long long)__popc(need);
    count = (unsigned)(want < left ? want : left);
    first = base;
    base += count;
    return true;
  }
};

// One iteration for the lanes of a warp that hold a sample (`held`, warp-uniform; every lane
// of the warp calls it). A lane whose next operation is a BLA block (s.on), or that has its
// outcome (done), waits until thr lanes wait or no lane steps plainly; the waiting lanes
// then apply their blocks together. The warp runs the block path for many lanes at a time
// instead of for one or two lanes on nearly every iteration, and each lane's own sequence of
// operations is unchanged. Returns the lanes that are done where the warp should look
// (warp-uniform): with BLA only when the waiting lanes have their turn, one vote a step.
template <bool EXT, bool D, bool L, bool B = false, bool T = false>
__device__ __forceinline__ unsigned warp_step(const Params &p, State<EXT> &s, Result &res, bool active, bool &done,
                                              unsigned held, uint32_t thr, ExactProduct &product,
                                              StripeTrace *tr = nullptr) {
  const unsigned FULL = 0xffffffffu;
  if (!L) {
    if (active) {
      plain_update<EXT, D, L, B>(p, s);
      done = post<EXT, D, L, B, T>(p, s, res, product, tr);
    }
    return __ballot_sync(FULL, done);
  }
  const bool wait = s.on | done;  // neither in a lane without a sample
  bool upd = active && !wait;
  if (upd) plain_update<EXT, D, L, B>(p, s);
  const unsigned waiting = __ballot_sync(FULL, wait);
  unsigned ended = 0;
  if ((uint32_t)__popc(waiting) >= thr || waiting == held) {
    ended = __ballot_sync(FULL, done);
    if (wait && !done) {
      uint32_t at;
      const int lv = block_level<EXT, T>(p, s, at);
      if (T)  // sample.rs:267-281: the block start, for a later replay
        tr->snap(StripeSnap{s.m, s.n, s.xr, s.xi, s.delta_exp, s.scale, s.dc_r, s.dc_i}, s.n + (2u << lv));
      apply_block<EXT, D>(p, s, lv, at, product);
      upd = true;
    }
  }
  if (upd) done = post<EXT, D, L, B, T>(p, s, res, product, tr);
  return ended;
}

// The threshold of warp_step: defer of 32 lanes, scaled to the lanes that hold a sample
// (once the queue runs dry lanes go idle, and a fixed threshold would hold every
// waiting lane until the last plain-stepping lane finds a block).
__device__ __forceinline__ uint32_t threshold(unsigned held, uint32_t defer) {
  return max(1u, ((uint32_t)__popc(held) * defer) >> 5);
}

// Series::eval (series.rs:247-271): Horner on x = dc / rho for p = sum b_k x^(k-1) and
// q = p'; delta = x p and, with D, dz/dc = (p + x q) / rho.
template <bool D>
__device__ __forceinline__ void series_start(const Params &p, double ar, double ai, double &xr, double &xi,
                                             double &dr, double &di) {
  const double sc = p.series_inv;
  const double ur = ar * sc, ui = ai * sc;
  double pr = 0.0, pi = 0.0, qr = 0.0, qi = 0.0;
  for (int k = (int)p.series_order - 1; k >= 0; --k) {
    const double2 c = __ldg(p.series_b + k);
    if (D) {
      const double nr = qr * ur - qi * ui + pr, ni = qr * ui + qi * ur + pi;
      qr = nr;
      qi = ni;
    }
    const double nr = pr * ur - pi * ui + c.x, ni = pr * ui + pi * ur + c.y;
    pr = nr;
    pi = ni;
  }
  xr = pr * ur - pi * ui;
  xi = pr * ui + pi * ur;
  if (D) {
    dr = (pr + qr * ur - qi * ui) * sc;
    di = (pi + qr * ui + qi * ur) * sc;
  } else {
    dr = 0.0;
    di = 0.0;
  }
}

// Start sample `slot` of the tile queue (one warp-sized tile per 32 slots, tiles in
// row-major order; 8x4 samples unless tuned). Returns
// false when the slot holds no sample to iterate (outside the grid, masked, or settled
// by the closed-form main-component test, whose result is written here).
template <bool EXT, bool D, bool L, bool B = false>
__device__ __forceinline__ void start_sample(const Params &p, State<EXT> &s, bool use_series, bool keep_counts);

template <bool EXT, bool D, bool L, bool S = false, bool B = false>
__device__ __forceinline__ int init(const Params &p, uint64_t slot, State<EXT> &s, Result &res) {
  uint32_t tile = (uint32_t)(slot >> 5);  // fewer than 2^31 samples
  if (p.tile_order) tile = __ldg(p.tile_order + tile);  // queue position -> row-major tile
  uint32_t w = (uint32_t)slot & 31u;
  const uint32_t ty = tile / p.tiles_x, tx = tile - ty * p.tiles_x;
  uint32_t ii = (tx << p.tile_shift) + (w & ((1u << p.tile_shift) - 1u));
  uint32_t jj = ty * (32u >> p.tile_shift) + (w >> p.tile_shift);
  if (ii >= p.cols || jj >= p.rows) return 0;
  uint32_t i = p.first_col + ii, j = p.first_row + jj;
  uint32_t idx = j * p.nx + i;
  const uint64_t in = (uint64_t)jj * p.in_pitch + ii;  // inputs hold the window only
  if (p.mask && !p.mask[in]) return 0;
  s.idx = idx;
  double ux, uy;
  if (p.offsets) {
    double2 o = p.offsets[in];
    ux = o.x;
    uy = o.y;
  } else {  // view.rs:118-122
    double x = (double)i + 0.5 - p.half_x;
    double y = (double)j + 0.5 - p.half_y;
    ux = p.cosr * x + p.sinr * y;
    uy = p.sinr * x - p.cosr * y;
  }
  if (EXT) {  // grid.rs:709-723
    s.ar = ux * p.h_m;
    s.ai = uy * p.h_m;
    s.offset_exp = (int32_t)p.h_e;
  } else {
    s.ar = ux * p.h;
    s.ai = uy * p.h;
    s.offset_exp = 0;
    if (p.tier == 0 && in_main_components(p.c_re + s.ar, p.c_im + s.ai)) {  // sample.rs:187-189
      res.kind = 1;
      res.n = 0;
      return 2;
    }
  }
  start_sample<EXT, D, L, B>(p, s, S, false);
  return 1;
}

// The iteration state of a sample whose offset (ar, ai, offset_exp) and index are set:
// the ordinary start at Z_0, or the series start when one is given and use_series.
// keep_counts keeps the block counters (a retry from zero after a series start counts
// both runs, grid.rs:623-648).
template <bool EXT, bool D, bool L, bool B>
__device__ __forceinline__ void start_sample(const Params &p, State<EXT> &s, bool use_series, bool keep_counts) {
  s.xr = 0.0;
  s.xi = 0.0;
  s.delta_exp = EXT ? s.offset_exp : 0;
  s.scale = EXT ? exp2i(s.delta_exp) : 1.0;
  s.dc_r = s.ar;
  s.dc_i = s.ai;
  s.dr = 0.0;
  s.di = 0.0;
  s.derivative_exp = 0;
  s.inverse = 1.0;
  s.m = 0;
  s.n = 0;
  s.Zr = p.z0r;
  s.Zi = p.z0i;
  s.r2a = -1.0;
  s.fr = EXT ? p.z0r + s.scale * 0.0 : p.z0r + 0.0;  // z of the first iteration
  s.fi = EXT ? p.z0i + s.scale * 0.0 : p.z0i + 0.0;
  save_point(s, 0.0, 0.0);
  s.chk = 16;
  s.replaying = false;
  s.limit = (uint32_t)p.max_iter;
  s.sn = EXT ? 0 : 8;
  s.returns = 0;
  s.pending = false;
  s.mu.reset();
  s.hold = 0;
  s.predicted = false;
  s.qr = 0.0;
  s.qi = 0.0;
  s.qstep = 0.0;
  s.adc = L ? sqrt(s.ar * s.ar + s.ai * s.ai) : 0.0;
  s.gate = p.nucleus >= 0 ? (uint32_t)p.nucleus + 1u : NO_GATE;
  s.ct.reset((int32_t)p.nucleus);
  s.on = false;
  if (!keep_counts) {
    s.blocks = 0;
    s.skipped = 0;
    s.shift = 0.0;
  }
  if (!EXT && use_series && p.series_n > 0) {
    // sample.rs:191-228 from the series' state: n = m = series_n, the state is the first
    // Brent save (saves resume at the next power of two), no nucleus contraction
    series_start<D>(p, s.ar, s.ai, s.xr, s.xi, s.dr, s.di);
    const uint32_t m = p.series_n;
    s.m = m;
    s.n = m;
    const Entry at = load_entry<L>(p, m);
    s.Zr = at.zr;
    s.Zi = at.zi;
    s.r2a = at.r2a;
    s.fr = s.Zr + s.xr;
    s.fi = s.Zi + s.xi;
    save_point(s, s.Zr + s.xr, s.Zi + s.xi);
    s.sn = m;
    const uint64_t np = next_pow2((uint64_t)m + 1);
    s.chk = np > 16 ? (uint32_t)np : 16u;
    s.gate = NO_GATE;
  }
  ahead<EXT, D, L>(p, s);
  if (B) {  // sample.rs:221-229: radii from zero; a bounded render has no nucleus heuristic
    s.e = 0.0;
    s.ed = 0.0;
    s.rc = 16.0 * U * (fabs(s.ar) + fabs(s.ai)) + 1e-300;
    s.gate = NO_GATE;
  }
  relimit(p, s);
  if (L && !EXT && use_series && p.series_n > 0) s.on = block_starts(s);
}

// Column encoder (store.rs:66-112, Bound absent) and raw state.
// store.rs:115-151 (B): Bounded evidence for an escaped sample with |z| = az, |dz/dc| = ad
// and radii ez, ed: the lower DE factor and the nu bound, or false unless the radii prove
// escape (|z| - ez > 2) and ed < ad / 2. CUDA's log / log1p / exp / exp2 (the columns
// within their ulps of the host's; byte-exact columns come from the raw radii).
__device__ __forceinline__ bool bounds(uint64_t n, double az, double ez, double ad, double ed, double &de_lo,
                                       double &bound) {
  const double lo = az - ez;
  if (!(lo > 2.0 && ed < 0.5 * ad)) return false;
  const double lnz = log(az), llo = log(lo), lhi = log(az + ez);
  const double nu = log1p(-log1p(-ez / az) / llo) / LN_2 + 8.0 * U * ((double)n + 8.0);
  const double g = lhi * exp2(-(double)n);
  de_lo = (lo * llo) / (az * lnz) * ad / (ad + ed) * exp(-g) * (1.0 - 4.0 / (lo * lo)) * (1.0 - 1e-6);
  const double de_hi = ((az + ez) * lhi) / (az * lnz) * ad / (ad - ed) * (1.0 + 1e-6);
  bound = nu * de_hi / de_lo * (1.0 + 1e-6);
  return true;
}

// nu, de and normal of an escaped sample (store.rs:66-112, 145-150; samples.rs:45-48):
// the Bounded evidence's lower DE factor de_lo scales de when bounded.
__device__ __forceinline__ void encode_columns(const Params &p, uint64_t idx, const Result &r, double z2,
                                               double log2z, bool bounded, double de_lo) {
  if (p.nu) p.nu[idx] = (double)r.n + 1.0 - log2(log2z);
  if (p.de) {  // store.rs:145-150
    double lnz = log2z * LN_2;
    double base = 2.0 * sqrt(z2) * lnz / (hypot(r.dr, r.di) * p.px_m);
    int64_t k = -(r.dexp + p.px_e);
    k = k < -4000 ? -4000 : (k > 4000 ? 4000 : k);
    const float d = (float)(base * exp2i(k / 2) * exp2i(k - k / 2));
    p.de[idx] = bounded ? (float)((double)d * de_lo) : d;
  }
  if (p.normal) {  // samples.rs:45-48 through view.rs:132-134
    double re = r.zr * r.dr + r.zi * r.di, im = r.zi * r.dr - r.zr * r.di;
    double x = p.cosr * re + p.sinr * im, y = p.sinr * re - p.cosr * im;
    double t = atan2(y, x) * (65536.0 / TAU);
    p.normal[idx] = (uint16_t)(int64_t)round(t);
  }
}

// A finished sample's outputs. R: only the raw state (status, count, class, z, dz/dc and
// its exponent, every pointer present) is stored here, and encode_kernel computes the
// columns of escaped samples afterwards from it, with all threads of a warp busy instead of
// the one lane that finishes.
template <bool B = false, bool T = false, bool R = false>
__device__ __forceinline__ void put(const Params &p, uint32_t sample, const Result &r, float stripe = 0.0f) {
  const uint32_t j = sample / p.nx, i = sample - j * p.nx;
  const uint64_t idx = (uint64_t)(j - p.first_row) * p.out_pitch + (i - p.first_col);
  if (p.status) p.status[idx] = 1;
  if (T && p.stripe_out) p.stripe_out[idx] = stripe;  // grid.rs:772: 0 unless escaped
  if (p.n_out) p.n_out[idx] = (uint32_t)(r.kind == 2 ? p.max_iter : r.n);
  if (r.kind != 0) {
    if (p.cls) p.cls[idx] = (uint8_t)(r.kind == 2 ? 2 : 1);
    return;
  }
  if (p.z_out) p.z_out[idx] = make_double2(r.zr, r.zi);
  if (p.dz_out) p.dz_out[idx] = make_double2(r.dr, r.di);
  if (p.dexp_out) p.dexp_out[idx] = r.dexp;
  if (R) {
    p.cls[idx] = 0;  // Escaped, heuristic evidence
    return;
  }
  double z2 = r.zr * r.zr + r.zi * r.zi;
  double log2z = 0.5 * log2(z2);
  double de_lo = 0.0, bnd = 0.0;
  bool bounded = false;
  if (B) {  // store.rs:88-106
    bounded = bounds(r.n, sqrt(z2), r.ez, hypot(r.dr, r.di), r.ed, de_lo, bnd);
    if (p.bound_out) p.bound_out[idx] = bounded ? (float)bnd : 0.0f;
    if (p.ez_out) p.ez_out[idx] = r.ez;
    if (p.ed_out) p.ed_out[idx] = r.ed;
  }
  if (p.cls) p.cls[idx] = bounded ? 4 : 0;  // Escaped | Bounded << 2
  encode_columns(p, idx, r, z2, log2z, bounded, de_lo);
}

// The columns of the escaped samples of a window whose persistent kernel stored only their
// raw state (put with R), samples t = start, start + stride, ... of the window: the same
// expressions as put.
__device__ __forceinline__ void encode_window(const Params &p, uint64_t start, uint64_t stride) {
  const uint64_t total = (uint64_t)p.rows * p.cols;
  for (uint64_t t = start; t < total; t += stride) {
    const uint64_t jj = t / p.cols, ii = t - jj * p.cols;
    const uint64_t idx = jj * p.out_pitch + ii;
    if (!p.status[idx] || p.cls[idx] != 0) continue;
    Result r;
    r.kind = 0;
    r.n = p.n_out[idx];
    const double2 z = p.z_out[idx], dz = p.dz_out[idx];
    r.zr = z.x;
    r.zi = z.y;
    r.dr = dz.x;
    r.di = dz.y;
    r.dexp = p.dexp_out[idx];
    const double z2 = r.zr * r.zr + r.zi * r.zi;
    encode_columns(p, idx, r, z2, 0.5 * log2(z2), false, 0.0);
  }
}

// One thread per sample of a frame job's window. (Templates, so that every translation unit
// including this header may hold them.)
template <int V = 0>
__global__ void encode_kernel(Params p) {
  encode_window(p, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, (uint64_t)gridDim.x * blockDim.x);
}

// The same for the jobs of a batch group after its persistent kernel: job blockIdx.y.
template <int V = 0>
__global__ void encode_jobs_kernel(const Params *__restrict__ jobs) {
  const Params &p = jobs[blockIdx.y];
  if (!(p.nu || p.de || p.normal)) return;
  encode_window(p, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, (uint64_t)gridDim.x * blockDim.x);
}

// S: the series-start variant (ordinary tiers, jobs with an admitted series); the others
// compile without the series start and its retry.
// B: the bounded variant (ordinary tiers, derivative on, no BLA or series): error radii,
// Bounded evidence and the Bound column.
// T: the stripe variant: every lane holds a Stripe recorder and writes the Stripe column.
template <bool T>
struct TraceSlot {
  __device__ __forceinline__ StripeTrace *get(const Params &) { return nullptr; }
};
template <>
struct TraceSlot<true> {
  StripeTrace t;
#if !defined(__CUDA_ARCH__)
  double2 units[StripeTrace::UNITS];  // host builds of this header
#endif
  __device__ __forceinline__ StripeTrace *get(const Params &p) {
#if defined(__CUDA_ARCH__)
    const size_t thread = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    t.at = p.stripe_traces + (thread / 32 * StripeTrace::UNITS * 32 + thread % 32 * StripeTrace::GROUP);
#else
    t.at = units;
#endif
    t.begin();
    t.end(0, 0.0, 0.0);
    return &t;
  }
};

// The BLA variants outside B and T store finished samples' raw state only (put's R: every
// raw pointer present) and encode_kernel fills nu, de and normal afterwards (measured on the
// 1920x1080 frame at a 1e-100 nucleus: 40.1 -> 39.2 ms, its fixed-tier variant 35.7 -> 33.8
// ms; without BLA the 480x270 1e-12 frame ran 3% slower, so those variants encode as they
// finish).
template <bool EXT, bool D, bool L, bool S = false, bool B = false, bool T = false>
__global__ void __launch_bounds__(128, Occupancy<EXT>::blocks) perturb_kernel(Params p) {
  const unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt = (1u << lane) - 1u;
  State<EXT> s;
  Result res;
  bool active = false, done = false, exhausted = false;
  Reservation slots;
  ExactProduct product;
  s.on = false;
  TraceSlot<T> trace;
  StripeTrace *tr = trace.get(p);
  uint64_t t0 = p.deadline_ns ? globaltimer() : 0;
  unsigned long long n_samples = 0, iters = 0, blocks = 0, skipped = 0, fallback = 0, closed = 0;
  double shift = 0.0;
  // Series start (grid.rs:623-648): the iterations a sample's count leaves out. The prefix
  // on a first run from the series (> 0); after an unresolved first run retried from zero,
  // prefix - max_iter, so that the first run counts max_iter - prefix.
  int64_t bias = 0;
  uint32_t blocks0 = 0, skipped0 = 0;  // S: the counts and the shift estimate the run from
  double shift0 = 0.0;                 // zero started with
  float stripe = 0.0f;  // T: of a sample that ends escaped
  auto finish = [&](uint32_t idx, const Result &r, uint64_t nblocks, uint64_t nskipped, double sh) {
    put<B, T, L && !B && !T>(p, idx, r, T && r.kind == 0 ? stripe : 0.0f);
    uint64_t spent = (uint64_t)((int64_t)(r.kind == 2 ? p.max_iter : r.n) - bias);
    bias = 0;
    if (L) {
      spent = spent - nskipped + nblocks;
      blocks += nblocks;
      skipped += nskipped;
      bool cf = r.kind == 1 && r.n == 0;
      closed += cf;
      fallback += (nblocks == 0 && !cf);
      shift = fmax(shift, sh);
    }
    iters += spent;
    n_samples += 1;
  };
  // an unresolved series start retries from zero, keeping the nucleus heuristic
  // (grid.rs:637-642); its count and blocks carry over
  auto retry = [&]() {
    bias -= (int64_t)p.max_iter;
    blocks0 = s.blocks;
    skipped0 = s.skipped;
    shift0 = s.shift;
    start_sample<EXT, D, L, B>(p, s, false, true);
    if (T) {  // grid.rs:638
      tr->begin();
      tr->start(s.n);
    }
  };
  const unsigned taking = FULL >> p.idle_lanes;
  slots.tail = p.idle_lanes != 0;
  for (;;) {
    unsigned need = __ballot_sync(FULL, !active) & taking;
    while (need && !exhausted) {
      if (p.deadline_ns) {
        uint64_t now = 0;
        if (lane == 0) now = globaltimer();
        now = __shfl_sync(FULL, now, 0);
        if (now - t0 > p.deadline_ns) {
          exhausted = true;
          if (lane == 0) atomicExch(p.timed_out, 1u);
          break;
        }
      }
      unsigned long long base = 0;
      unsigned take = 0;
      if (!slots.take(p.queue, p.total, p.tail, need, lane, base, take)) {
        exhausted = true;
        break;
      }
      if (!active && ((need >> lane) & 1u)) {
        const unsigned rank = __popc(need & lt);
        const uint64_t slot = base + rank;
        if (rank < take) {
          int got = init<EXT, D, L, S, B>(p, slot, s, res);
          if (got == 1) {
            if (S) {
              bias = p.series_n;
              blocks0 = skipped0 = 0;
              shift0 = 0.0;
            }
            if (T) {  // Job::one (grid.rs:630) and the loop's start (sample.rs:235)
              tr->begin();
              tr->start(s.n);
            }
            if (S && bias > 0 && s.n >= p.max_iter) retry();
            active = s.n < p.max_iter;
            if (!active) {  // no iteration to run
              res.kind = 2;
              finish(s.idx, res, s.blocks, s.skipped, s.shift);
            }
          } else if (got == 2) {
            finish(s.idx, res, 0, 0, 0.0);
          }
        }
      }
      need = __ballot_sync(FULL, !active) & taking;
    }
    // the lanes step until some of them have an outcome
    const unsigned held = __ballot_sync(FULL, active);
    if (!held) break;
    const uint32_t thr = threshold(held, p.defer);
    unsigned ended = 0;
    do {
      ended = warp_step<EXT, D, L, B, T>(p, s, res, active, done, held, thr, product, tr);
    } while (!ended);
    if (T) {  // the windows of the samples that end escaped, one after the other by the whole warp
#if defined(__CUDA_ARCH__)
      __syncwarp();  // their recorders are other lanes' writes
#endif
      unsigned todo = __ballot_sync(FULL, ((ended >> lane) & 1u) && res.kind == 0);
      while (todo) {
        const unsigned l = (unsigned)__ffs((int)todo) - 1u;
        todo &= todo - 1u;
        const float v = tr->average(lane, l, p.r2, p.stripe_window, p.stripe_freq);
        if (l == lane) stripe = v;
      }
    }
    if ((ended >> lane) & 1u) {
      done = false;
      if (S && bias > 0 && res.kind == 2) {
        retry();
      } else if (res.kind == 3) {  // once more, for Contraction's own product
        start_sample<EXT, D, L, B>(p, s, false, S);
        if (S) {
          s.blocks = blocks0;
          s.skipped = skipped0;
          s.shift = shift0;
        }
        if (T) {
          tr->begin();
          tr->start(s.n);
        }
        s.ct.take_exact();
        product.reset();
      } else {
        finish(s.idx, res, s.blocks, s.skipped, s.shift);
        active = false;
        s.on = false;
      }
    }
  }
  // warp reduction of the counters, one atomic per warp
  for (int o = 16; o > 0; o >>= 1) {
    n_samples += __shfl_down_sync(FULL, n_samples, o);
    iters += __shfl_down_sync(FULL, iters, o);
    blocks += __shfl_down_sync(FULL, blocks, o);
    skipped += __shfl_down_sync(FULL, skipped, o);
    fallback += __shfl_down_sync(FULL, fallback, o);
    closed += __shfl_down_sync(FULL, closed, o);
    shift = fmax(shift, __shfl_down_sync(FULL, shift, o));
  }
  if (lane == 0) {
    atomicAdd(&p.counters->samples, n_samples);
    atomicAdd(&p.counters->iterations, iters);
    if (L) {
      atomicAdd(&p.counters->blocks, blocks);
      atomicAdd(&p.counters->skipped, skipped);
      atomicAdd(&p.counters->fallback, fallback);
      atomicAdd(&p.counters->closed, closed);
      if (shift > 0.0 && !isnan(shift)) atomicMax(&p.counters->shift_bits, (unsigned long long)__double_as_longlong(shift));
    }
  }
}

}  // namespace fdk

namespace fdk {

// Batches: many jobs (frames, tiles, locations) in one persistent launch. Job j owns
// queue slots [starts[j], starts[j+1]); a lane takes a slot, finds its job by binary
// search, and runs the same init/step/put as the single-job kernel on that job's Params
// (read from global memory), so results equal fdc_render's bit for bit. Counters are
// kept per job, flushed with atomics when a lane moves to another job.
__device__ __forceinline__ uint32_t job_of(const unsigned long long *__restrict__ starts, uint32_t njobs,
                                           unsigned long long slot) {
  uint32_t lo = 0, hi = njobs;  // starts[lo] <= slot < starts[hi]
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (__ldg(starts + mid) <= slot) lo = mid;
    else hi = mid;
  }
  return lo;
}

struct LaneCounters {
  unsigned long long samples, iterations, blocks, skipped, fallback, closed;
  __device__ __forceinline__ void clear() { samples = iterations = blocks = skipped = fallback = closed = 0; }
  __device__ __forceinline__ void flush(Counters *c) {
    if (samples) atomicAdd(&c->samples, samples);
    if (iterations) atomicAdd(&c->iterations, iterations);
    if (blocks) atomicAdd(&c->blocks, blocks);
    if (skipped) atomicAdd(&c->skipped, skipped);
    if (fallback) atomicAdd(&c->fallback, fallback);
    if (closed) atomicAdd(&c->closed, closed);
    clear();
  }
};

template <bool EXT, bool D, bool L>
__global__ void __launch_bounds__(128, Occupancy<EXT>::blocks)
    perturb_batch_kernel(const Params *__restrict__ jobs, const unsigned long long *__restrict__ starts,
                         uint32_t njobs, unsigned long long total, unsigned long long *queue, Counters *per_job,
                         uint32_t defer) {
  const unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt = (1u << lane) - 1u;
  State<EXT> s;
  Result res;
  bool active = false, done = false, exhausted = false;
  uint32_t job = 0, counted = 0xffffffffu;
  Reservation slots;
  ExactProduct product;
  s.on = false;
  // over the last three waves of the grid, or the last eighth of the queue, a warp reserves
  // no slots ahead (as fdc_render's Params.tail)
  const unsigned long long waves = 3ull * gridDim.x * blockDim.x, last = waves > total / 8 ? waves : total / 8;
  LaneCounters lc;
  lc.clear();
  // the BLA variants store a finished sample's raw state; encode_jobs_kernel computes the
  // columns afterwards (every raw pointer present: fdc_batch_create provides scratch)
  auto finish = [&](const Params &p, uint32_t idx, const Result &r, uint64_t nblocks, uint64_t nskipped) {
    put<false, false, L>(p, idx, r);
    if (counted != job) {
      if (counted != 0xffffffffu) lc.flush(per_job + counted);
      counted = job;
    }
    uint64_t spent = r.kind == 2 ? p.max_iter : r.n;
    if (L) {
      spent = spent - nskipped + nblocks;
      lc.blocks += nblocks;
      lc.skipped += nskipped;
      bool cf = r.kind == 1 && r.n == 0;
      lc.closed += cf;
      lc.fallback += (nblocks == 0 && !cf);
    }
    lc.iterations += spent;
    lc.samples += 1;
  };
  for (;;) {
    unsigned need = __ballot_sync(FULL, !active);
    while (need && !exhausted) {
      unsigned long long base = 0;
      unsigned take = 0;
      if (!slots.take(queue, total, last, need, lane, base, take)) {
        exhausted = true;
        break;
      }
      if (!active) {
        const unsigned rank = __popc(need & lt);
        const unsigned long long slot = base + rank;
        if (rank < take) {
          job = job_of(starts, njobs, slot);
          const Params &p = jobs[job];
          int got = init<EXT, D, L>(p, slot - __ldg(starts + job), s, res);
          active = got == 1 && s.n < p.max_iter;
          if (got != 0 && !active) {  // settled, or no iteration to run
            if (got == 1) res.kind = 2;
            finish(p, s.idx, res, 0, 0);
          }
        }
      }
      need = __ballot_sync(FULL, !active);
    }
    const unsigned held = __ballot_sync(FULL, active);
    if (!held) break;
    const uint32_t thr = threshold(held, defer);
    const Params &p = jobs[job];
    unsigned ended = 0;
    do {
      ended = warp_step<EXT, D, L>(p, s, res, active, done, held, thr, product);
    } while (!ended);
    if ((ended >> lane) & 1u) {
      done = false;
      if (res.kind == 3) {  // once more, for Contraction's own product
        start_sample<EXT, D, L, false>(p, s, false, false);
        s.ct.take_exact();
        product.reset();
      } else {
        finish(p, s.idx, res, s.blocks, s.skipped);
        active = false;
        s.on = false;
      }
    }
  }
  if (counted != 0xffffffffu) lc.flush(per_job + counted);
}

}  // namespace fdk
