"""The calls whose speed matters to users of this package, as measurable cases.

Each case is one call (or one batch replay) through the package's public entry points:
render_with / render_bla (a frame from its orbit to host columns), Device.render_job (a
frame over an orbit that stays uploaded, as a viewer or a film renders) and
Device.batch / Batch.run (many frames or tiles in one replay). The views are the
benchmark configurations' (fractodactyl_b200.locations) at their own or smaller grids; the
seed turns and slightly rescales the view, so every seed iterates other samples.

listed() gives the fixed cases, draw() one more of the same ranges, prepare() what a program
holds before the call, run() one pass, work() the bytes and FP64 operations the pass cannot
do without, exact() the values by a plain NumPy iteration where that is quick.
"""
import ctypes
import dataclasses
import decimal
import functools
import math
import random

import numpy as np
import torch

import fractodactyl_b200 as fd
from fractodactyl_b200 import _lib
from fractodactyl_b200 import route
from fractodactyl_b200.locations import cached, jitter_offsets

DE = "nu,de,normal"

# (name, centre, log10 of the width at seed-independent scale, executed operations per sample
# with / without BLA): plain steps plus applied blocks, from the render counters, rounded.
VIEWS = {
    "valley": (lambda: ("-0.7453", "0.1127"), -2.2, 140, 140),
    "seahorse": (lambda: ("-0.7436438870371587", "0.1318259042053120"), -12.0, 1600, 1600),
    "c2": (lambda: _centre("c2", 0), -100.0, 700, 950),
    "c3": (lambda: _centre("c3", 0), -300.0, 680, 950),
    "c4": (lambda: _centre("c4", 0), -500.0, 575, 950),
    "c5a": (lambda: _centre("c5", 0), -211.0, 650, 950),
    "c5b": (lambda: _centre("c5", 1), -208.0, 4900, 950),
    "c5c": (lambda: _centre("c5", 2), None, 760, 950),
    "c5d": (lambda: _centre("c5", 3), None, 720, 950),
}
TILE_VIEWS = ("c5a", "c5b", "c5c", "c5d")


def _centre(name, k):
    d = cached(name)[k]
    return d["re"], d["im"]


def _log10_width(view):
    w = VIEWS[view][1]
    return w if w is not None else cached("c5")[TILE_VIEWS.index(view)]["log10_width"]


def _case(name, kind, view, nx, ny, max_iter, **kw):
    c = dict(name=name, kind=kind, view=view, nx=nx, ny=ny, ss=1, max_iter=max_iter, log10_width=_log10_width(view),
             escape_radius=1e10, columns=DE, bla=False, tier="auto", f32=False, frames=1)
    c.update(kw)
    return c


def listed():
    return [
        # a thumbnail of a shallow view, from a supplied orbit to host columns: launch and copy latency
        _case("thumb-64x36", "call", "valley", 64, 36, 2000),
        # an explorer's preview of a deep view, odd grid: orbit upload, table build, render, host columns
        _case("deep-preview-161x91", "call_bla", "c5a", 161, 91, 200_000, bla=True),
        # an ordinary shallow frame, counts and smooth iteration only (the first benchmark configuration)
        _case("frame-480x270-1e-12", "job", "seahorse", 480, 270, 20_000, escape_radius=256.0, columns="nu"),
        # a mid-depth frame without a table (film keyframes whose table has no level), odd grid
        _case("frame-401x227-1e-28-plain", "job", "c2", 401, 227, 50_000, log10_width=-28.0),
        # an ordinary deep frame on the Fixed tier with blocks
        _case("frame-1280x720-1e-100", "job", "c2", 1280, 720, 1_000_000, bla=True, tier="fixed"),
        # the headline frame: Scaled tier, blocks, every column
        _case("frame-1920x1080-1e-100", "job", "c2", 1920, 1080, 1_000_000, bla=True, tier="scaled"),
        # the precision form of the same view, columns kept on the device
        _case("f32-960x540-1e-100", "job_device", "c2", 960, 540, 1_000_000, bla=True, tier="scaled", f32=True),
        # the largest: jittered supersampling of a 1e-300 view, 2 x 2 samples a pixel
        _case("jitter-2880x1620-1e-300", "job_jitter", "c3", 2880, 1620, 1_000_000, ss=2, bla=True, tier="scaled"),
        # a zoom film's frames over one orbit in one batch replay
        _case("film-8x640x360", "film", "c4", 640, 360, 1_000_000, bla=True, frames=8),
        # tiles of several locations in one batch replay
        _case("tiles-4x512x256", "tiles", "c5a", 512, 256, 1_000_000, bla=True, frames=4),
        # certified escapes: the Bound column
        _case("bounded-320x180", "job_bounded", "seahorse", 320, 180, 5000, log10_width=-9.0),
        # the styling column over a deep frame with blocks
        _case("stripe-640x360-1e-100", "job_stripe", "c2", 640, 360, 1_000_000, bla=True, tier="fixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["call", "call_bla", "job", "job", "job_bla", "job_bla", "job_bla", "job_device", "job_jitter",
                       "film", "tiles", "job_bounded", "job_stripe"])
    nx, ny = _log_int(rng, 48, 1920), _log_int(rng, 27, 1080)
    columns = rng.choice([DE, DE, "nu", "nu,de"])
    if kind == "call":
        c = _case("", kind, rng.choice(["valley", "seahorse"]), min(nx, 400), min(ny, 300), rng.randrange(1500, 3000))
        c["log10_width"] = rng.uniform(-8.0, -2.2) if c["view"] == "seahorse" else rng.uniform(-3.0, -1.5)
    elif kind == "call_bla":
        c = _case("", kind, rng.choice(["c2", "c5a", "c5b"]), min(nx, 640), min(ny, 400), rng.randrange(50_000, 300_000),
                  bla=True)
    elif kind == "job":  # no table: F64, Fixed and Scaled tiers
        view, w, tier = rng.choice([("seahorse", rng.uniform(-12.0, -6.0), "auto"), ("c2", rng.uniform(-60.0, -16.0), "auto"),
                                    ("c2", rng.uniform(-60.0, -16.0), "scaled")])
        c = _case("", kind, view, min(nx, 480), min(ny, 270), rng.randrange(12_000, 20_000), tier=tier)
        c["log10_width"] = w
    elif kind == "job_bla":
        view, tier = rng.choice([("c2", "fixed"), ("c2", "scaled"), ("c3", "scaled"), ("c5b", "fixed"), ("c5a", "scaled")])
        c = _case("", "job", view, nx, ny, rng.randrange(200_000, 1_000_000), bla=True, tier=tier)
        if view == "c2":
            c["log10_width"] = rng.uniform(-100.0, -40.0)
    elif kind == "job_device":
        c = _case("", kind, "c2", min(nx, 960), min(ny, 540), rng.randrange(200_000, 1_000_000), bla=True,
                  tier=rng.choice(["fixed", "scaled"]), f32=rng.random() < 0.5)
    elif kind == "job_jitter":
        c = _case("", kind, rng.choice(["c2", "c3"]), 2 * (nx // 2), 2 * (ny // 2), 500_000, ss=2, bla=True, tier="scaled")
    elif kind == "film":
        c = _case("", kind, "c4", min(nx, 640), min(ny, 360), rng.randrange(200_000, 1_000_000), bla=True,
                  frames=rng.randrange(2, 9))
    elif kind == "tiles":
        s = rng.choice([64, 100, 128])
        c = _case("", kind, "c5a", 4 * s, 2 * s, rng.randrange(200_000, 1_000_000), bla=True, frames=rng.randrange(1, 5))
    elif kind == "job_bounded":
        c = _case("", kind, "seahorse", min(nx, 320), min(ny, 180), rng.randrange(3000, 5000))
        c["log10_width"] = rng.uniform(-9.0, -6.0)
    else:
        c = _case("", kind, "c2", min(nx, 640), min(ny, 360), rng.randrange(200_000, 1_000_000), bla=True,
                  tier=rng.choice(["fixed", "scaled"]))
    if kind not in ("job_bounded", "job_stripe"):
        c["columns"] = columns
    del c["name"]
    return c


@functools.lru_cache(maxsize=None)
def _orbit(re, im, bits, max_iter):
    return fd.Reference.from_fixed(re, im, bits, max_iter)


def _decimal(log10_value):
    e = math.floor(log10_value)
    return "%.9fe%d" % (10 ** (log10_value - e), e)


def _view(case, seed, log10_width=None):
    """The case's view turned by a seeded angle and rescaled by up to 5%."""
    rng = random.Random("%s %d" % (case["view"], seed))
    re, im = VIEWS[case["view"]][0]()
    w = (case["log10_width"] if log10_width is None else log10_width) + math.log10(rng.uniform(0.95, 1.05))
    width = _decimal(w)
    if w > -20.0:  # a binary fraction of few bits, so that exact() reads the same width
        m, e = math.frexp(10.0 ** w)
        width = "%.80e" % decimal.Decimal(math.ldexp(round(m * 2.0 ** 24), e - 24))
    return fd.View(re, im, width, rng.uniform(0.0, 2.0 * math.pi))


def _params(case, **kw):
    p = fd.Params(case["nx"], case["ny"], ss=case["ss"], max_iter=case["max_iter"], escape_radius=case["escape_radius"],
                  columns=tuple(case["columns"].split(",")), tier=None if case["tier"] == "auto" else case["tier"])
    return dataclasses.replace(p, **kw)


def _reference(view, p, bits=None):
    """The orbit of a view: binary64 on the F64 tier, else at its bits rounded up to a limb."""
    plane = fd.Plane.new(view, p.nx, p.ny)
    tier = plane.tier if p.tier is None else route.TIERS[p.tier]
    if tier == 0 and bits is None:
        return plane, tier, fd.Reference.new(plane.c_re, plane.c_im, p.max_iter, p.escape_radius)
    bits = bits or -(-plane.bits // 64) * 64
    r = _orbit(view.center_re, view.center_im, bits, p.max_iter)
    return plane, tier, fd.Reference(r.re, r.im, bits)


class Held:
    """What a program keeps between calls: uploaded orbits, a batch, its columns."""

    def __init__(self, case):
        self.case, self.dev, self.orbits, self.batch, self.keep = case, fd.device(0), [], None, []

    def upload(self, view, p, r, tier, bla):
        h = self.dev.upload(r)
        self.orbits.append(h)
        if not bla:
            return h, False
        dc, e = fd.bla_dc_bound(view, dataclasses.replace(p, tier={0: "f64", 1: "fixed", 2: "scaled"}[tier]))
        return h, self.dev.build_bla(h, fd.EPS, dc, e) > 0

    def __del__(self):
        try:
            if self.batch is not None:
                self.batch.free()
            for h in self.orbits:
                self.dev.free(h)
        except Exception:  # the interpreter is going down
            pass


def _job(s, view, p, plane, tier, r, bla, f32=False):
    h, levels = s.upload(view, p, r, tier, bla)
    flags = (_lib.DERIVATIVE if p.needs_derivative() else 0) | (_lib.BLA if levels else 0) | (_lib.F32 if f32 else 0)
    return route.make_job(plane, tier, p, h, r.nucleus_period(), flags)


def prepare(case, seed):
    kind = case["kind"]
    s = Held(case)
    if kind in ("call", "call_bla"):
        s.view, s.p = _view(case, seed), _params(case)
        _, _, s.r = _reference(s.view, s.p)
        return s
    if kind in ("film", "tiles"):
        jobs, groups = [], []
        n = case["frames"]
        if kind == "film":  # widths from 1e-10 down to the centre's own, one orbit at the deepest frame's bits
            logs = [-10.0 + (case["log10_width"] + 10.0) * k / max(1, n - 1) for k in range(n)]
            views = [_view(case, seed, w) for w in logs]
            ps = [_params(case) for _ in views]
            bits = -(-max(fd.Plane.new(v, p.nx, p.ny).bits for v, p in zip(views, ps)) // 64) * 64
        else:
            names = TILE_VIEWS[:n]
            views = [_view(dict(case, view=v, log10_width=_log10_width(v)), seed) for v in names]
            ps, bits = [_params(case) for _ in views], None
        for k, (v, p) in enumerate(zip(views, ps)):
            plane, tier, r = _reference(v, p, bits)
            j = _job(s, v, p, plane, max(tier, 1), r, True)
            if kind == "film":
                jobs.append(j)
                groups.append(k)
                continue
            tw, th = p.nx // 4, p.ny // 2
            for y in range(0, p.ny, th):
                for x in range(0, p.nx, tw):
                    t = _lib.Job()
                    ctypes.memmove(ctypes.byref(t), ctypes.byref(j), ctypes.sizeof(j))
                    t.first_col, t.cols, t.first_row, t.rows = x, min(tw, p.nx - x), y, min(th, p.ny - y)
                    jobs.append(t)
                    groups.append(k)
        s.batch = s.dev.batch(jobs, columns=tuple(case["columns"].split(",")), groups=groups)
        return s
    view, p = _view(case, seed), _params(case)
    plane, tier, r = _reference(view, p)
    if kind == "job_jitter":
        # the jitter reaches half a sample beyond the grid: a table for a grid 2 samples larger each way
        grown = _params(case, nx=p.nx + 4, ny=p.ny + 4)
        h, _ = s.upload(dataclasses.replace(view, width=_grown_width(plane, grown)), grown, r, tier, True)
        s.offsets = jitter_offsets(plane, p.nx, p.ny, seed)
        s.job = route.make_job(plane, tier, p, h, r.nucleus_period(),
                               (_lib.DERIVATIVE if p.needs_derivative() else 0) | _lib.BLA)
        s.job.offsets = s.offsets.ctypes.data
    else:
        s.job = _job(s, view, p, plane, tier, r, case["bla"], case["f32"])
    if kind == "job_bounded":
        s.dev.upload_error_radius(s.job.orbit, r.error_radius(None if tier == 0 else r.bits, plane.c_re, plane.c_im))
    n = p.nx * p.ny
    cols = {"cls": torch.uint8, "status": torch.uint8, "n": torch.int32, "nu": torch.float64, "de": torch.float32,
            "normal": torch.int16}
    want = ["cls", "status", "n"] + [c for c in ("nu", "de", "normal") if c in p.columns]
    if kind == "job_device":
        s.job.flags |= _lib.DEVICE_OUT
        s.columns = {k: torch.zeros(n, dtype=cols[k], device="cuda") for k in want}
        s.pointers = {k: t.data_ptr() for k, t in s.columns.items()}
    else:
        host = {"cls": np.uint8, "status": np.uint8, "n": np.uint32, "nu": np.float64, "de": np.float32,
                "normal": np.uint16}
        s.host = {k: np.zeros(n, host[k]) for k in want}
    return s


def _grown_width(plane, grown):
    """The decimal width at which a grid of grown.nx samples has the plane's spacing, 1% over."""
    return _decimal(math.log10(plane.h_m) + plane.h_e * math.log10(2.0) + math.log10(grown.nx * 1.01))


def _frame(samples):
    return {k: v for k, v in (("cls", samples.cls), ("n", samples.n), ("nu", samples.nu), ("de", samples.de),
                              ("normal", samples.normal)) if v is not None}


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "call":
        return _frame(fd.render_with(s.view, s.p, (s.r, s.r.bits), dev=s.dev)[1])
    if kind == "call_bla":
        return _frame(fd.render_bla(s.view, s.p, (s.r, s.r.bits), device_table=True, dev=s.dev)[1])
    if kind in ("film", "tiles"):
        s.batch.run()
        return s.batch.cols
    if kind == "job_device":
        s.dev.render_job(s.job, device_out=s.pointers)
        return s.columns
    if kind == "job_bounded":
        return s.dev.render_job(s.job, host_out=s.host, bounded=True)[0]
    if kind == "job_stripe":
        return s.dev.render_job(s.job, host_out=s.host, stripe=(16, 5.0))[0]
    return s.dev.render_job(s.job, host_out=s.host)[0]


def work(case):
    """Outputs written and orbit points read once; FP64 operations of the executed steps
    (40 a plain ordinary-tier step with the derivative, 47 floatexp, 31 / 38 without)."""
    n = case["nx"] * case["ny"] * case["frames"]
    cols = case["columns"].split(",")
    width = 1 + 1 + 4 + 8 * ("nu" in cols) + 4 * ("de" in cols) + 2 * ("normal" in cols)
    width += 4 * (case["kind"] == "job_stripe") + 20 * (case["kind"] == "job_bounded") + 16 * (case["kind"] == "job_jitter")
    views = TILE_VIEWS[:case["frames"]] if case["kind"] == "tiles" else (case["view"],)
    ops = sum(VIEWS[v][2 if case["bla"] else 3] for v in views) / len(views)
    ops = min(ops, case["max_iter"])
    d = "de" in cols or "normal" in cols
    step = (47 if d else 38) if case["tier"] == "scaled" or case["log10_width"] < -270 else (40 if d else 31)
    return {"bytes": float(n * width + 16 * min(case["max_iter"], 1 << 20)), "flops": float(n) * ops * step}


def exact(case, seed):
    """A plain NumPy iteration in binary64 of small F64-tier frames without blocks (the
    perturbation recurrence with rebasing; chaotic counts have no other 64-bit value):
    nu and de of escaped samples. The counts and classes are whole numbers."""
    if case["kind"] != "call" or case["log10_width"] < -9.0 or case["nx"] * case["ny"] > 40_000:
        return None
    view, nx, ny, cap = _view(case, seed), case["nx"], case["ny"], case["max_iter"]
    cr, ci, h = float(view.center_re), float(view.center_im), float(view.width) / nx
    co, si = math.cos(view.rotation), math.sin(view.rotation)
    zr, zi, Z = 0.0, 0.0, [(0.0, 0.0)]
    r2 = case["escape_radius"] ** 2
    while len(Z) < cap + 1 and zr * zr + zi * zi <= r2:
        zr, zi = zr * zr - zi * zi + cr, 2.0 * zr * zi + ci
        Z.append((zr, zi))
    Z = np.array(Z)
    last = len(Z) - 1
    x = np.arange(nx)[None, :] + 0.5 - nx / 2.0
    y = np.arange(ny)[:, None] + 0.5 - ny / 2.0
    a, b = ((co * x + si * y) * h).ravel(), ((si * x - co * y) * h).ravel()
    pr, pi = cr + a, ci + b
    q = (pr - 0.25) ** 2 + pi * pi
    live = np.flatnonzero(~((q * (q + (pr - 0.25)) <= 0.25 * pi * pi) | ((pr + 1.0) ** 2 + pi * pi <= 0.0625)))
    n_all = nx * ny
    nu, de = np.zeros(n_all), np.zeros(n_all)
    a, b = a[live], b[live]
    dr, di, ur, ui = (np.zeros(len(live)) for _ in range(4))
    m = np.zeros(len(live), np.int64)
    fr, fi = np.zeros(len(live)), np.zeros(len(live))
    with np.errstate(all="ignore"):
        for n in range(1, cap + 1):
            wr, wi = Z[m, 0], Z[m, 1]
            ur, ui = 2.0 * (fr * ur - fi * ui) + 1.0, 2.0 * (fr * ui + fi * ur)
            dr, di = 2.0 * (wr * dr - wi * di) + dr * dr - di * di + a, 2.0 * (wr * di + wi * dr + dr * di) + b
            m = m + 1
            fr, fi = Z[m, 0] + dr, Z[m, 1] + di
            f2 = fr * fr + fi * fi
            out = f2 > r2
            if out.any():
                k = live[out]
                l2 = 0.5 * np.log2(f2[out])
                nu[k] = n + 1.0 - np.log2(l2)
                de[k] = 2.0 * np.sqrt(f2[out]) * l2 * math.log(2.0) / (np.hypot(ur[out], ui[out]) * h * case["ss"])
                keep = ~out
                live, a, b, dr, di, ur, ui, m, fr, fi, f2 = (v[keep] for v in (live, a, b, dr, di, ur, ui, m, fr, fi, f2))
            back = (f2 < dr * dr + di * di) | (m == last)
            dr, di, m = np.where(back, fr, dr), np.where(back, fi, di), np.where(back, 0, m)
            if not len(live):
                break
    cols = case["columns"].split(",")
    got = {"cls": None, "n": None}
    for name, v in (("nu", nu), ("de", de), ("normal", None)):
        if name in cols:
            got[name] = v
    return got
