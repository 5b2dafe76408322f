"""The shift estimate (fdc_counters.shift, BlaStats.shift_px) of a series render with a table
whose samples are iterated a second time for the nucleus gate's own product: what the aborted
run added is not counted. The kernel's own source on the host, against the oracle, on the
2,535-period series frame: every sample through the second run (FDK_CONTRACTION_AGAIN), the
ordinary build, and a sample that the ordinary build sends there by itself."""
import ctypes as C
import json
import os
import subprocess

import numpy as np
import pytest

import fdref
import fractodactyl_b200 as fd

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
FRAME = json.load(open(os.path.join(HERE, "golden", "kats.json")))["series_frames"][-1]
EPS = 2.0 ** -26  # blocks enough for the estimate to differ from zero


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    out = {}
    for which, define in (("modulus", []), ("again", ["-DFDK_CONTRACTION_AGAIN=true"])):
        so = str(tmp_path_factory.mktemp("emu") / f"libshift_{which}.so")
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas",
                        *define, "-I", os.path.join(HERE, "emu"), "-I",
                        os.path.join(ROOT, "fractodactyl_b200", "csrc"), os.path.join(HERE, "emu", "emu_shift.cpp"),
                        "-o", so], check=True)
        L = C.CDLL(so)
        P, D, U32, U64, I32, I64 = C.c_void_p, C.c_double, C.c_uint32, C.c_uint64, C.c_int32, C.c_int64
        L.emu_render_shift.restype = C.c_int
        L.emu_render_shift.argtypes = [P, P, U64, P, P, U32, P, U32, U32, D, I32, U32, U32, D, D, D, I64, U32, D, I64, P, P,
                                       P, P, P, P, P]
        out[which] = L
    return out


@pytest.fixture(scope="module")
def frame():
    view3, nx, ny, it = (FRAME["re"], FRAME["im"], FRAME["width"]), 33, 19, 10_000
    v, p = fd.View(*view3), fd.Params(nx, ny, max_iter=it, columns=("nu", "de"))
    plane, tier = fd.route._setup(v, p)
    r, bits = fd.reference(v, p)
    rho, e = fd.bla_dc_bound(v, p)
    assert e == 0 and tier in (0, 1)
    series = fd.Series.build(r, rho, float(FRAME["width"]) / nx, it)
    table = fd.Bla.build_scaled(r, EPS, rho, 0)
    assert series.n > 0 and table.levels > 0
    ref = fdref.Ref.arrays(r.re, r.im, bits)
    job = fdref.make_job(*view3, nx, ny, it, escape_radius=p.escape_radius, columns=fdref.COL_NU | fdref.COL_DE, tier=tier)
    return dict(plane=plane, tier=tier, p=p, r=r, series=series, table=table, ref=ref, job=job, h=plane.h(),
                o_series=fdref.Series(ref, rho, float(FRAME["width"]) / nx, it), o_bla=fdref.Bla(ref, EPS, rho, 0))


def _emulate(L, f, nx, ny, mask=None, offsets=None, series=True):
    p, plane, n = f["p"], f["plane"], nx * ny
    re, im = np.ascontiguousarray(f["r"].re), np.ascontiguousarray(f["r"].im)
    blocks = np.ascontiguousarray(f["table"].blocks)
    offs = np.ascontiguousarray(f["table"].level_offsets, dtype=np.uint64)
    b = np.ascontiguousarray(f["series"].b, dtype=np.float64)
    out = dict(cls=np.zeros(n, np.uint8), n=np.zeros(n, np.uint32), z=np.zeros((n, 2)))
    cnt, shift = np.zeros(6, np.uint64), C.c_double()
    ptr = lambda a: None if a is None else a.ctypes.data
    rc = L.emu_render_shift(ptr(re), ptr(im), len(re), ptr(blocks), ptr(offs), f["table"].levels, ptr(b), len(b),
                            f["series"].n if series else 0, f["series"].rho, f["tier"], nx, ny, plane.c_re, plane.c_im,
                            plane.h_m, plane.h_e, p.max_iter, p.escape_radius, f["r"].nucleus_period(), ptr(mask),
                            ptr(offsets), ptr(out["cls"]), ptr(out["n"]), ptr(out["z"]), ptr(cnt), C.byref(shift))
    assert rc == 0
    names = ("samples", "iterations", "blocks", "skipped", "fallback_samples", "closed_form_samples")
    return out, dict(zip(names, (int(c) for c in cnt))), shift.value


@pytest.mark.parametrize("start", ["series", "zero"])
@pytest.mark.parametrize("which", ["modulus", "again"])
def test_frame_shift_equals_oracle(libs, frame, which, start):
    got, cnt, shift = _emulate(libs[which], frame, 33, 19, series=start == "series")
    if start == "series":
        want = fdref.render_series(frame["job"], frame["ref"], frame["o_series"], bla=frame["o_bla"], raw=True)
    else:
        want = fdref.render(frame["job"], frame["ref"], frame["o_bla"], raw=True)
    assert np.array_equal(got["cls"], want["cls"]) and np.array_equal(got["n"], want["n"].astype(np.uint32))
    esc = (want["cls"] & 3) == 0
    assert np.array_equal(got["z"][esc], want["z"][esc])
    for k in ("iterations", "blocks", "skipped", "fallback_samples", "closed_form_samples"):
        assert cnt[k] == want["stats"][k], k
    assert want["stats"]["shift_px"] > 0.0
    assert shift / frame["h"] == want["stats"]["shift_px"]  # in output pixels, one sample each here


def test_sample_sent_there_by_itself(libs, frame):
    """A sample whose modulus lies inside the band around the threshold: its estimate is its
    own run's from Z_0, second run forced or not (the run from the series, over the one
    iteration its start leaves, applies no block)."""
    nx, ny, k = 33, 19, 33 * 9 + 16
    assert frame["series"].n == 9_999
    mask, offsets = np.zeros(nx * ny, np.uint8), np.zeros((nx * ny, 2))
    mask[k] = 1
    offsets[k] = (0.05267262566412388, 0.0)
    want = fdref.iterate(frame["ref"], frame["o_bla"], ar=offsets[k, 0] * frame["h"], ai=0.0, max_iter=10_000,
                         r2=frame["p"].escape_radius ** 2, nucleus=frame["r"].nucleus_period())
    kinds = {"escaped": 0, "interior": 1, "unresolved": 2}
    for L in libs.values():
        got, cnt, shift = _emulate(L, frame, nx, ny, mask, offsets)
        assert (cnt["samples"], cnt["blocks"], cnt["skipped"]) == (1, want["blocks"], want["skipped"])
        assert want["blocks"] > 0 and got["cls"][k] & 3 == kinds[want["kind"]]
        assert shift == want["shift"] > 0.0
