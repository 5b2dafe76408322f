"""The second run for the nucleus gate's own product (Magnitude, kind 3) in the kernels that
restart a sample with code of their own: series starts with and without a table, the stripe
variant and batches, on the host with every sample sent through it (FDK_CONTRACTION_AGAIN):
values, columns and counters equal the oracle's or the ordinary build's."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import fdref
import fractodactyl_b200 as fd
from fractodactyl_b200.locations import cached
from test_kernel_emulation import (HERE, KATS, ROOT, Job, _check, _oracle_job, _outputs, _ptr, _setup, emu,  # noqa: F401
                                   emulate)


@pytest.fixture(scope="module")
def again(tmp_path_factory, emu):  # noqa: F811
    so = str(tmp_path_factory.mktemp("emu") / "libemu_users.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    "-DFDK_CONTRACTION_AGAIN=true", "-I", os.path.join(HERE, "emu"), "-I",
                    os.path.join(ROOT, "fractodactyl_b200", "csrc"), os.path.join(HERE, "emu", "emu.cpp"), "-o", so],
                   check=True)
    L = C.CDLL(so)
    L.emu_render.restype = C.c_int
    L.emu_render.argtypes = emu.emu_render.argtypes
    L.emu_render_batch.restype = C.c_int
    L.emu_render_batch.argtypes = emu.emu_render_batch.argtypes
    L.emu_set_stripe.argtypes = emu.emu_set_stripe.argtypes
    return L


def _gate_frame(tier):
    """The c2 nucleus's frame with multipliers on both sides of the threshold."""
    d = cached("c2")[0]
    view3, nx, ny, it = (d["re"], d["im"], "1e-104"), 25, 15, 4000
    v, p, plane, t, r = _setup(view3, nx, ny, it, tier)
    assert r.nucleus_period() == d["period"]
    dc, e = fd.bla_dc_bound(v, p)
    table = fd.Bla.build_scaled(r, fd.route.EPS, dc, e)
    assert table.levels > 0
    return view3, p, plane, t, r, table


@pytest.mark.parametrize("bla", [False, True])
@pytest.mark.parametrize("frame", [18, -1])
def test_series(again, frame, bla):
    f = KATS["series_frames"][frame]
    view3 = (f["re"], f["im"], f["width"])
    v, p, plane, t, r = _setup(view3, 33, 19, 10_000)
    rho, _ = fd.bla_dc_bound(v, p)
    series = fd.Series.build(r, rho, float(f["width"]) / 33, p.max_iter)
    ref = fdref.Ref.arrays(r.re, r.im, r.bits)
    o_series = fdref.Series(ref, rho, float(f["width"]) / 33, p.max_iter)
    table = ob = None
    if bla:
        eps = fd.route.EPS if frame == 18 else 2.0 ** -26
        table, ob = fd.Bla.build_scaled(r, eps, rho, 0), fdref.Bla(ref, eps, rho, 0)
        assert table.levels > 0
    got = emulate(again, r, plane, t, p, 1 | (2 if bla else 0) | 4, bla=table, series=series)
    want = fdref.render_series(_oracle_job(view3, p, t, fdref.COL_NU | fdref.COL_DE | fdref.COL_NORMAL), ref, o_series,
                               bla=ob, raw=True)
    _check(got, want, escaped=frame == 18)


@pytest.mark.parametrize("tier", ["fixed", "scaled"])
@pytest.mark.parametrize("bla", [False, True])
def test_stripe(emu, again, tier, bla):  # noqa: F811
    view3, p, plane, t, r, table = _gate_frame(tier)
    table = table if bla else None
    flags, out = 1 | (2 if bla else 0) | 32, []
    for L in (emu, again):
        stripe = np.zeros(p.nx * p.ny, np.float32)
        L.emu_set_stripe(16, 5.0, stripe.ctypes.data)
        try:
            got = emulate(L, r, plane, t, p, flags, bla=table)
        finally:
            L.emu_set_stripe(16, 5.0, None)
        got["stripe"] = stripe
        out.append(got)
    kinds = np.bincount(out[0]["cls"] & 3, minlength=3)
    assert kinds[1] > 20 and kinds[0] + kinds[2] > 20
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]) if isinstance(out[0][k], np.ndarray) else out[0][k] == out[1][k], k


@pytest.mark.parametrize("tier", ["fixed", "scaled"])
def test_batch(again, tier):
    view3, p, plane, t, r, table = _gate_frame(tier)
    ref = fdref.Ref.arrays(r.re, r.im, r.bits)
    ob = fdref.Bla(ref, fd.route.EPS, table.dc_max, table.dc_exp)
    re_, im_ = np.ascontiguousarray(r.re), np.ascontiguousarray(r.im)
    blocks = np.ascontiguousarray(table.blocks)
    offs = np.ascontiguousarray(table.level_offsets, dtype=np.uint64)
    outs = [_outputs(p.nx * p.ny) for _ in range(2)]
    jobs = (Job * 2)(*[Job(re=re_.ctypes.data, im=im_.ctypes.data, len=len(re_), blocks7=_ptr(blocks) if b else None,
                           level_offsets=_ptr(offs) if b else None, levels=table.levels if b else 0, tier=t,
                           flags=1 | (2 if b else 0), nx=p.nx, ny=p.ny, ss=p.ss, max_iter=p.max_iter, c_re=plane.c_re,
                           c_im=plane.c_im, h_m=plane.h_m, h_e=plane.h_e, cos_rot=plane.cos_rot,
                           sin_rot=plane.sin_rot, escape_radius=p.escape_radius, nucleus=r.nucleus_period(),
                           first_row=0, rows=0, first_col=0, cols=0, **{k: a.ctypes.data for k, a in outs[b].items()})
                       for b in range(2)])
    assert again.emu_render_batch(jobs, 2) == 0
    for b in range(2):
        want = fdref.render(_oracle_job(view3, p, t, fdref.COL_NU | fdref.COL_DE | fdref.COL_NORMAL), ref,
                            ob if b else None, raw=True)
        got = dict(outs[b], counters=dict(zip(("samples", "iterations", "blocks", "skipped", "fallback_samples",
                                               "closed_form_samples"), (int(c) for c in jobs[b].counters))))
        _check(got, want, escaped=False)
