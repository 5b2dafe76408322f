"""A sample whose nucleus product is lost (a zero factor: the centre sample of a frame around
the period-2 nucleus c = -1 has z_2 = 0) is iterated a second time for the product itself, in
every kernel that holds the gate: frames, stripe frames, batches and the allocation-free
entry point, with and without a table where they take one. Each equals the oracle."""
import ctypes as C

import numpy as np
import pytest

import fdref
import fractodactyl_b200 as fd
from fractodactyl_b200 import _lib

pytestmark = pytest.mark.gpu
NX, NY, IT = 9, 5, 300


def _noalloc(torch, job, r):
    n = NX * NY
    orbit = torch.from_numpy(np.ascontiguousarray(np.stack([r.re, r.im], 1).reshape(-1))).cuda()
    cols = {"cls": torch.zeros(n, dtype=torch.uint8, device="cuda"), "n": torch.zeros(n, dtype=torch.int32, device="cuda")}
    out = _lib.Out()
    for k, t in cols.items():
        setattr(out, k, t.data_ptr())
    cnt, err = _lib.Counters(), C.create_string_buffer(512)
    torch.cuda.synchronize()
    st = _lib.lib().fdc_render_noalloc(0, orbit.data_ptr(), len(r), C.byref(job), C.byref(out), None, C.byref(cnt), None,
                                       err, 512)
    assert st == _lib.OK, err.value.decode()
    return {k: t.cpu().numpy() for k, t in cols.items()}


@pytest.mark.parametrize("width,tier", [("1e-20", "fixed"), ("1e-20", "scaled")])
@pytest.mark.parametrize("user", ["frame", "frame-bla", "stripe", "stripe-bla", "batch", "batch-bla", "noalloc"])
def test_centre_sample(width, tier, user):
    torch = pytest.importorskip("torch")
    v, p = fd.View("-1", "0", width), fd.Params(NX, NY, max_iter=IT, columns=("nu",), tier=tier)
    plane, t = fd.route._setup(v, p)
    r, bits = fd.reference(v, p)
    r.bits = bits
    ref, table = fdref.Ref.arrays(r.re, r.im, r.bits), None
    bla = user.endswith("-bla")
    dc, e = fd.bla_dc_bound(v, p)
    if bla:
        table = fdref.Bla(ref, fd.route.EPS, dc, e)
    dev = fd.Device(0)
    try:
        h = dev.upload(r, fd.Bla.build_scaled(r, fd.route.EPS, dc, e) if bla else None)
        job = fd.route.make_job(plane, t, p, h, 2, _lib.BLA if bla else 0)
        if user == "noalloc":
            got = _noalloc(torch, job, r)
        elif user.startswith("batch"):
            b = dev.batch([job, job], columns=("nu",))
            b.run()
            got, twin = b.columns(0), b.columns(1)
            assert all(np.array_equal(got[k], twin[k]) for k in got)
            b.free()
        else:
            got, _, _ = dev.render_job(job, columns=("nu",), stripe=(16, 5.0) if user.startswith("stripe") else None)
    finally:
        dev.close()
    kinds = {"escaped": 0, "interior": 1, "unresolved": 2}
    h_ = np.ldexp(plane.h_m, plane.h_e)
    for k in range(NX * NY):
        x, y = k % NX + 0.5 - NX / 2.0, -(k // NX + 0.5 - NY / 2.0)
        where = dict(extended=True, ar=x * plane.h_m, ai=y * plane.h_m, offset_exp=plane.h_e) if t == 2 else \
            dict(ar=x * h_, ai=y * h_)
        o = fdref.iterate(ref, table, derivative=False, max_iter=IT, r2=p.escape_radius ** 2, nucleus=2, **where)
        assert (got["cls"][k] & 3, int(got["n"][k])) == (kinds[o["kind"]], IT if o["kind"] == "unresolved" else o["n"]), k
        if 2 * k == NX * NY - 1:
            assert o["kind"] == "interior" and o["n"] == 3
