"""The |dc| bound of a job with per-sample offsets (fdc_render's refusal beyond the BLA
table's dc_max, grid.rs:392-411) is h times the largest hypot of the rendered rows' offsets:
accepted at exactly that bound, refused one ulp above it, NaN offsets passed over as
before, an infinite one refused; few offsets and many (the threaded bound)."""
import ctypes as C

import numpy as np
import pytest

import fractodactyl_b200 as fd
from fractodactyl_b200 import _lib
from fractodactyl_b200.route import make_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(8, 4), (128, 96), (257, 130)])
@pytest.mark.parametrize("what", ["at", "above", "nan", "inf"])
def test_bound(nx, ny, what):
    v, p = fd.View("-0.743643887037158", "0.131825904205312", "1e-20"), fd.Params(nx, ny, max_iter=300)
    dev = fd.Device(0)
    try:
        plane, tier = fd.route._setup(v, p)
        r, bits = fd.reference(v, p)
        r.bits = bits
        offs = np.random.default_rng(nx).uniform(-nx, nx, (nx * ny, 2))
        half = max(float(_hypot(x, y)) for x, y in offs)
        bound = plane.h() * half
        if what == "above":
            bound = np.nextafter(bound, 0.0)
        if what == "nan":
            offs[3] = np.nan
        if what == "inf":
            offs[5, 1] = np.inf
        h = dev.upload(r)
        dev.build_bla(h, 2.0 ** -26, bound, 0)
        j = make_job(plane, tier, p, h, None, _lib.BLA)
        j.offsets = offs.ctypes.data
        if what in ("at", "nan"):
            assert dev.render_job(j)[2] == _lib.OK
        else:
            with pytest.raises(fd.RouteError, match="beyond the BLA table's dc_max"):
                dev.render_job(j)
    finally:
        dev.close()


_LIBM = C.CDLL("libm.so.6")
_LIBM.hypot.restype = C.c_double
_LIBM.hypot.argtypes = [C.c_double, C.c_double]


def _hypot(x, y):
    return _LIBM.hypot(x, y)
