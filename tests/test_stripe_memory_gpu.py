"""The stripe recorders are one buffer of the context, as large as its largest stripe launch:
frames on both kinds of tier and with every blocks_per_sm setting take no further memory, a
small frame takes little, and fdc_close gives it back."""
import numpy as np
import pytest

import fractodactyl_b200 as fd
from fractodactyl_b200 import _lib

pytestmark = pytest.mark.gpu
MB = 1 << 20
RECORDER = 2624  # bytes a thread


def test_one_buffer():
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info(0)[0]
    torch.cuda.synchronize()
    dev = fd.Device(0)
    try:
        frames = {}
        for name, tier, nx, ny in (("small", "scaled", 16, 8), ("scaled", "scaled", 640, 360), ("fixed", "fixed", 640, 360)):
            v, p = fd.View("0", "1", "1e-60"), fd.Params(nx, ny, max_iter=300, columns=("nu",), tier=tier)
            plane, t = fd.route._setup(v, p)
            r, bits = fd.reference(v, p)
            r.bits = bits
            h = dev.upload(r)
            job = fd.route.make_job(plane, t, p, h, r.nucleus_period(), 0)
            dev.render_job(job, columns=("nu",))  # everything but the recorders is allocated
            frames[name] = job, {}

        def render(name):
            job, first = frames[name]
            got, _, _ = dev.render_job(job, columns=("nu",), stripe=(16, 5.0))
            if not first:
                first.update({k: a.copy() for k, a in got.items()})
            assert all(np.array_equal(got[k], first[k]) for k in first)

        before = free()
        render("small")
        # 128 samples, one a warp: 32 blocks of 4 warps, whose 128 threads each have a recorder
        # (allocations round up to 2 MB)
        assert before - free() <= 32 * 128 * RECORDER + 4 * MB
        render("scaled")
        largest = before - free()
        assert largest <= 6 * 128 * 160 * RECORDER + 8 * MB
        for name in ("fixed", "scaled", "small"):
            for blocks in (0, 1, 2, 3, 4):
                dev.tune(blocks_per_sm=blocks)
                render(name)
        assert before - free() <= largest + 8 * MB
    finally:
        dev.close()
    assert free() >= before - 8 * MB
