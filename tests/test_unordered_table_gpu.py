"""An uploaded table in which a merged block's radius exceeds its first half's: legal
(fdc_upload_bla checks values and shape), so the kernels search it level by level. A table
whose second level holds no valid block hides all levels above it, however large their
radii: its frames are those of the table without them."""
import numpy as np
import pytest

import fractodactyl_b200 as fd
from fractodactyl_b200 import _lib

pytestmark = pytest.mark.gpu


def _frame(dev, view3, nx, ny, it, tier, blocks=None, stripe=None):
    v, p = fd.View(*view3), fd.Params(nx, ny, max_iter=it, tier=tier)
    plane, t = fd.route._setup(v, p)
    r, bits = fd.reference(v, p)
    r.bits = bits
    dc, e = fd.bla_dc_bound(v, p)
    table = fd.Bla.build_scaled(r, fd.route.EPS, dc, e)
    assert table.levels > 3
    rows = np.array(table.blocks).reshape(-1, 7)
    offs = [int(o) for o in table.level_offsets]
    if blocks is not None:
        rows = blocks(rows, offs)
    h = dev.upload(r, fd.Bla(rows, table.level_offsets, table.eps, dc, e, len(r)))
    job = fd.route.make_job(plane, t, p, h, r.nucleus_period(), _lib.DERIVATIVE | _lib.BLA)
    got, cnt, _ = dev.render_job(job, raw=True, stripe=stripe)
    dev.free(h)
    return got, (cnt.samples, cnt.iterations, cnt.blocks, cnt.skipped)


def _hidden(rows, offs):
    """Blocks of the second level with radius 0, and every radius above them enormous: out of
    order, and reached by no search that stops at the second level."""
    rows = rows.copy()
    rows[offs[1]:offs[2], 4] = 0.0
    rows[offs[2]:, 4] = 1e100
    return rows


def _cut(rows, offs):
    rows = rows.copy()
    rows[offs[1]:, 4] = 0.0
    return rows


@pytest.mark.parametrize("frame", [(("0", "1", "1e-300"), 96, 64, 5000, "scaled"), (("0", "1", "1e-60"), 96, 64, 5000, "fixed")],
                         ids=["scaled", "fixed"])
@pytest.mark.parametrize("stripe", [None, (16, 5.0)], ids=["plain", "stripe"])
def test_level_by_level(frame, stripe):
    dev = fd.Device(0)
    try:
        cut, c0 = _frame(dev, *frame, blocks=_cut, stripe=stripe)
        hidden, c1 = _frame(dev, *frame, blocks=_hidden, stripe=stripe)
        full, c2 = _frame(dev, *frame, stripe=stripe)
        assert c0 == c1 and c0[2] > c2[2] > 0  # the hidden levels were of use: fewer, longer blocks
        for k in cut:
            assert np.array_equal(cut[k], hidden[k]), k
    finally:
        dev.close()
