"""The shape of a frame launch (launch_shape): a launch of few samples leaves lanes idle only
for warps that are launched (fdc_tuning.blocks_per_sm), and a band that stands for a frame
(FDC_BAND, which the autotuner measures) takes the frame's shape."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from fractodactyl_b200 import _lib, tune

HERE = os.path.dirname(os.path.abspath(__file__))
SMS = 148


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu") / "libshape.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I",
                    os.path.join(os.path.dirname(HERE), "fractodactyl_b200", "csrc"),
                    os.path.join(HERE, "emu", "launch_shape.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    U64, U32 = ctypes.c_uint64, ctypes.c_uint32
    L.launch_shape_of.argtypes = [U64, U64, U32, U32, U32, U32, ctypes.POINTER(U32)]
    L.spread_warps.restype = U32
    return L


def shape(lib, slots, blocks, frame=None, resident=5, spread=None):
    out = (ctypes.c_uint32 * 2)()
    lib.launch_shape_of(slots, frame or slots, SMS, blocks, resident, spread or lib.spread_warps(0), out)
    return out[0], out[1]


@pytest.mark.parametrize("blocks", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("ext_plain", [0, 1])
def test_no_lane_idles_while_slots_wait(lib, blocks, ext_plain):
    """The lanes that take samples, over the warps launched an SM up to the spread, hold the
    whole queue, or every lane does."""
    spread = lib.spread_warps(ext_plain)
    warps = SMS * min(spread, 4 * blocks)
    for slots in (32, 64, 1024, 2304, 5664, 30720, 56800, 56832, 129600, 2073600, 1 << 36):
        idle, tail = shape(lib, slots, blocks, spread=spread)
        assert 0 <= idle < 32
        assert idle == 0 or (32 - idle) * warps >= slots
        assert idle == 0 or (31 - idle) * warps < slots or idle == 31
        assert tail == min(max(slots // 8, 3 * SMS * blocks * 128), 0xffffffff)


@pytest.mark.parametrize("blocks", [1, 5])
@pytest.mark.parametrize("frame", [2304, 14656, 2073600])
def test_band_takes_the_frames_shape(lib, blocks, frame):
    idle, tail = shape(lib, frame, blocks)
    for slots in (32, frame // 64 // 32 * 32 or 32, frame // 2):
        got_idle, got_tail = shape(lib, slots, blocks, frame=frame)
        assert got_idle == idle
        assert abs(got_tail / slots - min(tail, frame) / frame) < 2.0 / slots
    assert shape(lib, frame, blocks, frame=frame) == (idle, tail)


def test_tuner_measures_bands_as_the_frame():
    flags = []

    class Dev:
        tuning = tune.Setting()

        def tune(self, **kw):
            pass

        def render_job(self, job, columns=()):
            flags.append((int(job.flags), job.first_row, job.rows))
            n = job.nx * job.ny
            cnt = _lib.Counters(kernel_ms=1.0)
            return {"cls": np.zeros(n, np.uint8), "n": np.zeros(n, np.uint32)}, cnt, 0

    for nx, ny, launches in ((64, 128, 1), (1920, 1080, 1), (1920, 1200, 2)):
        flags.clear()
        job = _lib.Job(nx=nx, ny=ny, flags=_lib.DERIVATIVE | _lib.DEVICE_OUT)
        tune.Tuner(Dev(), settings=[tune.Setting(4), tune.Setting(8)], reps=1).choice(job)
        assert len(flags) == 3 * launches
        assert all(f & _lib.BAND and not f & _lib.DEVICE_OUT for f, _, _ in flags)
        assert job.flags == _lib.DERIVATIVE | _lib.DEVICE_OUT
        rows = sum(r for _, _, r in flags[:launches])
        assert rows == ny if launches == 1 else abs(rows * nx - (1 << 20)) <= 4 * nx
        assert all(0 <= f and f + r <= ny for _, f, r in flags)
