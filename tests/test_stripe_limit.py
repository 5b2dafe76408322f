"""A stripe replay that does not find the blocks' escape again (blocks and plain steps may
disagree by a table's eps, or by more with a table a caller made) gives up at its limit, 64
iterates past the escape, and the average covers what was recorded (sample.rs:397, 576-579):
the kernel's own loop on the host, with the block budget ending before, at and after the
limit."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu") / "libstripelimit.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", os.path.join(HERE, "emu"),
                    "-I", os.path.join(os.path.dirname(HERE), "fractodactyl_b200", "csrc"),
                    os.path.join(HERE, "emu", "stripe_limit.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.stripe_limit_check.restype = ctypes.c_uint32
    L.stripe_limit_check.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_uint32, ctypes.c_uint32]
    return L


@pytest.mark.parametrize("extended", [0, 1])
@pytest.mark.parametrize("derivative", [0, 1])
@pytest.mark.parametrize("limit,lim", [(64, 4), (64, 64), (64, 65), (64, 4096), (1, 4096), (141, 100000)])
def test_replay_ends_at_its_limit(lib, extended, derivative, limit, lim):
    assert lib.stripe_limit_check(extended, derivative, limit, lim) == limit
