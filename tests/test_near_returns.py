"""Once an extended-tier sample's four near returns are counted, its iterations take the
short path again: an interior sample that has settled on its cycle is near its save point at
every period, and must not run the full sequence each time."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu") / "libnear.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", os.path.join(HERE, "emu"),
                    "-I", os.path.join(os.path.dirname(HERE), "fractodactyl_b200", "csrc"),
                    os.path.join(HERE, "emu", "near_returns.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.near_returns_check.restype = ctypes.c_int
    L.near_returns_check.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.c_uint32, ctypes.POINTER(ctypes.c_uint32),
                                     ctypes.POINTER(ctypes.c_uint32)]
    return L


@pytest.mark.parametrize("ar,ai", [(1.2, 0.0), (1.0, 0.3), (1.1, 0.1), (1.3, -0.1)])
def test_no_full_sequence_after_the_fourth_return(lib, ar, ai):
    near, folded = ctypes.c_uint32(), ctypes.c_uint32()
    assert lib.near_returns_check(ar, ai, 20_000, ctypes.byref(near), ctypes.byref(folded)) == 4
    assert near.value > 15_000
    # the product shrinks by less than 2^5 an iteration here and leaves its 420 binades seldom
    assert folded.value < near.value // 20
