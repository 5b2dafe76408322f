"""The extended tier's quick block application (block_quick, perturb_f64.cuh) equals the full
one (block_full) bit for bit wherever it applies, over binary64's whole range of states and
coefficients: zeros, powers of two, mantissas just below 2, products that cancel, parts and
scalings that underflow. The kernel's own source, built for the host."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu") / "libblock.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", os.path.join(HERE, "emu"),
                    "-I", os.path.join(os.path.dirname(HERE), "fractodactyl_b200", "csrc"),
                    os.path.join(HERE, "emu", "block_quick.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.block_quick_check.restype = ctypes.c_int64
    L.block_quick_check.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int, ctypes.POINTER(ctypes.c_uint64)]
    return L


@pytest.mark.parametrize("derivative", [False, True])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_quick_equals_full(lib, seed, derivative):
    quick, n = ctypes.c_uint64(), 1_000_000
    assert lib.block_quick_check(seed, n, int(derivative), ctypes.byref(quick)) == 0
    assert quick.value > n // 20  # the quick path is taken often enough to be tested
