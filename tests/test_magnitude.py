"""The nucleus gate's squared modulus (Magnitude) against the reference's product of
multipliers (Contraction, sample.rs:658-698): wherever the modulus answers, the product
answers the same, over factors of any size. The product of a factor below 2^-1023 is NaN in
the reference (its rescaling by 2^k overflows) and never small, so the modulus leaves such
runs to the product itself. Frames over an orbit with such a point equal the oracle."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu") / "libmagnitude.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", os.path.join(HERE, "emu"),
                    "-I", os.path.join(os.path.dirname(HERE), "fractodactyl_b200", "csrc"),
                    os.path.join(HERE, "emu", "magnitude.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.magnitude_check.restype = ctypes.c_int64
    L.magnitude_check.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int, ctypes.POINTER(ctypes.c_uint64)]
    return L


@pytest.mark.parametrize("kind", range(6))
def test_answers_are_the_products(lib, kind):
    answered, n = ctypes.c_uint64(), 300_000
    assert lib.magnitude_check(kind + 1, n, kind, ctypes.byref(answered)) == 0
    assert (answered.value > n // 2) == (kind in (0, 2))
