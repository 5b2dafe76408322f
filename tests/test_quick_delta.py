"""The precision form's quick sums (quick_delta) and derivative blocks (block_dz_quick,
perturb_f32.cuh) leave the state that the wide-exponent ones leave, bit for bit, wherever
they apply: exponents apart and alike, cancelling terms, zeros, ties of the float rounding."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu") / "libdelta.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", os.path.join(HERE, "emu"),
                    "-I", os.path.join(os.path.dirname(HERE), "fractodactyl_b200", "csrc"),
                    os.path.join(HERE, "emu", "quick_delta.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("check", ["quick_delta_check", "quick_dz_check"])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_quick_equals_wide(lib, check, seed):
    f, quick, n = getattr(lib, check), ctypes.c_uint64(), 1_000_000
    f.restype = ctypes.c_int64
    assert f(ctypes.c_uint64(seed), ctypes.c_uint64(n), ctypes.byref(quick)) == 0
    assert quick.value > n // 20
