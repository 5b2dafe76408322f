"""The block search's forms (block_level, perturb_f64.cuh) against the reference's level by
level tests on random tables whose merged radii never exceed their first half's: table
lengths around powers of two, budgets that cut levels short, deltas exactly at a radius."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emu") / "liblevel.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", os.path.join(HERE, "emu"),
                    "-I", os.path.join(os.path.dirname(HERE), "fractodactyl_b200", "csrc"),
                    os.path.join(HERE, "emu", "block_level.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.block_level_check.restype = ctypes.c_int64
    L.block_level_check.argtypes = [ctypes.c_uint64, ctypes.c_uint32, ctypes.c_uint64]
    return L


@pytest.mark.parametrize("points", [4, 5, 9, 63, 66, 4097, 65538, 300_000, 1 << 20])
def test_search_equals_reference(lib, points):
    assert lib.block_level_check(points, points, 200_000) == 0
