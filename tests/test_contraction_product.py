"""The nucleus gate's product (Magnitude, fd_device.cuh): the kernels keep the product's
squared modulus alone and iterate a sample again with the reference's own product
(Contraction) where that modulus is too close to the threshold to tell. The kernel emulation
built so that every sample is iterated again (FDK_CONTRACTION_AGAIN) and the ordinary one
both equal the oracle bit for bit, on frames with samples on either side of the threshold."""
import os
import subprocess

import numpy as np
import pytest

import fdref
import fractodactyl_b200 as fd
from fractodactyl_b200.locations import cached
from test_kernel_emulation import HERE, ROOT, _check, _oracle_job, emu, emulate  # noqa: F401


@pytest.fixture(scope="module")
def again(tmp_path_factory, emu):  # noqa: F811
    import ctypes
    lib = str(tmp_path_factory.mktemp("emu") / "libemu_again.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas",
                    "-DFDK_CONTRACTION_AGAIN=true", "-I", os.path.join(HERE, "emu"), "-I",
                    os.path.join(ROOT, "fractodactyl_b200", "csrc"), os.path.join(HERE, "emu", "emu.cpp"), "-o", lib],
                   check=True)
    L = ctypes.CDLL(lib)
    L.emu_render.restype = ctypes.c_int
    L.emu_render.argtypes = emu.emu_render.argtypes
    return L


@pytest.mark.parametrize("tier", ["fixed", "scaled"])
@pytest.mark.parametrize("bla", [False, True])
@pytest.mark.parametrize("which", ["modulus", "again"])
def test_gate_equals_oracle(emu, again, tier, bla, which):  # noqa: F811
    d = cached("c2")[0]
    view3, nx, ny, it = (d["re"], d["im"], "1e-104"), 25, 15, 4000  # multipliers on both sides of 1e-3
    v, p = fd.View(*view3), fd.Params(nx, ny, max_iter=it, tier=tier)
    plane, t = fd.route._setup(v, p)
    r, bits = fd.reference(v, p)
    r.bits = bits
    assert r.nucleus_period() == d["period"]
    table = None
    if bla:
        dc, e = fd.bla_dc_bound(v, p)
        table = fd.Bla.build_scaled(r, fd.route.EPS, dc, e)
        assert table.levels > 0
    got = emulate(emu if which == "modulus" else again, r, plane, t, p, 1 | (2 if bla else 0), bla=table)
    ref = fdref.Ref.arrays(r.re, r.im, r.bits)
    ob = fdref.Bla(ref, fd.route.EPS, table.dc_max, table.dc_exp) if bla else None
    want = fdref.render(_oracle_job(view3, p, t, fdref.COL_NU | fdref.COL_DE | fdref.COL_NORMAL), ref, ob, raw=True)
    kinds = np.bincount(want["cls"] & 3, minlength=3)
    assert kinds[1] > 20 and kinds[0] + kinds[2] > 20  # on both sides of the gate
    _check(got, want, escaped=False)
