"""The block search over ordered tables in whole frames on the host: emu.cpp stages every table
as unordered; built here with the flag set by the rule of check_order (fdcuda.cu), the frames
equal the oracle's, as they do with the level by level search."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import fdref
import fractodactyl_b200 as fd
from test_kernel_emulation import HERE, KATS, ROOT, SEAHORSE, _check, _oracle_job, _setup, emu, emulate  # noqa: F401

STAGED = "  p.bla_ab = s.ab.data();\n"
ORDERED = STAGED + """  p.bla_ordered = 1;
  for (uint32_t i = 1; i < levels; ++i)
    for (uint32_t t = 0; t < p.bla_count[i]; ++t)
      if (!(s.r2[p.bla_off[i] + t] <= s.r2[p.bla_off[i - 1] + 2 * t])) p.bla_ordered = 0;
  g_ordered += p.bla_ordered;
"""


@pytest.fixture(scope="module")
def ordered(tmp_path_factory, emu):  # noqa: F811
    at = tmp_path_factory.mktemp("emu")
    with open(os.path.join(HERE, "emu", "emu.cpp")) as f:
        source = f.read()
    assert source.count(STAGED) == 1
    source = source.replace(STAGED, ORDERED).replace('extern "C" {', 'extern "C" { uint32_t g_ordered = 0; }\nextern "C" {', 1)
    (at / "emu_ordered.cpp").write_text(source)
    so = str(at / "libemu_ordered.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-Wno-unknown-pragmas", "-I",
                    os.path.join(HERE, "emu"), "-I", os.path.join(ROOT, "fractodactyl_b200", "csrc"),
                    str(at / "emu_ordered.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    L.emu_render.restype = C.c_int
    L.emu_render.argtypes = emu.emu_render.argtypes
    return L


@pytest.mark.parametrize("case", ["f64", "fixed", "scaled", "nucleus"])
def test_frames_equal_oracle(ordered, case):
    eps, tier = fd.route.EPS, None
    if case == "f64":
        view3, nx, ny, it, eps = (*SEAHORSE, "1e-10"), 40, 24, 20_000, 2.0 ** -30
    elif case == "fixed":
        f = KATS["series_frames"][18]
        view3, nx, ny, it = (f["re"], f["im"], f["width"]), 33, 19, 10_000
    elif case == "scaled":
        view3, nx, ny, it = ("0", "1", "1e-300"), 32, 16, 5_000
    else:
        d = fd.locations.cached("c2")[0]
        view3, nx, ny, it, tier = (d["re"], d["im"], "1e-100"), 16, 10, 20_000, "scaled"
    v, p, plane, t, r = _setup(view3, nx, ny, it, tier)
    dc, e = fd.bla_dc_bound(v, p)
    table = fd.Bla.build_scaled(r, eps, dc, e)
    assert table.levels > 3
    seen = C.c_uint32.in_dll(ordered, "g_ordered")
    before = seen.value
    got = emulate(ordered, r, plane, t, p, 1 | 2, bla=table)
    assert seen.value == before + 1  # the tables the library builds are ordered
    ref = fdref.Ref.arrays(r.re, r.im, r.bits)
    want = fdref.render(_oracle_job(view3, p, t, fdref.COL_NU | fdref.COL_DE | fdref.COL_NORMAL), ref,
                        fdref.Bla(ref, eps, table.dc_max, table.dc_exp), raw=True)
    _check(got, want, escaped=False)
    assert got["counters"]["blocks"] > 0 and np.any(got["cls"] == 0)
