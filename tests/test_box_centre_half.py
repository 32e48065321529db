"""Boxes as centre and half extent (csrc/layout.h): they hold the box they are made from, with room for the
slab test's rounding, and are no larger than that however far from the origin it lies."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def centre_half(tmp_path_factory):
    out = tmp_path_factory.mktemp("slab") / "libslab_check.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "three-mesh-bvh_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "slab_check.cpp"), "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    lib.centre_half.argtypes = [C.c_void_p] * 4 + [C.c_int64]

    def run(lo, hi):
        lo, hi = np.ascontiguousarray(lo, np.float32), np.ascontiguousarray(hi, np.float32)
        c, h = np.empty_like(lo), np.empty_like(lo)
        lib.centre_half(lo.ctypes.data, hi.ctypes.data, c.ctypes.data, h.ctypes.data, lo.size)
        return lo, hi, c, h

    return run


@pytest.mark.parametrize("offset", [0.0, 10.0, 1e4, -1e6, 3e8, 1e30])
@pytest.mark.parametrize("size", [1e-42, 1e-30, 1e-3, 1.0, 1e5, 1e20])
def test_holds_the_box_and_hugs_it(centre_half, offset, size):
    rng = np.random.default_rng(int(abs(offset) % 997) + 1)
    lo = (offset + rng.uniform(-1, 1, 20_000) * size).astype(np.float32)
    hi = np.maximum(lo, (lo.astype(np.float64) + rng.random(20_000) * size).astype(np.float32))
    lo, hi, c, h = centre_half(lo, hi)
    c, h, reach = c.astype(np.longdouble), h.astype(np.longdouble), np.maximum(hi.astype(np.longdouble) - c, c - lo)
    assert (h >= reach * (1 + 60 * 2.0**-24)).all()
    # at most half an ulp of the coordinates more than half of the box, and the slack
    half = (hi.astype(np.longdouble) - lo) / 2
    ulp = np.spacing(np.maximum(np.abs(lo), np.abs(hi))).astype(np.longdouble)
    assert (h <= (half + ulp) * (1 + 2.0**-17) + 2.0**-139).all()


def test_swapped_and_unusable_bounds(centre_half):
    nan, inf, big = np.nan, np.inf, 3.3e38
    _, _, c, h = centre_half([2, nan, 0, -inf, inf, -big], [1, 0, nan, inf, -inf, big])
    assert c[0] == 1.5 and 0.5 <= h[0] < 0.50001
    assert (c[1:] == 0).all() and (h[1:] > 2.9e38).all()
