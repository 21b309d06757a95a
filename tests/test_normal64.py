"""The integer Box-Muller transform (csrc/normal64.cuh), built for the host, against
extended-precision arithmetic: every returned part within 0.75 units in its last place
(0.5 of rounding, 2^-55 relative for the logarithm's and the square root's fixed point,
2^-56 for the angle's, and the host's own 64-bit mantissa)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def normals(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("normal64") / "libnormal64.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off",
                    os.path.join(HERE, "normal64_harness.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)

    def run(x, y):
        x, y = np.ascontiguousarray(x, np.uint32), np.ascontiguousarray(y, np.uint32)
        re, im = np.empty(x.size), np.empty(x.size)
        lib.normals(C.c_long(x.size), *(a.ctypes.data_as(C.c_void_p) for a in (x, y, re, im)))
        return re, im
    return run


def exact(x, y):
    L = np.longdouble
    pi = L("3.14159265358979323846264338327950288")
    r = np.sqrt(L(-2) * np.log((x.astype(L) + L(0.5)) * L(2) ** -32))
    # the nearest multiple of pi/4 split off the integer angle
    o = (((y.astype(np.int64) + (1 << 28)) >> 29) & 7)
    a = (((y.astype(np.int64) + (1 << 28)) & ((1 << 29) - 1)) - (1 << 28)).astype(L) * (2 * pi * L(2) ** -32)
    c, s, h = np.cos(a), np.sin(a), np.sqrt(L(0.5))
    co = np.array([1, h, 0, -h, -1, -h, 0, h], L)[o]
    so = np.array([0, h, 1, h, 0, -h, -1, -h], L)[o]
    return r * (co * c - so * s), r * (so * c + co * s)


EDGE = sorted({v & 0xFFFFFFFF for k in range(8) for b in (k << 29, (k << 29) + (1 << 28), 0xFF << 24, 0xFE << 24, 1 << 20)
               for v in (b - 2, b - 1, b, b + 1, b + 2)})


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no extended precision on this host")
@pytest.mark.parametrize("words", ["edges", "random", "near_one", "near_zero"])
def test_normal64_to_the_last_place(normals, words):
    rng = np.random.default_rng(7)
    x, y = (rng.integers(0, 1 << 32, 200000, dtype=np.uint64).astype(np.uint32) for _ in range(2))
    if words == "edges":
        x, y = (g.ravel().astype(np.uint32) for g in np.meshgrid(EDGE, EDGE))
    elif words == "near_one":      # u1 near 1: the logarithm and the radius are small
        x = ~(x >> (y % 33 % 32).astype(np.uint32))
    elif words == "near_zero":     # u1 and the angle near 0
        x, y = x >> (y % 31).astype(np.uint32), (y >> (x % 29).astype(np.uint32)) + ((x & 7) << np.uint32(29))
    got, want = normals(x, y), exact(x, y)
    for g, w in zip(got, want):
        ulp = np.spacing(np.abs(w).astype(np.float64))
        assert np.all(g[w == 0] == 0)
        assert np.max(np.abs(g.astype(np.longdouble) - w) / ulp) < 0.75


def test_no_undefined_behaviour(tmp_path):
    """Shifts and sums of every edge word (the word 0, whose remainder is exactly 0, among them)."""
    exe = str(tmp_path / "normal64")
    subprocess.run(["g++", "-O1", "-std=c++17", "-DNORMAL64_MAIN", "-fsanitize=undefined", "-fno-sanitize-recover=all",
                    os.path.join(HERE, "normal64_harness.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe] + [str(v) for v in EDGE], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
