"""The plans of csrc/tile_plan.h themselves (test_tile_plan.py restates the passes that use them): radices,
order of frequencies and pitch, at both precisions."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("tile") / "libtile.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-w",
                    "-I" + os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),
                    os.path.join(HERE, "tile_harness.cpp"), "-o", so], check=True)
    return C.CDLL(so)


LENGTHS = sorted({2 ** a * 3 ** b * 5 ** c for a in range(12) for b in range(8) for c in range(5)} & set(range(2, 2049)))
RADICES = {16: {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16}, 10: {2, 3, 4, 5, 6, 8, 9, 10}}   # FP32, FP64


@pytest.mark.parametrize("most", [16, 10])
def test_every_length_has_a_plan(lib, most):
    longest = 0
    for n in LENGTHS:
        fac = (C.c_int * 5)()
        nf = lib.tile_plan(n, most, fac)
        f = list(fac[:nf])
        assert 1 <= nf <= 5 and set(f) <= RADICES[most] and np.prod(f) == n and f == sorted(f, reverse=True)
        longest = max(longest, nf)
        # a transform whose passes leave frequency order[i] at position i: decimation in frequency
        order = (C.c_int * n)()
        lib.tile_frequencies(n, most, order)
        x = np.zeros(n, complex)
        x[1 % n] = 1.0
        y, L = x.copy(), n
        for r in f:
            y = y.reshape(n // L, r, L // r)
            w = np.exp(-2j * np.pi * np.outer(np.arange(r), np.arange(L // r)) / L)
            y = (np.fft.fft(y, axis=1) * w[None]).reshape(n)
            L //= r
        assert np.allclose(y, np.exp(-2j * np.pi * np.array(order) / n)), (n, f)
    assert longest == (4 if most == 16 else 5)


@pytest.mark.parametrize("elem", [8, 16])
def test_pitch_is_free_of_conflicts(lib, elem):
    """128 bytes a phase: 16 elements at FP32, 8 at FP64, of the tile's lines at neighbouring positions."""
    phase = 128 // elem
    for n in LENGTHS:
        for lines in range(1, 17):
            p = lib.tile_pitch_of(elem, n, lines)
            assert n <= p < n + 2 * phase
            k = 1
            while k < lines and k < phase:
                k *= 2
            if lines != k and lines < phase:
                continue                       # (the lines of a phase wrap to the next position)
            take = min(lines, phase)
            at = np.arange(phase)
            banks = ((at % take) * p + at // take) % phase
            assert np.unique(banks).size == phase, (n, lines, p)
