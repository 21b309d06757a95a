"""The reference model's drift (csrc/drift_math.cuh), built for the host, against extended precision,
also where one component is far above the others.  A term of K_a is rounded at most a dozen times on
its way into the sum, and the sums of it at most as often: 24 u of the terms' magnitudes, u the
working precision's 2^-53 or 2^-24.  The terms are those of the reference
(Propagator_without_cutoff.cu:24-128): the density of component 3 - a is not among K_a's."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("drift") / "libdrift.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-w",
                    "-I" + os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),
                    os.path.join(HERE, "drift_harness.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def terms(par, f):
    """The terms of K and Kbar (their sum is the drift), and their magnitudes' sum."""
    eps, ax, mu, P, Q, G = (np.longdouble(v) for v in par)
    pm, pc, pp, cc, cp, km, kp = f
    mus = [mu + P + Q, mu, mu, mu - P + Q]
    out = []
    for k, b, first, m, kin in ((pm, cc, pm - pc, pm, km), (cp, pc, cp - cc, pp, kp)):
        rows = []
        for a in range(4):
            p, q = ((1, 2) if a in (0, 3) else (0, 3))
            t = [eps * kin[a], eps * mus[a] * m[a], -2 * G * eps * k[p] * k[q] * b[3 - a]]
            t += [-2 * G * eps * k[c] * b[c] * k[a] for c in range(4) if c != 3 - a]
            rows.append((ax * (sum(t) + first[a]), abs(ax) * (sum(abs(v) for v in t) + abs(first[a]))))
        out.append(rows)
    return out


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("ax", [1.0, 0.5])
@pytest.mark.parametrize("large", [None, 0, 1, 2, 3])
def test_drift_to_rounding(lib, fp64, ax, large):
    n, rng = 400, np.random.default_rng(3)
    f = 0.4 + 0.2 * (rng.standard_normal((7, 4, n)) + 1j * rng.standard_normal((7, 4, n)))
    if large is not None:
        f[:, large] *= 3e3
    if not fp64:
        f = f.astype(np.complex64).astype(complex)
    par = np.array([0.0625, ax, -0.75, 0.0625, 0.03125, 0.25])   # exact at both precisions
    flat = np.ascontiguousarray(np.moveaxis(f, 2, 0))            # site, field, component
    k = np.empty((n, 2, 4), complex)
    lib.drift_ref4(int(fp64), C.c_long(n), *(v.ctypes.data_as(C.c_void_p) for v in (par, flat, k)))
    u = 2.0 ** (-53 if fp64 else -24)
    for side, rows in enumerate(terms(par, f.astype(np.clongdouble))):
        for a, (want, size) in enumerate(rows):
            assert np.all(np.abs(k[:, side, a] - want) < 24 * u * size), (side, a)
