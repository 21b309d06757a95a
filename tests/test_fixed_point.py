"""The FP64 line filters in block floating point (csrc/fft_int.cuh, k_tile.cuh), built for the host,
against extended precision and against FP64 butterflies of 8, 4, 2, 3 and 5: lines and slices
of every kind of plan, the exponential and the k^2 filter, condensates and single sites far above
the others."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LD = np.longdouble
pytestmark = pytest.mark.skipif(np.finfo(LD).nmant < 63, reason="no extended precision on this host")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("tile") / "libtile.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-w",
                    "-I" + os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),
                    os.path.join(HERE, "tile_harness.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def momenta(n):
    k = np.arange(n)
    return np.where(k < n // 2, 2 * np.pi * k / n, -2 * np.pi * (n - k) / n)


def filter_of(kind, n):
    p = momenta(n)
    return {"exp": np.exp(-0.025 * p * p), "k2": -p * p, "energy": 0.5 * p * p}[kind] / n


def field(kind, ns, dims, seed=1):
    rng = np.random.default_rng(seed)
    z = rng.standard_normal((ns,) + dims) + 1j * rng.standard_normal((ns,) + dims)
    if kind == "one_site":
        z = 1e-3 * (0.5 + 0.3 * z)
        z.reshape(ns, -1)[:, int(np.prod(dims)) // 3] = 3.0
        return z
    amp, width = {"condensate": (0.577, 0.1), "wide": (0.5, 0.25), "flat": (1.0, 0.003)}[kind]
    return amp + width * z


def integer(lib, x, filters, energy=False, cst=1.0):
    """The tile filter's slices, as many a tile as its size allows."""
    ns, dims = x.shape[0], x.shape[1:]
    d = (C.c_int * 3)(*(list(dims) + [1] * (3 - len(dims))))
    f = np.ascontiguousarray(np.concatenate([g for g in filters if g.size > 1]))
    out, per = np.empty_like(x), max(1, 2048 // int(np.prod(dims)))
    for i in range(0, ns, per):
        a, b = np.ascontiguousarray(x[i:i + per]), np.empty_like(x[i:i + per])
        assert lib.tile_filter(d, len(filters), a.shape[0], int(energy), C.c_double(cst), ptr(f), ptr(a), ptr(b))
        out[i:i + per] = b
    return out


def butterflies(lib, x, filters, energy=False):
    """The same by FP64 butterflies, axis by axis (energy: every axis of the slice, summed)."""
    out = np.zeros_like(x) if energy else x.copy()
    for a, f in enumerate(filters):
        if f.size == 1:
            continue
        y = np.ascontiguousarray(np.moveaxis(x if energy else out, a + 1, -1))
        lib.line_filter64(f.size, y.size // f.size, ptr(np.ascontiguousarray(f)), ptr(y))
        y = np.moveaxis(y, -1, a + 1)
        out = out + y if energy else y
    return out


def dft(n, sign):
    """exp(sign 2 pi i j k / n) in extended precision, the angle reduced to an octant."""
    m = np.outer(np.arange(n), np.arange(n)) % n
    t = 8 * m
    o = (t + n // 2) // n
    a = (t - o * n).astype(LD) / n * (LD("3.14159265358979323846264338327950288") / 4)
    h, c, s = np.sqrt(LD(0.5)), np.cos(a), np.sin(a)
    co = np.array([1, h, 0, -h, -1, -h, 0, h], LD)[o % 8]
    so = np.array([0, h, 1, h, 0, -h, -1, -h], LD)[o % 8]
    return co * c - so * s, sign * (so * c + co * s)


def exact(x, filters, energy=False):
    fft = pytest.importorskip("scipy.fft")
    out = np.zeros(x.shape, np.clongdouble) if energy else x.astype(np.clongdouble)
    for a, f in enumerate(filters):
        s = [1] * x.ndim
        s[a + 1] = f.size
        y = x.astype(np.clongdouble) if energy else out
        y = fft.ifft(fft.fft(y, axis=a + 1) * f.astype(LD).reshape(s), axis=a + 1) * f.size
        out = out + y if energy else y
    return out


def errors(got, want):
    e = np.abs(got - want).astype(float)
    return float(np.linalg.norm(e) / np.linalg.norm(np.abs(want).astype(float))), np.sqrt((e ** 2).mean(0))


@pytest.mark.parametrize("kind", ["exp"])
@pytest.mark.parametrize("n", [243, 729, 810, 900])
def test_no_site_is_worse_than_the_others(lib, n, kind):
    """Rounding errors are those of the transforms' frequencies, alike at every site: over 200
    lines the root mean square at a site scatters by 1 / 20 of itself (two parts each), so
    that of n sites' largest lies within six such steps, 1.3; a bias stands out at a few."""
    x, f = field("condensate", 200, (n,)), [filter_of(kind, n)]
    _, site = errors(integer(lib, x, f), exact(x, f))
    assert site.max() < 1.3 * np.sqrt((site ** 2).mean()), site.argmax()


@pytest.mark.parametrize("n", [2, 3, 8, 27, 48, 125, 900, 1875, 2048])
def test_twiddles_to_62_bits(lib, n):
    """Half a unit of rounding and 2^-80 of the series; 2^-2 units of the extended reference."""
    tab = np.empty((n, 2), np.int64)
    lib.fixed_twiddle_table(n, ptr(tab))
    c, s = dft(n, -1)
    got = tab.astype(LD)
    want = np.stack([c[1 % n], s[1 % n]], 1) * LD(2) ** 62
    assert np.abs(got - want).max() < 0.76


@pytest.mark.parametrize("kind", ["exp", "k2"])
@pytest.mark.parametrize("n", [9, 60, 192, 480, 729, 1152, 1728])
def test_one_site_far_above_the_others(lib, n, kind):
    """No further off than FP64 butterflies, at the worst site and in the 2-norm: with one site a
    thousand times the others every product of it carries its factor's error."""
    x, f = field("one_site", 48, (n,)), [filter_of(kind, n)]
    want = exact(x, f)
    (norm, site), (norm64, site64) = errors(integer(lib, x, f), want), errors(butterflies(lib, x, f), want)
    assert norm < norm64 and site.max() < site64.max()


@pytest.mark.parametrize("kind", ["condensate", "wide", "flat"])
@pytest.mark.parametrize("dims", [(8,), (48,), (60,), (250,), (600,), (729,), (810,), (900,), (1250,), (1875,), (2000,), (2048,),
                                  (30, 30), (27, 25), (8, 6, 4)], ids=lambda d: "x".join(map(str, d)))
def test_exponential_filter_against_butterflies(lib, dims, kind):
    """No further off than FP64 butterflies on a condensate, whose zero mode takes the top bits:
    plans of one to five radices, lines and slices."""
    x, f = field(kind, 48, dims), [filter_of("exp", n) for n in dims]
    want = exact(x, f)
    (norm, site), (norm64, site64) = errors(integer(lib, x, f), want), errors(butterflies(lib, x, f), want)
    assert norm < norm64 and site.max() < site64.max()


@pytest.mark.parametrize("n", [2, 3, 5, 9, 16, 48, 60, 243, 500, 900, 1875])
def test_single_modes_do_not_overflow(lib, n):
    """A line that is one mode grows by its whole radix in every pass; amplitudes along the binade
    and directions of up to sqrt(2) times a component.  An overflow would be an error of the
    line's size; roundings are 2^-50 of it at most."""
    k, j = np.arange(min(n, 40))[:, None], np.arange(n)[None, :]
    for amp in (1.0, 1.2, 1.5, 1.9999999, 2 - 2.0 ** -52):
        for turn in (1.0, 1j, np.exp(0.25j * np.pi), np.exp(1.0j)):
            x = amp * turn * np.exp(2j * np.pi * (k * j % n) / n)
            f = filter_of("exp", n)
            want = x * (f * n)[k]
            assert np.abs(integer(lib, x, [f]) - want).max() < 2.0 ** -50 * 2


@pytest.mark.parametrize("kind", ["condensate", "wide", "flat"])
@pytest.mark.parametrize("dims", [(8,), (48,), (60,), (250,), (600,), (729,), (810,), (900,), (1250,), (1875,), (2000,), (2048,),
                                  (30, 30), (27, 25), (8, 6, 4)], ids=lambda d: "x".join(map(str, d)))
def test_k2_filters_against_butterflies(lib, dims, kind):
    """The k^2 filter of lines and the kinetic energy of slices, which throw the condensate away."""
    energy = len(dims) > 1
    x, f = field(kind, 48, dims), [filter_of("energy" if energy else "k2", n) for n in dims]
    want = exact(x, f, energy)
    # (the kernel takes the product of all 1 / n into every axis of a sum)
    (norm, site), (norm64, site64) = errors(integer(lib, x, f, energy), want), errors(butterflies(lib, x, f, energy), want)
    assert norm < norm64 and site.max() < site64.max()


@pytest.mark.parametrize("scale", [1e-150, 1.0, 1e150])
def test_lines_of_one_value(lib, scale):
    """A constant line under a filter that vanishes at zero frequency gives exact zeros, also beside
    other lines of the tile."""
    x = np.ones((6, 60), complex) * (0.3 - 0.7j) * scale
    x[2:4] = field("condensate", 2, (60,)) * scale
    got = integer(lib, x, [filter_of("k2", 60)])
    assert np.all(got[[0, 1, 4, 5]] == 0) and np.all(got[2:4] != 0)


@pytest.mark.parametrize("kind", ["exp", "k2"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("site", [0, 7, 59])
def test_non_finite_lines_are_nan_and_alone(lib, kind, bad, site):
    x, f = field("wide", 5, (60,)), [filter_of(kind, 60)]
    want = integer(lib, x, f)
    y = x.copy()
    y[2, site] = bad
    got = integer(lib, y, f)
    assert np.all(np.isnan(got[2]))
    assert np.array_equal(got[[0, 1, 3, 4]], want[[0, 1, 3, 4]])


@pytest.mark.parametrize("n", [60, 300])
@pytest.mark.parametrize("kind", ["exp", "k2"])
def test_range_of_the_doubles(lib, n, kind):
    """A line times a power of two gives its result times it, bit for bit, wherever neither leaves the
    normal numbers: up to the last binade, and down to 2^-1022."""
    x, f = field("wide", 6, (n,)), [filter_of(kind, n)]
    want = integer(lib, x, f)
    low = lambda *a: min(np.abs(v[v != 0]).min() for z in a for v in (z.real, z.imag))
    high = lambda *a: max(np.abs(v).max() for z in a for v in (z.real, z.imag))
    # (the first site is subtracted: a difference of sites is a value, too)
    top = 1023 - int(np.floor(np.log2(max(2 * high(x), high(want)))))
    bottom = -1022 - int(np.floor(np.log2(min(low(x), low(want), low(x[:, 1:] - x[:, :1])))))
    for k in (top, top - 1, 900, -850, -900, bottom + 1, bottom):
        got = integer(lib, np.ldexp(x.real, k) + 1j * np.ldexp(x.imag, k), f)
        assert np.array_equal(got.real, np.ldexp(want.real, k)) and np.array_equal(got.imag, np.ldexp(want.imag, k)), k


def test_last_binade(lib):
    """Results of the last binade, [2^1023, 2^1024), are not infinite."""
    x = np.ldexp(1.75, 1023) * np.ones((3, 60), complex)
    got = integer(lib, x, [filter_of("exp", 60)])
    assert np.all(np.abs(got.real / x.real - 1) < 2.0 ** -50) and np.all(np.isfinite(got.imag))
