"""The tile filter's plans, addresses and passes (csrc/k_tile.cuh, clv_engine.cu tile_factors /
add_tile_slices / add_tile_axis) restated in numpy: every access inside the tile, every
element of the chain covered once, and the result the separable filter."""
import numpy as np
import pytest

RADICES = [16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2]


def factors(n):
    for want in range(1, 5):
        best = None

        def search(rest, most, cur):
            nonlocal best
            if len(cur) == want:
                if rest == 1 and (best is None or sum(cur) < sum(best)):
                    best = list(cur)
                return
            for r in RADICES:
                if r <= most and rest % r == 0:
                    search(rest // r, r, cur + [r])
        search(n, 16, [])
        if best:
            return best
    return None


def fast_div(x, d):
    """x / d by the reciprocal ceil(2^32 / d), as FastDiv."""
    m = (0xFFFFFFFF // d + 1) if d > 1 else 0
    x = np.asarray(x, np.uint64)
    return ((x * np.uint64(m)) >> np.uint64(32)).astype(np.int64) if m else x.astype(np.int64)


def order(n, fac):
    """Frequency at each position after the forward passes."""
    out = np.zeros(n, int)
    for i in range(n):
        rest, L, w = i, n, 1
        for r in fac:
            L //= r
            out[i] += rest // L * w
            rest %= L
            w *= r
    return out


class Lines:
    def __init__(self, rows, cols, PZ, n, I, along):
        self.n, self.PZ, self.I, self.cols, self.along = n, PZ, I, cols, along
        self.NL = rows if along else rows * cols // n
        self.es = 1 if along else PZ * (I // cols)

    def base(self, l):
        if self.along:
            return l * self.PZ
        hi = fast_div(l, self.I)
        lo = l - hi * self.I
        y = fast_div(lo, self.cols) if self.I > self.cols else 0
        return hi * self.n * self.es + y * (self.PZ - self.cols) + lo


def run_pass(t, g, R, kind, L, S, tw, f=None, fo=None):
    NB = g.NL * (g.n // R)
    b = np.arange(NB)
    j = fast_div(b, g.NL)
    l = b - j * g.NL
    blk = j if kind == "mid" else fast_div(j, S)
    k = 0 * j if kind == "mid" else j - blk * S
    p = g.base(l) + (blk * L + k) * g.es
    idx = p[:, None] + np.arange(R)[None, :] * (S * g.es)
    assert idx.min() >= 0 and idx.max() < t.size and np.unique(idx).size == idx.size
    v = t[idx]
    q = np.arange(R)
    w = tw[(q[None, :] * k[:, None] * (g.n // L))] if S > 1 else 1.0
    if kind == "dif":
        v = np.fft.fft(v, axis=1) * w
    elif kind == "dit":
        v = np.fft.ifft(v * np.conj(w), axis=1) * R
    else:
        h = f[blk[:, None] * R + q[None, :]] + (fo[l][:, None] if fo is not None else 0)
        v = np.fft.ifft(np.fft.fft(v, axis=1) * h, axis=1) * R
    t[idx] = v


def forward(t, g, fac, tw, whole):
    L = g.n
    for R in fac if whole else fac[:-1]:
        run_pass(t, g, R, "dif", L, L // R, tw)
        L //= R


def inverse(t, g, fac, tw, whole):
    S = 1 if whole else fac[-1]
    for R in reversed(fac if whole else fac[:-1]):
        run_pass(t, g, R, "dit", S * R, S, tw)
        S *= R


def run_tile(block, rows, cols, PZ, axes, energy):
    """axes: (n, I, along, filter); block: rows x cols, returned filtered."""
    t = np.full(rows * PZ + 1, np.nan, complex)
    addr = np.arange(rows)[:, None] * PZ + np.arange(cols)[None, :]
    t[addr] = block
    geo = [(Lines(rows, cols, PZ, n, I, along), factors(n), np.exp(-2j * np.pi * np.arange(n) / n), f[order(n, factors(n))])
           for n, I, along, f in axes]
    if not energy or len(geo) == 1:
        for g, fac, tw, f in geo:
            forward(t, g, fac, tw, False)
            run_pass(t, g, fac[-1], "mid", fac[-1], 1, tw, f)
            inverse(t, g, fac, tw, False)
    else:
        for g, fac, tw, f in geo[:-1]:
            forward(t, g, fac, tw, True)
        r = np.arange(rows)
        fo = sum(f[r // (g.I // cols) % g.n] for g, fac, tw, f in geo[:-1])
        g, fac, tw, f = geo[-1]
        assert g.along
        forward(t, g, fac, tw, False)
        run_pass(t, g, fac[-1], "mid", fac[-1], 1, tw, f, fo)
        inverse(t, g, fac, tw, False)
        for g, fac, tw, f in reversed(geo[:-1]):
            inverse(t, g, fac, tw, True)
    return t[addr]


def axis_filter(x, a, f):
    s = [1] * x.ndim
    s[a] = f.size
    return np.fft.ifft(np.fft.fft(x, axis=a) * f.reshape(s), axis=a)


def test_every_length_has_a_plan():
    for n in {2 ** a * 3 ** b * 5 ** c for a in range(12) for b in range(8) for c in range(5)}:
        if 2 <= n <= 2048:
            fac = factors(n)
            assert fac and np.prod(fac) == n and len(fac) <= 4
            assert sorted(order(n, fac)) == list(range(n))


@pytest.mark.parametrize("energy", [False, True])
@pytest.mark.parametrize("dims", [(60,), (2,), (135,), (30, 30), (24, 20), (8, 6, 4), (20, 1, 15), (2, 2)])
def test_whole_slices(dims, energy):
    rng = np.random.default_rng(1)
    ns = max(1, 400 // int(np.prod(dims)))
    x = rng.standard_normal((ns,) + dims) + 1j * rng.standard_normal((ns,) + dims)
    last = max(a for a in range(len(dims)) if dims[a] > 1)
    cols = dims[last]
    axes, want = [], np.zeros_like(x) if energy else x
    for a, n in enumerate(dims):
        if n == 1:
            continue
        f = rng.random(n)
        I = int(np.prod(dims[a + 1:]))
        axes.append((n, I, I == 1, f))
        want = want + axis_filter(x, a + 1, f) if energy else axis_filter(want, a + 1, f)
    total = np.prod([n for n, _, _, _ in axes])
    scaled = [(n, I, al, f / (total if energy else n)) for n, I, al, f in axes]
    rows = ns * int(np.prod(dims)) // cols
    got = run_tile(x.reshape(rows, cols), rows, cols, cols | 1, scaled, energy)
    assert np.max(np.abs(got.reshape(x.shape) - want)) < 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("n,inner,target", [(48, 1440, 4096), (100, 81, 2048), (20, 270, 4096), (16, 7, 4096), (500, 4, 2048)])
def test_strided_tiles(n, inner, target):
    rng = np.random.default_rng(2)
    hi = 2
    x = rng.standard_normal((hi, n, inner)) + 1j * rng.standard_normal((hi, n, inner))
    f = rng.random(n)
    W = target // n
    W = min(W // 16 * 16 if W >= 16 else (8 if W >= 8 else 4), inner)
    out, seen = np.zeros(x.size, complex), np.zeros(x.size, int)
    flat = x.reshape(-1)
    for h in range(hi):
        for l in range(0, inner, W):
            cols = min(W, inner - l)
            g = h * n * inner + l + np.arange(n)[:, None] * inner + np.arange(cols)[None, :]
            out[g] = run_tile(flat[g], n, cols, W | 1, [(n, cols, False, f / n)], False)
            seen[g] += 1
    assert np.all(seen == 1)
    want = axis_filter(x, 1, f)
    assert np.max(np.abs(out.reshape(x.shape) - want)) < 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("V,nt,L", [(60, 25, 4), (900, 50, 7), (1, 9, 2), (256, 32, 32), (600, 3, 1)])
def test_flattened_step_tasks_cover_every_site(V, nt, L):
    """k_tiled.cu: thread flat = flat0 + tid is site flat mod V of chunk flat / V."""
    nchunk = -(-nt // L)
    ntile = -(-V * nchunk // 256)
    assert ntile <= -(-V * nt // 256)          # the partials' capacity
    seen = np.zeros((nt, V), int)
    for flat in range(256 * ntile):
        k, s = divmod(flat, V)
        if k < nchunk:
            seen[nt * k // nchunk:nt * (k + 1) // nchunk, s] += 1
    assert np.all(seen == 1)
