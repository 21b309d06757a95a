"""The tile filter (csrc/k_tile.cuh) and the flattened step tasks: lines of every radix,
whole small slices, strided and contiguous tiles with remainders, mixed batches; steps and
observables against the FP64 oracle."""
import numpy as np
import pytest
from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def clv():
    import cl_var_dt_gb300 as m
    m.build()
    return m


def spin1(clv, **kw):
    base = dict(nx=60, ny=1, nz=1, nt=6, eps=0.05, mu=0.8, c0=0.3, c1=-0.05, q=0.02, K=0.05, dt_max=1e-3, seed=12)
    base.update(kw)
    return clv.ChainParams(**base)


def oracle_params(oracle, c):
    return oracle.spin1_params(nx=c.nx, ny=c.ny, nz=c.nz, nt=c.nt, eps=c.eps, mu=c.mu, c0=c.c0, c1=c.c1, q=c.q,
                               Kc=c.K, dt_max=c.dt_max)


# every radix alone and in two and three passes; slices of one and several per tile; tiles
# of lines with remainders (a last strided tile of one column: 81 = 5 x 16 + 1 at FP64)
SHAPES = [dict(nx=n, nt=5) for n in (2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 25, 27, 30, 45, 48, 50, 60, 81, 90,
                                     100, 135, 144, 150, 200, 225, 240, 250, 360, 375, 400, 480, 500)] + [
    dict(nx=30, ny=30, nt=7), dict(nx=24, ny=20, nt=5), dict(nx=2, ny=2, nt=2), dict(nx=100, ny=81, nt=2),
    dict(nx=100, ny=100, nt=2), dict(nx=8, ny=6, nz=4, nt=9), dict(nx=20, ny=18, nz=15, nt=3),
    dict(nx=6, ny=1, nz=10, nt=4), dict(nx=48, ny=20, nz=15, nt=2), dict(nx=3, ny=160, nz=50, nt=2)]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda d: "x".join(str(v) for v in d.values()))
def test_spin1_step_and_observables(clv, oracle, shape, prec):
    c = spin1(clv, **shape)
    p = oracle_params(oracle, c)
    tol = 1e-12 if prec == "f64" else 1e-5
    with clv.Engine(c, model=clv.MODEL_SPIN1, precision=clv.PREC_F64 if prec == "f64" else clv.PREC_F32) as e:
        assert e.plan()[0] == "tiled"
        e.init_spin1()
        psi, psic = oracle.spin1_init(p, c.seed, 0)
        e.step(1)
        psi, psic, dt, _, _ = oracle.step(p, psi, psic, seed=c.seed, chain=0, step_index=0)
        gp, gc = e.get_fields(0)
        assert rel_err(gp, psi) < tol and rel_err(gc, psic) < tol
        assert abs(e.step_info()["dt"][0] - dt) <= tol * dt
        e.evaluate()
        want, got = oracle.spin1_observables(p, gp, gc), e.spin1_samples(0)[0]
        assert np.max(np.abs(got - want)) < tol * max(1.0, float(np.max(np.abs(want))))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("chunk", [None, "1", "4"])
def test_mixed_batch(clv, oracle, monkeypatch, prec, chunk):
    """Shapes of different kinds in one engine; chains whose (chunk, site) pairs end inside a CTA."""
    if chunk:
        monkeypatch.setenv("CLV_CHUNK", chunk)
    shapes = [dict(nx=60, nt=25), dict(nx=128, nt=8), dict(nx=30, ny=30, nt=5), dict(nx=24, ny=20, nt=9),
              dict(nx=500, nt=3), dict(nx=64, ny=64, nt=2), dict(nx=100, ny=128, nt=2), dict(nx=2, nt=2)]
    chains = [spin1(clv, mu=0.4 + 0.1 * i, seed=3 + i, **s) for i, s in enumerate(shapes)]
    tol = 1e-12 if prec == "f64" else 1e-5
    with clv.Engine(chains, model=clv.MODEL_SPIN1, precision=clv.PREC_F64 if prec == "f64" else clv.PREC_F32) as e:
        e.init_spin1()
        e.step(1)
        for i, c in enumerate(chains):
            p = oracle_params(oracle, c)
            psi, psic = oracle.spin1_init(p, c.seed, i)
            psi, psic, _, _, _ = oracle.step(p, psi, psic, seed=c.seed, chain=i, step_index=0)
            gp, gc = e.get_fields(i)
            assert rel_err(gp, psi) < tol and rel_err(gc, psic) < tol, shapes[i]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [dict(nx=48, ny=10, nz=9, nt=4), dict(nx=90, nt=6), dict(nx=48, ny=40, nz=6, nt=2)],
                         ids=lambda d: "x".join(str(v) for v in d.values()))
def test_ref4_tile_filter_equals_line_filter(clv, monkeypatch, shape, prec):
    """The reference's kinetic term (x axis only) by the tile filter and by the separate
    line-filter, drift and update kernels."""
    c = clv.ChainParams(**shape, eps=0.02, a_x=1.0, G=0.1, Q=0.02, P=0.05, mu=-0.5, DT=0.002, seed=7)
    rng = np.random.default_rng(5)
    out = []
    for env in (None, "0"):
        if env:
            monkeypatch.setenv("CLV_FUSED", env)
            monkeypatch.setenv("CLV_TILED", env)
        with clv.Engine(c, model=clv.MODEL_REF4, precision=clv.PREC_F64 if prec == "f64" else clv.PREC_F32) as e:
            assert e.plan()[0] == ("unfused" if env else "tiled")
            if not out:
                f = (rng.standard_normal(e.shape(0)) + 1j * rng.standard_normal(e.shape(0))) * 0.3 + 0.5
            e.set_fields(0, f, np.conj(f))
            e.step(3)
            out.append(e.get_fields(0))
    tol = 1e-13 if prec == "f64" else 2e-6
    assert rel_err(out[0][0], out[1][0]) < tol and rel_err(out[0][1], out[1][1]) < tol


@pytest.mark.parametrize("kind", ["fluctuating", "one_site"])
@pytest.mark.parametrize("shape", [dict(nx=60, nt=8), dict(nx=128, ny=100, nt=2), dict(nx=30, ny=30, nt=4),
                                   dict(nx=243, nt=6), dict(nx=1500, nt=4), dict(nx=48, ny=20, nz=15, nt=2)],
                         ids=lambda d: "x".join(str(v) for v in d.values()))
def test_fp64_filter_to_rounding(clv, shape, kind):
    """The integer butterflies against long-double transforms: one step with dt = 1, no couplings
    and no noise gives psi + (kin(tau - 1) - psi).  The kinetic term, the drift and the sum
    are rounded once each (2^-53 of the field each), the transform adds 2^-55: 4e-16 in the
    2-norm."""
    fft = pytest.importorskip("scipy.fft")
    c = spin1(clv, **shape, mu=0.0, c0=0.0, c1=0.0, q=0.0, K=1e300, dt_max=1.0)
    rng = np.random.default_rng(3)
    with clv.Engine(c, model=clv.MODEL_SPIN1, precision=clv.PREC_F64) as e:
        f = (rng.standard_normal(e.shape(0)) + 1j * rng.standard_normal(e.shape(0))) * 0.3 + 0.5
        if kind == "one_site":
            f *= 1e-3
            f.reshape(3, c.nt, -1)[:, :, 5] = 3.0
        e.set_fields(0, f, np.conj(f))
        e.step_with_noise(np.zeros(2 * f.size))
        got = e.get_fields(0)[0]
    want = f.astype(np.clongdouble)
    for a, n in enumerate((c.nx, c.ny, c.nz)):
        if n > 1:
            k = np.arange(n)
            p = np.where(k < n // 2, 2 * np.pi * k / n, -2 * np.pi * (n - k) / n)
            s = [1] * 5
            s[2 + a] = n
            want = fft.ifft(fft.fft(want, axis=2 + a) * np.exp(-c.eps * 0.5 * p * p).reshape(s), axis=2 + a)
    want = np.roll(want, 1, 1)
    assert float(np.linalg.norm(np.abs(got - want).ravel().astype(float))) < \
        4e-16 * float(np.linalg.norm(np.abs(want).ravel().astype(float)))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("shape", [dict(nx=60, nt=6), dict(nx=30, ny=24, nt=4), dict(nx=100, ny=81, nt=2)],
                         ids=lambda d: "x".join(str(v) for v in d.values()))
def test_non_finite_field_flags_its_chain_only(clv, shape, bad, prec):
    chains = [spin1(clv, seed=3, **shape), spin1(clv, seed=4, **shape)]
    with clv.Engine(chains, model=clv.MODEL_SPIN1, precision=clv.PREC_F64 if prec == "f64" else clv.PREC_F32) as e:
        e.init_spin1()
        psi, psic = e.get_fields(0)
        e.step(1)
        want = e.get_fields(1)
        assert not any(e.chain_flags())
    with clv.Engine(chains, model=clv.MODEL_SPIN1, precision=clv.PREC_F64 if prec == "f64" else clv.PREC_F32) as e:
        e.init_spin1()
        psi[1, 1].flat[7] = bad
        e.set_fields(0, psi, psic)
        e.step(1)
        assert list(e.chain_flags()) == [1, 0]
        got = e.get_fields(1)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_zero_field_stays_zero(clv):
    """The reference's zero start: every line of the filter is zero."""
    c = clv.ChainParams(nx=60, ny=9, nt=6, eps=0.02, G=0.1, mu=-0.5, DT=0.002, seed=7)
    with clv.Engine(c, model=clv.MODEL_REF4, precision=clv.PREC_F64) as e:
        assert e.plan()[0] == "tiled"
        e.step_with_noise(np.zeros(2 * 4 * 60 * 9 * 6))
        assert all(np.all(f == 0) for f in e.get_fields(0)) and not any(e.chain_flags())


# lines of one to five radices at FP64, relative to their first site; strided tiles with a remainder;
# two-site lines, whose groups of a tile are the most there can be
@pytest.mark.parametrize("shape", [(2, 1, 1, 9), (48, 1, 1, 5), (729, 1, 1, 3), (810, 1, 1, 3), (900, 1, 1, 2), (1250, 1, 1, 2),
                                   (1875, 1, 1, 2), (2048, 1, 1, 2), (48, 20, 15, 2), (2, 60, 60, 2), (100, 81, 1, 2)], ids=str)
def test_ref4_kinetic_term_against_the_oracle(clv, oracle, shape):
    """(An odd extent has no momentum -k for its last one, so there the direction of the transform
    counts: the engine's is the oracle's for psibar and on the mirrored lattice for psi.)"""
    nx, ny, nz, nt = shape
    c = clv.ChainParams(nx=nx, ny=ny, nz=nz, nt=nt, eps=0.02, a_x=1.0, G=0.1, Q=0.02, P=0.05, mu=-0.5, DT=0.002, seed=7)
    p = oracle.Params(nx=nx, ny=ny, nz=nz, nt=nt, ncomp=4, eps=c.eps, a_x=c.a_x, mu=c.mu, P=c.P, Q=c.Q, G=c.G, DT=c.DT)
    rng = np.random.default_rng(5)
    with clv.Engine(c, model=clv.MODEL_REF4, precision=clv.PREC_F64) as e:
        f = 0.5 + 0.2 * (rng.standard_normal(e.shape(0)) + 1j * rng.standard_normal(e.shape(0)))
        e.set_fields(0, f, np.conj(f))
        zero = np.zeros(2 * f.size)
        e.step_with_noise(zero)
        gp, gc = e.get_fields(0)
        dt = e.step_info()["dt"][0]
    mirror = (lambda a: np.ascontiguousarray(np.roll(a[:, :, ::-1], 1, 2))) if nx % 2 else (lambda a: a)
    psi, psic, want, _, _ = oracle.step(p, mirror(f), mirror(np.conj(f)), noise=zero)
    assert abs(dt - want) <= 1e-12 * want
    assert rel_err(gp, mirror(psi)) < 1e-12
    if nx % 2 == 0:
        assert rel_err(gc, psic) < 1e-12


# kinetic energies of whole slices, summed over the axes at FP64, and axis by axis
@pytest.mark.parametrize("shape", [(729, 1, 1, 3), (1875, 1, 1, 2), (30, 30, 1, 5), (2, 2, 2, 9), (8, 6, 4, 5), (100, 81, 1, 2)],
                         ids=str)
def test_spin1_energies_at_fp64(clv, oracle, shape):
    c = spin1(clv, nx=shape[0], ny=shape[1], nz=shape[2], nt=shape[3])
    p = oracle_params(oracle, c)
    with clv.Engine(c, model=clv.MODEL_SPIN1, precision=clv.PREC_F64) as e:
        e.init_spin1()
        e.evaluate()
        psi, psic = e.get_fields(0)
        want, got = oracle.spin1_observables(p, psi, psic), e.spin1_samples(0)[0]
    assert np.max(np.abs(got - want)) < 1e-12 * max(1.0, float(np.max(np.abs(want))))


# the fused step's and its two-CTA form's lines (more chunks than SMs), and the step loop's
@pytest.mark.parametrize("kind", ["fluctuating", "one_site"])
@pytest.mark.parametrize("nx,count,nt", [(64, 1, 9), (128, 1, 9), (256, 1, 9), (64, 5, 40), (128, 5, 40), (256, 5, 40)])
def test_fp64_fused_lines_to_rounding(clv, nx, count, nt, kind):
    """As above for the lines of the fused kernels, and no site worse than the others: over the lines
    of the batch (81 at least) a site's root mean square scatters by 1 / 12 of itself, so the
    largest of 256 lies within five such steps."""
    fft = pytest.importorskip("scipy.fft")
    chains = [spin1(clv, nx=nx, nt=nt, mu=0.0, c0=0.0, c1=0.0, q=0.0, K=1e300, dt_max=1.0, seed=i) for i in range(count)]
    rng = np.random.default_rng(3)
    k = np.arange(nx)
    p = np.where(k < nx // 2, 2 * np.pi * k / nx, -2 * np.pi * (nx - k) / nx)
    err, size = [], 0.0
    with clv.Engine(chains, model=clv.MODEL_SPIN1, precision=clv.PREC_F64) as e:
        assert e.plan()[0] == "fused"
        fields = []
        for i in range(count):
            f = (rng.standard_normal(e.shape(i)) + 1j * rng.standard_normal(e.shape(i))) * 0.3 + 0.5
            if kind == "one_site":
                f *= 1e-3
                f[:, :, 5] = 3.0
            e.set_fields(i, f, np.conj(f))
            fields.append(f)
        e.step_with_noise(np.zeros(2 * sum(f.size for f in fields)))
        for i, f in enumerate(fields):
            got = e.get_fields(i)[0]
            want = fft.ifft(fft.fft(f.astype(np.clongdouble), axis=2) * np.exp(-0.05 * 0.5 * p * p).reshape(1, 1, nx, 1, 1), axis=2)
            want = np.roll(want, 1, 1)
            err.append(np.abs(got - want).astype(float).reshape(-1, nx))
            size += float((np.abs(want).astype(float) ** 2).sum())
    err = np.concatenate(err)
    assert np.sqrt((err ** 2).sum() / size) < 4e-16
    if kind == "fluctuating" and err.shape[0] >= 81:
        site = np.sqrt((err ** 2).mean(0))
        assert site.max() < 1.42 * np.sqrt((site ** 2).mean()), site.argmax()
