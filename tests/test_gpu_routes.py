"""Forms of the step chosen by size: planes of 32 to 128 and their energies, the next plane
prefetched, normals drawn in the reduce pass, two CTAs an SM at FP64, slices per tile of long
lines, 1D batches on the tiled path, and the reference observables' chunks.  Each against the
FP64 oracle (1e-12 FP64, 1e-5 FP32 a step, the engine's parity bounds) or, where the oracle
would take long, against the separate-kernel path, which has the same bounds: twice them."""
import numpy as np
import pytest
from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-12, "f32": 1e-5}


@pytest.fixture(scope="module")
def clv():
    import cl_var_dt_gb300 as m
    m.build()
    return m


@pytest.fixture(autouse=True)
def clean_env(monkeypatch):
    for k in ("CLV_FUSED", "CLV_TILED", "CLV_NO_TMA", "CLV_NO_SPECULATE", "CLV_CHUNK", "CLV_NO_PLANE",
              "CLV_NO_STATIC_PLAN", "CLV_NO_LOOP", "CLV_STORE_DRIFT"):
        monkeypatch.delenv(k, raising=False)


def spin1(clv, **kw):
    base = dict(nx=64, ny=1, nz=1, nt=6, eps=0.05, mu=0.8, c0=0.3, c1=-0.05, q=0.02, K=0.05, dt_max=1e-3, seed=12)
    base.update(kw)
    return clv.ChainParams(**base)


def ref4(clv, **kw):
    base = dict(nx=64, nt=16, eps=0.01, mu=-0.5, G=0.15, Q=0.02, P=0.1, DT=0.002, seed=3)
    base.update(kw)
    return clv.ChainParams(**base)


def prec_of(clv, prec):
    return clv.PREC_F64 if prec == "f64" else clv.PREC_F32


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(32, 32, 1, 3), (64, 64, 1, 2), (96, 96, 1, 2), (128, 128, 1, 27), (3, 32, 32, 3),
                                   (2, 64, 64, 2), (3, 96, 96, 2), (2, 128, 128, 2)], ids=str)
def test_planes_step_and_energies(clv, oracle, shape, prec):
    # (128 x 128 x 27: 162 planes of a launch, more than the SMs)
    c = spin1(clv, nx=shape[0], ny=shape[1], nz=shape[2], nt=shape[3])
    p = oracle.spin1_params(nx=c.nx, ny=c.ny, nz=c.nz, nt=c.nt, eps=c.eps, mu=c.mu, c0=c.c0, c1=c.c1, q=c.q, Kc=c.K,
                            dt_max=c.dt_max)
    with clv.Engine(c, model=clv.MODEL_SPIN1, precision=prec_of(clv, prec)) as e:
        e.init_spin1()
        psi, psic = oracle.spin1_init(p, c.seed, 0)
        e.step(1)
        psi, psic, _, _, _ = oracle.step(p, psi, psic, seed=c.seed, chain=0, step_index=0)
        gp, gc = e.get_fields(0)
        assert rel_err(gp, psi) < TOL[prec] and rel_err(gc, psic) < TOL[prec]
        e.evaluate()
        want, got = oracle.spin1_observables(p, gp, gc), e.spin1_samples(0)[0]
        assert np.max(np.abs(got - want)) < TOL[prec] * max(1.0, float(np.max(np.abs(want))))


def one_step(clv, chains, model, prec, start):
    with clv.Engine(chains, model=model, precision=prec_of(clv, prec)) as e:
        if model == clv.MODEL_SPIN1:
            e.init_spin1()
        else:
            for i, (a, b) in enumerate(start):
                e.set_fields(i, a, b)
        e.step(1)
        return [e.get_fields(i) for i in range(len(chains))], e.step_info(), e.plan()


def start_of(chains):
    rng = np.random.default_rng(8)
    out = []
    for c in chains:
        sh = (4, c.nt, c.nx, c.ny, c.nz)
        a = 0.4 + 0.2 * (rng.standard_normal(sh) + 1j * rng.standard_normal(sh))
        out.append((a, np.conj(a) + 0.05 * rng.standard_normal(sh)))
    return out


def against_separate_kernels(clv, monkeypatch, chains, model, prec, path):
    start = start_of(chains) if model == clv.MODEL_REF4 else None
    got, gi, plan = one_step(clv, chains, model, prec, start)
    monkeypatch.setenv("CLV_FUSED", "0")
    monkeypatch.setenv("CLV_TILED", "0")
    want, wi, other = one_step(clv, chains, model, prec, start)
    assert plan[0] == path and other[0] == "unfused", (plan, other)
    assert np.allclose(gi["dt"], wi["dt"], rtol=2 * TOL[prec], atol=0)
    for (a, b), (c, d) in zip(got, want):
        assert rel_err(a, c) < 2 * TOL[prec] and rel_err(b, d) < 2 * TOL[prec]


# 16 blocks of 256 sites an SM and more on up to 152 SMs: the reduce pass draws the normals;
# a spatial size that is not a multiple of 256, and several chains
@pytest.mark.parametrize("shapes", [[(128, 128, 39)], [(50, 30, 200), (27, 25, 300), (128, 64, 20)]], ids=str)
def test_normals_drawn_in_the_reduce_pass(clv, monkeypatch, shapes):
    chains = [ref4(clv, nx=x, ny=y, nt=t, mu=-0.5 + 0.1 * i, seed=5 + i) for i, (x, y, t) in enumerate(shapes)]
    against_separate_kernels(clv, monkeypatch, chains, clv.MODEL_REF4, "f64", "tiled")


def test_drawn_normals_give_the_update_kernels_bits(clv, monkeypatch):
    """A chain whose last block of 128 sites is partly empty (20 x 27 sites, 127 times), alone (the
    update draws its normals) and beside a chain that fills the GPU (the reduce pass draws them)."""
    monkeypatch.setenv("CLV_CHUNK", "8")   # the mean's order of summation
    small, large = ref4(clv, nx=20, ny=27, nt=127), ref4(clv, nx=128, ny=128, nt=48, seed=9)
    start = start_of([small, large])
    alone, ai, _ = one_step(clv, [small], clv.MODEL_REF4, "f64", start[:1])
    both, bi, _ = one_step(clv, [small, large], clv.MODEL_REF4, "f64", start)
    assert ai["dt"][0] == bi["dt"][0]
    assert np.array_equal(alone[0][0], both[0][0]) and np.array_equal(alone[0][1], both[0][1])


def test_fp64_spin1_with_two_ctas_an_sm_tiled(clv, monkeypatch):
    chains = [spin1(clv, nx=27, ny=20, nt=64 + i, mu=0.5 + 0.1 * i, seed=5 + i) for i in range(10)]
    against_separate_kernels(clv, monkeypatch, chains, clv.MODEL_SPIN1, "f64", "tiled")


# more chunks than SMs (two CTAs an SM, lines in place) and fewer
@pytest.mark.parametrize("nx", [64, 128, 256])
@pytest.mark.parametrize("count", [5, 3])
def test_fp64_spin1_fused_forms(clv, monkeypatch, nx, count):
    chains = [spin1(clv, nx=nx, nt=33, mu=0.5 + 0.1 * i, seed=5 + i) for i in range(count)]
    against_separate_kernels(clv, monkeypatch, chains, clv.MODEL_SPIN1, "f64", "fused")


@pytest.mark.parametrize("model,prec,nx,count,nt", [("ref4", "f32", 64, 3, 33), ("ref4", "f32", 256, 5, 17),
                                                    ("ref4", "f64", 64, 30, 65), ("ref4", "f64", 256, 8, 64),
                                                    ("spin1", "f64", 64, 30, 65), ("spin1", "f32", 64, 100, 101)])
def test_1d_batches_on_the_tiled_path(clv, monkeypatch, model, prec, nx, count, nt):
    make, m = (ref4, clv.MODEL_REF4) if model == "ref4" else (spin1, clv.MODEL_SPIN1)
    chains = [make(clv, nx=nx, nt=nt, seed=5 + i) for i in range(count)]
    against_separate_kernels(clv, monkeypatch, chains, m, prec, "tiled")
    monkeypatch.delenv("CLV_TILED")
    monkeypatch.setenv("CLV_FUSED", "1")
    with clv.Engine(chains, model=m, precision=prec_of(clv, prec)) as e:
        assert e.plan()[0] == "fused"


# one to four slices a tile, with a remainder, at 128 and 256 threads
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("nx,count,nt", [(1536, 1, 65), (1152, 20, 31), (960, 2, 5), (1500, 4, 33)])
def test_slices_per_tile_of_long_lines(clv, monkeypatch, nx, count, nt, prec):
    chains = [spin1(clv, nx=nx, nt=nt, seed=5 + i) for i in range(count)]
    against_separate_kernels(clv, monkeypatch, chains, clv.MODEL_SPIN1, prec, "tiled")


@pytest.mark.parametrize("nx,ny,nt", [(64, 1, 2), (60, 1, 9), (30, 9, 17), (128, 1, 100)])
def test_reference_observables_by_chunks(clv, oracle, nx, ny, nt):
    c = ref4(clv, nx=nx, ny=ny, nt=nt)
    with clv.Engine(c, model=clv.MODEL_REF4, precision=clv.PREC_F64) as e:
        (a, b), = start_of([c])
        e.set_fields(0, a, b)
        e.evaluate()
        n, F = e.ref_observables(0)
    p = oracle.Params(nx=nx, ny=ny, nz=1, nt=nt, ncomp=4, eps=c.eps, a_x=c.a_x, mu=c.mu, P=c.P, Q=c.Q, G=c.G)
    want_F, want_n = oracle.ref_observables(p, a, b)
    # (the engine reports means over the imaginary times, and over the sites for the densities)
    assert rel_err(n, want_n / nt / (nx * ny)) < TOL["f64"] and rel_err(F, want_F / nt) < TOL["f64"]


# few pairs (a thread per imaginary time) with chunks that end inside a CTA, and streaming
@pytest.mark.parametrize("nx,ny,nt", [(64, 1, 16), (30, 1, 25), (24, 9, 33), (128, 128, 40)])
def test_spin1_samples_at_fp32(clv, oracle, nx, ny, nt):
    c = spin1(clv, nx=nx, ny=ny, nt=nt)
    p = oracle.spin1_params(nx=nx, ny=ny, nt=nt, eps=c.eps, mu=c.mu, c0=c.c0, c1=c.c1, q=c.q, Kc=c.K, dt_max=c.dt_max)
    with clv.Engine(c, model=clv.MODEL_SPIN1, precision=clv.PREC_F32) as e:
        e.init_spin1()
        e.evaluate()
        psi, psic = e.get_fields(0)
        want, got = oracle.spin1_observables(p, psi, psic), e.spin1_samples(0)[0]
    assert np.max(np.abs(got - want)) < TOL["f32"] * max(1.0, float(np.max(np.abs(want))))


# a thread sums all imaginary times of its site (one chunk)
@pytest.mark.parametrize("nt,kind", [(24, "condensate"), (64, "random")])
def test_reference_profiles_round_once_a_time(clv, nt, kind):
    """F_x, F_y, F_z against extended precision.  A running sum over nt times rounds once a time
    at its own size: a variance of u^2 / 3 times its square, u = 2^-53, which for a random walk
    adds up to nt / 6 of the result's (a condensate's sum: nt / 9); a time's eight products add
    8 / 3 of their own."""
    c = ref4(clv, nx=300, ny=270, nt=nt)
    rng = np.random.default_rng(4)
    amp = 0.4 if kind == "condensate" else 0.0
    a, b = (amp + 0.2 * (rng.standard_normal((4, nt, 300, 270, 1)) + 1j * rng.standard_normal((4, nt, 300, 270, 1)))
            for _ in range(2))
    with clv.Engine(c, model=clv.MODEL_REF4, precision=clv.PREC_F64) as e:
        e.set_fields(0, a, b)
        e.evaluate()
        n, F = e.ref_observables(0)
    sites = rng.choice(300 * 270, 4000, replace=False)
    k = a.reshape(4, nt, -1)[:, :, sites].astype(np.clongdouble)
    m = np.roll(b.reshape(4, nt, -1)[:, :, sites].astype(np.clongdouble), -1, 1)
    t20, t02, t31, t13 = m[2] * k[0], m[0] * k[2], m[3] * k[1], m[1] * k[3]
    d = m * k
    want = np.stack([(t20 + t02 + t31 + t13).real, -(t20 - t02 + t31 - t13).imag, (d[0] + d[1] - d[2] - d[3]).real]).sum(1)
    err = F.reshape(3, -1)[:, sites] * np.longdouble(nt) - want
    rms = np.sqrt((err ** 2).sum(1) / (want ** 2).sum(1)).astype(float)
    # (the mean over the times divides once more: another third)
    assert np.all(rms < 2.0 ** -53 * np.sqrt(nt / 6 + 9 / 3)), rms


def test_spin1_sample_does_not_depend_on_the_batch(clv):
    """A chain's FP32 sample alone, in a batch of 0.5 and of 1.5 million sites: the same FP32 sums
    of 16 imaginary times, added in FP64 (5 000 of them: 5 000 2^-53 of the sum of magnitudes at
    the very most)."""
    c = spin1(clv, nx=60, nt=50)
    rng = np.random.default_rng(6)
    f = 0.6 + 0.1 * (rng.standard_normal((3, 50, 60, 1, 1)) + 1j * rng.standard_normal((3, 50, 60, 1, 1)))
    got = []
    for more in (0, 7, 23):
        with clv.Engine([c] + [spin1(clv, nx=512, nt=128, seed=i) for i in range(more)], model=clv.MODEL_SPIN1,
                        precision=clv.PREC_F32) as e:
            e.init_spin1()
            e.set_fields(0, f, np.conj(f))
            e.evaluate()
            got.append(e.spin1_samples(0)[0])
    for g in got[1:]:
        assert np.max(np.abs(g - got[0])) < 1e-12 * np.max(np.abs(got[0])), (got[0], g)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_engines_of_several_threads(clv, prec):
    """Engines whose tiles differ in size, created, stepped and closed by four threads at once."""
    from concurrent.futures import ThreadPoolExecutor

    shapes = [dict(nx=60, nt=6), dict(nx=48, ny=20, nt=3), dict(nx=600, nt=3), dict(nx=100, ny=81, nt=2)]

    def work(k):
        out = []
        for r in range(12):
            c = spin1(clv, seed=7 + k, **shapes[(k + r * (k % 2)) % 4])
            with clv.Engine(c, model=clv.MODEL_SPIN1, precision=prec_of(clv, prec)) as e:
                e.init_spin1()
                e.step(2)
                out.append(e.get_fields(0)[0])
        return out

    want = [work(k) for k in range(4)]
    with ThreadPoolExecutor(4) as pool:
        got = list(pool.map(work, range(4)))
    for a, b in zip(want, got):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))


def test_the_sizes_above_take_the_forms_they_are_for():
    """plan() names the path, not the form: the sizes of this file against the thresholds of
    clv_engine.cu in blocks of 256 sites an SM (16: normals in the reduce pass, 8: two CTAs an SM,
    3: FP64 lines on the tiled path; more chunks of 33 times than SMs for the fused form)."""
    sms = pytest.importorskip("torch").cuda.get_device_properties(0).multi_processor_count
    per_sm = lambda sites: sites // 256 / sms
    assert per_sm(128 * 128 * 39) >= 16 and per_sm(50 * 30 * 200 + 27 * 25 * 300 + 128 * 64 * 20) >= 16
    assert per_sm(20 * 27 * 127) < 8 and per_sm(20 * 27 * 127 + 128 * 128 * 48) >= 16
    assert 8 <= per_sm(27 * 20 * sum(64 + i for i in range(10)))
    assert 5 * 33 > sms > 3 * 33
    assert per_sm(30 * 64 * 65) >= 3 and per_sm(8 * 256 * 64) >= 3 and per_sm(100 * 64 * 101) >= 16
