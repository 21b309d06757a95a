"""The tiled path without memory for kinbar: chains stepped in windows of as many as kin holds twice,
with the bits of the step that holds all at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def clv():
    import cl_var_dt_gb300 as m
    m.build()
    return m


def batch(clv, model):
    shapes = [dict(nx=60, nt=25), dict(nx=30, ny=30, nt=5), dict(nx=64, ny=64, nt=3), dict(nx=500, nt=9),
              dict(nx=48, ny=16, nz=16, nt=3), dict(nx=100, ny=128, nt=2), dict(nx=8, ny=6, nz=4, nt=9), dict(nx=96, ny=96, nt=2)]
    if model == "ref4":
        return [clv.ChainParams(**s, eps=0.02, G=0.1, Q=0.02, P=0.05, mu=-0.5 + 0.05 * i, DT=0.002, seed=3 + i)
                for i, s in enumerate(shapes)]
    # (a small K rejects the speculative step of every other chain)
    return [clv.ChainParams(**s, eps=0.05, mu=0.4 + 0.1 * i, c0=0.3, c1=-0.05, q=0.02, K=0.05 if i % 2 else 1e-4, dt_max=1e-3,
                            seed=3 + i) for i, s in enumerate(shapes)]


def run(clv, chains, model, prec, tune=False):
    out = {}
    with clv.Engine(chains, model=clv.MODEL_REF4 if model == "ref4" else clv.MODEL_SPIN1,
                    precision=clv.PREC_F64 if prec == "f64" else clv.PREC_F32) as e:
        assert e.plan()[0] == "tiled"
        rng = np.random.default_rng(2)
        for i in range(len(chains)):
            f = 0.5 + 0.2 * (rng.standard_normal(e.shape(i)) + 1j * rng.standard_normal(e.shape(i)))
            e.set_fields(i, f, np.conj(f))
        out["bytes"] = e.device_bytes()
        e.step(3)
        e.evaluate()
        if tune:
            e.autotune(1)
        e.step_with_noise(rng.standard_normal(2 * sum(int(np.prod(e.shape(i))) for i in range(len(chains)))))
        out["phases"] = len(e.step_timed()), len(e.plan()[1])
        out["late"] = e.device_bytes()
        out["fields"] = [e.get_fields(i) for i in range(len(chains))]
        out["info"] = e.step_info()
        out["obs"] = [e.ref_observables(i) if model == "ref4" else e.spin1_samples(i) for i in range(len(chains))]
        out["elems"] = sum(int(np.prod(e.shape(i))) for i in range(len(chains))) * (16 if prec == "f64" else 8)
    return out


def same(a, b):
    for (x, xc), (y, yc) in zip(a["fields"], b["fields"]):
        assert np.array_equal(x, y) and np.array_equal(xc, yc)
    for k in a["info"]:
        assert np.array_equal(a["info"][k], b["info"][k]), k
    for x, y in zip(a["obs"], b["obs"]):
        assert all(np.array_equal(p, q) for p, q in zip(x, y))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("model", ["spin1", "ref4"])
@pytest.mark.parametrize("stored", [None, "0"])
def test_windows_give_the_same_bits(clv, monkeypatch, model, prec, stored):
    monkeypatch.setenv("CLV_CHUNK", "4")     # the order of the mean's sums
    if stored:
        monkeypatch.setenv("CLV_STORE_DRIFT", stored)
    chains = batch(clv, model)
    a = run(clv, chains, model, prec)
    monkeypatch.setenv("CLV_TEST_NO_KINBAR", "1")
    b = run(clv, chains, model, prec)
    same(a, b)
    assert a["phases"][0] == a["phases"][1] == b["phases"][0] == b["phases"][1]
    assert a["bytes"] - b["bytes"] == a["elems"]
    monkeypatch.setenv("CLV_TEST_NO_KINBAR", "2")   # given back for the injected noise
    c = run(clv, chains, model, prec)
    same(a, c)
    assert c["bytes"] == a["bytes"] and c["late"] == a["late"] - a["elems"]


def test_kinbar_given_back_for_the_autotuner(clv, monkeypatch):
    chains = batch(clv, "spin1")
    a = run(clv, chains, "spin1", "f64", tune=True)
    monkeypatch.setenv("CLV_TEST_NO_KINBAR", "2")
    b = run(clv, chains, "spin1", "f64", tune=True)
    same(a, b)
    assert b["late"] == a["late"] - a["elems"]


def test_a_chain_of_more_than_half_needs_its_kinbar(clv, monkeypatch):
    """Refused with the allocation's error, and the next engine works."""
    c = batch(clv, "spin1")[:1]
    monkeypatch.setenv("CLV_TEST_NO_KINBAR", "1")
    with pytest.raises(Exception, match="kinbar"):
        clv.Engine(c, model=clv.MODEL_SPIN1)
    monkeypatch.delenv("CLV_TEST_NO_KINBAR")
    with clv.Engine(c, model=clv.MODEL_SPIN1) as e:
        e.init_spin1()
        e.step(2)


# (the second: large enough for the normals to be drawn in the reduce pass, on up to 152 SMs)
@pytest.mark.parametrize("shape", [dict(nx=60, nt=25), dict(nx=128, ny=128, nt=39)], ids=["small", "drawn"])
def test_a_chain_of_more_than_half_gives_its_stored_drift(clv, monkeypatch, shape):
    c = [clv.ChainParams(**shape, eps=0.02, G=0.1, Q=0.02, P=0.05, mu=-0.5, DT=0.002, seed=3)]
    a = run(clv, c, "ref4", "f64")
    monkeypatch.setenv("CLV_TEST_NO_KINBAR", "1")
    b = run(clv, c, "ref4", "f64")
    same(a, b)
    assert a["bytes"] - b["bytes"] > 1.9 * a["elems"]    # (16 bytes stay in the arrays' place or none)
