"""The work a user of this framework has it do, as cases with sizes, inputs and exact values.

A pass is a block of a run: n Langevin steps of every chain of an engine, one observable
evaluation, and the fields read back into the caller's device buffers (a snapshot or the
hand-over to the caller's own analysis).  Chains continue from pass to pass, as a run's do.

Kinds of chains: the reference's 4-component model under its own kinetic term and step rule
("ref4": the drop-in), and the spin-1 model with the exponential kinetic factor and the
K/max step rule ("spin1").  A case is

  model, precision ("f64" or "f32"), chains, dims, sides and nts (texts: what a chain's
  extents are picked from, by the chain's place in the batch), eps, steps per pass.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import cl_var_dt_gb300 as clv

STEP_K, DT_MAX = 0.05, 1e-3          # spin-1 step rule dt = min(dt_max, K / max|drift|)
DT, DT_MIN, DT_CLAMP, ALPHA = 0.002, 1e-8, 0.01, 0.9   # the reference's step rule
G, A_X = 0.1, 1.0


def listed():
    def case(name, model, precision, chains, dims, sides, nts, eps, steps):
        return dict(name=name, model=model, precision=precision, chains=chains, dims=dims, sides=sides, nts=nts,
                    eps=eps, steps=steps)

    return [
        # the plain FP64 single chain (64 sites, 64 imaginary times), observables every 10 steps:
        # the smallest run, bound by latencies
        case("single-f64-1d64", "spin1", "f64", 1, 1, "64", "64", 4 / 64, 10),
        # the reference program's shipped Parameters.h: 256 x 32, observables every 100 steps
        case("dropin-f64-1d256", "ref4", "f64", 1, 1, "256", "32", 0.01, 100),
        # the same model as a scan of chemical potentials at FP32, uneven lines
        case("scan-f32-ref4", "ref4", "f32", 48, 1, "128,200,256", "32,48,64", 0.01, 20),
        # the benchmark line: 256 chains of 256 sites, 128 imaginary times, FP32-mixed
        case("batch-f32-1d256", "spin1", "f32", 256, 1, "256", "128", 6 / 128, 10),
        # the same lattice in plain FP64, a batch of 32
        case("batch-f64-1d256", "spin1", "f64", 32, 1, "256", "128", 6 / 128, 5),
        # odd and ragged lines and small 2D slices in one batch (slices up to 1024 sites)
        case("ragged-f32-small", "spin1", "f32", 64, 0, "60x1,100x1,135x1,250x1,30x30,24x20,48x15,600x1",
             "25,50,96", 0.05, 10),
        # one 2D chain of 128 x 128 sites, observables every 20 steps
        case("plane-f32-2d128", "spin1", "f32", 1, 2, "128", "128", 8 / 128, 20),
        # density tuning: 64 uneven 2D chains
        case("uneven-f32-2d", "spin1", "f32", 64, 2, "32,64,96,128", "32,64,128,256", 0.05, 5),
        # one large 3D chain, 64^3 sites, 64 imaginary times
        case("cube-f32-3d64", "spin1", "f32", 1, 3, "64", "64", 4 / 64, 5),
        # the drop-in on a 2D lattice and on a ragged 3D one, FP64
        case("dropin-f64-2d128", "ref4", "f64", 1, 2, "128", "128", 0.0625, 2),
        case("dropin-f64-3d", "ref4", "f64", 1, 0, "48x40x36", "24", 0.0625, 4),
        # long lines, beyond the sizes of the tiled filters
        case("long-f32-1d", "spin1", "f32", 4, 1, "1500", "96", 0.05, 10),
    ]


# Sizes a lattice can have (products of 2, 3, 5).
_SMOOTH = sorted(a * b * c for a in (2 ** i for i in range(12)) for b in (1, 3, 9, 27) for c in (1, 5, 25)
                 if 8 <= a * b * c <= 2048)


def _near(rng, lo, hi):
    """A lattice extent, spread over the logarithm of [lo, hi]."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return rng.choice([n for n in _SMOOTH if lo <= n <= hi and abs(math.log(n / x)) < 0.35])


def draw(rng):
    model, precision = rng.choice([("spin1", "f32"), ("spin1", "f32"), ("spin1", "f64"), ("ref4", "f64"), ("ref4", "f32")])
    shape = rng.choice(["line", "line", "small", "plane", "square", "cube", "long"])
    chains = round(math.exp(rng.uniform(0, math.log(256))))
    nts = rng.sample([4, 10, 16, 25, 32, 48, 50, 64, 96, 100, 128, 256], 3)
    if shape == "line":
        dims, sides = 1, [_near(rng, 16, 512) for _ in range(rng.choice([1, 3]))]
        sides = [rng.choice([64, 128, 256])] if rng.random() < 0.4 else sides
    elif shape == "small":
        dims, sides = 0, ["%dx%d" % (_near(rng, 8, 32), _near(rng, 8, 32)) for _ in range(3)]
    elif shape == "plane":
        dims, sides = 0, ["%dx%d" % (_near(rng, 32, 256), _near(rng, 32, 160)) for _ in range(2)]
    elif shape == "square":
        dims, sides = 2, rng.sample([32, 48, 64, 96, 100, 128], rng.choice([1, 3]))
    elif shape == "cube":
        dims, sides = 0, ["%dx%dx%d" % (_near(rng, 8, 96), _near(rng, 8, 64), _near(rng, 8, 64))]
        sides = ["64x64x%d" % rng.choice([32, 64])] if rng.random() < 0.4 else sides
    else:
        dims, sides = 1, [_near(rng, 640, 2048)]
    case = dict(model=model, precision=precision, chains=chains, dims=dims, sides=",".join(map(str, sides)),
                nts=",".join(map(str, nts)), eps=round(rng.uniform(0.01, 0.0625), 4), steps=rng.choice([1, 2, 5, 10, 20]))
    # at most a ninth of the largest listed case's site-updates, FP64 ones counting forty times
    limit = 2 * 64 ** 4
    weight = 40 if precision == "f64" else 1

    def cost():
        return sum(np.prod(s, dtype=float) for s in _shapes(case)) * case["steps"] * weight

    while cost() > limit and case["chains"] > 1:
        case["chains"] = max(1, case["chains"] // 2)
    while cost() > limit and case["steps"] > 1:
        case["steps"] = max(1, case["steps"] // 2)
    while cost() > limit:
        case["nts"] = ",".join(str(max(4, int(n) // 2)) for n in case["nts"].split(","))
        if all(int(n) <= 4 for n in case["nts"].split(",")):
            break
    return case


def _shapes(case):
    """(nx, ny, nz, nt) of every chain."""
    r = random.Random(20261203)
    sides, nts = case["sides"].split(","), case["nts"].split(",")
    out = []
    for _ in range(case["chains"]):
        s = r.choice(sides)
        ext = [int(v) for v in s.split("x")] if case["dims"] == 0 else [int(s)] * case["dims"]
        out.append(tuple(ext + [1] * (3 - len(ext))) + (int(r.choice(nts)),))
    return out


def _params(case, seed):
    """Couplings of every chain: the ranges of the configurations, drawn from the seed."""
    r = random.Random(seed * 1000003 + 17)
    out = []
    for nx, ny, nz, nt in _shapes(case):
        c0 = r.uniform(0.2, 0.6)
        p = dict(nx=nx, ny=ny, nz=nz, nt=nt, eps=case["eps"], seed=r.getrandbits(63))
        if case["model"] == "ref4":
            p.update(mu=r.uniform(-1.5, -0.5), P=r.uniform(0, 0.1), Q=r.uniform(0, 0.05), G=G, a_x=A_X, DT=DT,
                     dt_min=DT_MIN, dt_max_clamp=DT_CLAMP, alpha=ALPHA)
        else:
            p.update(mu=c0 * r.uniform(0.5, 2.0), c0=c0, c1=r.uniform(-0.2, 0.1), q=r.uniform(0, 0.1), K=STEP_K, dt_max=DT_MAX)
        out.append(p)
    return out


def _ncomp(case):
    return 4 if case["model"] == "ref4" else 3


def _fields(case, seed):
    """psi and psibar of all chains, one after another in the [c][tau][x][y][z] layout: a
    condensate with fluctuations, psibar near psi's conjugate as on a chain under way."""
    n = sum(math.prod(s) for s in _shapes(case)) * _ncomp(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    real, kind = (torch.float64, torch.complex128) if case["precision"] == "f64" else (torch.float32, torch.complex64)
    amp, width = (math.sqrt(1 / 3), 0.1) if case["model"] == "spin1" else (0.4, 0.2)
    x = torch.randn(n, 2, generator=g, device="cuda", dtype=real) * width
    x[:, 0] += amp
    y = torch.randn(n, 2, generator=g, device="cuda", dtype=real) * (0.2 * width)
    psi = torch.view_as_complex(x)
    return psi, torch.conj_physical(psi) + torch.view_as_complex(y).to(kind)


def _where(case):
    return clv.DEVICE | (clv.C64 if case["precision"] == "f32" else 0)


def prepare(case, seed):
    chains = [clv.ChainParams(**p) for p in _params(case, seed)]
    e = clv.Engine(chains, model=clv.MODEL_REF4 if case["model"] == "ref4" else clv.MODEL_SPIN1,
                   precision=clv.PREC_F64 if case["precision"] == "f64" else clv.PREC_F32)
    psi, psic = _fields(case, seed)
    torch.cuda.synchronize()
    _check(clv.lib().clv_set_fields(e.h, -1, psi.data_ptr(), psic.data_ptr(), _where(case)))
    return dict(case=case, engine=e, psi=torch.empty_like(psi), psic=torch.empty_like(psic), sample=np.zeros(8))


def _check(rc):
    if rc:
        raise RuntimeError(clv.lib().clv_last_error().decode())


def run(state):
    e, case = state["engine"], state["case"]
    e.step(case["steps"])
    e.evaluate()
    out = dict(psi=state["psi"], psic=state["psic"])
    _check(clv.lib().clv_get_fields(e.h, -1, state["psi"].data_ptr(), state["psic"].data_ptr(), _where(case)))
    if case["chains"] == 1 and case["model"] == "ref4":
        # the drop-in reads its running means at every snapshot; a batch's samples stay on
        # the device and are read once, at the end of a run
        out["n"], out["F"] = e.ref_observables(0)
    elif case["chains"] == 1:
        # a monitor's fixed-size read: the sample of the run's first evaluation
        _check(clv.lib().clv_read_spin1_samples(e.h, 0, state["sample"].ctypes.data_as(C.POINTER(C.c_double)), 1, C.byref(C.c_int())))
        out["sample"] = state["sample"]
    return out


def work(case):
    """Every step reads both fields and writes them, all components, once; a state that the
    on-chip memory holds (128 MB) is read and written once a pass.  Operations: per
    component and field the transforms of the filtered axes, the filter and the update, the
    drift's products, and Box-Muller's transcendentals counted as 40."""
    c, comp = _ncomp(case), 16 if case["precision"] == "f64" else 8
    sites = sum(math.prod(s) for s in _shapes(case))
    state = 2 * c * comp * sites
    passes = case["steps"] if state > 128e6 else 1
    flops = 0.0
    for nx, ny, nz, nt in _shapes(case):
        axes = [nx] if case["model"] == "ref4" else [nx, ny, nz]
        per = 2 * c * (sum(10 * math.log2(n) + 2 for n in axes if n > 1) + 14) + (180 if c == 4 else 170) + 40 * c
        flops += per * nx * ny * nz * nt
    # the evaluation reads both fields once more, the read-back writes them once
    return {"bytes": 2.0 * state * passes + 2.0 * state, "flops": flops * case["steps"]}


# ------------------------------------------------- the same steps in 64 bits, plain torch
def _philox(c, k):
    """Philox4x32-10: c and k lists of int64 tensors or ints holding 32-bit words."""
    m = 0xFFFFFFFF
    for _ in range(10):
        p, q = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((q >> 32) & m) ^ c[1] ^ k[0], q & m, ((p >> 32) & m) ^ c[3] ^ k[1], p & m]
        k = [(k[0] + 0x9E3779B9) & m, (k[1] + 0xBB67AE85) & m]
    return c


def _normal(x, y):
    """Box-Muller of two words: u1 = (x + 1/2) 2^-32, u2 = y 2^-32."""
    r = torch.sqrt(-2.0 * torch.log((x.double() + 0.5) * 2.0 ** -32))
    o = ((y + (1 << 28)) >> 29) & 7                       # nearest multiple of pi/4
    a = (((y + (1 << 28)) & ((1 << 29) - 1)) - (1 << 28)).double() * (2 * math.pi * 2.0 ** -32)
    s, c, h = torch.sin(a), torch.cos(a), math.sqrt(0.5)
    co = torch.tensor([1, h, 0, -h, -1, -h, 0, h], dtype=torch.float64, device=x.device)[o]
    so = torch.tensor([0, h, 1, h, 0, -h, -1, -h], dtype=torch.float64, device=x.device)[o]
    return torch.complex(r * (co * c - so * s), r * (so * c + co * s))


def _noise(p, chain, step, ncomp, device):
    n = p["nx"] * p["ny"] * p["nz"] * p["nt"]
    site = torch.arange(n, dtype=torch.int64, device=device)
    key = [p["seed"] & 0xFFFFFFFF, p["seed"] >> 32]
    out = []
    for c in range(ncomp):
        lone = ncomp % 2 == 1 and c == ncomp - 1
        at = site >> 1 if lone else site
        zero = torch.zeros_like(at)
        w = _philox([at, zero + step, zero, zero + chain + ((c >> 1) << 24)], key)
        if lone:
            hi = (site & 1).bool()
            out.append(_normal(torch.where(hi, w[2], w[0]), torch.where(hi, w[3], w[1])))
        else:
            out.append(_normal(w[2], w[3]) if c & 1 else _normal(w[0], w[1]))
    return torch.stack(out)


def _momenta(n, device):
    k = np.arange(n)
    return torch.tensor(np.where(k < n // 2, 2 * np.pi * k / n, -2 * np.pi * (n - k) / n), device=device)


def _kinetic(p, model, f):
    if model == "ref4":
        k = _momenta(p["nx"], f.device).view(-1, 1, 1)
        return torch.fft.ifft(torch.fft.fft(f, dim=2) * (-(k * k) / p["a_x"]), dim=2)
    for a, n in enumerate((p["nx"], p["ny"], p["nz"])):
        if n > 1:
            k = _momenta(n, f.device)
            shape = [1] * 5
            shape[2 + a] = n
            f = torch.fft.ifft(torch.fft.fft(f, dim=2 + a) * torch.exp(-p["eps"] * 0.5 * k * k).view(shape), dim=2 + a)
    m2 = torch.tensor([1.0, 0.0, 1.0], dtype=torch.float64, device=f.device).view(3, 1, 1, 1, 1)
    return f * torch.exp(p["eps"] * (p["mu"] + p["q"] * m2))


def _drift(p, model, psi, psic):
    kin, kinc = _kinetic(p, model, psi), _kinetic(p, model, psic)
    prev, cur = lambda f: torch.roll(f, 1, 1), lambda f: f
    nxt = lambda f: torch.roll(f, -1, 1)
    if model == "ref4":
        mu = [p["mu"] + p["P"] + p["Q"], p["mu"], p["mu"], p["mu"] - p["P"] + p["Q"]]

        def contact(b, k, first):
            n = [b[a] * k[a] for a in range(4)]
            t = k if first else b                          # the field the term multiplies
            o = b if first else k
            return torch.stack([(n[0] + n[1] + n[2]) * t[0] + t[1] * o[3] * t[2], (n[0] + n[1] + n[3]) * t[1] + t[0] * o[2] * t[3],
                                (n[0] + n[2] + n[3]) * t[2] + t[3] * o[1] * t[0], (n[1] + n[2] + n[3]) * t[3] + t[2] * o[0] * t[1]])

        mus = torch.tensor(mu, dtype=torch.float64, device=psi.device).view(4, 1, 1, 1, 1)
        pm, cp = prev(psi), nxt(psic)
        K = p["a_x"] * (pm - psi + p["eps"] * (mus * pm - 2 * p["G"] * contact(psic, pm, True) + prev(kin)))
        Kc = p["a_x"] * (cp - psic + p["eps"] * (mus * nxt(psi) - 2 * p["G"] * contact(cp, psi, False) + nxt(kinc)))
        return K, Kc

    def pair(b, k):
        n = b[0] * k[0] + b[1] * k[1] + b[2] * k[2]
        return n, b[0] * k[0] - b[2] * k[2], b[0] * k[1] + b[1] * k[2], b[1] * k[0] + b[2] * k[1]

    e, c0, c1 = p["eps"], p["c0"], p["c1"]
    b, k = cur(psic), prev(psi)
    n, z, u, d = pair(b, k)
    K = prev(kin) - psi - e * (c0 * n * k + c1 * torch.stack([z * k[0] + d * k[1], u * k[0] + d * k[2], u * k[1] - z * k[2]]))
    b, k = nxt(psic), psi
    n, z, u, d = pair(b, k)
    Kc = nxt(kinc) - psic - e * (c0 * n * b + c1 * torch.stack([z * b[0] + u * b[1], d * b[0] + u * b[2], d * b[1] - z * b[2]]))
    return K, Kc


def _step_size(p, model, K, Kc):
    if model == "spin1":
        return min(p["dt_max"], p["K"] / max(float(K.abs().max()), float(Kc.abs().max())))
    a = K[0].abs()
    mean, most = float(a.sum()) / K.numel(), float(a.max())
    dt = min(max(mean / most * p["DT"] if most > 0 else p["DT"], p["dt_min"]), p["dt_max_clamp"])
    return (1 - p["alpha"]) * p["DT"] + p["alpha"] * dt


def _ref_observables(p, psi, psic):
    b, k = torch.roll(psic, -1, 1), psi
    d = [(b[a] * k[a]).real for a in range(4)]
    n = [float(x.sum()) * p["a_x"] / p["nt"] for x in d]
    t20, t02, t31, t13 = b[2] * k[0], b[0] * k[2], b[3] * k[1], b[1] * k[3]
    F = torch.stack([(t20 + t02 + t31 + t13).real, -(t20 - t02 + t31 - t13).imag, d[0] + d[1] - d[2] - d[3]])
    return np.array([sum(n)] + n), (F.sum(1) / p["nt"]).reshape(3, -1).cpu().numpy()


def _spin1_observables(p, psi, psic):
    b, k = torch.roll(psic, -1, 1), psi
    kinetic = torch.zeros_like(k)
    for a, n in enumerate((p["nx"], p["ny"], p["nz"])):
        if n > 1:
            shape = [1] * 5
            shape[2 + a] = n
            kinetic += torch.fft.ifft(torch.fft.fft(k, dim=2 + a) * (0.5 * _momenta(n, k.device) ** 2).view(shape), dim=2 + a)
    n = (b * k).sum(0)
    z = b[0] * k[0] - b[2] * k[2]
    f2 = z * z + 2 * (b[0] * k[1] + b[1] * k[2]) * (b[1] * k[0] + b[2] * k[1])
    energy = (b * kinetic).sum(0) - p["q"] * (b[0] * k[0] + b[2] * k[2]) + 0.5 * p["c0"] * n * n + 0.5 * p["c1"] * f2
    return np.array([v for x in (n, z, f2, energy) for v in (float(x.real.mean()), float(x.imag.mean()))])


def exact(case, seed):
    psi_all, psic_all = (f.to(torch.complex128) for f in _fields(case, seed))
    off, out, outc, obs = 0, [], [], {}
    for i, p in enumerate(_params(case, seed)):
        shape = (_ncomp(case), p["nt"], p["nx"], p["ny"], p["nz"])
        m = math.prod(shape)
        psi, psic = psi_all[off:off + m].reshape(shape), psic_all[off:off + m].reshape(shape)
        off += m
        for k in range(case["steps"]):
            K, Kc = _drift(p, case["model"], psi, psic)
            dt = _step_size(p, case["model"], K, Kc)
            z = _noise(p, i, k, shape[0], psi.device).reshape(shape) * math.sqrt(dt)
            psi, psic = psi + dt * K + z, psic + dt * Kc + z.conj()
        out.append(psi.reshape(-1))
        outc.append(psic.reshape(-1))
        if case["chains"] == 1 and case["model"] == "ref4":
            obs["n"], obs["F"] = _ref_observables(p, psi, psic)
        elif case["chains"] == 1:
            obs["sample"] = _spin1_observables(p, psi, psic)
    return dict(psi=torch.cat(out), psic=torch.cat(outc), **obs)
