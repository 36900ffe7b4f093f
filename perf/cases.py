"""Performance cases: what a partial-wave fit asks of this library.

A fit of an amplitude model evaluates the likelihood and its gradient hundreds
of times over fixed samples (phase space, data, subtracted background) and takes
the exact Hessian at its minimum, or at every step of a Newton fit. Toy studies
repeat this for many small samples, so the analysis object itself is built again
and again, and its per-event intensities drive the accept-reject draw. Every
case is one such call through the public API.

A case is a dict: `op` (the call), `model` (a bundled workload model), the
sample sizes `n_phsp`, `n_data`, `n_bkg`, and `precision` ("fp64", the default
of the API, or "mixed").

``exact`` restates the models in plain torch FP64 (helicity sums of spinless
three-body decays), with gradients and Hessians by autograd; the inputs are
drawn with it as well, so they depend on the seed alone.
"""
from __future__ import annotations

import itertools
import math
import os
import tempfile

import numpy as np
import torch

import ctpwa_b200
from ctpwa_b200 import workloads


def listed():
    def case(name, op, model, n_phsp, n_data, n_bkg, precision="fp64"):
        return dict(name=name, op=op, model=model, n_phsp=n_phsp, n_data=n_data, n_bkg=n_bkg, precision=precision)

    return [
        # one evaluation of the single-resonance model at its benchmark size: the smallest fit, all latency
        case("nll_rho", "nll", "pipi_rho", 200_000, 20_000, 0),
        # one evaluation inside the native fit driver of a small toy fit: parameters in and result out through
        # host memory, ragged sample sizes
        case("host_3rho_toy_mixed", "host", "pipi_3rho", 100_003, 10_007, 1_001, "mixed"),
        # identical final-state particles (every amplitude a sum over their exchange), an ordinary size
        case("nll_ksks", "nll", "ksks", 1_000_000, 100_000, 0),
        # the three-chain model at its benchmark size: getNLL and autograd, as the drop-in user calls it
        case("nll_3rho", "nll", "pipi_3rho", 5_000_000, 500_000, 50_000),
        # an ordinary mixed-form fit, sizes off every tile
        case("nll_3rho_mixed", "nll", "pipi_3rho", 1_234_567, 123_457, 12_347, "mixed"),
        # the headline evaluation in both forms: 11.1 million events, 7 amplitudes, 9 free resonance parameters
        case("nll_kkpi", "nll", "kkpi", 10_000_000, 1_000_000, 100_000),
        case("nll_kkpi_mixed", "nll", "kkpi", 10_000_000, 1_000_000, 100_000, "mixed"),
        # the Hessian that ends every toy fit, and the one of the full fit (the largest case)
        case("hessian_3rho_toy", "hessian", "pipi_3rho", 1_000_000, 100_000, 10_000),
        case("hessian_kkpi", "hessian", "kkpi", 10_000_000, 1_000_000, 100_000),
        # a toy job's set-up: the analysis over events already on the GPU, and its first evaluation
        case("create_3rho", "create", "pipi_3rho", 1_000_000, 100_000, 10_000, "mixed"),
        # intensities of accept-reject candidates
        case("intensity_kkpi", "intensity", "kkpi", 1_000, 1_210_000, 0),
        # the start of a fit at fixed resonance parameters: the normalisation matrices and an evaluation from them
        case("fixed_kkpi", "fixed", "kkpi", 10_000_000, 1_000_000, 100_000, "mixed"),
    ]


def draw(rng):
    """A case of the same ranges: toy jobs of 10k data events up to the benchmark size of the model, sizes log-uniform."""
    op = rng.choice(("nll", "nll", "nll", "host", "hessian", "create", "intensity", "fixed"))
    model = rng.choice(("pipi_rho", "pipi_3rho", "pipi_3rho", "kkpi", "kkpi", "ksks"))
    top = {"pipi_rho": 500_000, "pipi_3rho": 500_000, "kkpi": 1_000_000, "ksks": 300_000}[model]
    n_data = int(math.exp(rng.uniform(math.log(5_000), math.log(top))))
    n_phsp = min(10 * top, int(n_data * rng.uniform(3.0, 10.0)))
    n_bkg = int(n_data * rng.uniform(0.02, 0.1)) if rng.random() < 0.6 else 0
    if op == "intensity":
        n_phsp, n_data, n_bkg = 1_000, int(n_data * rng.uniform(1.0, 4.0)), 0
    precision = "fp64" if op in ("hessian", "intensity") else rng.choice(("fp64", "mixed"))
    return dict(op=op, model=model, n_phsp=n_phsp, n_data=n_data, n_bkg=n_bkg, precision=precision)


# --------------------------------------------------------------------------- inputs

_DEV = "cuda"
_BKG_WEIGHT = {"pipi_rho": 0.5, "pipi_3rho": 0.8, "kkpi": 0.3, "ksks": 0.5}
_CHUNK = 1 << 19
_tmp = None


def _config(case):
    """config.yml of the model; its Data entries name no files that are read."""
    global _tmp
    if _tmp is None:
        _tmp = tempfile.TemporaryDirectory(prefix="ctpwa_cases_")
    path = os.path.join(_tmp.name, case["model"] + ("_bkg" if case["n_bkg"] else "") + ".yml")
    if not os.path.exists(path):
        with open(path, "w") as f:
            f.write(workloads.config_text(case["model"], "in-memory-phsp", "in-memory-data"))
    return path


def _phase_space(model, n, gen):
    """Uniform three-body phase space [n, 3, 4] (E, px, py, pz) in the rest frame of the parent."""
    M, (m1, m2, m3) = workloads.M_JPSI, workloads.MASSES[model]
    f64 = dict(dtype=torch.float64, device=_DEV)

    def brk(m, a, b):
        return torch.sqrt(torch.clamp((m * m - (a + b) ** 2) * (m * m - (a - b) ** 2), min=0.0)) / (2.0 * m)

    def direction(k):
        c = torch.rand(k, generator=gen, **f64) * 2.0 - 1.0
        phi = torch.rand(k, generator=gen, **f64) * (2.0 * math.pi)
        s = torch.sqrt(1.0 - c * c)
        return torch.stack([s * torch.cos(phi), s * torch.sin(phi), c], dim=1)

    lo, hi = m1 + m2, M - m3
    grid = torch.linspace(lo, hi, 20001, **f64)[1:-1]
    top = 1.02 * (brk(M, grid, m3) * brk(grid, m1, m2)).max()
    out, have = [], 0
    while have < n:
        k = min(4 * _CHUNK, int((n - have) * 1.8) + 4096)
        m12 = lo + (hi - lo) * torch.rand(k, generator=gen, **f64)
        m12 = m12[torch.rand(k, generator=gen, **f64) * top < brk(M, m12, m3) * brk(m12, m1, m2)]
        k = m12.numel()
        q3, q12, d3, d1 = brk(M, m12, m3), brk(m12, m1, m2), direction(k), direction(k)
        beta = d3 * (q3 / torch.sqrt(m12 * m12 + q3 * q3))[:, None]
        gamma = torch.sqrt(m12 * m12 + q3 * q3) / m12

        def boost(m, sign):
            e, p = torch.sqrt(m * m + q12 * q12), sign * q12[:, None] * d1
            bp = (beta * p).sum(1)
            return torch.cat([(gamma * (e + bp))[:, None],
                              p + (gamma * gamma / (gamma + 1.0) * bp + gamma * e)[:, None] * beta], dim=1)

        p3 = torch.cat([torch.sqrt(m3 * m3 + q3 * q3)[:, None], -q3[:, None] * d3], dim=1)
        out.append(torch.stack([boost(m1, 1.0), boost(m2, -1.0), p3], dim=1))
        have += k
    return torch.cat(out)[:n].contiguous()


def _signal(model, n, p, gen):
    """n events drawn against the model's intensity at the parameters p."""
    top, out, have = None, [], 0
    while have < n:
        cand = _phase_space(model, _CHUNK, gen)
        with torch.no_grad():
            f = _intensity(model, _Events(model, cand), p)
        top = 1.2 * f.max() if top is None else top
        out.append(cand[torch.rand(f.numel(), generator=gen, dtype=torch.float64, device=_DEV) * top < f])
        have += out[-1].shape[0]
    return torch.cat(out)[:n]


def _inputs(case, seed):
    """Samples, background weights and the point of evaluation: couplings of a seeded truth, the data drawn there
    (with the background events that the background sample subtracts), the parameters some steps away from it."""
    model = case["model"]
    gen = torch.Generator(device=_DEV)
    gen.manual_seed(1_000_003 * (seed + 1) + 17)
    rng = np.random.default_rng(7_000 + seed)
    nV, theta = _MODELS[model]["n_amp"], np.array(_MODELS[model]["theta"])
    mag, phase = rng.uniform(0.1, 1.0, nV), rng.uniform(0.0, 2.0 * math.pi, nV)
    mag[0], phase[0] = 1.0, 0.0
    truth = np.concatenate([mag * np.cos(phase), mag * np.sin(phase), theta])
    step = np.concatenate([rng.uniform(-0.05, 0.05, 2 * nV), theta * rng.uniform(-0.02, 0.02, theta.size)])
    truth_t = torch.tensor(truth, dtype=torch.float64, device=_DEV)
    p = torch.tensor(truth + step, dtype=torch.float64, device=_DEV)
    phsp = _phase_space(model, case["n_phsp"], gen)
    if case["op"] == "intensity":
        return dict(p=p, phsp=phsp, data=_phase_space(model, case["n_data"], gen), bkg=None, wb=None)
    nb, wb = case["n_bkg"], _BKG_WEIGHT[model]
    n_in = round(wb * nb)
    data = _signal(model, case["n_data"] - n_in, truth_t, gen)
    if n_in:
        data = torch.cat([data, _phase_space(model, n_in, gen)])
    bkg = _phase_space(model, nb, gen) if nb else None
    return dict(p=p, phsp=phsp, data=data, bkg=bkg,
                wb=torch.full((nb,), wb, dtype=torch.float64, device=_DEV) if nb else None)


# --------------------------------------------------------------------------- the measured calls


def _analysis(case, x):
    weights = [None, None, x["wb"]] if x["wb"] is not None else None
    return ctpwa_b200.analysis.from_device(_config(case), x["phsp"], x["data"], x["bkg"], weights=weights,
                                           precision=case["precision"])


def prepare(case, seed):
    x = _inputs(case, seed)
    state = dict(op=case["op"], case=case, p=x["p"])
    if case["op"] == "create":
        state["x"] = x
        return state
    state["ana"] = _analysis(case, x)
    if case["op"] == "nll":
        state["p"].requires_grad_(True)
    if case["op"] == "host":
        state["p"] = x["p"].cpu().numpy()
    return state


def run(state):
    op, p = state["op"], state["p"]
    if op == "create":
        return _analysis(state["case"], state["x"]).getNLLAndGrad(p)
    ana = state["ana"]
    if op == "nll":
        nll = ana.getNLL(p)
        (grad,) = torch.autograd.grad(nll, p)
        return nll.detach(), grad
    if op == "host":
        return ana.getNLLHost(p)
    if op == "hessian":
        return ana.getHessian(p)
    if op == "intensity":
        return ana.getIntensity(p, kind=1)
    if op == "fixed":
        ana.cacheNormalisation(p)
        return ana.getNLLAndGrad(p, cached=True)
    raise ValueError(op)


def work(case):
    """Bytes: the angular values of one helicity per conjugate pair (and the unpaired one) and the invariant masses of
    every event once (momenta for the set-up), FP64 or FP32. Flops: lineshapes with the derivatives that the call
    needs, coherent sums, the adjoint."""
    m = _MODELS[case["model"]]
    size = 4 if case["precision"] == "mixed" else 8
    n = case["n_phsp"] + case["n_data"] + case["n_bkg"]
    terms, planes, nP = len(m["terms"]), m["planes"], 2 * m["n_amp"] + len(m["theta"])
    per = planes * 2 * 2 * size + m["masses"] * size
    value = terms * (20 + 8 * 3) + planes * 24
    grad = value + terms * (8 + 2 * 20)
    if case["op"] == "intensity":
        n = case["n_data"]
        return {"bytes": float(n * (per + 8)), "flops": float(n * value)}
    if case["op"] == "hessian":
        # rank-1 updates of a symmetric nP x nP matrix: Re and Im of three helicities and the gradient
        return {"bytes": float(n * per), "flops": float(n * (grad + terms * 60 + 7 * nP * (nP + 1)))}
    if case["op"] == "create":
        return {"bytes": float(n * (96 + 2 * per)), "flops": float(n * (grad + planes * 400))}
    if case["op"] == "fixed":
        # FP64 quadratic forms over phase space, one evaluation over the rest
        d = case["n_data"] + case["n_bkg"]
        per64 = planes * 2 * 2 * 8 + m["masses"] * 8
        forms = 8 * terms * (terms + 2 * len(m["theta"]))
        return {"bytes": float(case["n_phsp"] * per64 + d * per),
                "flops": float(case["n_phsp"] * (grad + forms) + d * grad)}
    return {"bytes": float(n * per), "flops": float(n * grad)}


def tolerance(case):
    # FP64: sums of up to 10^7 terms that partly cancel, in another order (against exact: up to 3e-13). Mixed: FP32
    # lineshapes and angular values, the error of the gradient an unbiased walk (against exact: up to 6e-7, in the
    # gradient of small samples).
    return {"rel": 5e-6} if case["precision"] == "mixed" else {"rel": 5e-12}


# --------------------------------------------------------------------------- plain torch FP64 restatement

# terms: (amplitude, bachelor, daughter 1, daughter 2, spin, index of the first resonance parameter, lineshape);
# the final-state particles by their index in Data.order
_BW, _FLATTE = "bwr", "flatte"
_RHO = [0.775, 0.149, 1.465, 0.400, 1.720, 0.250]
_MODELS = {
    "pipi_rho": dict(n_amp=1, theta=_RHO[:2], planes=1, masses=1, terms=[(0, 2, 0, 1, 1, 0, _BW)]),
    "pipi_3rho": dict(n_amp=9, theta=_RHO, planes=3, masses=3,
                      terms=[(3 * c + r, b, i, j, 1, 2 * r, _BW)
                             for c, (b, i, j) in enumerate(((2, 0, 1), (1, 0, 2), (0, 1, 2))) for r in range(3)]),
    "kkpi": dict(n_amp=7, theta=[0.8955, 0.047, 1.414, 0.232, 1.4256, 0.0985, 1.68, 0.3, 0.1], planes=5, masses=3,
                 terms=[(3 * c + r, b, i, j, (1, 1, 2)[r], 2 * r, _BW)
                        for c, (b, i, j) in enumerate(((1, 0, 2), (0, 1, 2))) for r in range(3)]
                 + [(6, 2, 0, 1, 1, 6, _FLATTE)]),
    "ksks": dict(n_amp=2, theta=[0.8955, 0.047, 1.5174, 0.086], planes=4, masses=3,
                 terms=[(0, 1, 0, 2, 1, 0, _BW), (0, 0, 1, 2, 1, 0, _BW), (1, 2, 0, 1, 2, 2, _BW),
                        (1, 2, 1, 0, 2, 2, _BW)]),
}


def _clebsch(j1, m1, j2, m2, J, M):
    """<j1 m1 j2 m2 | J M> for integer spins (Racah's formula)."""
    if m1 + m2 != M or abs(m1) > j1 or abs(m2) > j2 or abs(M) > J:
        return 0.0
    f = math.factorial
    a = math.sqrt((2 * J + 1) * f(j1 + j2 - J) * f(j1 - j2 + J) * f(-j1 + j2 + J) / f(j1 + j2 + J + 1))
    b = math.sqrt(f(J + M) * f(J - M) * f(j1 - m1) * f(j1 + m1) * f(j2 - m2) * f(j2 + m2))
    s = 0.0
    for k in range(max(0, j2 - J - m1, j1 - J + m2), min(j1 + j2 - J, j1 - m1, j2 + m2) + 1):
        s += (-1) ** k / (f(k) * f(j1 + j2 - J - k) * f(j1 - m1 - k) * f(j2 + m2 - k) * f(J - j2 + m1 + k)
                          * f(J - j1 - m2 + k))
    return a * b * s


def _harmonic(l, m, d):
    """Y_l^m(theta, -phi) of the unit vectors d [n, 3]."""
    x, y, z = d[:, 0], d[:, 1], d[:, 2]
    w = torch.complex(x, -y if m >= 0 else y) ** abs(m)
    if l == 1:
        poly = {0: math.sqrt(3 / (4 * math.pi)) * z, 1: math.sqrt(3 / (8 * math.pi)) * torch.ones_like(z)}[abs(m)]
    else:
        poly = {0: math.sqrt(5 / (16 * math.pi)) * (3 * z * z - 1), 1: math.sqrt(15 / (8 * math.pi)) * z,
                2: math.sqrt(15 / (32 * math.pi)) * torch.ones_like(z)}[abs(m)]
    return w * poly * (-1.0 if m > 0 and m % 2 else 1.0)


def _mass2(p):
    return p[:, 0] ** 2 - (p[:, 1:] ** 2).sum(1)


def _frame(p1, p2):
    """Direction and momentum of p1 in the rest frame of p1 + p2."""
    P = p1 + p2
    m = torch.sqrt(_mass2(P))
    a = ((P[:, 1:] * p1[:, 1:]).sum(1) / (P[:, 0] + m) - p1[:, 0]) / m
    k = p1[:, 1:] + a[:, None] * P[:, 1:]
    q = torch.sqrt((k * k).sum(1))
    return k / q[:, None], q


class _Events:
    """Parameter-independent values of a sample: per topology the angular amplitude of each helicity, the masses."""

    def __init__(self, model, p4):
        self.n = p4.shape[0]
        self.sl, self.kin = {}, {}
        for _, b, i, j, spin, _, _ in _MODELS[model]["terms"]:
            if (b, i, j, spin) in self.sl:
                continue
            pb, pi, pj = p4[:, b], p4[:, i], p4[:, j]
            pr = pi + pj
            d1, q1 = _frame(pb, pr)
            d2, q2 = _frame(pi, pj)
            top = {m: _harmonic(spin, m, d1) for m in range(-spin, spin + 1)}
            dec = {s: _harmonic(spin, s, d2) for s in range(-spin, spin + 1)}
            norm = 100.0 * (q1 ** spin) * (q2 ** spin) / math.sqrt(3.0 * (2 * spin + 1))
            self.sl[b, i, j, spin] = torch.stack(
                [norm * sum(_clebsch(spin, s, spin, M - s, 1, M) * top[M - s] * dec[s]
                            for s in range(-spin, spin + 1) if abs(M - s) <= spin) for M in (1, 0, -1)])
            self.kin[b, i, j, spin] = (torch.sqrt(_mass2(pr)), q1, q2)


def _barrier(spin, z2):
    return 1.0 + z2 if spin == 1 else 9.0 + 3.0 * z2 + z2 * z2


def _q2(m, a, b):
    return (m * m - (a + b) ** 2) * (m * m - (a - b) ** 2) / (4.0 * m * m)


def _lineshape(model, term, ev, theta):
    _, b, i, j, spin, k, kind = term
    masses = workloads.MASSES[model]
    m, q1, q2 = ev.kin[b, i, j, spin]
    m0 = theta[k]
    d2 = 9.0  # radius 3 / GeV squared
    q0, q01 = _q2(m0, masses[i], masses[j]), _q2(torch.as_tensor(workloads.M_JPSI, dtype=torch.float64), masses[b], m0)
    bf2 = _barrier(spin, q0 * d2) / _barrier(spin, q2 * q2 * d2)
    bf = torch.sqrt(bf2 * _barrier(spin, q01 * d2) / _barrier(spin, q1 * q1 * d2))
    x = m0 * m0 - m * m
    if kind == _BW:
        gamma = theta[k + 1] * (q2 * q2 / q0) ** spin * (q2 / torch.sqrt(q0)) * (m0 / m) * bf2
        y = m0 * gamma
    else:
        s, y, g = m * m, 0.0, 0.0
        for c, mc in enumerate((0.493677, 0.13957)):
            f1 = 1.0 - 4.0 * mc * mc / s
            rho = torch.sqrt(f1.abs())
            y = y + theta[k + 1 + c] * 0.5 * m0 * torch.where(f1 >= 0, rho, torch.zeros_like(rho))
            g = g + theta[k + 1 + c] * 0.5 * m0 * torch.where(f1 < 0, rho, torch.zeros_like(rho))
        x = x + g
    return torch.complex(x, y) * (bf / (x * x + y * y))


def _intensity(model, ev, p):
    M = _MODELS[model]
    nV = M["n_amp"]
    v, theta = torch.complex(p[:nV], p[nV:2 * nV]), p[2 * nV:]
    S = 0.0
    for key, terms in itertools.groupby(M["terms"], key=lambda t: t[1:5]):
        F = 0.0
        for t in terms:
            F = F + v[t[0]] * _lineshape(model, t, ev, theta)
        S = S + F[None] * ev.sl[key]
    return (S.real ** 2 + S.imag ** 2).sum(0)


def _sums(model, p4, w, p, log, order):
    """Sum over the events of w log f (log) or f, with its gradient and, for order 2, its Hessian."""
    P = p.numel()
    val, grad = torch.zeros((), dtype=torch.float64, device=_DEV), torch.zeros(P, dtype=torch.float64, device=_DEV)
    hess = torch.zeros((P, P), dtype=torch.float64, device=_DEV)
    for e0 in range(0, p4.shape[0], _CHUNK):
        ev = _Events(model, p4[e0:e0 + _CHUNK])
        q = p.detach().clone().requires_grad_(True)
        f = _intensity(model, ev, q)
        s = (torch.log(f) if w is None else w[e0:e0 + _CHUNK] * torch.log(f)).sum() if log else f.sum()
        (g,) = torch.autograd.grad(s, q, create_graph=order > 1)
        val += s.detach()
        grad += g.detach()
        if order > 1:
            for i in range(P):
                hess[i] += torch.autograd.grad(g[i], q, retain_graph=i + 1 < P)[0]
    return val, grad, hess


def exact(case, seed):
    x = _inputs(case, seed)
    model, p = case["model"], x["p"]
    if case["op"] == "intensity":
        with torch.no_grad():
            return torch.cat([_intensity(model, _Events(model, x["data"][e:e + _CHUNK]), p)
                              for e in range(0, case["n_data"], _CHUNK)])
    order = 2 if case["op"] == "hessian" else 1
    nd, wb = case["n_data"], float(x["wb"].sum()) if x["wb"] is not None else 0.0
    d = _sums(model, x["data"], None, p, True, order)
    f = _sums(model, x["phsp"], None, p, False, order)
    r = f[1] / f[0]
    nll = -d[0] + (nd - wb) * torch.log(f[0] / case["n_phsp"])
    grad = -d[1] + (nd - wb) * r
    hess = -d[2] + (nd - wb) * (f[2] / f[0] - torch.outer(r, r))
    if x["bkg"] is not None:
        b = _sums(model, x["bkg"], x["wb"], p, True, order)
        nll, grad, hess = nll + b[0], grad + b[1], hess + b[2]
    if order == 2:
        return hess
    return (float(nll), grad.cpu().numpy()) if case["op"] == "host" else (nll, grad)
