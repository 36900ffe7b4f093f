"""The one-pass Hessian sums (kernels/hessgram.cuh) against forward mode.

getHessian takes the one pass, getHessianVectorProduct along the unit
directions recomputes every event in dual numbers; both are FP64 sums of the
same terms, so they differ by rounding only: 1e-11 of the largest entry (the
bound the linearity test of the products uses)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _many_resonances(nres):
    """Three chains x nres resonances: 3 nres amplitudes, 2 nres free resonance parameters."""
    from ctpwa_b200 import workloads

    names = [f"r{i}" for i in range(nres)]
    txt = workloads.config_text("pipi_3rho", "p", "d")
    txt = txt[:txt.index("Resonances:")].replace("rho770, rho1450, rho1700", ", ".join(names))
    return txt + "Resonances:\n" + "".join(
        f"  {n}: {{J: 1, P: -1, model: BWR, parameters: [{0.8 + 0.13 * i:.3f}, {0.15 + 0.02 * i:.3f}], free: [0, 1]}}\n"
        for i, n in enumerate(names))


def _setup(tmp_path, text, masses, sizes, weights=(False, False, False), seed=1, few=()):
    """An analysis over phase-space samples, and its parameters. few: weights of the first data events."""
    import torch

    import ctpwa_b200
    from ctpwa_b200 import toymc, workloads

    cfg = tmp_path / "c.yml"
    cfg.write_text(text)
    rng = np.random.default_rng(seed)
    dev = "cuda:0"
    s = [torch.tensor(toymc.phase_space(workloads.M_JPSI, masses, n, 100 + seed + k), device=dev) if n else None
         for k, n in enumerate(sizes)]
    # signed weights: data and background events of negative weight enter with the opposite sign, zero drops out
    w = [torch.tensor(np.where(np.arange(n) % 7 == 3, 0.0, rng.uniform(0.5 if k == 0 else -0.4, 1.5, n)), device=dev)
         if use else None for k, (n, use) in enumerate(zip(sizes, weights))]
    if len(few):
        w[1][::5][:len(few)] = torch.tensor(few, dtype=torch.float64, device=dev)
    ana = ctpwa_b200.analysis.from_device(str(cfg), s[0], s[1], s[2], weights=w)
    p = torch.tensor(workloads.true_params(ana.getNVector(), ana.getFreeResParams()[0].numpy(), seed=seed) *
                     rng.uniform(0.97, 1.03, ana.getNParams()), device=dev)
    return ana, p


def _check(ana, p):
    import torch

    H = ana.getHessian(p)
    F = ana.getHessianVectorProduct(p, torch.eye(p.numel(), dtype=torch.float64, device=p.device))
    F = 0.5 * (F + F.T)
    assert torch.isfinite(F).all() and float(F.abs().max()) > 0
    assert float((H - F).abs().max()) <= 1e-11 * float(F.abs().max())
    assert torch.equal(H, ana.getHessian(p))  # fixed summation order


def _compare(tmp_path, text, masses, sizes, weights=(False, False, False), seed=1):
    _check(*_setup(tmp_path, text, masses, sizes, weights, seed))


@pytest.mark.parametrize("sizes", [(1, 1, 0), (31, 33, 1), (32, 32, 32), (129, 127, 63), (40_000, 4_001, 395)])
def test_tile_edges(tmp_path, sizes):
    from ctpwa_b200 import workloads

    _compare(tmp_path, workloads.config_text("kkpi", "p", "d"), workloads.MASSES["kkpi"], sizes)


@pytest.mark.parametrize("model", ["pipi_rho", "pipi_3rho", "ksks", "kkpi"])
@pytest.mark.parametrize("paired", [True, False])
def test_models_and_weights(tmp_path, monkeypatch, model, paired):
    from ctpwa_b200 import workloads

    if not paired:
        monkeypatch.setenv("CTPWA_NO_POL_PAIRING", "1")
    _compare(tmp_path, workloads.config_text(model, "p", "d"), workloads.MASSES[model], (3001, 517, 130),
             weights=(True, True, True), seed=3)


@pytest.mark.parametrize("nres", [6, 7])
def test_largest_matrix_and_beyond(tmp_path, nres):
    """48 rows, the largest matrix of the one-pass kernel, and 56, which takes forward mode."""
    from ctpwa_b200 import workloads

    _compare(tmp_path, _many_resonances(nres), workloads.MASSES["pipi_3rho"], (2000, 300, 40), seed=5)


def test_capture_of_the_first_call(tmp_path):
    """A first getHessian inside a graph capture, after products on the same handle, replays to the eager result."""
    import torch

    import ctpwa_b200
    from ctpwa_b200 import toymc, workloads

    cfg = tmp_path / "c.yml"
    cfg.write_text(workloads.config_text("pipi_rho", "p", "d"))
    s = [torch.tensor(toymc.phase_space(workloads.M_JPSI, workloads.MASSES["pipi_rho"], n, n), device="cuda:0")
         for n in (2000, 300)]
    ana = ctpwa_b200.analysis.from_device(str(cfg), *s)
    p = torch.tensor(workloads.true_params(ana.getNVector(), ana.getFreeResParams()[0].numpy()), device="cuda:0")
    ana.getHessianVectorProduct(p, torch.ones_like(p))
    ana.getNLL(p)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        H = ana.getHessian(p)
    p.mul_(1.01)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(H, ana.getHessian(p))


# Clamped events: components of w S / f beyond 1e10 count as constants. Weights
# of 1e12 clamp some of an event's components, 1e18 all of them.
CLAMPING = {"some": [1e12, -1e12, 3e12, 1e10, -2e11, 1e12], "all": [1e18, -1e18, 1e18, 1.0, 1e18]}


@pytest.mark.parametrize("few", list(CLAMPING))
@pytest.mark.parametrize("model", ["pipi_3rho", "ksks", "kkpi"])
@pytest.mark.parametrize("paired", [True, False])
def test_clamped_by_weight(tmp_path, monkeypatch, model, paired, few):
    from ctpwa_b200 import workloads

    if not paired:
        monkeypatch.setenv("CTPWA_NO_POL_PAIRING", "1")
    _check(*_setup(tmp_path, workloads.config_text(model, "p", "d"), workloads.MASSES[model], (1001, 217, 40),
                   weights=(False, True, False), seed=7, few=CLAMPING[few]))


@pytest.mark.parametrize("paired", [True, False])
def test_clamped_at_an_amplitude_zero(tmp_path, monkeypatch, paired):
    """One coupling set so that the amplitude of one data event vanishes to rounding: its S / f lies beyond 1e10 at
    unit weight, and what it would add to the Hessian unclamped is 1e20 times what the other events add."""
    import torch

    from ctpwa_b200 import workloads

    if not paired:
        monkeypatch.setenv("CTPWA_NO_POL_PAIRING", "1")
    ana, p = _setup(tmp_path, workloads.config_text("kkpi", "p", "d"), workloads.MASSES["kkpi"], (1001, 217, 40), seed=9)
    nV = ana.getNVector()

    def f(z):  # all amplitudes of one event share one angular vector: f = |A + z B|^2
        q = p.clone()
        q[1], q[nV + 1] = z.real, z.imag
        return float(ana.getIntensity(q, kind=1)[3])

    a, k, b = f(0j), f(1 + 0j), f(1j)
    bb = (f(1 + 0j) + f(-1 + 0j) - 2 * a) / 2  # |B|^2
    z = -complex(k - a - bb, b - a - bb) / (2 * bb)
    p[1], p[nV + 1] = z.real, z.imag
    assert f(z) < 1e-20 * a
    _check(ana, p)


def test_clamped_products_are_rows(tmp_path):
    """With clamped events the matrix of second derivatives is not symmetric. Only getHessian symmetrises it: the
    sums of a shard along several directions are those of each direction alone, and the resonance rows of the
    Gram-based Hessian are the products."""
    import torch

    from ctpwa_b200 import workloads

    ana, p = _setup(tmp_path, workloads.config_text("kkpi", "p", "d"), workloads.MASSES["kkpi"], (1001, 217, 40),
                    weights=(False, True, False), seed=7, few=CLAMPING["some"])
    n, nV = p.numel(), ana.getNVector()
    d = torch.tensor(np.random.default_rng(3).standard_normal((6, n)), device=p.device)
    for dirs in (d, torch.eye(n, dtype=torch.float64, device=p.device)):
        many = ana.getShardHvpSums(p, dirs).view(dirs.shape[0], -1)
        one = torch.stack([ana.getShardHvpSums(p, u[None]).view(-1) for u in dirs])
        assert float((many - one).abs().max()) <= 1e-11 * float(one.abs().max())
    rows = ana.getHessianVectorProduct(p, torch.eye(n, dtype=torch.float64, device=p.device))[2 * nV:]
    G = ana.getHessian(p, method="gram")[2 * nV:]
    assert float((rows[:, :2 * nV] - G[:, :2 * nV]).abs().max()) <= 1e-11 * float(rows.abs().max())


def test_many_polarisations(tmp_path):
    """27 polarisation states (a vector decaying to two vectors and a pseudoscalar), whose components a 32-bit mask
    does not hold: forward mode."""
    text = """Particles:
  Jpsi: {J: 1, P: -1, mass: 3.0969}
  V1:   {J: 1, P: -1, mass: 0.78265}
  V2:   {J: 1, P: -1, mass: 0.77526}
  pi0:  {J: 0, P: -1, mass: 0.13495}
Data:
  order: [V1, V2, pi0]
  data: [npy, "d"]
  phsp: [npy, "p"]
DecayChains:
  c:
    Jpsi: [[pi0, R]]
    R: [V1, V2]
    intermediates:
      R:
        - [J: 0, P: -1]: [eta1760, eta2225]
Resonances:
  eta1760: {J: 0, P: -1, model: BWR, parameters: [1.76, 0.24], free: [0, 1]}
  eta2225: {J: 0, P: -1, model: BWR, parameters: [2.22, 0.18], free: [0, 1]}
"""
    ana, p = _setup(tmp_path, text, (0.78265, 0.77526, 0.13495), (301, 97, 0), weights=(False, True, False), seed=7,
                    few=CLAMPING["some"])
    assert ana.getNPolarizations() == 27
    _check(ana, p)
