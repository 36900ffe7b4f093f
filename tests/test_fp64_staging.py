"""The plain kernel's per-thread asynchronous copies and its table of reals
against direct loads and the full complex table, at sizes around a launch's
tiles, with and without weights: the same FP64 sums with, at most, another
rounding per event (1e-12 of the NLL, 1e-10 of the largest gradient entry, the
bounds of the other staging modes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(tmp_path, model, sizes, weighted):
    import torch
    from ctpwa_b200 import toymc, workloads

    cfg = tmp_path / "c.yml"
    cfg.write_text(workloads.config_text(model, "p", "d"))
    rng = np.random.default_rng(11)
    s = [torch.tensor(toymc.phase_space(workloads.M_JPSI, workloads.MASSES[model], n, 40 + k), device="cuda:0") if n else None
         for k, n in enumerate(sizes)]
    w = [torch.tensor(rng.uniform(0.2, 1.5, n), device="cuda:0") if weighted and n else None for n in sizes]
    return str(cfg), s, w


@pytest.mark.parametrize("model", ["pipi_rho", "pipi_3rho", "ksks", "kkpi"])
@pytest.mark.parametrize("sizes,weighted", [((1, 1, 0), False), ((191, 193, 1), True), ((56_833, 5_001, 385), False),
                                            ((170_003, 17_001, 1_003), True)])
def test_copies_and_reals_match_direct_loads(tmp_path, monkeypatch, model, sizes, weighted):
    import torch
    import ctpwa_b200
    from ctpwa_b200 import workloads

    cfg, s, w = _setup(tmp_path, model, sizes, weighted)

    def evaluate():
        ana = ctpwa_b200.analysis.from_device(cfg, s[0], s[1], s[2], weights=w)
        p = torch.tensor(workloads.true_params(ana.getNVector(), ana.getFreeResParams()[0].numpy()) * 1.01, device="cuda:0")
        n, g = ana.getNLLAndGrad(p)
        return ana.launchShape()["fp64"], float(n), g, ana.getIntensity(p, kind=1), ana.getNLLHost(p.cpu().numpy())

    shape, n1, g1, f1, (nh, gh) = evaluate()
    assert shape["pol_paired"] == 1 and shape["stage"] == 4, shape
    assert nh == n1 and np.array_equal(gh, g1.cpu().numpy())  # host-buffer path: the same launches
    monkeypatch.setenv("CTPWA_STAGE", "0")
    direct = evaluate()
    monkeypatch.setenv("CTPWA_NO_POL_PAIRING", "1")
    full = evaluate()
    assert direct[0]["stage"] == 0 and direct[0]["pol_paired"] == 1 and full[0]["pol_paired"] == 0
    for _, n0, g0, f0, _ in (direct, full):
        assert abs(n1 - n0) <= 1e-12 * max(1.0, abs(n0))
        assert float((g1 - g0).abs().max()) <= 1e-10 * float(g0.abs().max())
        assert float((f1 - f0).abs().max()) <= 1e-12 * float(f0.abs().max())


def test_two_of_three_polarisations(tmp_path):
    """m = +-1 only: pairs alone, no polarisation paired with itself; against the oracle's FP64 result."""
    import torch
    import ctpwa_b200
    from ctpwa_b200 import workloads
    from oracle.binding import Oracle

    cfg = workloads.make("kkpi", tmp_path, n_phsp=4001, n_data=700, n_bkg=0, accept_reject=False, seed=3, gpu_generator=False)
    text = open(cfg).read().replace("Jpsi: {J: 1, P: -1, mass: 3.0969}", "Jpsi: {J: 1, P: -1, mass: 3.0969, polarization: [1, -1]}")
    open(cfg, "w").write(text)
    ana = ctpwa_b200.analysis(cfg)
    assert ana.getNPolarizations() == 2 and ana.launchShape()["fp64"]["pol_paired"] == 1
    p = workloads.true_params(ana.getNVector(), ana.getFreeResParams()[0].numpy())
    n, g = ana.getNLLAndGrad(torch.tensor(p, device="cuda:0"))
    onll, og, _ = Oracle(cfg).nll_grad(p)
    assert abs(float(n) - onll) <= 1e-10 * abs(onll)
    assert np.max(np.abs(g.cpu().numpy() - og)) <= 1e-9 * np.max(np.abs(og))


@pytest.mark.parametrize("model", ["pipi_rho", "pipi_3rho", "ksks"])
@pytest.mark.parametrize("sizes,weighted", [((1, 1, 0), False), ((191, 193, 1), True), ((255, 257, 129), False),
                                            ((170_003, 17_001, 1_003), True)])
def test_copies_of_the_complex_table(tmp_path, monkeypatch, model, sizes, weighted):
    """Samples whose polarisations are not paired: copies of the complex angular values against direct loads."""
    import torch
    import ctpwa_b200
    from ctpwa_b200 import workloads

    cfg, s, w = _setup(tmp_path, model, sizes, weighted)
    monkeypatch.setenv("CTPWA_NO_POL_PAIRING", "1")

    def evaluate():
        ana = ctpwa_b200.analysis.from_device(cfg, s[0], s[1], s[2], weights=w)
        p = torch.tensor(workloads.true_params(ana.getNVector(), ana.getFreeResParams()[0].numpy()) * 1.01, device="cuda:0")
        n, g = ana.getNLLAndGrad(p)
        return ana.launchShape()["fp64"], float(n), g

    shape, n1, g1 = evaluate()
    assert shape["pol_paired"] == 0 and shape["stage"] == 4, shape
    monkeypatch.setenv("CTPWA_STAGE", "0")
    direct, n0, g0 = evaluate()
    assert direct["stage"] == 0 and direct["pol_paired"] == 0
    assert abs(n1 - n0) <= 1e-12 * max(1.0, abs(n0))
    assert float((g1 - g0).abs().max()) <= 1e-10 * float(g0.abs().max())


# resonances per chain -> threads, copies; reverse mode up to 8 (88 sums), beyond it symbolic derivatives (72 sums)
MANY = {5: (128, 4), 7: (128, 4), 8: (128, 4), 9: (128, 4)}


@pytest.mark.parametrize("nres", list(MANY))
def test_many_sums_stay_in_shared_memory(tmp_path, nres):
    """Three chains of several resonances: the per-thread gradient sums and the copies of an event fit twice per SM at
    128 threads; against the oracle's FP64 result."""
    import torch
    import ctpwa_b200
    from ctpwa_b200 import workloads
    from oracle.binding import Oracle

    cfg = workloads.make("pipi_3rho", tmp_path, n_phsp=2003, n_data=301, n_bkg=0, accept_reject=False, seed=3,
                         gpu_generator=False)
    names = [f"r{i}" for i in range(nres)]
    text = open(cfg).read()
    text = text[:text.index("Resonances:")].replace("rho770, rho1450, rho1700", ", ".join(names)) + "Resonances:\n"
    for i, n in enumerate(names):
        text += f"  {n}: {{J: 1, P: -1, model: BWR, parameters: [{0.8 + 0.13 * i:.3f}, {0.15 + 0.02 * i:.3f}], free: [0, 1]}}\n"
    open(cfg, "w").write(text)
    ana = ctpwa_b200.analysis(cfg)
    shape = ana.launchShape()["fp64"]
    assert shape["acc_smem"] == 1 and (shape["block"], shape["stage"]) == MANY[nres], shape
    p = workloads.true_params(ana.getNVector(), ana.getFreeResParams()[0].numpy())
    n, g = ana.getNLLAndGrad(torch.tensor(p, device="cuda:0"))
    onll, og, _ = Oracle(cfg).nll_grad(p)
    assert abs(float(n) - onll) <= 1e-10 * abs(onll)
    assert np.max(np.abs(g.cpu().numpy() - og)) <= 1e-9 * np.max(np.abs(og))
