"""Kernel modules that pass from a destroyed handle to the next one: live
handles of one model never share a module (its constant block holds the
parameters of a call), and a handle on a module that another has used gives
the results of one on a fresh module."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_handles_on_reused_modules(tmp_path):
    import torch
    import ctpwa_b200
    from ctpwa_b200 import toymc, workloads

    cfg = tmp_path / "c.yml"
    cfg.write_text(workloads.config_text("pipi_3rho", "p", "d"))
    s = [torch.tensor(toymc.phase_space(workloads.M_JPSI, workloads.MASSES["pipi_3rho"], n, n), device="cuda:0")
         for n in (30_001, 3_001)]

    def make():
        return ctpwa_b200.analysis.from_device(str(cfg), *s)

    first = make()
    base = torch.tensor(workloads.true_params(first.getNVector(), first.getFreeResParams()[0].numpy()), device="cuda:0")
    points = [base * (1.0 + 0.003 * k) for k in range(6)]
    want = [[x.clone() for x in first.getNLLAndGrad(p)] + [first.getHessian(p)] for p in points]
    torch.cuda.synchronize()
    del first
    bad = []

    def work(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for r in range(8):
                ana = make()  # takes over a module that another thread's handle has left, or loads one
                for j in range(6):
                    i = (k + r + j) % 6
                    n, g = ana.getNLLAndGrad(points[i])
                    H = ana.getHessian(points[i])
                    stream.synchronize()
                    if not (torch.equal(n, want[i][0]) and torch.equal(g, want[i][1]) and torch.equal(H, want[i][2])):
                        bad.append((k, r, i))
                del ana

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def _model(tmp_path):
    import torch
    from ctpwa_b200 import toymc, workloads

    cfg = tmp_path / "c.yml"
    cfg.write_text(workloads.config_text("pipi_rho", "p", "d"))
    s = [torch.tensor(toymc.phase_space(workloads.M_JPSI, workloads.MASSES["pipi_rho"], n, n), device="cuda:0")
         for n in (400_001, 40_001)]
    return str(cfg), s


def test_destroyed_while_its_work_is_queued(tmp_path):
    """Evaluations queued on a stream nobody waits for, the handle destroyed, and the next one evaluating at other
    parameters on the module it took over: the queued ones keep their own parameters."""
    import torch
    import ctpwa_b200
    from ctpwa_b200 import workloads

    cfg, s = _model(tmp_path)
    make = lambda: ctpwa_b200.analysis.from_device(cfg, *s)
    ana = make()
    base = torch.tensor(workloads.true_params(ana.getNVector(), ana.getFreeResParams()[0].numpy()), device="cuda:0")
    other = base * 1.05
    want = [float(ana.getNLLAndGrad(p)[0]) for p in (base, other)]
    assert want[0] != want[1]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(4):
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            got = [ana.getNLLAndGrad(base)[0] for _ in range(50)]
        lib, h = ana._lib, ana._h
        ana._h = None
        lib.ctpwa_destroy(h)
        ana = make()
        n2 = ana.getNLLAndGrad(other)[0]
        torch.cuda.synchronize()
        assert [float(x) for x in got] == [want[0]] * 50 and float(n2) == want[1]


def test_changed_kernel_sources_are_compiled(tmp_path, monkeypatch):
    """A handle created after the kernel folder was set, or a file in it edited, runs the new code and not a module
    that an earlier handle of the same model has left."""
    import shutil
    from pathlib import Path

    import torch
    import ctpwa_b200
    from ctpwa_b200 import workloads

    cfg, s = _model(tmp_path)

    def nll():
        ana = ctpwa_b200.analysis.from_device(cfg, *s)
        p = torch.tensor(workloads.true_params(ana.getNVector(), ana.getFreeResParams()[0].numpy()), device="cuda:0")
        return float(ana.getNLL(p))

    first = nll()
    kernels = tmp_path / "kernels"
    shutil.copytree(Path(ctpwa_b200.__file__).parent / "csrc" / "kernels", kernels)
    src = kernels / "fused_nll.cuh"
    text = src.read_text()
    line = "accd[0] += -log((double)f) * we;"
    assert text.count(line) == 1
    monkeypatch.setenv("CTPWA_JIT_CACHE_DIR", str(tmp_path / "jit"))
    src.write_text(text.replace(line, "accd[0] += -2.0 * log((double)f) * we;"))
    monkeypatch.setenv("CTPWA_B200_KERNEL_DIR", str(kernels))
    second = nll()
    src.write_text(text.replace(line, "accd[0] += -3.0 * log((double)f) * we;"))
    third = nll()
    monkeypatch.delenv("CTPWA_B200_KERNEL_DIR")
    assert nll() == first
    assert abs((third - second) - (second - first)) <= 1e-9 * abs(first) and abs(second - first) > 1e-3 * abs(first)
