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
