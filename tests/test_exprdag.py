"""Derivatives of the expression graph's kept products, compiled with the host compiler."""
import subprocess
from pathlib import Path

import ctpwa_b200

MAIN = r"""
#include "exprdag.hpp"
#include <cmath>
#include <cstdio>
using namespace ctpwa::dag;
static double ev(const Graph& g, int n, double t0, double t1, double k)
{
    const Node& d = g.nodes[n];
    auto a = [&] { return ev(g, d.a, t0, t1, k); };
    auto b = [&] { return ev(g, d.b, t0, t1, k); };
    switch (d.op) {
    case Const: return d.v;
    case Theta: return d.idx ? t1 : t0;
    case Kin: return k;
    case Add: return a() + b();
    case Sub: return a() - b();
    case Mul: return a() * b();
    case Recip: return 1 / a();
    case Neg: return -a();
    default: return NAN;
    }
}
int main()
{
    // a product of parameters alone, one of parameters and an event value, an event value times each
    for (int kind = 0; kind < 4; ++kind) {
        Graph g;
        const int x = g.theta(0), y = g.theta(1), e = g.kin(0);
        int n = g.mul(g.add(x, y), g.mul(x, g.recip(y)));
        if (kind % 2) n = g.mul(n, g.recip(g.add(g.mul(x, e), g.mul(e, e))));
        n = g.keepLog(n);
        if (kind >= 2) n = g.mul(g.sub(e, y), n);
        for (int j = 0; j < 2; ++j) {
            const int d = g.deriv(n, j);
            const double h = 1e-5, t0 = 1.3, t1 = 0.7, k = 0.4;
            const double num = (ev(g, n, t0 + (j ? 0 : h), t1 + (j ? h : 0), k) -
                                ev(g, n, t0 - (j ? 0 : h), t1 - (j ? h : 0), k)) / (2 * h);
            const double sym = ev(g, d, t0, t1, k);
            std::printf("%d %d %.12g %.12g\n", kind, j, sym, num);
            if (!(std::fabs(sym - num) <= 1e-8 * (1 + std::fabs(num)))) return 1;
        }
    }
    return 0;
}
"""


def test_kept_products(tmp_path):
    """From the logarithm where event and parameters mix, by the product rule where a kept product has parameters
    alone (whose logarithm's derivative is formed from the derivative itself)."""
    csrc = Path(ctpwa_b200.__file__).parent / "csrc"
    (tmp_path / "m.cpp").write_text(MAIN)
    exe = tmp_path / "m"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(csrc), "-o", str(exe), str(tmp_path / "m.cpp"),
                    str(csrc / "exprdag.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
