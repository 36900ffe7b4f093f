"""The theta gradient of the FP64 likelihood kernel in reverse mode, on the CPU.

The generated model code is plain arithmetic, so it is compiled here with the
host compiler: the theta sums from model_adjoint and the Jacobian
(model_theta_sum) against the symbolic derivatives of model_columns, for random
per-event values, parameters and seeds. Both are FP64 sums of the same few dozen
products, so they agree to 1e-12 of the sum of the terms' magnitudes."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from ctpwa_b200 import workloads

HARNESS = r"""
#include <cmath>
#include <cstring>
using std::sqrt; using std::log; using std::exp; using std::sin; using std::cos; using std::atan2;
#define __device__
#define __forceinline__ inline
#define __restrict__
static float ct_rcpf(float x) { return 1.0f / x; }
static float ct_sqrtf(float x) { return std::sqrt(x); }
static double ct_rho(bool im, double s, double ma, double mb)
{
    double f1 = 1 - (ma + mb) * (ma + mb) / s, f2 = 1 - (ma - mb) * (ma - mb) / s;
    f2 = f2 > 0 ? std::sqrt(f2) : 0;
    return im ? (f1 >= 0 ? 0 : std::sqrt(-f1) * f2) : (f1 >= 0 ? std::sqrt(f1) * f2 : 0);
}
#include "model.cuh"
struct Sink {
    const double* w; double a[M_NADJ + 1] = {};
    void value(int, double, double) {}
    bool sums() { return true; }
    double wr(int t) const { return w[2 * t]; }
    double wi(int t) const { return w[2 * t + 1]; }
    void adj(int k, double x) { a[k] += x; }
};
extern "C" void dims(int* o) { o[0] = M_NEV; o[1] = M_NTH; o[2] = M_NTERM; o[3] = M_NADJ; }
// per theta: reverse mode, symbolic, sum of the magnitudes of the symbolic terms
extern "C" void grads(const double* ev, const double* th, const double* w, double* out)
{
    double C[M_NCONST + M_NJAC + 1], Fr[M_NTERM], Fi[M_NTERM], dr[M_NDER + 1], di[M_NDER + 1];
    for (int q = 0; q < M_NPRO; ++q) model_prologue(q, th, C);
    Sink s; s.w = w;
    model_adjoint(ev, C, s);
    model_columns(ev, C, Fr, Fi, dr, di);
    std::memset(out, 0, sizeof(double) * 3 * M_NTH);
    for (int j = 0; j < M_NTH; ++j) out[3 * j] = model_theta_sum(j, C + M_NCONST, s.a);
    for (int k = 0; k < M_NDER; ++k) {
        const int t = der_term(k); double* o = out + 3 * der_th(k);
        o[1] += dr[k] * w[2 * t] - di[k] * w[2 * t + 1];
        o[2] += std::fabs(dr[k] * w[2 * t]) + std::fabs(di[k] * w[2 * t + 1]);
    }
}
"""

CUSTOM = ("rho770: {J: 1, P: -1, model: Custom, paramValues: [0.775, 0.149], paramNames: [mass, width], free: [0, 1], "
          'expr: "EXPR"}')
EXPRS = {  # the last reads log(0), guarded, where m is the mass
    "custom_division": "1.0 / (mass * mass - m * m - csqrt(0.0 - 1.0) * mass * width * q) + width * q",
    "custom_abs": "width * abs(m - mass + csqrt(0.0 - 1.0) * q)",
    "custom_log": "width * Re(log((m - mass) * (m - mass)))",
}


def _compile(tmp_path, name):
    import ctpwa_b200

    base = "pipi_rho" if name in EXPRS else name
    text = workloads.config_text(base, "p", "d")
    if name in EXPRS:
        text = text[:text.index("  rho770:")] + "  " + CUSTOM.replace("EXPR", EXPRS[name]) + "\n"
    (tmp_path / "c.yml").write_text(text)
    (tmp_path / "h.cpp").write_text(HARNESS)
    os.environ["CTPWA_MODEL_SOURCE_OUT"] = str(tmp_path / "model.cuh")
    try:
        ctpwa_b200.precompile(str(tmp_path / "c.yml"))
    finally:
        del os.environ["CTPWA_MODEL_SOURCE_OUT"]
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-shared", "-fPIC", "-I", str(tmp_path), "-o", str(tmp_path / "h.so"),
                    str(tmp_path / "h.cpp")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "h.so"))
    d = (ctypes.c_int * 4)()
    lib.dims(d)
    ptr = lambda x: x.ctypes.data_as(ctypes.POINTER(ctypes.c_double))

    def grads(ev, th, w):
        out = np.zeros((d[1], 3))
        lib.grads(ptr(ev), ptr(th), ptr(w), ptr(out))
        return out

    init = np.array([x["init"] for x in ctpwa_b200.describe(str(tmp_path / "c.yml"))["slots"]])
    return list(d), init, grads


@pytest.mark.parametrize("name", ["pipi_rho", "pipi_3rho", "kkpi", "ksks", *EXPRS])
def test_matches_symbolic_derivatives(tmp_path, name):
    (nev, nth, nterm, _), init, grads = _compile(tmp_path, name)
    rng = np.random.default_rng(5)
    for _ in range(50):
        o = grads(rng.uniform(0.3, 2.0, nev), init * rng.uniform(0.9, 1.1, nth), rng.uniform(-1, 1, 2 * nterm))
        assert np.isfinite(o).all()
        assert (np.abs(o[:, 0] - o[:, 1]) <= 1e-12 * o[:, 2].max() * (1 + nth)).all(), o


def test_guarded_branch_that_is_not_taken(tmp_path):
    """At m == mass the logarithm's argument is replaced by a constant: no derivative comes through it, in particular
    none of the root of zero that was replaced."""
    (nev, _, nterm, _), init, grads = _compile(tmp_path, "custom_log")
    o = grads(np.full(nev, init[0]), init, np.ones(2 * nterm))
    assert np.isfinite(o[:, 1]).all() and np.array_equal(o[:, 0], o[:, 1]), o
