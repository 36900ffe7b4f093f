"""Which compact angular tables the maxima over the events allow (csrc/pairing.hpp, host-compiled): the dropped
component of the polarisation paired with itself is bounded by its own plane's size."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import ctpwa_b200

SRC = r"""
#include "pairing.hpp"
extern "C" int decide(int nplane, int npol, const double* m)
{
    const ctpwa::Pairing p = ctpwa::pairingOf(nplane, npol, m);
    return p.pairs + 2 * p.reals + 4 * p.mid_im;
}
"""


@pytest.fixture(scope="module")
def decide(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairing")
    (d / "p.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", str(Path(ctpwa_b200.__file__).parent / "csrc"),
                    "-o", str(d / "p.so"), str(d / "p.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "p.so"))

    def f(npol, planes, pairs=None):
        """planes: (|SL|, |Re|, |Im|) per plane; pairs: (distance to the conjugate, to minus it)"""
        n, npair = len(planes), npol // 2
        m = np.array((pairs or [(0.0, 1.0)] * (n * npair)) + []).ravel()
        m = np.ascontiguousarray(np.concatenate([m, np.array(planes, dtype=float).ravel()]))
        r = lib.decide(n, npol, m.ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
        return bool(r & 1), bool(r & 2), bool(r & 4)

    return f


def test_tables(decide):
    big, small = (1.0, 1.0, 1e-16), (1e-6, 1e-6, 1e-22)
    assert decide(3, [big, small]) == (True, True, False)
    assert decide(3, [(1.0, 1e-16, 1.0), (1e-6, 1e-22, 1e-6)]) == (True, True, True)
    # a small plane whose dropped component is below 1e-12 of the large one but not of its own
    assert decide(3, [big, (1e-6, 1e-6, 1e-13)]) == (True, False, True)
    assert decide(3, [(1.0, 1e-16, 1.0), (1e-6, 1e-13, 1e-6)])[:2] == (True, False)
    # a plane that cancels to rounding is neither real nor imaginary
    assert decide(3, [big, (3e-17, 2e-17, 3e-17)]) == (True, True, False)
    # real in one plane, imaginary in another
    assert decide(3, [big, (0.5, 1e-17, 0.5)])[:2] == (True, False)
    # two polarisations: pairs alone
    assert decide(2, [(1.0, 0.0, 0.0)]) == (True, True, False)
    # not conjugates (or only up to a sign), nothing there, one polarisation
    assert decide(3, [big], [(1e-11, 1.0)])[0] is False
    assert decide(3, [big], [(1.0, 0.0)])[0] is False
    assert decide(3, [(0.0, 0.0, 0.0)])[0] is False
    assert decide(1, [big], [])[0] is False
