"""What a search pays on the host for an origin grid that its context has not seen: the basis takes the time
of a few ten thousand cosines, against searches of about a millisecond."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SHIM = r"""
#include <chrono>
#include <cmath>
#include "origin_basis.h"
static double now() { return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count(); }
extern "C" double basis_time(int n, int min_r, int R, float omax, float step, int n1, int f8) {
    double best = 1e9;
    for (int k = 0; k < 9; ++k) {
        const double t = now();
        const auto b = cryoim::make_origin_basis(n, min_r, R, omax, step, n1, f8 != 0);
        const double d = now() - t + (b.nb > 0 ? 0.0 : 1e9);
        best = d < best ? d : best;
    }
    return best;
}
extern "C" double cosine_time(int count) {
    double best = 1e9;
    for (int k = 0; k < 9; ++k) {
        volatile double s = 0.0;
        const double t = now();
        for (int i = 0; i < count; ++i) s = s + std::cos(0.0245436926 * (i % 129 - 64) * (0.5 * (i % 25) - 6.0));
        const double d = now() - t;
        best = d < best ? d : best;
    }
    return best;
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("obcost")
    (d / "shim.cpp").write_text(SHIM)
    csrc = os.path.join(ROOT, "cryoim_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", csrc, str(d / "shim.cpp"),
                    os.path.join(csrc, "origin_basis.cpp"), "-o", str(d / "shim.so")], check=True)
    lib = C.CDLL(str(d / "shim.so"))
    lib.basis_time.restype = lib.cosine_time.restype = C.c_double
    lib.basis_time.argtypes = [C.c_int] * 3 + [C.c_float] * 2 + [C.c_int] * 2
    return lib


# (the basis of the second grid by cosines alone, one for each of its sums' terms, is 750,000 of them)
@pytest.mark.parametrize("n,r0,R,omax,cosines", [(256, 7, 64, 6.0, 60_000), (512, 13, 128, 12.0, 250_000)])
def test_basis_costs_few_cosines(shim, n, r0, R, omax, cosines):
    n1 = int(np.float32(2 * omax / 0.5) + np.float32(0.5)) + 1
    assert shim.basis_time(n, r0, R, omax, 0.5, n1, 0) < shim.cosine_time(cosines)
