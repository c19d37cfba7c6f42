"""The origin grid's basis (csrc/origin_basis.cpp) on the CPU: the phase of every origin of a
grid, at every band sample, comes back from the basis to the error it promises, for grids of one origin, even and odd ones, coarser and finer than the band,
and ranges that take several tiles of rows."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SHIM = r"""
#include "origin_basis.h"
using namespace cryoim;
static OriginBasis B;
extern "C" int ob_make(int n, int min_r, int R, float omax, float step, int n1, int f8, int* out) {
    B = make_origin_basis(n, min_r, R, omax, step, n1, f8 != 0);
    out[0] = B.nb; out[1] = B.slots; out[2] = B.layout; return B.units;
}
extern "C" void ob_get(float* q, float* f, int* row, float* mid) {
    for (size_t i = 0; i < B.q.size(); ++i) q[i] = B.q[i];
    for (size_t i = 0; i < B.f.size(); ++i) f[i] = B.f[i];
    for (int i = 0; i < B.slots; ++i) { row[3 * i] = B.mx[i]; row[3 * i + 1] = B.my[i]; row[3 * i + 2] = B.part[i]; }
    *mid = B.mid;
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("ob")
    src = d / "shim.cpp"
    src.write_text(SHIM)
    csrc = os.path.join(ROOT, "cryoim_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", csrc, str(src),
                    os.path.join(csrc, "origin_basis.cpp"), "-o", str(d / "shim.so")], check=True)
    return C.CDLL(str(d / "shim.so"))


@pytest.mark.parametrize("n,r0,R,omax,step", [
    (256, 7, 64, 6.0, 0.5), (64, 4, 22, 2.0, 0.5), (64, 4, 12, 2.0, 0.7), (64, 4, 22, 0.0, 0.5), (64, 2, 20, 1.0, 2.0),
    (128, 4, 26, 6.0, 0.25), (64, 2, 30, 6.0, 0.5), (100, 3, 20, 15.0, 1.0)])
@pytest.mark.parametrize("f8", [0, 1])
def test_phases_come_back(shim, n, r0, R, omax, step, f8):
    n1 = int(np.float32(2 * omax / step) + np.float32(0.5)) + 1
    dims = (C.c_int * 3)()
    units = shim.ob_make(n, r0, R, C.c_float(omax), C.c_float(step), n1, f8, dims)
    nb, slots, layout = dims
    q, f = np.zeros((nb, n1), np.float32), np.zeros((nb, 2 * R + 1), np.float32)
    row, mid = np.zeros((slots, 3), np.int32), C.c_float()
    shim.ob_get(q.ctypes.data_as(C.c_void_p), f.ctypes.data_as(C.c_void_p), row.ctypes.data_as(C.c_void_p),
                C.byref(mid))
    assert slots % (32 * units) == 0 and slots // units <= 160 and (layout < 0 or units == 1)
    x = -omax + step * np.arange(n1)
    ky, hx = np.meshgrid(np.arange(-R, R + 1), np.arange(0, R + 1), indexing="ij")
    d2 = hx ** 2 + ky ** 2
    keep = ((hx > 0) | (ky > 0)) & (d2 >= r0 * r0) & (d2 <= R * R)
    hx, ky = hx[keep], ky[keep]
    use = [(m, k) for m, k, part in row if m >= 0 and part == 0]
    second = {(m, k) for m, k, part in row if m >= 0 and part == 1}
    assert len(set(use)) == len(use) and second <= set(use)
    M, K = (np.array(v) for v in zip(*use))
    i4 = np.array([1, 1j, -1, -1j])
    w = 2 * np.pi / n
    got = np.zeros((n1, n1, len(hx)), complex)
    for m, k in zip(M, K):
        g = f[m][R + hx].astype(float) * f[k][R + ky] * i4[(m & 1) + (k & 1)] * np.exp(1j * w * mid.value * (hx + ky))
        got += q[k].astype(float)[:, None, None] * q[m].astype(float)[None, :, None] * g
    want = np.exp(1j * w * (x[None, :, None] * hx + x[:, None, None] * ky))
    # what is left out: a root mean square of 5e-5 (BF16) or 4e-4 (e4m3) of a phase (|value| = 1)
    assert np.mean(np.abs(got - want) ** 2) <= 1.02 * (4e-4 if f8 else 5e-5) ** 2
    # and the functions in use are the whole space where the grid has no more of them
    if n1 <= 8:
        assert np.abs(got - want).max() < 2e-6
