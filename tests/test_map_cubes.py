"""Cubes of frequencies cut from a map's transform, and from that of the map padded to twice its side, have
a margin of cells beyond the band: at every box and band that is accepted each cell's place in the
transform is inside it and is its frequency modulo the transform's size."""
import ctypes as C
import os
import subprocess

from conftest import ROOT


def test_every_cell_is_inside_the_transform(tmp_path):
    (tmp_path / "shim.cpp").write_text('#include "kernels.h"\nextern "C" {\n'
                                       "int at(int k, int n) { return cryoim::freq_index(k, n); }\n"
                                       "int radius(int r) { return cryoim::render_cube_radius(r); }\n}\n")
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "cryoim_gb300", "csrc"), "-I", inc, str(tmp_path / "shim.cpp"), "-o",
                    str(tmp_path / "shim.so")], check=True)
    lib = C.CDLL(str(tmp_path / "shim.so"))
    for n in list(range(8, 130, 2)) + [256, 384, 512]:
        for r in {0, 1, n // 4, n // 2 - 3, n // 2 - 2}:
            # the plain map's, the twice-oversampled one's, the renderer's: transform size, cube radius
            for m, rc in ((n, r), (2 * n, 2 * r + 1), (2 * n, lib.radius(r))):
                assert rc + 1 <= m // 2
                for k in (-rc - 1, -1, 0, rc, rc + 1):
                    i = lib.at(k, m)
                    assert 0 <= i < m and (i - m // 2 - k) % m == 0
