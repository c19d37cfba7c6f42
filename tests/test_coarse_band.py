"""The coarse level's band lies within the search's own at every pair of radii: samples beyond it are
outside the particle's window, its ramps' table and the map's cube."""
import ctypes as C
import os
import subprocess

from conftest import ROOT


def test_coarse_radius_is_within_the_band(tmp_path):
    (tmp_path / "shim.cpp").write_text(
        '#include "kernels.h"\nextern "C" int radius(int a, int b) { return cryoim::coarse_radius(a, b); }\n')
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "cryoim_gb300", "csrc"), "-I", inc, str(tmp_path / "shim.cpp"), "-o",
                    str(tmp_path / "shim.so")], check=True)
    lib = C.CDLL(str(tmp_path / "shim.so"))
    for max_r in range(0, 130):
        for min_r in range(0, max_r + 1):
            rc = lib.radius(min_r, max_r)
            assert min_r <= rc <= max_r
            if min_r < max_r:
                assert rc == max(min_r + 1, max_r // 2)
