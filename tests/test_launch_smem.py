"""A kernel's shared-memory permission is one state of the device for all host threads (csrc/launch.h): a
launch's request never lowers it, counts the kernel's static memory, and is the only place that sets it."""
import ctypes as C
import glob
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "cryoim_gb300", "csrc")
# a runtime of one kernel: its static memory, the dynamic memory it may have, how often that was set
SHIM = r"""
#include "launch.h"
extern "C" {
size_t fixed_bytes; int allowed = 49152, sets = 0;
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    *a = cudaFuncAttributes(); a->sharedSizeBytes = fixed_bytes; a->maxDynamicSharedSizeBytes = allowed; return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 232448; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) { allowed = v; ++sets; return cudaSuccess; }
void reset(size_t fixed) { fixed_bytes = fixed; allowed = 49152; sets = 0; }
int ask(size_t bytes) { return cryoim::allow_smem_of(nullptr, bytes); }
// a launch is accepted if its dynamic memory is allowed and all of it fits what is allowed beside it
int launch(size_t bytes) { return allowed > 49152 - (int)fixed_bytes && sets ? bytes <= (size_t)allowed : bytes + fixed_bytes <= 49152; }
int nsets() { return sets; }
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    d = tmp_path_factory.mktemp("smem")
    (d / "shim.cpp").write_text(SHIM)
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", inc, str(d / "shim.cpp"), "-o",
                    str(d / "shim.so")], check=True)
    lib = C.CDLL(str(d / "shim.so"))
    lib.ask.argtypes = lib.launch.argtypes = lib.reset.argtypes = [C.c_size_t]
    return lib


def test_a_smaller_request_leaves_the_larger_one_in_force(fake):
    fake.reset(1024)
    assert fake.ask(217000) == 0   # one lane, about to launch
    assert fake.ask(184000) == 0   # another lane's call comes between
    assert fake.ask(100) == 0
    assert fake.launch(217000) and fake.launch(184000) and fake.launch(100)
    assert fake.nsets() == 1


def test_static_memory_counts(fake):
    for fixed in (0, 264, 2048):
        for more in (-64, 0, 64, 4096):
            fake.reset(fixed)
            want = 49152 - fixed + more
            assert fake.ask(want) == 0 and fake.launch(want)
    fake.reset(264)
    assert fake.ask(232448 - 264) == 0 and fake.launch(232448 - 264)
    assert fake.ask(232448 - 263) != 0


def test_nothing_else_sets_it():
    users = [os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "**", "*.*"), recursive=True)
             if "cudaFuncSetAttribute" in open(f).read()]
    assert users == ["launch.h"]
