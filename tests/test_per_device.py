"""Set-up that belongs to a kernel on a device (csrc/per_device.h) is done on each device, against a fake runtime of three
devices, and no source file keeps such a flag for the whole process."""
import ctypes
import glob
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "glm_asr_stack_b200", "csrc")
SOURCE = r"""
#include "per_device.h"
static int current = 0, fail = 0, set_ups[3] = {0, 0, 0}, cleared = 0;
extern "C" cudaError_t cudaGetDevice(int *d) { *d = current; return current == 7 ? cudaErrorInvalidDevice : cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { ++cleared; return cudaSuccess; }
extern "C" int use(int device, int failing) {
    static glmasr::PerDevice<bool> done;
    current = device;
    fail = failing;
    return (int)glmasr::once_per_device(done, [] { ++set_ups[current]; return fail ? cudaErrorInvalidValue : cudaSuccess; });
}
extern "C" int count(int device) { return device < 0 ? cleared : set_ups[device]; }
"""


def test_once_per_device(tmp_path):
    (tmp_path / "p.cpp").write_text(SOURCE)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", os.path.join(cuda, "include"), "-o",
                    str(tmp_path / "p.so"), str(tmp_path / "p.cpp")], check=True, capture_output=True)
    lib = ctypes.CDLL(str(tmp_path / "p.so"))
    assert lib.use(0, 0) == 0 and lib.use(0, 0) == 0 and lib.count(0) == 1
    assert lib.use(1, 1) != 0 and lib.count(-1) == 1          # a failure is returned, cleared and tried again
    assert lib.use(1, 0) == 0 and lib.use(1, 0) == 0 and lib.count(1) == 2
    assert lib.use(2, 0) == 0 and lib.use(0, 0) == 0 and [lib.count(i) for i in range(3)] == [1, 2, 1]
    assert lib.use(7, 0) != 0


def test_no_process_wide_opt_in():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        src = open(path).read()
        assert not re.search(r"static\s+(bool|int)\s+\w*(configured|ready)\w*(\[\d+\])?\s*=", src.replace("g_tail_ready[64]", "")), path
