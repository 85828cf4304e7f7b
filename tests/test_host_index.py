"""Index arithmetic shared by host and device (csrc/device_math.cuh), compiled
for the host and checked against Python's whole numbers at the ends of its
ranges."""
import ctypes
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "water-sim-cuda_b200", "csrc")

SOURCE = """
#include "device_math.cuh"
extern "C" int t_in_range(int b, int o, int n) { return mpm::in_range(b, o, n); }
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    nvcc = shutil.which("nvcc")
    if not nvcc:
        pytest.skip("nvcc is not on PATH")
    folder = tmp_path_factory.mktemp("host_index")
    src, so = folder / "host_index.cu", folder / "host_index.so"
    src.write_text(SOURCE)
    made = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC",
                           "-I", CSRC, "-o", str(so), str(src)], capture_output=True, text=True)
    assert made.returncode == 0, made.stderr
    return ctypes.CDLL(str(so))


def test_stencil_base_in_a_run_of_cells(host):
    top, bottom = 2 ** 31 - 1, -2 ** 31
    for o in (-2, -1, 0, 1, 2, 3, 6, 126, 2 ** 27):
        for n in (0, 1, 3, 4, 8):
            for b in [bottom, bottom + 1, bottom + 2, top - 2, top - 1, top, -3, -2, -1, 0, 1, 7] + [o + d for d in range(-2, n + 2)]:
                assert host.t_in_range(b, o, n) == (o <= b < o + n), (b, o, n)
