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
extern "C" int t_quotient(int n, int d) { return mpm::bin_quotient(n, mpm::bin_reciprocal(d)); }
extern "C" void t_origin(int bin, int nbx, int nby, int* xyz) {
    mpm::SimParams p{};
    p.nbx = nbx, p.nby = nby;
    p.inv_nbx = mpm::bin_reciprocal(nbx), p.inv_nby = mpm::bin_reciprocal(nby);
    mpm::bin_origin(p, bin, xyz, xyz + 1, xyz + 2);
}
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


def test_quotients(host):
    top = 2 ** 31 - 1
    for d in [1, 2, 3, 5, 7, 17, 18, 33, 66, 138, 255, 256, 257, 4097, 65535, 65536, 65537, 2 ** 24 - 1, 2 ** 24, top - 1, top]:
        some = {0, 1, d - 2, d - 1, d, d + 1, 65535, 65536, 2 ** 24 - 1, top // d * d - 1, top // d * d, top - 1, top}
        some |= {k * d + r for k in (top // d // 3, top // d // 2) for r in (-1, 0, 1)}
        for n in sorted(n for n in some if 0 <= n <= top):
            assert host.t_quotient(n, d) == n // d, (n, d)


@pytest.mark.parametrize("size", [(1, 1, 1), (6, 1100, 1100), (64, 1024, 1024), (128, 1024, 1024), (1024, 64, 1024),
                                  (40, 21, 23), (256, 256, 256), (2 ** 27 - 16, 1, 1), (5, 3, 2 ** 25)])
def test_origin_of_the_bins(host, size):
    nb = [(s + 2 + e - 1) // e for s, e in zip(size, (8, 4, 4))]
    out = (ctypes.c_int * 3)()
    total = nb[0] * nb[1] * nb[2]
    for bin in sorted({0, 1, nb[0] - 1, nb[0], total // 3, total // 2, total - nb[0] - 1, total - 2, total - 1} & set(range(total))
                      if total < 10 ** 6 else [0, 1, nb[0], 65535, 65536, total // 3, total // 2, total - nb[0] - 1, total - 2, total - 1]):
        if not 0 <= bin < total:
            continue
        host.t_origin(bin, nb[0], nb[1], out)
        want = (bin % nb[0] * 8 - 2, bin // nb[0] % nb[1] * 4 - 2, bin // (nb[0] * nb[1]) * 4 - 2)
        assert tuple(out) == want, (bin, tuple(out), want)
