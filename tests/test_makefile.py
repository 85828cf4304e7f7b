"""A change of any header rebuilds every object whose source includes it."""
import os
import re
import shutil
import subprocess

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "water-sim-cuda_b200")
CSRC = os.path.join(PKG, "csrc")
HEADERS = sorted(f for f in os.listdir(CSRC) if f.endswith((".h", ".cuh")))


def _includes(name, seen):
    with open(os.path.join(CSRC, name)) as f:
        for inc in re.findall(r'#include "([^"]+)"', f.read()):
            inc = os.path.basename(inc)
            if inc not in seen and os.path.exists(os.path.join(CSRC, inc)):
                seen.add(inc)
                _includes(inc, seen)
    return seen


@pytest.mark.parametrize("header", HEADERS)
def test_header_is_a_prerequisite(header):
    if not shutil.which("make"):
        pytest.skip("make is not on PATH")
    plan = subprocess.run(["make", "-n", "-C", PKG, "-W", f"csrc/{header}", "NVCC=nvcc", "lib/libmpm_b200.so"], capture_output=True, text=True)
    assert plan.returncode == 0, plan.stderr
    for src in sorted(os.listdir(CSRC)):
        if src.endswith((".cu", ".cpp")) and src != "cli.cpp" and header in _includes(src, set()):
            assert re.search(rf"-c csrc/{re.escape(src)}\b", plan.stdout), f"{src} includes {header} but would not be rebuilt"
