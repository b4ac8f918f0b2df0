"""The frame scheduler (csrc/frame.cpp) on the CPU: its passes, run thread by thread
as the kernels address them, against the circuit applied gate by gate.  Rings,
growing ranges and random permutations with gaps; statevectors (one bit a gate)
in whole-state and partial tiles, Pauli coefficients (two bits a gate); every
element size the kernels have; odd sizes.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = str(tmp_path_factory.mktemp("frame") / "frame_schedule_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(CUDA, "include"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "frame_schedule_check.cpp"),
                    os.path.join(ROOT, "jaqsi_b200", "csrc", "frame.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("bits,nb,t,low,elem", [
    (1, 9, 9, 3, 8), (1, 9, 9, 3, 16), (1, 12, 12, 3, 8), (1, 13, 11, 3, 8), (1, 13, 11, 3, 16), (1, 14, 11, 4, 8),
    (1, 15, 11, 3, 16),
    (2, 10, 10, 3, 4), (2, 10, 10, 3, 8), (2, 12, 11, 3, 4), (2, 12, 11, 3, 8), (2, 14, 11, 3, 4), (2, 14, 11, 3, 8),
])
def test_schedule_is_the_circuit(check, bits, nb, t, low, elem, kind):
    for seed in (1, 2):
        r = subprocess.run([check] + [str(v) for v in (bits, nb, t, low, elem, kind, seed)], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
