"""The row bands of the small-level multigrid kernel stay inside their levels, for
every height and cluster size (host code, no GPU).  A band beyond the end of
its level would write past the level's arrays."""
import os
import shutil
import subprocess

import pytest

from stz_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bands_stay_inside_their_levels(tmp_path):
    cxx = shutil.which("g++")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    if not cxx or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("needs g++ and CUDA's headers")
    exe = str(tmp_path / "bands")
    subprocess.run([cxx, "-O1", "-std=c++17", "-w", "-I", cuda, "-I", os.path.join(ROOT, "stz_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "bands_main.cc"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
