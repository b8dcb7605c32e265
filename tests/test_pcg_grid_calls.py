"""The host side of the one-launch PCG solver over a stand-in CUDA runtime (tests/cpp/pcg_grid_calls.cpp): a cooperative launch
that the driver refuses leaves the system to the passes."""
import os
import shutil
import subprocess

import pytest

from lapis_b200 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_refused_launch_is_left_to_the_passes(tmp_path):
    nvcc, gxx = _build._nvcc(), shutil.which("g++")
    if shutil.which(nvcc) is None or gxx is None:
        pytest.skip("needs nvcc and g++")
    env = {k: v for k, v in os.environ.items() if k not in ("CC", "CXX")}
    obj, exe = str(tmp_path / "pcg_grid.o"), str(tmp_path / "pcg_grid_calls")
    subprocess.run([nvcc, *_build.NVCC_FLAGS, "-c", os.path.join(_build.CSRC, "pcg_grid.cu"), "-o", obj], check=True, env=env)
    include = os.path.join(os.path.dirname(os.path.dirname(shutil.which(nvcc))), "include")
    subprocess.run([gxx, "-std=c++17", "-I", include, os.path.join(ROOT, "tests", "cpp", "pcg_grid_calls.cpp"), obj, "-o", exe], check=True, env=env)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
