"""The calls on host arrays over a stand-in CUDA runtime (tests/cpp/host_calls.cpp): no GPU is involved, so that what must
not reach one can be tried."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.isdir(os.path.join(CUDA, "include")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("host_calls") / "host_calls")
    env = {k: v for k, v in os.environ.items() if k not in ("CC", "CXX")}
    subprocess.run([gxx, "-std=c++17", "-O2", "-pthread", "-rdynamic", "-I", os.path.join(CUDA, "include"),
                    os.path.join(ROOT, "tests", "cpp", "host_calls.cpp"), "-o", exe, "-ldl"], check=True, env=env)
    return exe


# offsets: differences that wrap around the index type must not pass as row lengths
# in_flight: a call that fails behind the upload leaves no copy from the caller's page-locked arrays under way
# exhausted: memory or threads that cannot be had; no exception may leave a C entry point
# fork_exit: a child process forked behind a large call exits
# full_device: idle memory of the pool goes to an allocation that fails without it, and back to the device
# threads: four threads in calls at once
@pytest.mark.parametrize("scenario", ["offsets", "in_flight", "exhausted", "fork_exit", "full_device", "threads"])
def test_host_calls(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
