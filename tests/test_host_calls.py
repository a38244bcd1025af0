"""The library's host code without a GPU: tests/cpp/host_calls.cpp defines the CUDA runtime functions
that the library imports and runs scenarios against them (what a batch's device table points to, what
happens when an allocation fails, which kernel a call comes to)."""
import os
import shutil
import subprocess

import pytest

from range_libc_gb300 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host_calls(tmp_path_factory):
    _lib.lib()   # built
    path = _lib.library_path()
    nvcc = os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")
    include = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        pytest.skip("CUDA headers not found")
    exe = tmp_path_factory.mktemp("host_calls") / "host_calls"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-rdynamic", "-I", os.path.join(ROOT, "include"), "-I", include,
                           os.path.join(HERE, "cpp", "host_calls.cpp"), "-o", str(exe), "-L", os.path.dirname(path),
                           "-lrangelibc_gb300", f"-Wl,-rpath,{os.path.dirname(path)}", "-Wl,--allow-shlib-undefined"])
    return exe


@pytest.mark.parametrize("scenario", ["batch_tables", "batch_in_flight", "bresenham_memory", "occupancy",
                                      "shared_memory_limits", "learned_timeouts", "autotune"])
def test_host_calls(host_calls, scenario):
    r = subprocess.run([str(host_calls), scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
