"""The distance transform's per-cell searches, run on the host against the oracle.

edt_col_search and edt_row_search (rlc_map.cu) are __host__ __device__: the harness is compiled for
the host with nvcc, beside the oracle's C restatement of the reference's transform, and compares
every cell bit for bit on seeded maps -- tile and block edges, empty and full columns, obstacles far
enough apart that whole blocks are searched, and sides from 4096 to 16384 whose keys round.  The
GPU tests run the kernels themselves.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HERE = os.path.dirname(os.path.abspath(__file__))


def test_searches_equal_the_oracle(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    orc, exe = tmp_path / "rlc_oracle.o", tmp_path / "edt_search_check"
    subprocess.check_call(["gcc", "-O2", "-ffp-contract=off", "-c", os.path.join(ROOT, "oracle", "rlc_oracle.c"),
                           "-o", str(orc)])
    subprocess.check_call([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                           "-Xcompiler", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(ROOT, "range_libc_gb300", "csrc"),
                           os.path.join(HERE, "cpp", "edt_search_check.cu"), str(orc), "-o", str(exe), "-lpthread"])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith(" 0 mismatches"), r.stdout
