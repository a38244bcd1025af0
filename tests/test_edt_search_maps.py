"""The distance transform's searches on whole maps, on the host against the oracle: the reference's
benchmark map from the golden fixture, the generated workload maps, and large sparse ones."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from range_libc_gb300 import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HERE = os.path.dirname(os.path.abspath(__file__))


def test_searches_on_whole_maps(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    orc, exe = tmp_path / "rlc_oracle.o", tmp_path / "edt_search_maps"
    subprocess.check_call(["gcc", "-O2", "-ffp-contract=off", "-c", os.path.join(ROOT, "oracle", "rlc_oracle.c"),
                           "-o", str(orc)])
    subprocess.check_call([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                           "-Xcompiler", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(ROOT, "range_libc_gb300", "csrc"),
                           os.path.join(HERE, "cpp", "edt_search_maps.cu"), str(orc), "-o", str(exe), "-lpthread"])
    maps = {"corridor_512": W.corridor_map(512, 5), "rect_disk_1024": W.rect_disk_map(1024, 31),
            "corridor_300x410": np.ascontiguousarray(W.corridor_map(512, 78)[:300, :410]),
            "basement_hallways_5cm": np.load(os.path.join(HERE, "golden", "reference_vectors.npz"))["basement/occ"]}
    args = []
    for name, occ in maps.items():
        o = np.ascontiguousarray(occ, np.uint8)
        o.tofile(tmp_path / name)
        args += [str(tmp_path / name), str(o.shape[0]), str(o.shape[1])]
    r = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith(" 0 mismatches"), r.stdout
