"""The rule by which the one walk over a cell's face slopes decides the limiter
(limit_left: k_plm_r, k_plm_z and, by branch, the reverse step's a_gather_plm) against
the reference's face-by-face loop, on the host: slopes of mixed sizes, whose
products with the running slope underflow in one order and not in another."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")


def test_walk_ends_where_the_loop_ends(tmp_path):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "check_limiter")
    subprocess.run([NVCC, "-std=c++17", "-O2", "-Wno-deprecated-gpu-targets", "-Xcompiler", "-ffp-contract=off",
                    "-o", exe, os.path.join(HERE, "limiter_local", "check_limiter.cu")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    print(out.stdout)
    assert out.returncode == 0, out.stdout + out.stderr
    n = dict(zip(out.stdout.split()[::2], map(int, out.stdout.split()[1::2])))
    assert n["decided"] > 0 and n["left"] > 0
