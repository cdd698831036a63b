"""Scaling of the fixed-point operator rows (sse_fixed_ops.cuh), compiled by
nvcc as host code (no GPU)."""
import json
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_rows_next_to_a_power_of_two_keep_their_value(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "fixed_point_operators_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    os.path.join(HERE, "fixed_point_operators_check.cu"), "-o", exe], check=True, capture_output=True)
    assert json.loads(subprocess.run([exe], check=True, capture_output=True, text=True).stdout)["mismatches"] == 0
