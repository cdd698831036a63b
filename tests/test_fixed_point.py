"""Block fixed-point arithmetic of the FP64 form (sse_fixed.cuh), compiled by
nvcc as host code, against long double (no GPU)."""
import json
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.fail("nvcc is required")
    exe = str(tmp_path_factory.mktemp("fixed") / "fixed_point_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off",
                    os.path.join(HERE, "fixed_point_check.cu"), "-o", exe], check=True, capture_output=True)
    return json.loads(subprocess.run([exe], check=True, capture_output=True, text=True).stdout)


def test_flux_is_at_least_as_accurate_as_fp64(results):
    # rms error over random states, largest over components, Mach numbers 1e-3
    # to 3 and jumps 1e-5 to 0.4, relative to the FP64 algebra's own
    assert results["flux_error_ratio"] < 1.0
    # 60 fraction bits below scales that exceed the values by up to 2^6
    assert results["flux_relative"] < 2.0 ** -51


def test_means(results):
    # FP32 pairs below z = 1e-4, FP64 series and logarithm above: an FP64
    # evaluation's few units of 2^-53
    assert results["mean"] < 8 * 2.0 ** -53


def test_conversions_are_exact(results):
    assert results["conversion_mismatches"] == 0
