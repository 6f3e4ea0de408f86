"""The natural-word engine and the exact slices' twiddle sums run without a
signed overflow, at their largest operands and in every compiled plan of
N >= 64 (tests/host/overflow_check.cu under the compiler's sanitizer)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def report():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out_dir = os.path.join(ROOT, "tests", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "overflow_check")
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-Xcompiler", "-fsanitize=signed-integer-overflow -fno-sanitize-recover=all",
                    "-lubsan", "-I" + os.path.join(ROOT, "fft_onchip_gb300", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-o", exe, os.path.join(ROOT, "tests", "host", "overflow_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return {k: float(v) for k, v in (line.split() for line in r.stdout.strip().splitlines())}


def test_twiddle_sums(report):
    assert report["tw_sum_bad"] == 0


def test_every_compiled_plan_at_the_largest_scale(report):
    assert report["plans"] >= 15
    # the bound of test_natural_engine.py's plans, for a fourth pass: 7 units of
    # 2^-49 of the largest input a pass with twiddles, at most three of them
    assert report["compiled_plans_rel"] < 2e-15
