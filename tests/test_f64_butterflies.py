"""The binary64 engine's twiddled butterflies on tangent-form table entries.

CPU: tests/host/tangent_check.cu compiles them as host code and runs every
radix behind every span up to 4096 points, each k, against long double."""
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
    exe = os.path.join(out_dir, "tangent_check")
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I" + os.path.join(ROOT, "fft_onchip_gb300", "csrc"), "-I" + os.path.join(ROOT, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "host", "tangent_check.cu")], check=True)
    r = subprocess.run([exe], check=True, capture_output=True, text=True)
    return {k: float(v) for k, v in (line.split() for line in r.stdout.strip().splitlines())}


# With u = 2^-53: a twiddled term is off by at most 4 u |x_m| (entry, tangent,
# two roundings), the R terms by 4 u sqrt(R) |x|, each of the log2 R sums by
# u sqrt(R) |x|, and the constant products of radix 8 and 16 by 3 u sqrt(R) |x|.
@pytest.mark.parametrize("radix,units", [(2, 5), (4, 6), (8, 10), (16, 11)])
def test_twiddled_butterfly(report, radix, units):
    assert report["radix%d" % radix] < units * radix ** 0.5 * 2.0 ** -53
