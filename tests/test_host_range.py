"""CPU test of the decision that hands a host buffer to a kernel: the whole
buffer lies in mapped registrations (tests/host/host_range_check.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_byte_is_looked_at():
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    out_dir = os.path.join(ROOT, "tests", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "host_range_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I" + os.path.join(ROOT, "fft_onchip_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "host", "host_range_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
