"""The natural-word fixed-point arithmetic (EngFxN, the plans of N >= 64).

CPU: tests/host/natural_check.cu compiles it as host code: products at their
largest operands, the small DFTs, and whole plans at the largest input scale.
GPU: transforms at the edges of what the conversions and tiles take, against
the long-double oracle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from fft_onchip_gb300 import inputs
from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def report():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out_dir = os.path.join(ROOT, "tests", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "natural_check")
    csrc = os.path.join(ROOT, "fft_onchip_gb300", "csrc")
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I" + csrc, "-I" + os.path.join(ROOT, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "host", "natural_check.cu")], check=True)
    r = subprocess.run([exe], check=True, capture_output=True, text=True)
    return {k: float(v) for k, v in (line.split() for line in r.stdout.strip().splitlines())}


# In units of the last place.  A product is floored (1) and drops its low * low
# terms: two of at most 2^31 * 2^31 / 2^64 = 1/4 at quarter scale, and the
# table's rounding moves it by less than 1/4; at full scale all but the floor
# is four times that.  The constant products drop less than 0.02 (mulh) and 0.3
# (rot8) and their constants' rounding moves them by less than 1/8.  A dft8
# output takes two mulh, a dft16 output two rot8 and one mulh on its k1.
@pytest.mark.parametrize("name,bound", [("cmul_quarter_units", 1.75), ("cmul_units", 4.0), ("mulh_units", 1.15),
                                        ("rot8_units", 1.43), ("dft2_units", 0.1), ("dft4_units", 0.1),
                                        ("dft8_units", 2.3), ("dft16_units", 4.1)])
def test_products_and_small_dfts(report, name, bound):
    assert report[name] < bound


def test_far_input_conversion(report):
    assert report["in_far_mismatch"] == 0


def test_whole_plans_at_the_largest_scale(report):
    # at most 7 units a pass at the last pass's scale (2^-49 of the largest
    # input), three passes with twiddles, outputs of at least sqrt(N) times the
    # inputs' magnitude: below 7 * 3 * 2^-49 * sqrt(2) / 32; an overflow is O(1)
    assert report["plans_rel"] < 2e-15


def _fft(cuda, x):
    import fft_onchip_gb300 as F
    y = F.fft(cuda.from_numpy(np.ascontiguousarray(x)).cuda(), engine="fx")
    cuda.cuda.synchronize()
    return y.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024, 2048, 4096])
def test_values_and_partial_tiles(cuda, n):
    """Every plan, one transform past a tile and alone, values of one and of
    twelve decades: each transform to 4e-15 (7 units a component of the last
    pass, 2^-49 of the largest input at N = 4096 and 2^-53 at N = 64, over
    outputs of sqrt(N) times the inputs' rms, a fifth of the largest or more)."""
    import fft_onchip_gb300 as F
    cur = F.plan_query(n, F.ENGINE_FX)
    try:
        for v in range(cur["variants"]):
            F.plan_select(n, F.ENGINE_FX, v)
            tpb = F.plan_query(n, F.ENGINE_FX)["transforms_per_block"]
            for batch in (1, tpb + 1):
                x = np.concatenate([inputs.normal(n, batch, seed=n + v), inputs.loguniform(n, batch, seed=n + v)])[::2]
                y, ref = _fft(cuda, x), O.fft_f64(x)
                err = np.linalg.norm(y - ref, axis=1) / np.linalg.norm(ref, axis=1)
                assert err.max() < 4e-15, (n, v, batch, err.max())
    finally:
        F.plan_select(n, F.ENGINE_FX, cur["variant"])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 512, 4096])
def test_extreme_exponents(cuda, n):
    """Exponent fields that read as binary32 infinities and NaNs (values from
    2^1017 up), as binary32 subnormals (below 2^-1015), and both in one
    transform: a few points each, so that no output overflows."""
    rng = np.random.default_rng(n)
    rows = []
    for e in (1016, 1017, 1018, 1020, 1021, -1014, -1015, -1016, -1018):
        for spread in (0, 40, 1900):
            x = np.zeros(n, dtype=np.complex128)
            at = rng.choice(n, 3, replace=False)
            x[at] = np.ldexp(rng.uniform(0.5, 1.0, 3), e) + 1j * np.ldexp(rng.uniform(-1.0, -0.5, 3), e)
            if spread and abs(e - spread) < 1060:
                x[(at[0] + 1) % n] = np.ldexp(0.75, e - spread)
            rows.append(x)
    x = np.array(rows)
    y = _fft(cuda, x)
    assert np.isfinite(y.view(np.float64)).all()
    # the same transforms at an ordinary scale, scaled back exactly
    e = np.frexp(np.abs(x.view(np.float64)).max(axis=1))[1]
    down = np.ldexp(x.view(np.float64), -e[:, None]).view(np.complex128)
    ref = O.fft_f64(down)
    got = np.ldexp(y.view(np.float64), -e[:, None]).view(np.complex128)
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    # subnormal results keep the binary64 grid: 2^-1074 against 2^-1018
    # 7 units of 2^-49 a component over values of at least the largest input
    assert err[e > -1000].max() < 2e-14 and err[e <= -1000].max() < 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 1024, 4096])
def test_non_finite_and_zero(cuda, n):
    x = inputs.uniform(n, 4, seed=3)
    x[0] = 0.0
    x[1, n // 3] = np.inf
    x[2, 5] = complex(0.0, np.nan)
    y = _fft(cuda, x)
    assert (y[0] == 0).all() and np.isnan(y[1:3].view(np.float64)).all() and np.isfinite(y[3].view(np.float64)).all()
