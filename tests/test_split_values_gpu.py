"""Split-form transforms whose values or outputs leave the conversions' fast
forms: zeros, values below the FP32 range beside ordinary ones, outputs that
are exactly zero, and non-finite rows beside finite ones in one tile."""
import numpy as np
import pytest

from fft_onchip_gb300 import inputs
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = {"split_bf16x3": 5e-6, "split_tf32x2": 5e-6, "split_exact": 1e-11}


@pytest.mark.parametrize("n", [16, 32, 512, 2048, 4096])
@pytest.mark.parametrize("engine", sorted(TOL))
def test_rows_off_the_fast_forms(cuda, fftoc_lib, n, engine):
    import fft_onchip_gb300 as F
    tpb = F.plan_query(n, F.ENGINES[engine])["transforms_per_block"]
    rows = 8 * max(1, tpb) + 3
    x = inputs.normal(n, rows, seed=n)
    x[0::8] = 1.0                                 # constant: one output, the others zero
    x[1::8, n // 2:] = 0.0                        # half zeros
    x[2::8, 1::2] *= 1e-60                        # below the FP32 range beside ordinary values
    x[3::8] = 0.0
    x[4::8, 3] = -0.0
    x[5::8] *= 1e25                               # out of the unscaled range
    x[6::8, n - 1] = np.inf
    y = F.fft(cuda.from_numpy(x).cuda(), engine=engine)
    cuda.cuda.synchronize()
    y = y.cpu().numpy()
    bad = np.arange(rows) % 8 == 6
    zero = np.arange(rows) % 8 == 3
    assert (y[zero] == 0).all()
    assert not np.isfinite(y[bad].view(np.float64)).all(axis=1).any()
    ok = ~(bad | zero)
    ref = O.fft_f64(x[ok])
    err = np.linalg.norm(y[ok] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    # FP32 data and accumulation (24 bits a product) over at most three passes
    assert err.max() < TOL[engine], (n, engine, err.max())
    assert fftoc_lib.fftoc_device_error_check() == 0
