"""fft_ptr's integer arguments may be anything that int() takes: Python, numpy
(scalars and arrays of one value) and torch integers, and integral floats."""
import numpy as np
import pytest
import torch

from fft_onchip_gb300 import _lib


@pytest.mark.parametrize("kind", [int, np.int32, np.int64, np.array, np.float64, float, torch.tensor, str])
@pytest.mark.parametrize("n,status", [(48, 1), (64, 2)])
def test_sizes(fftoc_lib, kind, n, status):
    import fft_onchip_gb300 as F
    for engine in ("auto", 0, "fx", np.int64(2)):
        with pytest.raises(F.FftocError) as e:  # no such size; a negative batch
            F.fft_ptr(kind(n), 1 << 20, 1 << 20, -1, engine=engine)
        assert e.value.status == status
