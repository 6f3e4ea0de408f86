import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300); run with -m gpu")


@pytest.fixture(scope="session")
def fftoc_lib():
    """libfftoc.so, built in-tree if it is not there yet (nvcc cross-compiles)."""
    from fft_onchip_gb300 import _lib, build
    if not os.path.exists(_lib.LIB_PATH):
        build.build()
    return _lib.load()


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.fixture(autouse=True)
def plan_selections():
    """Each test starts with the library's own choice of plans: a selection holds
    for the rest of the process."""
    yield
    from fft_onchip_gb300 import _lib
    if _lib._lib is not None:
        for n in _lib.SIZES:
            for engine in (_lib.ENGINE_F64, _lib.ENGINE_FX):
                _lib.plan_restore(n, engine, None)
