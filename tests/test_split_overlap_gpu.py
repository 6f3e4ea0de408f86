"""The split-form kernels' overlapped launches: one CTA, the largest grid below
and the first inside the sizes launched without overlap, a few tiles a CTA, and
the first batch with too many tiles for it: chains of calls against the
synchronised sequence, bit for bit, and under capture."""
import pytest

from test_overlap_gpu import test_chain_in_place as chain_in_place

pytestmark = pytest.mark.gpu

# N, transforms per CTA, CTAs per SM
PLANS = [("split_bf16x3", 16, 16, 2), ("split_bf16x3", 1024, 2, 4), ("split_tf32x2", 4096, 2, 2), ("split_exact", 64, 32, 2),
         ("split_exact", 4096, 2, 1)]


@pytest.mark.parametrize("engine,n,tpb,per_sm", PLANS)
def test_grids(cuda, fftoc_lib, engine, n, tpb, per_sm):
    wave = cuda.cuda.get_device_properties(0).multi_processor_count * per_sm
    for tiles in (1, wave // 2, wave // 2 + 1, 3 * wave - 1, 16 * wave + 1):
        chain_in_place(cuda, fftoc_lib, n, tiles * tpb, engine)
