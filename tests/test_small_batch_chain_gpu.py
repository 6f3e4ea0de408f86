"""Small-batch plans in chains of overlapped launches, in place and under
capture, bit for bit against the synchronised sequence: one transform, a ragged
second CTA and the largest batch of each plan."""
import pytest

from test_overlap_gpu import test_chain_in_place as chain_in_place
from test_small_batch_gpu import PLANS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine,n", sorted(PLANS))
def test_chain(cuda, fftoc_lib, engine, n):
    import fft_onchip_gb300 as F
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    for per_sm, v in PLANS[engine, n]:
        assert F.plan_for_batch(n, F.ENGINES[engine], per_sm * sms, sms)["variant"] == v
        tpb = F.plan_query(n, F.ENGINES[engine], variant=v)["transforms_per_block"]
        for batch in {1, tpb + 1, per_sm * sms}:
            chain_in_place(cuda, fftoc_lib, n, batch, engine)
