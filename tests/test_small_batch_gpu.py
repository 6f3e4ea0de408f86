"""The fixed-point engine's plans for small batches: while no plan is selected,
batches up to a per-size number of transforms per SM run the size's
small-batch plan, larger ones variant 0.  Each is compared bit for bit with the
same plan selected, in a process of its own (a selection holds for the rest of
the process)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# transforms per SM, variant
PLANS = {8: (512, 4), 16: (128, 5), 32: (512, 6), 64: (32, 8), 128: (512, 8), 256: (256, 8), 512: (5, 8), 1024: (3, 9),
         2048: (6, 1)}

SCRIPT = """
import sys, torch
import fft_onchip_gb300 as F
n, per_sm, small = map(int, sys.argv[1:])
limit = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
q = F.plan_query(n, F.ENGINE_FX)
assert q["variant"] == 0
tpb = F.plan_query(n, F.ENGINE_FX, variant=small)["transforms_per_block"]
torch.manual_seed(n)
x = torch.randn(limit + 1, n, dtype=torch.complex128, device="cuda")
batches = sorted({1, tpb + 1, limit - 1, limit, limit + 1})
bits = lambda y: torch.view_as_real(y).view(torch.int64)
default = {b: F.fft(x[:b], engine="fx") for b in batches}
ref = torch.fft.fft(x)
for b in batches:
    assert ((default[b] - ref[:b]).norm() / ref[:b].norm()).item() < 1e-13, b
    v = small if b <= limit else 0
    F.plan_select(n, F.ENGINE_FX, v)
    assert torch.equal(bits(F.fft(x[:b], engine="fx")), bits(default[b])), (b, v)
F.plan_select(n, F.ENGINE_FX, 0)  # a selected plan serves every batch
y = F.fft(x, engine="fx")
assert torch.equal(bits(F.fft(x[:1], engine="fx")), bits(y[:1]))
"""


@pytest.mark.gpu
@pytest.mark.parametrize("n", sorted(PLANS))
def test_plan_by_batch(cuda, fftoc_lib, n):
    per_sm, variant = PLANS[n]
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(n), str(per_sm), str(variant)], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
