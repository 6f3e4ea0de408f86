"""The plans for small batches: while no plan is selected, batches up to a
per-size number of transforms per SM run the size's small-batch plan, larger
ones the next or variant 0.  Each is compared bit for bit with the
same plan selected, in a process of its own (a selection holds for the rest of
the process)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# engine, n: ((transforms per SM, variant), ...) by rising limit
PLANS = {
    ("fx", 8): ((512, 4),), ("fx", 16): ((128, 5),), ("fx", 32): ((512, 6),), ("fx", 64): ((32, 8),),
    ("fx", 128): ((16, 9), (512, 8)), ("fx", 256): ((8, 9), (256, 8)), ("fx", 512): ((5, 8),), ("fx", 1024): ((3, 9),),
    ("fx", 2048): ((6, 1),),
    ("f64", 8): ((192, 4),), ("f64", 16): ((48, 5),), ("f64", 32): ((48, 6),), ("f64", 64): ((24, 8),),
    ("f64", 128): ((12, 8),), ("f64", 256): ((12, 8),), ("f64", 512): ((7, 8),), ("f64", 1024): ((16, 10),),
}

SCRIPT = """
import sys, torch
import fft_onchip_gb300 as F
engine, n = sys.argv[1], int(sys.argv[2])
plans = [tuple(map(int, a.split(","))) for a in sys.argv[3:]]
eng = F.ENGINES[engine]
sms = torch.cuda.get_device_properties(0).multi_processor_count
assert F.plan_query(n, eng)["variant"] == 0
batches = {1}
for per_sm, v in plans:
    tpb = F.plan_query(n, eng, variant=v)["transforms_per_block"]
    batches |= {tpb + 1, per_sm * sms - 1, per_sm * sms, per_sm * sms + 1}
most = max(batches)
torch.manual_seed(n)
x = torch.randn(most, n, dtype=torch.complex128, device="cuda")
bits = lambda y: torch.view_as_real(y).view(torch.int64)
default = {b: F.fft(x[:b], engine=engine) for b in sorted(batches)}
ref = torch.fft.fft(x)
for b in sorted(batches):
    assert ((default[b] - ref[:b]).norm() / ref[:b].norm()).item() < 1e-13, b
    v = next((v for per_sm, v in plans if b <= per_sm * sms), 0)
    F.plan_select(n, eng, v)
    assert torch.equal(bits(F.fft(x[:b], engine=engine)), bits(default[b])), (b, v)
F.plan_select(n, eng, 0)  # a selected plan serves every batch
y = F.fft(x, engine=engine)
assert torch.equal(bits(F.fft(x[:1], engine=engine)), bits(y[:1]))
"""


@pytest.mark.gpu
@pytest.mark.parametrize("engine,n", sorted(PLANS))
def test_plan_by_batch(cuda, fftoc_lib, engine, n):
    plans = ["%d,%d" % p for p in PLANS[engine, n]]
    r = subprocess.run([sys.executable, "-c", SCRIPT, engine, str(n)] + plans, cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
