"""The workloads whose speed counts, as a user's program runs them through the public entry points.

Every case is one call: a batch of equal transforms on device buffers (``kind`` "batch"), a mixed-size batch with
an offset table ("uneven"), or a batch in pinned host memory ("host").  ``engine`` is the arithmetic asked for.
Sizes are those of the benchmark's configurations (64-point batch of 65,536; the 1 GiB sweep; the split-precision
families; 200,000 mixed transforms) and, between them, generic ones: a single transform, a few dozen, ragged counts.
"""
import math

import numpy as np
import torch

import fft_onchip_gb300 as F
from fft_onchip_gb300 import inputs

SIZES = (8, 16, 32, 64, 128, 256, 512, 1024, 2048, 4096)
GIB = 1 << 30
LOG_RANGE = math.log(1e6)  # |z| of the log-uniform family in [1e-6, 1e6]


def _batch(name, n, batch, engine="auto", family="normal"):
    return {"name": name, "kind": "batch", "n": n, "batch": batch, "engine": engine, "family": family}


def listed():
    return [
        # one transform: an interactive call, all latency
        _batch("single_n64", 64, 1, family="uniform"),
        # a handful of long transforms, e.g. the channels of one frame: far fewer than the SMs can hold
        _batch("frame_n4096_b24", 4096, 24),
        # the small configuration: 65,536 64-point transforms, uniform values
        _batch("small_n64_b65536", 64, 65536, family="uniform"),
        # an ordinary batch with a count that no tile divides, of a size between the sweep's
        _batch("ragged_n1024_b5003", 1024, 5003),
        # the sweep's ends and middle, 1 GiB of input: streaming use
        _batch("sweep_n16", 16, GIB // (16 * 16)),
        _batch("sweep_n512", 512, GIB // (512 * 16)),
        _batch("sweep_n4096", 4096, GIB // (4096 * 16)),
        # callers that want IEEE binary64 arithmetic throughout
        _batch("ieee_n256_b16411", 256, 16411, engine="f64"),
        # the split-precision form: values over twelve decades at the BF16x3 accuracy, and the exact-slice form
        _batch("split_bf16x3_n4096", 4096, GIB // (4096 * 16), engine="split_bf16x3", family="loguniform"),
        _batch("split_exact_n512", 512, GIB // (512 * 16), engine="split_exact"),
        # 200,000 transforms of mixed sizes, packed back to back, in one call on a plan kept between batches
        {"name": "uneven_200k", "kind": "uneven", "count": 200000, "engine": "auto", "family": "uniform"},
        # data in pinned host memory in and out: a call of some 80 MB each way
        {"name": "host_n256_b20011", "kind": "host", "n": 256, "batch": 20011, "engine": "auto", "family": "normal"},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(("uniform", "normal", "loguniform"))
    kind = rng.choice(("auto",) * 5 + ("f64", "split_bf16x3", "split_tf32x2", "split_exact", "uneven", "host"))
    if kind == "uneven":
        return {"kind": "uneven", "count": _spread(rng, 100, 200000), "engine": "auto", "family": family}
    n = rng.choice(SIZES[1:] if kind.startswith("split") else SIZES)
    if kind == "host":
        most = (128 << 20) // (16 * n)
        return {"kind": "host", "n": n, "batch": _spread(rng, 1, most), "engine": "auto", "family": family}
    # IEEE arithmetic runs at a tenth of the memory's rate: 64 MiB of it cost what 1 GiB costs elsewhere
    most = ((64 << 20) if kind == "f64" else GIB) // (16 * n)
    return {"kind": "batch", "n": n, "batch": _spread(rng, 1, most), "engine": kind, "family": family}


def _values(count, family, seed):
    """`count` complex128 values on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if family == "loguniform":
        x = torch.empty(count, 2, dtype=torch.float64, device="cuda").uniform_(0.0, 1.0, generator=g)
        return torch.polar(torch.exp((2.0 * x[:, 0] - 1.0) * LOG_RANGE), 2.0 * math.pi * x[:, 1])
    x = torch.empty(count, 2, dtype=torch.float64, device="cuda")
    if family == "uniform":
        x.uniform_(-1.0, 1.0, generator=g)
    else:
        x.normal_(generator=g)
    return torch.view_as_complex(x)


def _layout(case, seed):
    """The same sizes for every seed, in the seed's order."""
    ns = np.random.default_rng(seed).permutation(inputs.uneven_sizes(case["count"], 0))
    offsets, total = inputs.uneven_layout(ns)
    return ns, offsets, total


def prepare(case, seed):
    if case["kind"] == "uneven":
        ns, offsets, total = _layout(case, seed)
        x = _values(total, case["family"], seed)
        return {"kind": "uneven", "plan": F.UnevenPlan(case["count"], case["engine"]), "x": x, "out": torch.empty_like(x),
                "offsets": torch.from_numpy(offsets).cuda(), "ns": torch.from_numpy(ns).cuda()}
    x = _values(case["batch"] * case["n"], case["family"], seed).reshape(case["batch"], case["n"])
    if case["kind"] == "host":
        h = torch.empty(tuple(x.shape), dtype=x.dtype, pin_memory=True)
        h.copy_(x)
        out = torch.empty(tuple(x.shape), dtype=x.dtype, pin_memory=True)
        return {"kind": "host", "x": h, "out": out, "engine": case["engine"]}
    return {"kind": "batch", "x": x, "out": torch.empty_like(x), "engine": case["engine"]}


def run(state):
    if state["kind"] == "uneven":
        return state["plan"](state["x"], state["offsets"], state["ns"], out=state["out"])
    if state["kind"] == "host":
        return F.fft_host(state["x"], out=state["out"], engine=state["engine"])
    return F.fft(state["x"], out=state["out"], engine=state["engine"])


def exact(case, seed):
    if case["kind"] == "uneven":
        ns, offsets, total = _layout(case, seed)
        x = _values(total, case["family"], seed)
        out = torch.empty_like(x)
        for n in np.unique(ns):
            at = torch.from_numpy(offsets[ns == n]).cuda().unsqueeze(1) + torch.arange(int(n), device="cuda")
            out[at] = torch.fft.fft(x[at])
        return out
    x = _values(case["batch"] * case["n"], case["family"], seed).reshape(case["batch"], case["n"])
    y = torch.fft.fft(x)
    return y.cpu() if case["kind"] == "host" else y


def work(case):
    """Each complex128 point read once and written once (over the host link too, for host data), and 5 n log2 n
    operations a transform."""
    if case["kind"] == "uneven":
        ns = _layout(case, 0)[0].astype(np.float64)
        # an int64 offset and an int32 size for each transform
        return {"bytes": float(32.0 * ns.sum() + 12.0 * len(ns)), "flops": float((5.0 * ns * np.log2(ns)).sum())}
    points = case["batch"] * case["n"]
    return {"bytes": 32.0 * points, "flops": 5.0 * points * math.log2(case["n"])}
