"""fftoc_c2c_fwd_host on pinned buffers: the direct launch (binary64 and
fixed-point engines) and the staged chunks (split engines, pageable memory)
give the device-buffer call's bits, for one transform, ragged counts and
several chunks, in place and out of place, and inside a pinned allocation."""
import pytest

from fft_onchip_gb300 import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,engine", [(8, 1, "fx"), (16, 5003, "fx"), (32, 700, "f64"), (64, 40001, "fx"),
                                            (256, 20011, "fx"), (512, 3, "fx"), (1024, 1000, "f64"), (2048, 777, "fx"),
                                            (4096, 161, "fx"), (256, 20011, "split_bf16x3"), (512, 3001, "split_exact"),
                                            (8, 3000, "dmma")])
def test_pinned_matches_device_call(cuda, n, batch, engine):
    import fft_onchip_gb300 as F
    x = cuda.from_numpy(inputs.normal(n, batch + 2, seed=n)).pin_memory()
    want = F.fft(x[1:-1].cuda(), engine=engine).cpu()
    guard = cuda.full_like(x, float("nan")).pin_memory()
    out = guard[1:-1]                                       # inside a pinned allocation
    F.fft_host(x[1:-1], out=out, engine=engine)
    eq = lambda a, b: cuda.equal(cuda.view_as_real(a), cuda.view_as_real(b))
    assert eq(out, want)
    assert cuda.isnan(guard[0]).all() and cuda.isnan(guard[-1]).all()
    F.fft_host(x[1:-1], out=x[1:-1], engine=engine)         # in place
    assert eq(x[1:-1], want)


def test_pinned_and_pageable_mixed(cuda):
    import fft_onchip_gb300 as F
    n, batch = 128, 3000
    x = cuda.from_numpy(inputs.uniform(n, batch, seed=2))
    want = F.fft(x.cuda()).cpu()
    for a, b in ((x.pin_memory(), cuda.empty_like(x)), (x, cuda.empty_like(x).pin_memory()), (x, cuda.empty_like(x))):
        F.fft_host(a, out=b)
        assert cuda.equal(cuda.view_as_real(b), cuda.view_as_real(want))


def test_order_on_the_callers_stream(cuda):
    """After earlier work on the stream, before later work, and under capture."""
    import fft_onchip_gb300 as F
    n, batch = 512, 2000
    src = cuda.from_numpy(inputs.uniform(n, batch, seed=5)).cuda()
    h = cuda.empty(batch, n, dtype=src.dtype, pin_memory=True)
    o = cuda.empty_like(h).pin_memory()
    want = F.fft(src)
    got = cuda.empty_like(src)
    s = cuda.cuda.Stream()
    s.wait_stream(cuda.cuda.current_stream())

    def body():
        h.copy_(src, non_blocking=True)
        F.fft_host_ptr(n, h.data_ptr(), o.data_ptr(), batch, cuda.cuda.current_stream().cuda_stream)
        got.copy_(o, non_blocking=True)

    with cuda.cuda.stream(s):
        cuda.cuda._sleep(1000000)
        body()
    s.synchronize()
    assert cuda.equal(cuda.view_as_real(got), cuda.view_as_real(want))
    got.zero_()
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g):
        body()
    g.replay()
    cuda.cuda.synchronize()
    assert cuda.equal(cuda.view_as_real(got), cuda.view_as_real(want))
