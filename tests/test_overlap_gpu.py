"""Launches that may be scheduled while the kernel before them drains: every
result must be what a synchronised sequence of the same calls gives, bit for
bit, in a chain of calls, with other kernels in between, and under capture."""
import pytest

from fft_onchip_gb300 import inputs

pytestmark = pytest.mark.gpu

# one transform, a partial wave, several waves
CASES = [(8, 700, "fx"), (64, 1, "fx"), (64, 20000, "fx"), (256, 3000, "f64"), (512, 900, "fx"), (1024, 1500, "fx"),
         (4096, 3, "fx"), (4096, 700, "fx"), (4096, 400, "split_bf16x3"), (512, 2000, "split_exact")]


@pytest.mark.parametrize("n,batch,engine", CASES)
def test_chain_in_place(cuda, fftoc_lib, n, batch, engine):
    import fft_onchip_gb300 as F
    x = cuda.from_numpy(inputs.normal(n, batch, seed=n)).cuda()
    steps = 6

    def chain(buf, sync):
        for _ in range(steps):
            F.fft(buf, out=buf, engine=engine)
            if sync:
                cuda.cuda.synchronize()
            buf.mul_(1.0 / n ** 0.5)  # another library's kernel between two of ours
            F.fft(buf, out=buf, engine=engine)  # and ours right behind it, then behind ours
            if sync:
                cuda.cuda.synchronize()
            F.fft(buf, out=buf, engine=engine)
            if sync:
                cuda.cuda.synchronize()
            buf.mul_(1.0 / n)
        return buf

    want = chain(x.clone(), True)
    got = chain(x.clone(), False)
    cuda.cuda.synchronize()
    assert cuda.equal(cuda.view_as_real(got), cuda.view_as_real(want))
    # the same chain captured once and replayed on other data
    buf = x.clone()
    s = cuda.cuda.Stream()
    s.wait_stream(cuda.cuda.current_stream())
    with cuda.cuda.stream(s):
        chain(buf, False)
    cuda.cuda.current_stream().wait_stream(s)
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g):
        chain(buf, False)
    for _ in range(2):
        buf.copy_(x)
        g.replay()
    cuda.cuda.synchronize()
    assert cuda.equal(cuda.view_as_real(buf), cuda.view_as_real(want))
    assert fftoc_lib.fftoc_device_error_check() == 0


def test_two_streams_and_refilled_inputs(cuda):
    """Two streams of calls over buffers that are refilled between calls."""
    import fft_onchip_gb300 as F
    n, batch, rounds = 512, 3000, 8
    src = [cuda.from_numpy(inputs.uniform(n, batch, seed=k)).cuda() for k in range(rounds)]
    want = []
    for k in range(rounds):
        want.append(F.fft(src[k], engine="fx"))
        cuda.cuda.synchronize()
    streams = [cuda.cuda.Stream() for _ in range(2)]
    bufs = [cuda.empty_like(src[0]) for _ in streams]
    outs = [[cuda.empty_like(src[0]) for _ in range(rounds)] for _ in streams]
    cuda.cuda.synchronize()
    for k in range(rounds):
        for i, st in enumerate(streams):
            with cuda.cuda.stream(st):
                bufs[i].copy_(src[k])
                F.fft(bufs[i], out=outs[i][k], engine="fx")
                F.fft(bufs[i], out=bufs[i], engine="fx")
    cuda.cuda.synchronize()
    for i in range(len(streams)):
        for k in range(rounds):
            assert cuda.equal(cuda.view_as_real(outs[i][k]), cuda.view_as_real(want[k])), (i, k)
