"""The plan of a call: the library's choice by batch while none is selected,
a selected one for every batch, and the way back to the library's choice."""
import pytest

from fft_onchip_gb300 import _lib
from test_small_batch_gpu import PLANS

SMS = 152


def by_batch(n, engine, batch):
    return _lib.plan_for_batch(n, _lib.ENGINES[engine], batch, SMS)["variant"]


@pytest.mark.parametrize("engine", ["fx", "f64"])
@pytest.mark.parametrize("n", _lib.SIZES)
def test_choice_by_batch_and_back(fftoc_lib, n, engine):
    """At each limit, the batch that it still takes and the first that it does not."""
    eng = _lib.ENGINES[engine]
    plans = PLANS.get((engine, n), ())
    batches = [0, 1, 1 << 40] + [p * SMS + d for p, _ in plans for d in (-1, 0, 1)]
    want = {b: next((v for p, v in plans if b <= p * SMS), 0) for b in batches}
    assert _lib.plan_selected(n, eng) is None
    assert {b: by_batch(n, engine, b) for b in batches} == want
    other = _lib.plan_query(n, eng)["variants"] - 1
    for v in (0, other):  # 0 is a selection like the others
        _lib.plan_select(n, eng, v)
        assert _lib.plan_selected(n, eng) == v
        assert {by_batch(n, engine, b) for b in batches} == {v}
    _lib.plan_restore(n, eng, None)
    assert _lib.plan_selected(n, eng) is None
    assert {b: by_batch(n, engine, b) for b in batches} == want
    _lib.plan_restore(n, eng, other)
    assert _lib.plan_selected(n, eng) == other


def test_engines_with_one_plan(fftoc_lib):
    for n, engine in ((8, _lib.ENGINE_DMMA), (512, _lib.ENGINE_SPLIT_EXACT)):
        _lib.plan_select(n, engine, 0)
        assert _lib.plan_selected(n, engine) is None
        _lib.plan_restore(n, engine, None)
        assert _lib.plan_for_batch(n, engine, 1, SMS) == _lib.plan_query(n, engine)


def test_errors(fftoc_lib):
    import ctypes
    info, v = _lib.PlanInfo(), ctypes.c_int()
    L, fx = fftoc_lib, _lib.ENGINE_FX
    assert L.fftoc_plan_query_batch(60, fx, 1, SMS, ctypes.byref(info)) == 1
    assert L.fftoc_plan_query_batch(64, fx, -1, SMS, ctypes.byref(info)) == 2
    assert L.fftoc_plan_query_batch(64, fx, 1, 0, ctypes.byref(info)) == 2
    assert L.fftoc_plan_query_batch(64, fx, 1, SMS, None) == 2
    assert L.fftoc_plan_selected(60, fx, ctypes.byref(v)) == 1
    assert L.fftoc_plan_selected(64, fx, None) == 2
    assert L.fftoc_plan_unselect(60, fx) == 1
    assert L.fftoc_plan_unselect(64, 99) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("n,engine,batch", [(8, "fx", 1000), (32, "f64", 700), (64, "f64", 3648), (256, "fx", 1), (512, "fx", 761),
                                            (256, "fx", 38912), (256, "fx", 38913), (1024, "f64", 33), (2048, "fx", 777)])
def test_all_buffers_take_one_plan(cuda, fftoc_lib, n, engine, batch):
    """Device, pinned, pageable and allocation-free calls give the same bits."""
    import fft_onchip_gb300 as F
    from fft_onchip_gb300 import inputs
    x = cuda.from_numpy(inputs.normal(n, batch, seed=n)).pin_memory()
    want = cuda.view_as_real(F.fft(x.cuda(), engine=engine).cpu())
    same = lambda y: cuda.equal(cuda.view_as_real(y), want)
    assert same(F.fft_host(x, out=cuda.empty_like(x).pin_memory(), engine=engine))
    assert same(cuda.from_numpy(F.fft_host(x.numpy().copy(), engine=engine)))
    if x.numel() * 16 <= 32 << 20:
        y = cuda.empty_like(x)
        s = cuda.cuda.current_stream()
        assert fftoc_lib.fftoc_c2c_fwd_host_noalloc(n, x.data_ptr(), y.data_ptr(), batch, F.ENGINES[engine], s.cuda_stream) == 0
        s.synchronize()
        assert same(y)


@pytest.mark.gpu
@pytest.mark.parametrize("selected", [None, 0, 3])
def test_tuner_puts_the_selection_back(cuda, fftoc_lib, selected):
    from fft_onchip_gb300 import tune
    _lib.plan_restore(128, _lib.ENGINE_FX, selected)
    tune.time_variants(128, "fx", gib=0.001, reps=1, warmup=1, rounds=1)
    assert _lib.plan_selected(128, _lib.ENGINE_FX) == selected
