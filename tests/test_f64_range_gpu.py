"""The binary64 engine up to the largest values: every output that is
representable is computed, whatever the intermediate values of the butterflies
would reach, and transforms beside such a one keep their bits."""
import numpy as np
import pytest

from fft_onchip_gb300 import _lib, inputs
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOP = np.finfo(np.float64).max
DOWN = 2.0 ** -600  # squares stay representable


def large_rows(n):
    """Transforms whose outputs are representable, the largest near TOP."""
    rng = np.random.default_rng(n)
    at = np.unique(np.r_[0, 1, n - 1, rng.integers(0, n, 12)])
    rows = np.zeros((3 * len(at) + 4, n), dtype=np.complex128)
    for k, i in enumerate(at):  # impulses: every output of modulus 0.9 TOP
        rows[3 * k, i] = 0.9 * TOP
        rows[3 * k + 1, i] = 0.9j * TOP
        rows[3 * k + 2, i] = 0.9 * TOP * (0.8 - 0.6j)
    rows[-4] = 0.9 * TOP / n
    rows[-3] = 0.9 * TOP / n * np.exp(2j * np.pi * 3 * np.arange(n) / n)
    rows[-2] = 0.6 * TOP / n * (rng.choice((-1, 1), n) + 1j * rng.choice((-1, 1), n))
    rows[-1] = np.where(np.arange(n) % 2 == 0, 0.9 * TOP / n, 1e-300)
    return rows


def check(y, x):
    assert np.isfinite(y.view(np.float64)).all()
    for a, b in zip(y * DOWN, x * DOWN):
        assert O.rel_l2(a[None], O.fft_f64(b[None])) < 1e-14


@pytest.mark.parametrize("n", _lib.SIZES)
def test_every_plan(cuda, fftoc_lib, n):
    import fft_onchip_gb300 as F
    x = large_rows(n)
    d = cuda.from_numpy(x).cuda()
    check(F.fft(d, engine="f64").cpu().numpy(), x)
    for v in range(F.plan_query(n, F.ENGINE_F64)["variants"]):
        F.plan_select(n, F.ENGINE_F64, v)
        check(F.fft(d, engine="f64").cpu().numpy(), x)


@pytest.mark.parametrize("n", _lib.SIZES)
def test_neighbours_keep_their_bits_and_overflows_stay(cuda, fftoc_lib, n):
    import fft_onchip_gb300 as F
    plain = inputs.normal(n, 64, seed=n)
    plain[1::4] *= 1e-306  # sums down to the subnormals
    plain[2::4] *= 1e300 / n
    want = F.fft(cuda.from_numpy(plain).cuda(), engine="f64").cpu().numpy()
    mixed = plain.copy()
    big = large_rows(n)
    where = np.arange(0, 64, 3)
    mixed[where] = big[where % len(big)]
    mixed[3], mixed[6, n // 2], mixed[9, 1] = TOP, np.inf, np.nan
    y = F.fft(cuda.from_numpy(mixed).cuda(), engine="f64").cpu().numpy()
    rest = np.setdiff1d(np.arange(64), where)
    assert np.array_equal(y[rest].view(np.int64), want[rest].view(np.int64))
    assert y[3, 0] == complex(np.inf, 0) and not np.isfinite(y[6]).any() and not np.isfinite(y[9]).any()
    check(y[where[4:]], mixed[where[4:]])


def test_other_entry_points(cuda, fftoc_lib):
    import fft_onchip_gb300 as F
    from fft_onchip_gb300 import onchip
    rows = [large_rows(n)[k] for n in _lib.SIZES for k in (0, 2, -4, -2)]
    ns = np.array([len(r) for r in rows], dtype=np.int32)
    off = np.concatenate([[0], np.cumsum(ns[:-1])]).astype(np.int64)
    y = F.UnevenPlan(len(rows), "f64")(cuda.from_numpy(np.concatenate(rows)).cuda(), cuda.from_numpy(off).cuda(),
                                       cuda.from_numpy(ns).cuda()).cpu().numpy()
    for r, o in zip(rows, off):
        check(y[None, o:o + len(r)], r[None])
    for n in (8, 64, 1024):
        x = large_rows(n)
        check(F.fft_host(x, engine="f64"), x)
        tpb = F.plan_query(n, F.ENGINE_F64)["transforms_per_block"]
        x = np.resize(x, (tpb, n))
        d = cuda.from_numpy(x).cuda()
        _lib.check(fftoc_lib.fftoc_onchip_run(n, F.ENGINE_F64, d.data_ptr(), 1, 1, cuda.cuda.current_stream().cuda_stream))
        check(d.cpu().numpy(), x)


@pytest.mark.parametrize("n", _lib.SIZES)
def test_in_place(cuda, fftoc_lib, n):
    """Tiles that are redone read their inputs again: nothing of them is stored before."""
    import fft_onchip_gb300 as F
    x = large_rows(n)
    x = np.concatenate([x, inputs.normal(n, len(x) // 2, seed=n), x[::-1]])
    for v in range(F.plan_query(n, F.ENGINE_F64)["variants"]):
        F.plan_select(n, F.ENGINE_F64, v)
        d = cuda.from_numpy(x).cuda()
        want = F.fft(d, engine="f64")
        F.fft(d, out=d, engine="f64")
        assert cuda.equal(cuda.view_as_real(d), cuda.view_as_real(want)), v
        check(d.cpu().numpy(), x)
