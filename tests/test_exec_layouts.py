"""Twiddle tables of the device-side executors by layout: objects compiled with
an older <fftoc/exec.cuh> ask for the layout that they know, by the old entry's
name, and get it; a layout from a newer header is refused."""
import ctypes
import re
import os

import numpy as np
import pytest

from fft_onchip_gb300 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_unknown_layouts_are_refused(fftoc_lib):
    out, r = ctypes.c_void_p(1), (ctypes.c_int * 4)(8, 8, 1, 1)
    for layout in (-1, 0, _lib.EXEC_LAYOUT + 1):
        assert fftoc_lib.fftoc_exec_table(64, _lib.ENGINE_FX, r, layout, ctypes.byref(out)) == 7
    assert fftoc_lib.fftoc_exec_table(60, _lib.ENGINE_FX, r, 1, ctypes.byref(out)) == 1


def test_header_and_python_agree():
    header = open(os.path.join(ROOT, "include", "fftoc.h")).read()
    assert int(re.search(r"#define FFTOC_EXEC_LAYOUT (\d+)", header).group(1)) == _lib.EXEC_LAYOUT
    # executors ask for the layout of the header that they are compiled with
    text = open(os.path.join(ROOT, "include", "fftoc", "exec.cuh")).read()
    assert len(re.findall(r"fftoc_exec_table\(N, \w+, radix, FFTOC_EXEC_LAYOUT, ", text)) == 2


def _table(cuda, call, ints):
    out = ctypes.c_void_p()
    assert call(ctypes.byref(out)) == 0
    host = np.empty(ints, dtype=np.int32)
    rt = ctypes.CDLL("libcudart.so.13")
    assert rt.cudaMemcpy(ctypes.c_void_p(host.ctypes.data), out, ctypes.c_size_t(4 * ints), 2) == 0
    return host


@pytest.mark.gpu
@pytest.mark.parametrize("n,radix", [(16, [8, 2]), (64, [8, 8]), (1024, [16, 16, 4]), (4096, [16, 16, 16])])
def test_contents(cuda, fftoc_lib, n, radix):
    r = (ctypes.c_int * 4)(*(radix + [1] * (4 - len(radix))))
    c, s, p = [], [], radix[0]  # entry (m - 1) p + k of each pass: the twiddle of k m
    for R in radix[1:]:
        ang = 2 * np.pi * (np.arange(1, R)[:, None] * np.arange(p)[None, :]).ravel() / (R * p)
        c.append(np.cos(ang))
        s.append(np.sin(ang))
        p *= R
    w = np.stack([np.concatenate(c), -np.concatenate(s)], axis=1)
    old = lambda e, count: _table(cuda, lambda out: fftoc_lib.fftoc_exec_twiddles(n, e, r, out), count)
    new = lambda e, layout, count: _table(cuda, lambda out: fftoc_lib.fftoc_exec_table(n, e, r, layout, out), count)
    # the old entry: 16 bytes each, (cos, -sin) or limbs h 2^30 + l of 2^60 times them
    f64 = old(_lib.ENGINE_F64, 4 * len(w)).view(np.float64).reshape(-1, 2)
    assert np.abs(f64 - w).max() < 1e-15
    limbs = old(_lib.ENGINE_FX, 4 * len(w)).reshape(-1, 2, 2).astype(np.float64)
    assert limbs[..., 1].min() >= 0 and limbs[..., 1].max() < 2 ** 30
    assert np.abs((limbs[..., 0] + limbs[..., 1] / 2 ** 30) / 2 ** 30 - w).max() < 1e-15
    assert np.array_equal(old(_lib.ENGINE_FX, 4 * len(w)), new(_lib.ENGINE_FX, 1, 4 * len(w)))
    # natural words from n = 64 up: the real part's limbs of 2^62 times it come first
    if n >= 64:
        nat = new(_lib.ENGINE_FX, 2, 6 * len(w))[:4 * len(w)].reshape(-1, 4).astype(np.float64)
        assert np.abs((nat[:, 0] + nat[:, 1] / 2 ** 32) / 2 ** 30 - w[:, 0]).max() < 1e-15
    else:
        assert np.array_equal(new(_lib.ENGINE_FX, 2, 4 * len(w)), old(_lib.ENGINE_FX, 4 * len(w)))
