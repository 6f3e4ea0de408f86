"""Kernels that are resident while the one before them still writes their input
(launches with the overlap attribute) read the caller's data with coherent
loads: a non-coherent one (__ldg) is defined only for memory that nothing
writes during the kernel's lifetime.  __ldg is left to the constant tables and
to the split forms' kernels of plain launches."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fft_onchip_gb300", "csrc")
TABLES = re.compile(r"^(bmat|tw|c\.tws?|base|sums)\b")
PLAIN = re.compile(r"if constexpr \(OVERLAP\) return load_point\(p\);\s*else return __ldg\(p\);")


def source(name, start=None):
    """A file's text from `start` on, comments removed."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    return text[text.index(start):] if start else text


@pytest.mark.parametrize("name,start", [("fft_split.cuh", "struct SplitCtx"), ("fft_exact.cuh", "struct ExactCtx"),
                                        ("fft_kernel.cuh", "fft_fwd_kernel("), ("fft_persistent.cuh", "fft_fwd_persistent(")])
def test_read_only_loads_are_of_tables(name, start):
    text = source(name, start)
    assert "after_previous();" in text
    loads = re.findall(r"__ldg\(\s*([^()]*)", PLAIN.sub("", text))
    assert [a for a in loads if not TABLES.match(a)] == []


def test_split_kernel_of_each_launch():
    """Only the kernel compiled with coherent loads is launched with the overlap."""
    assert PLAIN.search(source("fft_split.cuh"))
    kernels = source("kernels_split.cu")
    assert re.findall(r"d\.(fn\w*) = \(const void\*\)&\w+<[^;]*?(true|false)>;", kernels) == \
        [("fn", "false"), ("fn_overlap", "true")] * 2
    launch = source("api_split.cu", "fftoc_status launch_split(")
    assert re.findall(r"launch_overlapped\(([^,]*),.*?(\w+)\);", launch) == [("overlap ? d.fn_overlap : d.fn", "overlap")]


@pytest.mark.parametrize("name", ["fft_split.cuh", "fft_exact.cuh"])
def test_no_load_past_the_batch(name):
    """A clamped load would read a transform that another CTA may be storing."""
    assert not re.search(r"batch - 1\)? \* N", source(name, "after_previous();"))
