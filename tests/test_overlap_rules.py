"""Kernels whose launch overlaps the kernel before them: the compiler may move
the loads of the cache-hint intrinsics above the wait at their start, so the
files that hold such kernels use the loads of gb_common.cuh instead."""
import os
import re

import pytest

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libgrid_b200", "csrc", "cuda")


def _code(name):
    with open(os.path.join(CUDA, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _overlapping():
    return sorted(n for n in os.listdir(CUDA) if n != "gb_common.cuh" and "grid_wait(" in _code(n))


def test_files_found():
    assert "gb_cn.cu" in _overlapping() and "gb_fft_impl.cuh" in _overlapping()


@pytest.mark.parametrize("name", _overlapping())
def test_no_cache_hint_intrinsics(name):
    assert not re.findall(r"__ld(?:cg|cs|ca|cv|lu)\(", _code(name))


def test_tables_built_on_the_stream_are_read_after_a_plain_launch():
    """Every sweep's launch takes the word of the function that builds tables."""
    code = _code("gb_cn.cu")
    launches = re.findall(r"cn_launch\w*(?:<\w+>)?\((.*?)\)+;", code.split("int gb_cn_step")[1])
    assert len(launches) == 2 and all(a.split(",")[-1].strip() == "built" for a in launches)
    assert "overlap = !built &&" in code
