"""A kernel that may start before its predecessor in the stream has ended (it calls mb_grid_dep_wait) reads its operands by
ordinary loads: PTX's read-only path (ld.global.nc, which __ldg and const __restrict__ pointers become) wants data that do
not change while the kernel runs, and nothing keeps such a load behind the wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mace_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


SOURCES = sorted(n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh")))
# the headers whose device functions those kernels are made of have no wait of their own
CHAINED = [n for n in SOURCES if "mb_grid_dep_wait();" in _code(n) or n in ("gemm_u8_tail.cuh", "common.cuh", "sm100_ptx.cuh")]


def test_the_chained_kernels_are_found():
    assert {"gemm_f32_gather.cu", "dwconv_u8.cu", "net_ops_f32.cu", "gemm_u8_tc.cuh", "winograd_f32.cu"} <= set(CHAINED)


@pytest.mark.parametrize("name", CHAINED)
def test_chained_kernels_use_ordinary_loads(name):
    code = _code(name)
    assert not re.findall(r"__ldg\s*\(|ld\.global\.nc|__ldlu", code)
    assert not re.findall(r"\bconst\s+[\w:]+\s*\*\s*__restrict__", code)
