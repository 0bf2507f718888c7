"""The GEMM planner (tile shape, how many parts the last round's tiles are cut into) is host code in the kernel
library; without a device it plans for a B200's 148 SMs, so its choices are checked here on CPU."""

import ctypes
import os

import pytest

LIB = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tandem_b200", "libtb200_cuda.so")
pytestmark = pytest.mark.skipif(not os.path.exists(LIB), reason="the kernel library has not been built")


def plan(m, n, k):
    lib = ctypes.CDLL(LIB)
    out = (ctypes.c_int * 4)()
    lib.tb_gemm_plan(m, n, k, out)
    bm, bn, parts, whole = out
    return bm, bn, parts, whole


def test_whole_rounds_are_never_split():
    for m, n, k in [(8192, 768, 3072), (8192, 3072, 768), (8192, 2304, 768), (3072, 768, 8192), (768, 768, 8192), (1024, 768, 3072)]:
        bm, bn, parts, whole = plan(m, n, k)
        rows, units = (256, 74) if bm == 512 else (bm, 148)  # 512 marks the 256-row tiles of a CTA pair
        tiles = -(-m // rows) * -(-n // bn)
        assert parts >= 1 and 0 <= whole <= tiles
        if parts > 1:
            tail = tiles - whole
            assert whole % units == 0 and 0 < tail and tail * parts <= units  # the parts run on the SMs the last round leaves idle
            assert -(-k // 64) // parts >= 2  # every part keeps at least two k-blocks
        else:
            assert whole == 0


def test_long_reductions_with_few_tiles_are_split():
    assert plan(768, 768, 8192)[2] >= 3      # 36 tiles, 128 k-blocks: the square weight gradient
    assert plan(3072, 768, 8192)[2] == 2     # 72 tiles of 128 x 256, or 36 of a CTA pair
    assert plan(1024, 768, 3072)[2] >= 2     # 48 tiles, 48 k-blocks: one rank's share at 8 GPUs


def test_short_reductions_are_not_split():
    assert plan(1024, 768, 768)[2] == 1      # twelve k-blocks: folding would cost more than it saves
    assert plan(8192, 3072, 768)[:3] == (128, 256, 1) or plan(8192, 3072, 768)[2] <= 2


def test_narrow_outputs_get_narrow_tiles():
    assert plan(8192, 128, 768)[1] == 128


def cut(m, n, k):
    """Which sums a plan cuts: parts, and the uncut region as (full columns, upper rows of the next tile column, its right edge)."""
    bm, bn, parts, whole = plan(m, n, k)
    if parts == 1:
        return 1
    bm = 256 if bm == 512 else bm  # 512 marks the 256-row tiles of a CTA pair
    columns, rows = whole // -(-m // bm) * bn, whole % -(-m // bm) * bm
    return parts, columns, rows, min(columns + bn, n) if rows else columns


@pytest.mark.parametrize("shape,want", [
    ((1024, 768, 2304), (2, 0, 0, 0)), ((8192, 768, 2304), (2, 512, 2560, 768)), ((2304, 768, 8192), (2, 0, 0, 0)),
    ((8192, 768, 3072), (3, 512, 2560, 768)), ((3072, 768, 8192), (2, 0, 0, 0)), ((50304, 1024, 4096), 1),
    ((1024, 1024, 2560), (2, 0, 0, 0)), ((256, 1024, 2560), (3, 0, 0, 0)), ((8192, 2048, 16384), (2, 1536, 7680, 1792)),
    ((16384, 50304, 2048), (2, 50176, 9216, 50304)), ((768, 768, 8192), (4, 0, 0, 0)), ((8192, 3072, 768), 1), ((1537, 1003, 768), 1),
])
def test_the_cuts_of_a_reduction_do_not_depend_on_the_kernel(shape, want):
    """The order in which a product is added up is part of its result (training is compared bit for bit): it belongs to the
    sizes, and a faster tile shape or kernel leaves it alone.  The pinned cuts are those of the first planner."""
    assert cut(*shape) == want
