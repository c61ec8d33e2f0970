"""Alias blocks around the least table size that gets them: the samples of the table alone, whichever
side of the line, for every way a block's aliases are encoded or not, in both generator modes."""
from __future__ import annotations

import pytest

from test_gpu_alias_blocks import GENS, _check

pytestmark = pytest.mark.gpu

LINE = 5 << 20  # the largest table without blocks


@pytest.mark.parametrize("rng", [0, 1])
@pytest.mark.parametrize("gen", sorted(GENS))
def test_blocks_equal_the_table(pkg, cuda, gen, rng):
    _check(pkg, cuda, LINE + 4096 + 33, gen, rng, pkg.wrs.SCAN_FLOAT_FLOAT, 12, 0)


@pytest.mark.parametrize("rest", [0, 1, 31, 32, 33, 4095])
def test_around_the_line(pkg, cuda, rest):
    _check(pkg, cuda, LINE + rest, "uniform", 1, pkg.wrs.SCAN_COMPENSATED, 8, (1 << 32) - 77)


def test_bytes_begin_above_the_line(pkg, cuda):
    """Blocks and heavy bits: 1 byte per weight and 1 bit, above the line only."""
    W = pkg.wrs
    handle = W.Handle(W.AliasTableConfig(2, scan_precision=W.SCAN_COMPENSATED))
    at, above, far = (W.lib().wrs_buffers_bytes(handle.ptr, n) for n in (LINE, LINE + 1, 2 * LINE))
    per_weight = (far - above) / (LINE - 1)  # with the blocks
    assert 0 <= above - at - LINE * 9 // 8 < 8192
    assert abs(per_weight - (at / LINE + 9 / 8)) < 0.01
