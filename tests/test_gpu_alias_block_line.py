"""Alias blocks around the least table size that gets them: the samples of the table alone, whichever
side of the line, for every way a block's aliases are encoded or not, in both generator modes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import weights_lognormal, weights_uniform
from gpu_util import d2h, h2d
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


def _unencodable(n, seed):
    """Periods of 11 heavy items and 21 zeros, with half a period's heavy items moved to the start: a
    block's light items go through 11 switches over a gap, which neither steps nor distances hold."""
    w = np.where(np.arange(n) % 32 < 11, np.float32(2.9), np.float32(0.0)).astype(np.float32)
    w[11:17] = 2.9
    last = n // 32 * 32 - 32
    w[last + 5:last + 11] = 0.0
    return w


def _reads_in_eighths(internals) -> int:
    """the control block's count of expected entry reads, two words behind the mean"""
    return int(d2h(internals.views()["mean64"] + 16, 1, np.uint64)[0])


@pytest.mark.parametrize("gen", [weights_uniform, _unencodable])
def test_only_a_build_counts_reads(pkg, cuda, gen):
    """The entry reads the build's blocks cost decide how the table is sampled; total-mass passes into
    the same buffers, alone or in a scan, leave them."""
    W = pkg.wrs
    n, s = LINE + 32, 1 << 18
    # (float-float: FP32 prefixes drift by parts of an item, and with them the periods' phase)
    cfg = W.AliasTableConfig(12, rng=W.RNG_PHILOX4X32_10, scan_precision=W.SCAN_FLOAT_FLOAT,
                             split_full_light=True)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, s, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(gen(n, 1)))
    for _ in range(2):
        wrs.build(None, b, n)
    reads = _reads_in_eighths(b.internals)
    assert (6 * n < reads <= 8 * n) if gen is _unencodable else (n <= reads < 2 * n)
    other = h2d(weights_lognormal(n, 2))
    wrs.total_mass(None, other, n, b.internals)
    wrs.prefix_sum(None, other, n, cuda.empty_like(other), b.internals)
    assert _reads_in_eighths(b.internals) == reads
    wrs.sample(None, b, n, s, seed=3)
    ref = cuda.empty_like(b.samples)
    wrs.alias_sample(None, b.internals.views()["alias_table"], n, s, 3, 0, ref.data_ptr())
    assert cuda.equal(b.samples, ref)


def _denormal(n, seed):
    """A total so small that the mean rounds to zero: every p is infinite or NaN."""
    w = np.zeros(n, np.float32)
    w[np.random.default_rng(seed).choice(n, 50, replace=False)] = np.float32(2.0**-149)
    return w


def _eighths(n, seed):
    """A mean of one and light weights at multiples of an eighth, where the blocks' codes begin, or one
    step of the float beside them."""
    rng = np.random.default_rng(seed)
    eighth = rng.integers(0, 9, n // 2) / np.float32(8.0)
    beside = rng.integers(0, 3, n // 2)
    light = np.where(beside == 0, np.nextafter(eighth, np.float32(0.0)),
                     np.where(beside == 1, eighth, np.nextafter(eighth, np.float32(1.0))))
    return np.concatenate([light, 2.0 - light, np.ones(n - 2 * (n // 2))]).astype(np.float32)


@pytest.mark.parametrize("rng", [0, 1])
@pytest.mark.parametrize("gen", [_denormal, _eighths, _unencodable])
def test_values_at_the_codes_edges(pkg, cuda, monkeypatch, gen, rng):
    monkeypatch.setitem(GENS, "edge", gen)
    _check(pkg, cuda, LINE + 64, "edge", rng, pkg.wrs.SCAN_FLOAT_FLOAT, 12, 0)
