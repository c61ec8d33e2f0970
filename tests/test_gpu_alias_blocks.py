"""Alias sampling through the table's alias blocks (tables of more than 2^22 entries) against
sampling from the table alone: the same samples, bit for bit, at block and tile edges, for every
way the aliases of a block can be encoded or not, in both generator modes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import weights_lognormal, weights_precision, weights_uniform, weights_zipf
from gpu_util import h2d

pytestmark = pytest.mark.gpu

BASE = 1 << 22


def _equal(n, seed):
    return np.full(n, 0.75, np.float32)  # no heavy item: every bucket keeps itself


def _two_values(n, seed):
    w = np.ones(n, np.float32)
    w[np.random.default_rng(seed).random(n) < 0.5] = 3.0
    return w


def _few_lights(n, seed):
    """Almost all items slightly heavy: light buckets far apart, long runs of heavy ones."""
    w = np.full(n, 1.0, np.float32)
    w[np.random.default_rng(seed).random(n) < 0.02] = 0.01
    return w


def _one_giant(n, seed):
    w = np.full(n, 1e-3, np.float32)
    w[n // 3] = np.float32(n)  # every light bucket aliases one far item
    return w


GENS = {"uniform": weights_uniform, "zipf": weights_zipf, "lognormal": weights_lognormal,
        "precision": weights_precision, "equal": _equal, "two_values": _two_values,
        "few_lights": _few_lights, "one_giant": _one_giant}


def _check(pkg, torch, n, gen, rng, precision, split, offset, s=200_003):
    W = pkg.wrs
    cfg = W.AliasTableConfig(split, rng=rng, scan_precision=precision,
                             split_full_light=precision == W.SCAN_FLOAT_FLOAT)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(GENS[gen](n, n & 0xffff)))
    wrs.build(None, b, n)
    table = b.internals.views()["alias_table"]
    # an output that is only 4-byte aligned, and one that is 16-byte aligned
    for shift in (1, 0):
        out = torch.full((2, s + 1), -1, dtype=torch.int32, device="cuda")
        got, ref = out[0][shift:shift + s - shift], out[1][shift:shift + s - shift]
        m = got.numel()
        pkg.wrs.check(pkg.wrs.lib().wrs_sample_at(wrs.handle.ptr, None, b.internals.ptr, n, m, 7,
                                                  offset, got.data_ptr()))
        wrs.alias_sample(None, table, n, m, 7, offset, ref.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(out[0], out[1])
        assert int(got.min()) >= 0 and int(got.max()) < n


@pytest.mark.parametrize("rng", [0, 1])
@pytest.mark.parametrize("gen", sorted(GENS))
def test_blocks_equal_the_table(pkg, cuda, gen, rng):
    W = pkg.wrs
    _check(pkg, cuda, BASE + 4096 + 33, gen, rng, W.SCAN_FLOAT_FLOAT, 12, 0)


@pytest.mark.parametrize("rest", [1, 31, 32, 33, 4095])
def test_block_edges(pkg, cuda, rest):
    _check(pkg, cuda, BASE + rest, "uniform", 1, pkg.wrs.SCAN_COMPENSATED, 8, (1 << 32) - 77)


def test_overlapping_subproblems(pkg, cuda):
    """FP32 prefixes: splits step back and subproblems overlap, so aliases break the order."""
    for rng in (0, 1):
        _check(pkg, cuda, (1 << 25) + 17, "uniform", rng, pkg.wrs.SCAN_FP32, 2, 5)
