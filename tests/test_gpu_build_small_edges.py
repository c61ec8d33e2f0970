"""The one-launch build where its pieces take their other ways: shares of more items than its staging
holds, one subproblem for everything, and FP32 carries over several tiles (which go tile by tile)."""
from __future__ import annotations

import numpy as np
import pytest

import test_gpu_build_small as small
from test_gpu_parity import Built, GENS, same_table

pytestmark = pytest.mark.gpu

# (n, split size): a CTA's share above 5212 items, subproblems larger than the distribution
WIDE = [(6000, 6000), (20_000, 7000), (32_768, 8192), (32_768, 5213), (20_000, 40_000)]


@pytest.mark.parametrize("gen", ["uniform", "zipf", "one_giant", "two_values"])
@pytest.mark.parametrize("precision", ["SCAN_COMPENSATED", "SCAN_FLOAT_FLOAT"])
def test_shares_beyond_the_staging(pkg, monkeypatch, gen, precision):
    monkeypatch.setattr(small, "SIZES", WIDE)
    small.test_against_the_stages(pkg, gen, precision)


@pytest.mark.parametrize("gen", sorted(GENS))
@pytest.mark.parametrize("N,split", [(4097, 3), (8192, 8), (20_000, 12), (32_768, 16), (32_768, 8192)])
def test_fp32_over_several_tiles(pkg, cuda, oracle, gen, N, split):
    """The partition as the oracle's, prefixes within FP32's bound of the FP64 ones, the same from build
    to build, and the table that the oracle packs from them."""
    w = GENS[gen](N, N + split)
    b = Built(pkg, w, pkg.AliasTableConfig(split_size=split))
    assert b.status == 0
    idx, elems, hc = oracle.partition(w, b.mean)
    assert b.hc == hc
    assert np.array_equal(b.idx, idx)
    assert np.array_equal(b.elems.view(np.uint32), elems.view(np.uint32))
    ref = oracle.partition_prefix_f64(w, b.mean)
    err = np.abs(b.prefix.astype(np.float64) - ref) / np.maximum(np.abs(ref), 1e-30)
    assert err.max() <= 1e-4, err.max()
    again = Built(pkg, w, pkg.AliasTableConfig(split_size=split))
    assert np.array_equal(again.prefix.view(np.uint32), b.prefix.view(np.uint32))
    table = oracle.split_pack(w, b.idx, b.prefix, b.hc, b.mean, split, elems=b.elems)
    assert same_table(b.table, table)
    assert same_table(again.table, table)
