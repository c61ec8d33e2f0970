"""Cutpoint sampling on the compensated CMF by groups (wrs_sample, many samples) against the
per-sample bisection (the primitive): the same indices for ranges of every width class (below 64,
below 256 and wider candidates), empty cells, ragged ends and offsets, in both generator modes."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import weights_lognormal, weights_precision, weights_uniform, weights_zipf
from gpu_util import h2d

pytestmark = pytest.mark.gpu

GENS = {"uniform": weights_uniform, "zipf": weights_zipf, "lognormal": weights_lognormal,
        "precision": weights_precision}


@pytest.mark.parametrize("rng", [0, 1])
@pytest.mark.parametrize("gen", sorted(GENS))
@pytest.mark.parametrize("n,entry", [(1, 32), (40, 1), (5000, 32), (300_007, 60), (300_007, 130),
                                     (300_007, 400)])
@pytest.mark.parametrize("rest", [0, 37])
def test_groups_equal_the_bisection(pkg, cuda, n, entry, gen, rng, rest):
    W = pkg.wrs
    cfg = W.CutpointConfig(entry, rng=rng, scan_precision=W.SCAN_COMPENSATED)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(GENS[gen](n, n)))
    wrs.build(None, b, n)
    v = b.internals.views()
    s, offset = (1 << 19) + rest, (1 << 32) - 200_000
    out = cuda.full((2, s), -1, dtype=cuda.int32, device="cuda")
    W.check(W.lib().wrs_sample_at(wrs.handle.ptr, None, b.internals.ptr, n, s, 11, offset,
                                  out[0].data_ptr()))
    wrs.cutpoint_sample(None, v["cmf"], n, v["guide_table"], s, 11, offset, out[1].data_ptr())
    cuda.cuda.synchronize()
    assert cuda.equal(out[0], out[1])
    assert int(out[0].min()) >= 0 and int(out[0].max()) < n


@pytest.mark.parametrize("rng", [0, 1])
@pytest.mark.parametrize("entry", [32, 400])
def test_infinite_total(pkg, cuda, entry, rng):
    """Finite weights whose sum exceeds FP32's range: ranges that end in an infinite value."""
    W = pkg.wrs
    n, s = 6 * 4096 + 17, 1 << 19
    w = weights_uniform(n, 3)
    w[7::4096] = 1e38
    cfg = W.CutpointConfig(entry, rng=rng, scan_precision=W.SCAN_COMPENSATED)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, s, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(w))
    wrs.build(None, b, n)
    v = b.internals.views()
    wrs.sample(None, b, n, s, seed=3)
    ref = cuda.empty_like(b.samples)
    wrs.cutpoint_sample(None, v["cmf"], n, v["guide_table"], s, 3, 0, ref.data_ptr())
    cuda.cuda.synchronize()
    assert cuda.equal(b.samples, ref)
