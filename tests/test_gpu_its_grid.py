"""ITS on the compensated CMF through its grid of cells against the bisection of the CMF alone: the
same indices at totals of every magnitude (the grid's power of two is capped for tiny ones), with
items that share a step with the target, cells with more items than parts, and empty cells."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import weights_lognormal, weights_precision, weights_uniform, weights_zipf
from gpu_util import d2h, h2d

pytestmark = pytest.mark.gpu


def _giants(n, seed):
    """A few items hold nearly all the mass: most cells are empty, the others crowded."""
    w = np.full(n, 1e-6, np.float32)
    w[np.random.default_rng(seed).integers(0, n, 5)] = 1.0
    return w


def _zero_runs(n, seed):
    w = weights_uniform(n, seed)
    w[np.random.default_rng(seed).random(n) < 0.7] = 0.0
    w[n // 2] = 0.5
    return w


GENS = {"uniform": weights_uniform, "zipf": weights_zipf, "lognormal": weights_lognormal,
        "precision": weights_precision, "giants": _giants, "zero_runs": _zero_runs}


@pytest.mark.parametrize("rng", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 2.0**-126, 2.0**-80, 2.0**90])
@pytest.mark.parametrize("gen", sorted(GENS))
@pytest.mark.parametrize("n,entry", [(1, 4), (27, 4), (8193, 1), (300_007, 4), (1_000_003, 40)])
def test_grid_equals_the_bisection(pkg, cuda, n, entry, gen, scale, rng):
    W = pkg.wrs
    cfg = W.ITSConfig(guiding_entry_size=entry, rng=rng, scan_precision=W.SCAN_COMPENSATED)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(GENS[gen](n, n) * np.float32(scale)))
    wrs.build(None, b, n)
    s, offset = 50_001, (1 << 32) - 1234
    out = cuda.full((2, s + 1), -1, dtype=cuda.int32, device="cuda")
    for shift in (1, 0):  # an output that is only 4-byte aligned, and one that is 8-byte aligned
        got, ref = out[0][shift:shift + s], out[1][shift:shift + s]
        W.check(W.lib().wrs_sample_at(wrs.handle.ptr, None, b.internals.ptr, n, s, 9, offset,
                                      got.data_ptr()))
        wrs.its_sample(None, b.internals.views()["cmf"], n, s, 9, offset, ref.data_ptr())
        cuda.cuda.synchronize()
        assert cuda.equal(out[0], out[1])
        assert int(got.min()) >= 0 and int(got.max()) < n


@pytest.mark.parametrize("rng", [0, 1])
@pytest.mark.parametrize("n", [4 * 8192 - 7, 4 * 8192, 4 * 8192 + 1])
def test_grid_around_the_cached_size(pkg, cuda, n, rng):
    """Grids of up to 4096 cells are read through the L1s, larger ones around them."""
    W = pkg.wrs
    cfg = W.ITSConfig(rng=rng, scan_precision=W.SCAN_COMPENSATED)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    s = 200_001
    out = cuda.full((2, s), -1, dtype=cuda.int32, device="cuda")
    for seed in (1, 2):  # the second build's grid, not the first one's lines
        b.weights.copy_(h2d(weights_lognormal(n, seed)))
        wrs.build(None, b, n)
        W.check(W.lib().wrs_sample_at(wrs.handle.ptr, None, b.internals.ptr, n, s, 9, 0,
                                      out[0].data_ptr()))
        wrs.its_sample(None, b.internals.views()["cmf"], n, s, 9, 0, out[1].data_ptr())
        cuda.cuda.synchronize()
        assert cuda.equal(out[0], out[1])


@pytest.mark.parametrize("rng", [0, 1])
@pytest.mark.parametrize("entry", [1, 4, 40, 20_000])  # the last: one cell
def test_infinite_total(pkg, cuda, entry, rng):
    """Finite weights whose sum exceeds FP32's range (no tile's does): the CMF ends in infinities, the
    Philox stream's targets spread over the finite values all the same."""
    W = pkg.wrs
    n = 6 * 4096 + 17
    w = weights_uniform(n, 3)
    w[7::4096] = 1e38
    cfg = W.ITSConfig(guiding_entry_size=entry, rng=rng, scan_precision=W.SCAN_COMPENSATED)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(w))
    wrs.build(None, b, n)
    cmf = d2h(b.internals.views()["cmf"], n, np.float32)
    assert np.isinf(cmf[-1]) and np.isfinite(cmf[3 * 4096 + 6]) and np.isinf(cmf[3 * 4096 + 7])
    s = 100_001
    out = cuda.full((2, s), -1, dtype=cuda.int32, device="cuda")
    W.check(W.lib().wrs_sample_at(wrs.handle.ptr, None, b.internals.ptr, n, s, 9, 0,
                                  out[0].data_ptr()))
    wrs.its_sample(None, b.internals.views()["cmf"], n, s, 9, 0, out[1].data_ptr())
    cuda.cuda.synchronize()
    assert cuda.equal(out[0], out[1])
    assert rng == 0 or len(out[0].unique()) >= 4
