"""Sampling from buffers whose CMF is no longer the one that the build wrote: what the build stored
beside it to steer the search must not be followed past its bounds."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import weights_lognormal, weights_uniform
from gpu_util import cudart, d2h, h2d

pytestmark = pytest.mark.gpu


def test_grid_walk_ends_with_its_cell(pkg, cuda):
    """The caller overwrites the CMF through its pointer.  A grid cell of single items ends at most
    27 items behind its first, wherever the new CMF reaches the target: here at its last item."""
    W = pkg.wrs
    n, heads, s = 4096, 16, 1 << 18
    cfg = W.ITSConfig(rng=W.RNG_PHILOX4X32_10, scan_precision=W.SCAN_COMPENSATED)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, s, cfg, handle=wrs.handle)
    b.weights.zero_()
    b.weights[:heads] = 1.0
    wrs.build(None, b, n)
    cmf = b.internals.views()["cmf"]
    assert np.array_equal(d2h(cmf, heads, np.float32), np.arange(1, heads + 1, dtype=np.float32))
    other = np.full(n, 2.0**-20, np.float32)
    other[-1] = heads
    assert cudart().cudaMemcpy(cmf, other.ctypes.data, other.nbytes, 1) == 0
    wrs.sample(None, b, n, s, seed=3)
    cuda.cuda.synchronize()
    got = b.samples.cpu().numpy()
    assert got.min() >= 0 and got.max() < heads + 27
    # about one sample in 2000 shares a step with an item and walks from it to its cell's end
    assert (got >= 27).sum() > s // 10000


def _sampled(W, cuda, wrs, b, n, s, primitive):
    """wrs_sample's samples and the primitive's on the CMF that the buffers hold now"""
    out = cuda.full((2, s), -1, dtype=cuda.int32, device="cuda")
    W.check(W.lib().wrs_sample_at(wrs.handle.ptr, None, b.internals.ptr, n, s, 11, 5,
                                  out[0].data_ptr()))
    primitive(out[1])
    cuda.cuda.synchronize()
    return out


def _rewrite(W, how, wrs, b, n, w):
    """Another CMF into the buffers: whole, piece by piece behind its start (so that it falls at each
    piece), by the block-wise baseline, or by a build that does not store what the first one did."""
    cmf = b.internals.views()["cmf"]
    if how == "scan":
        wrs.prefix_sum(None, w, n, cmf, b.internals)
    elif how == "pieces":
        for at in range(1000, n - 500, 500):
            wrs.prefix_sum(None, w[at:], 500, cmf + 4 * at, b.internals)
    elif how == "blockwise":
        wrs.prefix_sum_blockwise(None, w, n, cmf, b.internals)
    else:
        b.weights.copy_(w)
        W.WRS(W.ITSConfig(guiding_entry_size=0, rng=wrs.handle.config.rng,
                          scan_precision=wrs.handle.config.scan_precision)).build(None, b, n)


@pytest.mark.parametrize("how", ["scan", "pieces", "blockwise", "unguided_build"])
@pytest.mark.parametrize("precision,entry", [(1, 4), (0, 4), (0, 0)])
def test_its_follows_the_cmf(pkg, cuda, precision, entry, how):
    W = pkg.wrs
    n, s = 70_001, 100_003
    cfg = W.ITSConfig(guiding_entry_size=entry, rng=W.RNG_PHILOX4X32_10, scan_precision=precision)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(weights_uniform(n, 1)))
    wrs.build(None, b, n)
    _rewrite(W, how, wrs, b, n, h2d(weights_lognormal(n, 2)))
    out = _sampled(W, cuda, wrs, b, n, s, lambda o: wrs.its_sample(
        None, b.internals.views()["cmf"], n, s, 11, 5, o.data_ptr()))
    assert cuda.equal(out[0], out[1])


@pytest.mark.parametrize("how", ["scan", "pieces", "blockwise"])
def test_cutpoint_follows_the_cmf(pkg, cuda, how):
    W = pkg.wrs
    n, s = 70_001, 1 << 19
    cfg = W.CutpointConfig(32, rng=W.RNG_PHILOX4X32_10, scan_precision=W.SCAN_COMPENSATED)
    wrs = W.WRS(cfg)
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(weights_uniform(n, 1)))
    wrs.build(None, b, n)
    _rewrite(W, how, wrs, b, n, h2d(weights_lognormal(n, 2)))
    v = b.internals.views()
    out = _sampled(W, cuda, wrs, b, n, s, lambda o: wrs.cutpoint_sample(
        None, v["cmf"], n, v["guide_table"], s, 11, 5, o.data_ptr()))
    assert cuda.equal(out[0], out[1])
