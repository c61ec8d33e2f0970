"""Sampling from buffers whose CMF is no longer the one that the build wrote: what the build stored
beside it to steer the search must not be followed past its bounds."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import cudart, d2h

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
