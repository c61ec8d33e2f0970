"""Guiding table and ITS cells around the number of cells up to which the cells' brackets are found
without a pass of their own, against the plain bisection of the whole CMF."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import weights_lognormal, weights_precision, weights_zipf
from gpu_util import d2h, empty, h2d, t2h

pytestmark = pytest.mark.gpu

GENS = {"lognormal": weights_lognormal, "precision": weights_precision, "zipf": weights_zipf}
LINE = 32768  # cells


@pytest.mark.parametrize("gen", sorted(GENS))
@pytest.mark.parametrize("cells", [1, 31, 33, 4097, LINE - 1, LINE, LINE + 1])
def test_cutpoint_guide(pkg, cells, gen):
    W = pkg.wrs
    cfg = W.CutpointConfig(guiding_entry_size=3, scan_precision=W.SCAN_COMPENSATED)
    wrs = W.WRS(cfg)
    n = 3 * cells - 1 if cells > 1 else 1
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(GENS[gen](n, n)))
    wrs.build(None, b, n)
    v = b.internals.views()
    ref = empty(cells, "i32")
    wrs.cutpoint_guide(None, v["cmf"], n, ref)
    assert np.array_equal(d2h(v["guide_table"], cells, np.uint32), t2h(ref, np.uint32))


@pytest.mark.parametrize("gen", sorted(GENS))
@pytest.mark.parametrize("precision,per", [("SCAN_COMPENSATED", 8), ("SCAN_FP32", 4)])
@pytest.mark.parametrize("cells", [33, LINE, LINE + 1])
def test_its(pkg, cuda, cells, precision, per, gen):
    W = pkg.wrs
    cfg = W.ITSConfig(guiding_entry_size=4, scan_precision=getattr(W, precision))
    wrs = W.WRS(cfg)
    n = per * cells - 3
    b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
    b.weights.copy_(h2d(GENS[gen](n, n)))
    wrs.build(None, b, n)
    s = 300_001
    out = cuda.full((2, s), -1, dtype=cuda.int32, device="cuda")
    W.check(W.lib().wrs_sample_at(wrs.handle.ptr, None, b.internals.ptr, n, s, 5, 11,
                                  out[0].data_ptr()))
    wrs.its_sample(None, b.internals.views()["cmf"], n, s, 5, 11, out[1].data_ptr())
    cuda.cuda.synchronize()
    assert cuda.equal(out[0], out[1])
