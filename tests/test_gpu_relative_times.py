"""Times that must stand in proportion: where a smaller piece of work once took longer than a larger
one.  Least times of several rounds, on the device, with wide margins."""
from __future__ import annotations

import pytest

from conftest import weights_uniform
from gpu_util import h2d

pytestmark = pytest.mark.gpu


def _least_ms(torch, call, rounds=12, calls=8):
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    call()
    best = float("inf")
    for _ in range(rounds):
        start.record()
        for _ in range(calls):
            call()
        end.record()
        torch.cuda.synchronize()
        best = min(best, start.elapsed_time(end) / calls)
    return best


def test_its_small_grid_is_not_slower(pkg, cuda):
    """2^23 samples through a grid of 4 KB against one of 256 KB: about the same time (0.198 ms and
    0.047 when every SM read the small one's few sectors from L2)."""
    W = pkg.wrs
    s, took = 1 << 23, {}
    for n in (1000, 65536):
        cfg = W.ITSConfig(rng=W.RNG_PHILOX4X32_10, scan_precision=W.SCAN_COMPENSATED)
        wrs = W.WRS(cfg)
        b = W.WRSBuffers.allocate(n, s, cfg, handle=wrs.handle)
        b.weights.copy_(h2d(weights_uniform(n, n)))
        wrs.build(None, b, n)
        took[n] = _least_ms(cuda, lambda: wrs.sample(None, b, n, s, seed=1))
    assert took[1000] < 2.0 * took[65536], took
