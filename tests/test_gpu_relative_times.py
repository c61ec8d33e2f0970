"""Times that must stand in proportion: where a smaller piece of work once took longer than a larger
one.  Least times of several rounds, on the device, with wide margins."""
from __future__ import annotations

import pytest

from conftest import weights_uniform, weights_zipf
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


def test_smaller_build_takes_less(pkg, cuda):
    """Partitions of 757 and 1465 tiles against one of 2051: 0.38 and 0.73 of its time (0.99 and 1.1
    when the smaller ones let the kernels after them start early)."""
    W = pkg.wrs
    cfg = W.AliasTableConfig(2)
    wrs = W.WRS(cfg)
    took = {}
    for n in (3_100_003, 6_000_001, 8_400_003):
        b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
        b.weights.copy_(h2d(weights_zipf(n, n)))
        took[n] = _least_ms(cuda, lambda: wrs.build(None, b, n))
    assert took[3_100_003] < 0.65 * took[8_400_003], took
    assert took[6_000_001] < 0.92 * took[8_400_003], took
