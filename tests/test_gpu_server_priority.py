"""Small batches that go ahead of a larger one in flight, some of them drawing from the table that it
builds: every request's samples equal those of the request alone."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_small_batches_beside_a_large_one(pkg, cuda):
    W = pkg.wrs
    cfg = pkg.AliasTableConfig(split_size=8, rng=W.RNG_PHILOX4X32_10,
                               scan_precision=W.SCAN_FLOAT_FLOAT, split_residual_f64=True,
                               split_full_light=True)
    h = W.Handle(cfg)
    big, rounds = 1 << 20, 12
    server = W.Server(h, memory_budget=512 << 20, slots=3, max_batch_dists=32,
                      max_batch_weights=big, max_batch_samples=1 << 18)
    pool = cuda.rand(2 * big, device="cuda", generator=cuda.Generator("cuda").manual_seed(5))
    rng = np.random.default_rng(5)
    rows, at = [], 0
    for r in range(rounds):
        large = (100 * r, int(rng.integers(0, big // 32)) * 32, big)
        small = [(100 * r + 1 + k, int(rng.integers(0, big // 32)) * 32, int(rng.integers(1, 3000)))
                 for k in range(20)]
        for table, off, n in [large] + small + [large] * 3 + small[:4]:
            s = int(rng.integers(1, 4097))
            rows.append((table, off, at, n, s, 7 + len(rows)))
            at += (s + 31) // 32 * 32
    out = cuda.full((at,), -1, dtype=cuda.int32, device="cuda")
    reqs = W.Server.requests((t, pool.data_ptr() + 4 * off, out.data_ptr() + 4 * a, n, s, seed)
                             for t, off, a, n, s, seed in rows)
    comps = server.run_trace(reqs, [0.0] * len(rows))
    cuda.cuda.synchronize()
    assert all(c.status == 0 for c in comps)
    assert server.stats()["device_status"] == 0 and server.stats()["batches"] >= 2 * rounds
    table = cuda.empty(2 * big, dtype=cuda.int32, device="cuda")
    alone = cuda.empty(4096, dtype=cuda.int32, device="cuda")
    one = W.Batch(h, 1, big, 4096)
    for t, off, a, n, s, seed in rows:
        one.set(None, [(pool.data_ptr() + 4 * off, table, alone, n, s, seed)])
        one.build(None)
        one.sample(None)
        assert cuda.equal(out[a:a + s], alone[:s]), (t, n, s)
