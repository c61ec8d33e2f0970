"""The one-launch build of a small distribution against the staged entry points (total mass,
prefix partition, split-pack), which launch the general kernels: every output the same, bit for bit,
at the edges of tiles, clusters and subproblem shares.  (FP32 carries follow the lookback's order
beyond one tile, so FP32 is compared on one tile.)"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import weights_lognormal, weights_precision, weights_uniform, weights_zipf
from gpu_util import d2h, empty, h2d, t2h

pytestmark = pytest.mark.gpu


def _equal(n, seed):
    return np.full(n, 0.75, np.float32)  # no heavy item


def _zeros(n, seed):
    return np.zeros(n, np.float32)


def _one_giant(n, seed):
    w = np.full(n, 1e-3, np.float32)
    w[n // 3] = np.float32(n + 1)
    return w


def _two_values(n, seed):
    w = np.ones(n, np.float32)
    w[np.random.default_rng(seed).random(n) < 0.5] = 3.0
    return w


def _not_finite(n, seed):
    w = weights_uniform(n, seed)
    w[n // 2] = np.nan if n & 1 else np.inf
    return w


GENS = {"uniform": weights_uniform, "zipf": weights_zipf, "lognormal": weights_lognormal,
        "precision": weights_precision, "equal": _equal, "zeros": _zeros,
        "one_giant": _one_giant, "two_values": _two_values, "not_finite": _not_finite}

# (n, split size): one tile and several, one share and several, the last sizes before the general path
SIZES = [(1, 2), (2, 2), (31, 32), (33, 32), (446, 2), (448, 2), (1000, 2), (3569, 2), (4095, 2),
         (4096, 2), (4097, 12), (4096, 3), (8192, 32), (12289, 32), (20481, 10), (24575, 12),
         (28672, 64), (32767, 32), (32768, 16), (32768, 500)]


@pytest.mark.parametrize("gen", sorted(GENS))
@pytest.mark.parametrize("precision", ["SCAN_FP32", "SCAN_COMPENSATED", "SCAN_FLOAT_FLOAT"])
def test_against_the_stages(pkg, gen, precision):
    import torch
    W = pkg.wrs
    prec = getattr(W, precision)
    ff = prec == W.SCAN_FLOAT_FLOAT
    for e, (n, split) in enumerate(SIZES):
        if prec == W.SCAN_FP32 and n > 4096:
            continue
        cfg = W.AliasTableConfig(split, use_partition_elements=e % 3 != 1, scan_precision=prec,
                                 split_residual_f64=e % 2 == 0, split_full_light=ff or e % 4 == 2)
        wrs = W.WRS(cfg)
        shift = e & 1  # weights that are only 4-byte aligned too
        w = torch.zeros(n + 1, device="cuda")[shift:shift + n]
        w.copy_(h2d(GENS[gen](n, n)))
        b = W.WRSBuffers.allocate(n, 1, cfg, handle=wrs.handle)
        b.weights.copy_(w)
        b.weights = w
        wrs.build(None, b, n)
        v = b.internals.views()
        i2 = W.Internals(wrs.handle, n)
        elems = empty(n) if cfg.use_partition_elements else None
        idx, prefix, lo = empty(n, "u32"), empty(n), empty(n) if ff else None
        table = torch.full((2 * n,), -1, dtype=torch.int32, device="cuda")
        wrs.total_mass(None, w, n, i2)
        wrs.prefix_partition(None, w, n, idx, prefix, elems, i2, prefix_lo=lo)
        wrs.split_pack(None, w, idx, prefix, elems, n, table, i2, prefix_lo=lo)
        where = f"{gen} {precision} n={n} split={split}"
        v2 = i2.views()
        for key, t in (("mean", np.uint32), ("mean64", np.uint64), ("total", np.uint64),
                       ("heavy_count", np.uint32)):
            assert d2h(v[key], 1, t) == d2h(v2[key], 1, t), (where, key)
        for key, t in (("partition_indices", idx), ("partition_prefix", prefix),
                       ("partition_elements", elems), ("partition_prefix_lo", lo)):
            if t is not None:
                assert np.array_equal(d2h(v[key], n, np.uint32), t2h(t, np.uint32)), (where, key)
        got = d2h(v["alias_table"], 2 * n, np.uint32)
        assert np.array_equal(got, t2h(table, np.uint32)), where
        assert b.internals.status() == i2.status(), where
