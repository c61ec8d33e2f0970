"""The work a user of this library has it do, as timed cases.

A case names a path (`kind`), its sizes, the weights' distribution and the options that matter.
Every path goes through the Python mirror of the C ABI (`WRS`, `Batch`, `Server`), as a program
that owns its weights and sample buffers calls it.  Distributions are those of the benchmark:
uniform (0, 1] on a 2^-24 grid, Zipf-like (i + 1)^-1.1 permuted, log-normal(0, 2), and the
precision configuration's log-normal(0, 3) with zeros and 1e6 outliers.

Alias tables come back as (p, alias index), the CMF and samples as they are.  Alias, ITS and
Cutpoint paths whose tiles exchange FP32 carries are run in the compensated precisions, whose
results repeat bit for bit from run to run; the FP32 carry is timed on one tile and on the scan,
whose outputs are floats.
"""
import importlib
import math

import numpy as np
import torch

W = importlib.import_module("merian-wrs_gb300").wrs

PRECISION = {"fp32": W.SCAN_FP32, "comp": W.SCAN_COMPENSATED, "ff": W.SCAN_FLOAT_FLOAT}
RNG = {"ref": W.RNG_REFERENCE, "philox": W.RNG_PHILOX4X32_10}


def listed():
    return [
        # one material or one light list of a renderer: the reference's defaults as they are, a
        # single tile, all latency (its CPU reference is pinned at this size)
        {"name": "alias_1k_defaults", "kind": "alias", "n": 1024, "s": 4096, "dist": "uniform",
         "split": 2, "precision": "fp32", "rng": "ref"},
        # the small configuration: a distribution rebuilt for every frame, 16 samples per weight
        {"name": "alias_64k", "kind": "alias", "n": 65536, "s": 1 << 20, "dist": "uniform",
         "split": 2, "precision": "comp", "rng": "philox"},
        # an environment map's texels (an odd size): the shaders' own random streams, 10 samples
        # per weight, a table that stays in L2
        {"name": "alias_1m_ref_rng", "kind": "alias", "n": 1000003, "s": 10000019,
         "dist": "lognormal", "split": 8, "precision": "comp", "rng": "ref"},
        # a mid-size table just beyond L2, drawn from a few times per weight
        {"name": "alias_16m_lognormal", "kind": "alias", "n": (1 << 24) + 5, "s": 1 << 26,
         "dist": "lognormal", "split": 12, "precision": "ff", "rng": "philox"},
        # the headline: one large distribution, built and drawn from (4 samples per weight)
        {"name": "alias_64m_uniform", "kind": "alias", "n": 1 << 26, "s": 1 << 28,
         "dist": "uniform", "split": 12, "precision": "ff", "rng": "philox"},
        # heavy-tailed data (word or item frequencies): most buckets are light, few draws keep
        {"name": "alias_50m_zipf", "kind": "alias", "n": 50000017, "s": 200000003, "dist": "zipf",
         "split": 12, "precision": "ff", "rng": "philox"},
        # weights that change often: the table is rebuilt and drawn from only a little
        {"name": "alias_64m_rebuild", "kind": "alias", "n": (1 << 26) - 3, "s": 1 << 20,
         "dist": "precision", "split": 12, "precision": "ff", "rng": "philox"},
        # many distributions of uneven sizes in one launch per stage
        {"name": "batch_1024", "kind": "batch", "dists": 1024, "n_max": 1 << 18, "s": 1 << 26,
         "split": 12, "precision": "ff", "rng": "philox"},
        # a burst of build + sample requests through the server, 30 % on tables of the burst
        {"name": "served_512", "kind": "served", "requests": 512, "n_max": 1 << 20,
         "s_max": 65536, "split": 12, "precision": "ff", "rng": "philox"},
        # inverse transform sampling of a large distribution
        {"name": "its_16m", "kind": "its", "n": (1 << 24) + 5, "s": 1 << 26, "dist": "lognormal",
         "precision": "comp", "rng": "philox"},
        # Cutpoint at the reference's guiding entry size and random streams
        {"name": "cutpoint_4m", "kind": "cutpoint", "n": 1 << 22, "s": 1 << 26, "dist": "uniform",
         "entry": 32, "precision": "comp", "rng": "ref"},
        # the scan by itself, the reference's precision
        {"name": "scan_128m_fp32", "kind": "scan", "n": (1 << 27) - 7, "dist": "uniform",
         "precision": "fp32"},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["alias"] * 6 + ["batch", "served", "its", "its", "cutpoint", "scan"])
    dist = rng.choice(["uniform", "zipf", "lognormal", "precision"])
    stream = rng.choice(["ref", "philox"])
    if kind == "scan":
        return {"kind": kind, "n": _size(rng, 1 << 16, 1 << 27), "dist": dist,
                "precision": rng.choice(["fp32", "comp"])}
    if kind == "batch":
        return {"kind": kind, "dists": _size(rng, 64, 2048),
                "n_max": _size(rng, 1 << 12, 1 << 18), "s": _size(rng, 1 << 22, 1 << 27),
                "split": rng.choice([8, 12, 16]), "precision": rng.choice(["comp", "ff"]),
                "rng": stream}
    if kind == "served":
        return {"kind": kind, "requests": _size(rng, 32, 768), "n_max": _size(rng, 1 << 12, 1 << 20),
                "s_max": _size(rng, 1 << 10, 1 << 16), "split": rng.choice([8, 12]),
                "precision": rng.choice(["comp", "ff"]), "rng": stream}
    if kind == "cutpoint":
        return {"kind": kind, "n": _size(rng, 1 << 12, 1 << 26), "s": _size(rng, 1 << 16, 1 << 27),
                "dist": dist, "entry": rng.choice([16, 32, 128]), "precision": "comp",
                "rng": stream}
    if kind == "its":
        return {"kind": kind, "n": _size(rng, 1 << 10, 1 << 26), "s": _size(rng, 1 << 14, 1 << 27),
                "dist": dist, "precision": "comp", "rng": stream}
    n = _size(rng, 1 << 10, 1 << 26)
    return {"kind": kind, "n": n, "s": min(1 << 28, max(1024, int(n * 2.0 ** rng.uniform(-6, 6)))),
            "dist": dist, "split": rng.choice([2, 4, 8, 12, 16]),
            "precision": rng.choice(["comp", "ff", "ff"]), "rng": stream}


# ---- inputs -----------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _weights(dist, n, seed):
    g = _generator(seed)
    if dist == "uniform":
        x = torch.randint(1, (1 << 24) + 1, (n,), generator=g, device="cuda", dtype=torch.int32)
        return x.float() * 2.0 ** -24
    if dist == "zipf":
        w = torch.arange(1, n + 1, device="cuda", dtype=torch.float32).pow(-1.1)
        return w[torch.randperm(n, generator=g, device="cuda")]
    if dist == "lognormal":
        return torch.exp(2.0 * torch.randn(n, generator=g, device="cuda"))
    w = torch.exp(3.0 * torch.randn(n, generator=g, device="cuda"))
    w[torch.rand(n, generator=g, device="cuda") < 0.01] = 0.0
    w[torch.rand(n, generator=g, device="cuda") < 1e-4] *= 1e6
    return w


class _DeviceArray:
    """A library-owned device array, for torch; `owner` lives as long as a tensor on it does."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr,
                                         "strides": None, "version": 3}


def _view(owner, ptr, shape, typestr):
    return torch.as_tensor(_DeviceArray(owner, ptr, shape, typestr), device="cuda")


def _config(case):
    common = {"scan_precision": PRECISION[case["precision"]]}
    if "rng" in case:
        common["rng"] = RNG[case["rng"]]
    if case["kind"] in ("its", "scan"):
        return W.ITSConfig(**common)
    if case["kind"] == "cutpoint":
        return W.CutpointConfig(case["entry"], **common)
    ff = case["precision"] == "ff"  # the benchmark's options go with its precision
    return W.AliasTableConfig(case["split"], split_residual_f64=ff, split_full_light=ff, **common)


def _spread(seed, count, n_max, n_min=64):
    """Sizes log-uniform in [n_min, n_max], seeded."""
    rng = np.random.default_rng(seed)
    lo = min(n_min, n_max)
    return rng, np.floor(np.exp(rng.uniform(math.log(lo), math.log(n_max + 1.0), count))
                         ).astype(np.int64).clip(lo, n_max)


def _offsets(sizes):
    return np.concatenate([[0], np.cumsum((np.asarray(sizes) + 31) // 32 * 32)]).astype(np.int64)


def _batch_sizes(case):
    # the sizes belong to the case, as a program's set of distributions does
    rng, sizes = _spread(case["dists"] * 7919 + case["n_max"], case["dists"], case["n_max"])
    counts = np.maximum(1, np.floor(sizes * (case["s"] / sizes.sum()))).astype(np.int64)
    return sizes, counts, rng.random(case["dists"]) < 0.5


def _served_sizes(case):
    R = case["requests"]
    rng, n = _spread(R * 104729 + case["n_max"], R, case["n_max"], 256)
    s = np.floor(np.exp(rng.uniform(0.0, math.log(case["s_max"] + 1.0), R))).astype(np.int64)
    table = np.arange(R, dtype=np.int64)
    reuse, back = rng.random(R) < 0.3, rng.integers(1, 65, R)
    for i in range(1, R):
        if reuse[i]:
            table[i] = table[max(0, i - int(back[i]))]
    return n[table], s.clip(1, case["s_max"]), table


def prepare(case, seed):
    cfg = _config(case)
    wrs = W.WRS(cfg)
    st = {"kind": case["kind"], "wrs": wrs, "stream": torch.cuda.current_stream(),
          "seed": seed * 2654435761 % (1 << 32)}
    if case["kind"] == "scan":
        st["n"] = case["n"]
        st["in"] = _weights(case["dist"], case["n"], seed)
        st["out"] = torch.empty_like(st["in"])
        st["internals"] = W.Internals(wrs.handle, case["n"])
        return st
    if case["kind"] == "batch":
        sizes, counts, zipf = _batch_sizes(case)
        w_off, s_off = _offsets(sizes), _offsets(counts)
        w = _weights("uniform", int(w_off[-1]), seed)
        for d in np.nonzero(zipf)[0]:
            a, n = int(w_off[d]), int(sizes[d])
            w[a:a + n] = w[a:a + n].argsort().add_(1).float().pow_(-1.1)
        st["weights"] = w
        st["table"] = torch.zeros((int(w_off[-1]), 2), dtype=torch.int32, device="cuda")
        st["samples"] = torch.zeros(int(s_off[-1]), dtype=torch.int32, device="cuda")
        st["batch"] = W.Batch(wrs.handle, case["dists"], int(sizes.sum()), int(counts.sum()))
        st["batch"].set(st["stream"], [
            (w.data_ptr() + 4 * int(w_off[d]), st["table"].data_ptr() + 8 * int(w_off[d]),
             st["samples"].data_ptr() + 4 * int(s_off[d]), int(sizes[d]), int(counts[d]),
             st["seed"] + d) for d in range(case["dists"])])
        return st
    if case["kind"] == "served":
        n, s, table = _served_sizes(case)
        R = case["requests"]
        pool = (1 << 22) + case["n_max"]
        s_off = _offsets(s)
        st["pool"] = torch.exp(1.5 * torch.randn(pool, generator=_generator(seed), device="cuda"))
        st["samples"] = torch.zeros(int(s_off[-1]), dtype=torch.int32, device="cuda")
        at = np.random.default_rng(seed).integers(0, (1 << 22) // 32, R)[table] * 32
        st["reqs"] = W.Server.requests(
            (int(table[i]), st["pool"].data_ptr() + 4 * int(at[i]),
             st["samples"].data_ptr() + 4 * int(s_off[i]), int(n[i]), int(s[i]), st["seed"] + i)
            for i in range(R))
        # a request names its table by id; every pass is a burst of new tables
        st["ids"] = np.frombuffer(st["reqs"], dtype=np.uint64).reshape(R, -1)[:, 0]
        st["arrivals"] = [0.0] * R
        st["server"] = W.Server(wrs.handle, memory_budget=4 << 30)
        return st
    n, s = case["n"], case["s"]
    b = W.WRSBuffers.allocate(n, s, cfg, handle=wrs.handle)
    b.weights.copy_(_weights(case["dist"], n, seed))
    views = b.internals.views()
    st.update(n=n, s=s, buffers=b)
    if case["kind"] == "alias":
        table = _view(b.internals, views["alias_table"], (n, 2), "<i4")
        st["out"] = (table.view(torch.float32)[:, 0], table[:, 1])
    elif case["kind"] == "its":
        st["out"] = (_view(b.internals, views["cmf"], (n,), "<f4"),)
    else:
        entries = (n + case["entry"] - 1) // case["entry"]
        st["out"] = (_view(b.internals, views["cmf"], (n,), "<f4"),
                     _view(b.internals, views["guide_table"], (entries,), "<i4"))
    return st


def run(st):
    wrs, stream = st["wrs"], st["stream"]
    if st["kind"] == "scan":
        wrs.prefix_sum(stream, st["in"], st["n"], st["out"], st["internals"])
        return [st["out"]]
    if st["kind"] == "batch":
        st["batch"].build(stream)
        st["batch"].sample(stream)
        return [st["table"].view(torch.float32)[:, 0], st["table"][:, 1], st["samples"]]
    if st["kind"] == "served":
        st["ids"] += np.uint64(len(st["arrivals"]))
        st["server"].run_trace(st["reqs"], st["arrivals"])
        return [st["samples"]]
    wrs.build(stream, st["buffers"], st["n"])
    wrs.sample(stream, st["buffers"], st["n"], st["s"], st["seed"])
    return [*st["out"], st["buffers"].samples]


def exact(case, seed):
    if case["kind"] not in ("scan", "its", "cutpoint"):
        return None  # alias tables, and indices drawn from them
    cmf = torch.cumsum(_weights(case["dist"], case["n"], seed).double(), 0)
    return {"scan": [cmf], "its": [cmf, None], "cutpoint": [cmf, None, None]}[case["kind"]]


def work(case):
    """Weights read, table or CMF (and guiding table) written, samples written, each once."""
    if case["kind"] == "scan":
        return {"bytes": 8 * case["n"], "flops": case["n"]}
    if case["kind"] == "batch":
        sizes, counts, _ = _batch_sizes(case)
        return {"bytes": 12 * int(sizes.sum()) + 4 * int(counts.sum()), "flops": 0}
    if case["kind"] == "served":
        n, s, table = _served_sizes(case)
        built = n[table == np.arange(len(table))]
        return {"bytes": 12 * int(built.sum()) + 4 * int(s.sum()), "flops": 0}
    n, s = case["n"], case["s"]
    out = {"alias": 8 * n, "its": 4 * n,
           "cutpoint": 4 * n + 4 * (n // case.get("entry", 1))}[case["kind"]]
    return {"bytes": 4 * n + out + 4 * s, "flops": 0}
