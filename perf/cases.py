"""Timed cases of the framework's main path: histogram, index gather, triangle
counting, the graph build that feeds it, a batch of many small instances, and
the drop-in calls on host arrays.

A case is a dict of plain values.  `listed()` gives the named ones, `draw(rng)`
one more of the same ranges; `prepare` makes what a caller has in hand,
`run` is one call through the public entry points, `work` what that call has
to move, and `exact` its result in plain torch or numpy where that is quick.
"""
import math
import random

import numpy as np
import torch

import bale_old_gb300 as bale
from bale_old_gb300 import batch as bale_batch

QUADRANTS = (0.57, 0.19, 0.19)  # R-MAT a, b, c of every graph here
EDGE_FACTOR = 16
PAD = 32  # a batch's outputs share one tensor, each from a multiple of 32 entries (256 bytes)


def listed():
    return [
        # the smallest calls of the batched and served mixes: 10K updates into
        # 1K counters, where launch latency is what a caller sees
        {"name": "histo_small", "kind": "histo", "n": 10_007, "size": 1_000, "zipf": 0.0, "packed": False},
        # the plain histogram: 10^7 uniform updates into 10^6 counters (a table that fits L2)
        {"name": "histo_l2", "kind": "histo", "n": 10_000_000, "size": 1_000_000, "zipf": 0.0, "packed": False},
        # the largest histogram of the mixes: 64M updates into 16M counters (a table about L2's size)
        {"name": "histo_large", "kind": "histo", "n": 1 << 26, "size": 1 << 24, "zipf": 0.0, "packed": False},
        # an ordinary gather with the packed indices of the exstack variants, its table in L2, an odd count
        {"name": "ig_l2", "kind": "ig", "n": 4_000_003, "size": 1 << 20, "zipf": 0.0, "packed": True},
        # a request stream of middling length against the full 512 MiB table, as one serving request
        {"name": "ig_mid", "kind": "ig", "n": 20_000_001, "size": 1 << 26, "zipf": 0.0, "packed": False},
        # the index gather's own configuration: 2^28 uniform requests, 2^26 entries
        {"name": "ig_large", "kind": "ig", "n": 1 << 28, "size": 1 << 26, "zipf": 0.0, "packed": False},
        # ... and its skewed variant: Zipf(1.1) over a permutation of the table
        {"name": "ig_zipf", "kind": "ig", "n": 1 << 28, "size": 1 << 26, "zipf": 1.1, "packed": False},
        # triangles of the degree-ordered R-MAT graph of scale 22, the whole call
        {"name": "tri_rmat", "kind": "tri", "graph": "rmat", "scale": 22, "n": 1 << 22, "degree": 32,
         "prepared": False},
        # triangles of an Erdos-Renyi graph: 2^20 vertices of average degree 32, labels as drawn
        {"name": "tri_er", "kind": "tri", "graph": "er", "scale": 0, "n": 1 << 20, "degree": 32, "prepared": False},
        # the triangle kernels' input built from an edge list (R-MAT scale 20, 16M edges)
        {"name": "build", "kind": "build", "scale": 20, "edges": 1 << 24},
        # 512 small instances (256 histograms, 192 gathers, 64 graphs) replayed as one batch
        {"name": "batch_small", "kind": "batch", "histos": 256, "igs": 192, "tris": 64, "largest": 1 << 20,
         "scale": 14, "sizes": 1},
        # the drop-in gather a ported app calls, host arrays in and out (chunked pipeline)
        {"name": "ig_host", "kind": "host", "op": "ig", "n": 50_000_000, "size": 1 << 24, "packed": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["histo", "histo", "ig", "ig", "ig", "tri", "tri", "build", "batch", "host"])
    if kind == "histo":
        return {"kind": kind, "n": _log(rng, 10_000, 1 << 26), "size": _log(rng, 1_000, 1 << 24),
                "zipf": rng.choice([0.0, 0.0, 0.0, 1.1]), "packed": rng.random() < 0.3}
    if kind == "ig":
        return {"kind": kind, "n": _log(rng, 10_000, 1 << 28), "size": _log(rng, 1_000, 1 << 26),
                "zipf": rng.choice([0.0, 0.0, 0.8, 1.1, 1.3]), "packed": rng.random() < 0.3}
    if kind == "tri":
        if rng.random() < 0.6:
            scale = rng.randint(10, 21)
            return {"kind": kind, "graph": "rmat", "scale": scale, "n": 1 << scale, "degree": 2 * EDGE_FACTOR,
                    "prepared": rng.random() < 0.4}
        return {"kind": kind, "graph": "er", "scale": 0, "n": _log(rng, 1_000, 1 << 20), "degree": rng.randint(4, 48),
                "prepared": rng.random() < 0.2}
    if kind == "build":
        scale = rng.randint(10, 20)
        return {"kind": kind, "scale": scale, "edges": int((1 << scale) * rng.uniform(4, 16)) | 1}
    if kind == "batch":
        return {"kind": kind, "histos": rng.randint(1, 256), "igs": rng.randint(1, 192), "tris": rng.randint(0, 32),
                "largest": _log(rng, 1 << 16, 1 << 20), "scale": rng.randint(9, 14), "sizes": rng.randint(2, 1 << 20)}
    return {"kind": kind, "op": rng.choice(["ig", "ig", "histo"]), "n": _log(rng, 10_000, 50_000_000),
            "size": _log(rng, 1_000, 1 << 24), "packed": rng.random() < 0.5}


# ---------------------------------------------------------------- inputs
def _gen(seed, k=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1_000_003 + k)


def _values(n, g):
    return torch.randint(-(1 << 62), 1 << 62, (n,), dtype=torch.int64, device="cuda", generator=g)


def _index(n, size, zipf, packed, g):
    """n indices in [0, size): uniform, or Zipf(zipf) ranks (the continuous
    inverse distribution, cut to whole ranks) sent through a permutation."""
    if zipf:
        u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
        u.mul_((size + 1.0) ** (1.0 - zipf) - 1.0).add_(1.0).pow_(1.0 / (1.0 - zipf))
        rank = u.to(torch.int64).sub_(1).clamp_(0, size - 1)
        del u
        ix = torch.randperm(size, dtype=torch.int64, device="cuda", generator=g)[rank]
    else:
        ix = torch.randint(0, size, (n,), dtype=torch.int64, device="cuda", generator=g)
    return ix << 16 if packed else ix


def _rmat_edges(scale, m, g):
    a, b, c = QUADRANTS
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        x = torch.rand(m, device="cuda", generator=g)
        u.mul_(2).add_(x >= a + b)
        v.mul_(2).add_(((x >= a) & (x < a + b)) | (x >= a + b + c))
    return u, v


def _edge_list(scale, m, g):
    """m R-MAT edges in random order and direction: _distinct(m) different ones,
    the others repeats and a few self loops: the graph built
    from them has as many nonzeros whatever the seed."""
    n, want = 1 << scale, _distinct(m)
    key = torch.zeros(0, dtype=torch.int64, device="cuda")
    while key.numel() < want:
        u, v = _rmat_edges(scale, m, g)
        key = torch.unique(torch.cat([key, (torch.minimum(u, v) * n + torch.maximum(u, v))[u != v]]))
    key = key[torch.randperm(key.numel(), device="cuda", generator=g)[:want]]
    again = key[torch.randint(0, want, (m - want,), device="cuda", generator=g)]
    loops = torch.randint(0, n, ((m - want) // 16,), device="cuda", generator=g)
    again[:loops.numel()] = loops * n + loops
    key = torch.cat([key, again])[torch.randperm(m, device="cuda", generator=g)]
    lo, hi = torch.div(key, n, rounding_mode="floor"), key % n
    turn = torch.rand(m, device="cuda", generator=g) < 0.5
    return torch.where(turn, lo, hi), torch.where(turn, hi, lo)


def _distinct(m):
    return m - m // 8


def _er_lower(n, degree, g):
    """The strictly lower CSR of n * degree / 2 random edges, repeats and
    self loops dropped."""
    m = n * degree // 2
    u = torch.randint(0, n, (m,), dtype=torch.int64, device="cuda", generator=g)
    v = torch.randint(0, n, (m,), dtype=torch.int64, device="cuda", generator=g)
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.maximum(u, v) * n + torch.minimum(u, v))
    row = torch.div(key, n, rounding_mode="floor")
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return off, (key - row * n).contiguous()


def _batch_sizes(case):
    rng = random.Random(case["sizes"])
    top = case["largest"]
    histos = [(_log(rng, 1_000, top), _log(rng, 10_000, top)) for _ in range(case["histos"])]
    igs = [(_log(rng, 1_000, 4 * top), _log(rng, 10_000, top)) for _ in range(case["igs"])]
    tris = [rng.randint(8, case["scale"]) for _ in range(case["tris"])]
    return histos, igs, tris


def _prepare_batch(case, seed):
    g = _gen(seed)
    histos, igs, tris = _batch_sizes(case)
    at, places = 0, []
    for length in [t for t, _ in histos] + [n for _, n in igs] + [1] * len(tris):
        places.append((at, length))
        at += -(-length // PAD) * PAD
    out = torch.zeros(at, dtype=torch.int64, device="cuda")
    outs = [out[a:a + length] for a, length in places]
    inst = [bale_batch.histo(outs[k], _index(n, t, 0.0, False, g)) for k, (t, n) in enumerate(histos)]
    for t, n in igs:
        inst.append(bale_batch.ig(outs[len(inst)], _index(n, t, 0.0, False, g), _values(t, g)))
    for k, scale in enumerate(tris):
        off, col = bale.gen_rmat_dev(scale, EDGE_FACTOR, *QUADRANTS, seed * 1000 + k)
        inst.append(bale_batch.triangles(off, col.contiguous(), outs[len(inst)]))
    torch.cuda.synchronize()
    return {"batch": bale_batch.Batch(inst), "out": out}


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": dict(case)}
    if kind == "ig":
        g = _gen(seed)
        s["table"] = _values(case["size"], g)
        s["index"] = _index(case["n"], case["size"], case["zipf"], case["packed"], g)
        s["tgt"] = torch.empty(case["n"], dtype=torch.int64, device="cuda")
    elif kind == "histo":
        g = _gen(seed)
        # counts carry over from earlier models, as in the reference's app
        s["counts"] = torch.randint(0, 100, (case["size"],), dtype=torch.int64, device="cuda", generator=g)
        s["index"] = _index(case["n"], case["size"], case["zipf"], case["packed"], g)
    elif kind == "tri":
        if case["graph"] == "rmat":
            s["offset"], s["nonzero"] = bale.gen_rmat_dev(case["scale"], EDGE_FACTOR, *QUADRANTS, seed)
        else:
            s["offset"], s["nonzero"] = _er_lower(case["n"], case["degree"], _gen(seed))
        s["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        s["resident"] = bale.TrianglePrepared(s["offset"], s["nonzero"]) if case["prepared"] else None
    elif kind == "build":
        s["u"], s["v"] = _edge_list(case["scale"], case["edges"], _gen(seed))
    elif kind == "batch":
        s.update(_prepare_batch(case, seed))
    else:
        rng = np.random.default_rng(seed)
        ix = rng.integers(0, case["size"], case["n"], dtype=np.int64)
        s["index"] = ix << 16 if case["packed"] else ix
        if case["op"] == "ig":
            s["table"] = rng.integers(-(1 << 62), 1 << 62, case["size"], dtype=np.int64)
            s["tgt"] = np.zeros(case["n"], np.int64)
        else:
            s["counts"] = rng.integers(0, 100, case["size"], dtype=np.int64)
    return s


# ---------------------------------------------------------------- one call
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ig":
        bale.ig_dev(s["tgt"], s["index"], s["table"], shift=16 if case["packed"] else 0)
        return s["tgt"]
    if kind == "histo":
        bale.histo_dev(s["counts"], s["index"], shift=16 if case["packed"] else 0)
        return s["counts"]
    if kind == "tri":
        if s["resident"] is not None:
            s["resident"].count(s["count"])
        else:
            bale.triangle_dev(s["offset"], s["nonzero"], s["count"])
        return s["count"]
    if kind == "build":
        return bale.graph_build_dev(s["u"], s["v"], 1 << case["scale"])
    if kind == "batch":
        s["batch"].run()
        return s["out"]
    if case["op"] == "ig":
        (bale.ig_exstack if case["packed"] else bale.ig_agi)(s["tgt"], s["index"], s["table"])
        return s["tgt"]
    (bale.histo_exstack if case["packed"] else bale.histo_agi)(s["index"], s["counts"])
    return s["counts"]


# ---------------------------------------------------------------- what a call has to do
def _ig_bytes(n, size):
    return 8 * n + 8 * n + 8 * min(n, size)


def _histo_bytes(n, size):
    return 8 * n + 16 * min(n, size)


def work(case):
    kind = case["kind"]
    flops = 0
    if kind == "ig" or (kind == "host" and case["op"] == "ig"):
        nbytes = _ig_bytes(case["n"], case["size"])
    elif kind in ("histo", "host"):
        nbytes, flops = _histo_bytes(case["n"], case["size"]), case["n"]
    elif kind == "tri":
        # offsets and columns once; a few per cent of the drawn edges are repeats
        nbytes = 8 * (case["n"] + 1) + 8 * (case["n"] * case["degree"] // 2)
    elif kind == "build":
        nbytes = 16 * case["edges"] + 8 * ((1 << case["scale"]) + 1) + 8 * _distinct(case["edges"])
    else:
        histos, igs, tris = _batch_sizes(case)
        flops = sum(n for _, n in histos)
        nbytes = sum(_histo_bytes(n, t) for t, n in histos) + sum(_ig_bytes(n, t) for t, n in igs)
        nbytes += sum(8 * ((1 << c) + 1) + 8 * (EDGE_FACTOR << c) for c in tris)
    return {"bytes": int(nbytes), "flops": int(flops)}


def exact(case, seed):
    """The gathers' and histograms' results in plain torch and numpy; graphs
    and batches have none this quick."""
    kind = case["kind"]
    if kind not in ("ig", "histo", "host"):
        return None
    s = prepare(case, seed)
    k = s["index"] >> 16 if case["packed"] else s["index"]
    if "table" in s:
        return s["table"][k]
    if kind == "host":
        return s["counts"] + np.bincount(k, minlength=case["size"])
    return s["counts"] + torch.bincount(k, minlength=case["size"])
