"""The work a user has this framework do, as cases that can be timed.

A case is a dict of plain values. `prepare` builds what a program holds before
the call (the index, the queries), `run` makes the call through the public
Python API and returns its results, `work` counts the bytes and operations the
call cannot do without, `exact` gives the 64-bit value of a result where it has
one. Four kinds:

* flat     - search of a flat index: device buffers, or host buffers as numpy
* build    - create, calibrate, add, prepare and a first small search
* bucketed - search of the bucketed (IVF) index, with a fixed n_probe or with
             the learned per-query n_probe
* multi    - one launch over several flat indexes, queries and results on the host

Data: rows with power-law coordinate variances under a random rotation
(embeddings; `data="embedding"`), a clipped Gaussian mixture (SIFT-like;
`data="mixture"`), clusters on the unit sphere with Zipf sizes (word vectors;
the bucketed index).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vectorcache_b200 import BucketedTurboQuantIndex, BucketParams, TurboQuantIndex
from vectorcache_b200.multi import MultiIndex
from vectorcache_b200.probe import ProbeMLP
from vectorcache_b200.synthetic import haar_orthogonal, power_law_spectrum

DEVICE = "cuda:0"
CALIBRATION_ROWS = 10_000
ADD_ROWS = 262_144  # rows handed to add_device at a time
PROBE_CLASSES = (1, 2, 4, 8, 16, 32, 64, 96, 128, 160, 192, 224, 256, 320, 384, 512)


def _flat(name, n, dim, bits, nq, k, tqplus=True, data="embedding", host=False):
    return {"name": name, "kind": "flat", "n": n, "dim": dim, "bits": bits, "nq": nq, "k": k, "tqplus": tqplus,
            "data": data, "host": host}


def listed():
    return [
        # One lookup in a small index, numpy in and out: the call's latency and its launches.
        _flat("flat_1q_100k_128_b4_host", 100_000, 128, 4, 1, 10, tqplus=False, data="mixture", host=True),
        # One interactive query over an embedding collection: a pass over the codes.
        _flat("flat_1q_1M_1536_b4", 1_000_000, 1536, 4, 1, 10),
        # A burst of requests on the largest serving index.
        _flat("flat_16q_10M_768_b3", 10_000_000, 768, 3, 16, 10),
        # A ragged batch: sizes that are no multiple of any tile, more results a query.
        _flat("flat_257q_300007_392_b3_k64", 300_007, 392, 3, 257, 64),
        # A batch over a small low-dimensional index.
        _flat("flat_1000q_100k_128_b4", 100_000, 128, 4, 1000, 10, tqplus=False, data="mixture"),
        # A batch over coarse codes, candidates for a later re-rank.
        _flat("flat_2048q_1M_1536_b2_k64", 1_000_000, 1536, 2, 2048, 64),
        # The offline batch: ten thousand queries over a million embeddings.
        _flat("flat_10000q_1M_1536_b4", 1_000_000, 1536, 4, 10_000, 10),
        # Ingest: a new collection from raw rows to its first results.
        {"name": "build_262144_1536_b4", "kind": "build", "n": 262_144, "dim": 1536, "bits": 4, "nq": 64, "k": 10,
         "tqplus": True},
        # Word vectors, the whole query set at the probe count that reaches Recall@10 0.95, with re-rank.
        {"name": "bucketed_10000q_1200k_100_p464", "kind": "bucketed", "n": 1_200_000, "dim": 100, "bits": 4,
         "nq": 10_000, "k": 10, "n_probe": 464, "rerank_k": 100, "learned": False},
        # The same index behind an interactive service: a handful of queries.
        {"name": "bucketed_16q_1200k_100_p128", "kind": "bucketed", "n": 1_200_000, "dim": 100, "bits": 4,
         "nq": 16, "k": 10, "n_probe": 128, "rerank_k": 100, "learned": False},
        # The same index with the probe network choosing each query's n_probe.
        {"name": "bucketed_2048q_1200k_100_learned", "kind": "bucketed", "n": 1_200_000, "dim": 100, "bits": 4,
         "nq": 2048, "k": 10, "n_probe": 512, "rerank_k": 100, "learned": True},
        # Several tenants' indexes of uneven size, width and batch, answered by one launch.
        {"name": "multi_8", "kind": "multi", "n_indexes": 8, "n_min": 10_000, "n_max": 1_000_000, "nq_max": 300,
         "layout": 7},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case. Costs stay below the listed 10,000-query searches."""
    kind = rng.choices(["flat", "build", "bucketed", "multi"], [10, 2, 4, 1])[0]
    if kind == "flat":
        dim = 8 * _log_int(rng, 8, 192)
        n = _log_int(rng, 10_000, min(4_000_000, 1_536_000_000 // dim))
        nq = _log_int(rng, 1, 10_000)
        data = rng.choice(["embedding", "embedding", "mixture"])
        case = _flat("", n, dim, rng.choice([2, 3, 4, 4]), nq, _log_int(rng, 1, 128),
                     tqplus=data == "embedding" and rng.random() < 0.75, data=data, host=rng.random() < 0.3)
    elif kind == "build":
        dim = 8 * _log_int(rng, 8, 192)
        case = {"kind": kind, "n": _log_int(rng, 20_000, min(1_000_000, 400_000_000 // dim)), "dim": dim,
                "bits": rng.choice([2, 3, 4]), "nq": _log_int(rng, 1, 64), "k": rng.choice([1, 10, 64]),
                "tqplus": rng.random() < 0.75}
    elif kind == "bucketed":
        learned = rng.random() < 0.3
        n = _log_int(rng, 200_000 if learned else 50_000, 1_200_000)
        k = _log_int(rng, 1, 64)
        case = {"kind": kind, "n": n, "dim": rng.randint(48, 200), "bits": rng.choice([2, 3, 4, 4]),
                "nq": _log_int(rng, 1, 10_000), "k": k,
                "n_probe": 512 if learned else _log_int(rng, 8, max(16, n // 2600)),
                "rerank_k": rng.choice([0, k + _log_int(rng, 10, 100)]), "learned": learned}
    else:
        case = {"kind": kind, "n_indexes": rng.randint(2, 12), "n_min": 10_000, "n_max": _log_int(rng, 50_000, 500_000),
                "nq_max": _log_int(rng, 4, 300), "layout": rng.randint(100, 1_000_000)}
    case.pop("name", None)
    return case


# ---- data -------------------------------------------------------------------

_rotations: dict = {}


def _gen(*key):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(np.random.SeedSequence([int(v) for v in key]).generate_state(1)[0]))
    return g


def _embedding_rows(n, dim, gen):
    """Unit rows of power-law variances under one rotation per dim."""
    if dim not in _rotations:
        sd = np.sqrt(power_law_spectrum(dim))
        _rotations[dim] = torch.as_tensor(sd[:, None] * haar_orthogonal(dim, 1234).T, dtype=torch.float32,
                                          device=DEVICE)
    x = torch.randn((n, dim), generator=gen, device=DEVICE) @ _rotations[dim]
    return x / torch.linalg.vector_norm(x, dim=1, keepdim=True)


def _mixture_rows(n, dim, gen, centers):
    """256 isotropic Gaussians clipped to [0, inf), spanning about 0..255."""
    lab = torch.randint(0, centers.shape[0], (n,), generator=gen, device=DEVICE)
    x = centers[lab] + 0.35 * torch.randn((n, dim), generator=gen, device=DEVICE)
    return x.clamp_(min=0.0) * (255.0 / 4.5)


def _sphere_rows(n, dim, gen, centers, spread, weights):
    """Clusters on the unit sphere: Zipf sizes, spread per cluster."""
    lab = torch.multinomial(weights, n, replacement=True, generator=gen)
    x = centers[lab] + spread[lab, None] * torch.randn((n, dim), generator=gen, device=DEVICE)
    return x / torch.linalg.vector_norm(x, dim=1, keepdim=True)


def _source(case, seed):
    """rows(n, part): n rows of the case's law; other parts are other draws."""
    dim = case["dim"]
    if case["kind"] == "bucketed":
        g = _gen(seed, 1)
        centers = torch.randn((2000, dim), generator=g, device=DEVICE)
        centers /= torch.linalg.vector_norm(centers, dim=1, keepdim=True)
        kappa = torch.exp(math.log(20.0) + math.log(10.0) * torch.rand(2000, generator=g, device=DEVICE))
        weights = torch.arange(1, 2001, device=DEVICE, dtype=torch.float32) ** -1.1
        return lambda n, part: _sphere_rows(n, dim, _gen(seed, 2, part), centers, kappa.rsqrt(), weights)
    if case.get("data", "embedding") == "mixture":
        centers = torch.randn((256, dim), generator=_gen(seed, 1), device=DEVICE)
        return lambda n, part: _mixture_rows(n, dim, _gen(seed, 2, part), centers)
    return lambda n, part: _embedding_rows(n, dim, _gen(seed, 2, part))


def _flat_index(n, dim, bits, tqplus, rows):
    """An index of n generated rows, added a chunk at a time."""
    index = TurboQuantIndex(dim, bits)
    for part, at in enumerate(range(0, n, ADD_ROWS)):
        x = rows(min(ADD_ROWS, n - at), part)
        if at == 0:
            if tqplus:
                index.calibrate_device(x[:CALIBRATION_ROWS])
            index.add_device(x)
            index.prepare()
        else:
            index.add_device(x)
    return index


def _results(nq, k):
    return (torch.empty((nq, k), dtype=torch.float32, device=DEVICE),
            torch.empty((nq, k), dtype=torch.int64, device=DEVICE))


def _multi_shapes(case):
    """(n, dim, bits, nq, k) of every index; the layout number fixes them."""
    rng = np.random.default_rng(case["layout"])
    shapes = []
    for _ in range(case["n_indexes"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        nq = int(round(math.exp(rng.uniform(0.0, math.log(case["nq_max"])))))
        shapes.append((n, int(rng.choice([128, 384, 768, 1536])), int(rng.choice([2, 3, 4])), nq,
                       int(rng.choice([10, 64]))))
    return shapes


def _probe_network(index, rows, n_train=4096):
    """A probe network trained for a short while: a query is labelled with the
    class covering the buckets whose routing score is near its best one."""
    mlp = ProbeMLP(classes=PROBE_CLASSES, seed=3)
    q = rows(n_train, 1 << 20)
    top = torch.empty((n_train, 256), dtype=torch.float32, device=DEVICE)
    ids = torch.empty((n_train, 256), dtype=torch.int32, device=DEVICE)
    index.route_device(q, 256, top, ids)
    near = (top > top[:, :1] - 0.55).sum(1, dtype=torch.int32)
    classes = torch.tensor(PROBE_CLASSES, dtype=torch.int32, device=DEVICE)
    label = torch.searchsorted(classes, near).clamp_(max=len(PROBE_CLASSES) - 1).to(torch.int32)
    f = torch.cat([top, top - torch.cat([top[:, 1:], top[:, -1:]], 1)], 1)
    mlp.set_normalization(f.mean(0).cpu().numpy(), f.std(0).clamp_(min=1e-6).cpu().numpy())
    for step in range(60):
        at = (step * 512) % n_train
        mlp.train_step_device(top[at:at + 512], label[at:at + 512], 512, 256, 1e-3)
    return mlp


# ---- the cases --------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "multi":
        indexes, queries, ks = [], [], []
        for i, (n, dim, bits, nq, k) in enumerate(_multi_shapes(case)):
            rows = _source({"kind": "flat", "dim": dim}, seed * 64 + i)
            indexes.append(_flat_index(n, dim, bits, True, rows))
            queries.append(rows(nq, 1 << 20).cpu().numpy())
            ks.append(k)
        multi = MultiIndex(indexes)
        multi.plan([len(q) for q in queries], ks, autotune=True)
        return {"kind": kind, "indexes": indexes, "queries": queries, "multi": multi}
    rows = _source(case, seed)
    queries = rows(case["nq"], 1 << 21)
    if kind == "flat":
        index = _flat_index(case["n"], case["dim"], case["bits"], case["tqplus"], rows)
        if case["host"]:
            return {"kind": "host", "index": index, "queries": queries.cpu().numpy(), "k": case["k"]}
        return {"kind": kind, "index": index, "queries": queries, "k": case["k"],
                "out": _results(case["nq"], case["k"])}
    if kind == "build":
        return {"kind": kind, "rows": rows(case["n"], 0), "queries": queries, "k": case["k"], "dim": case["dim"],
                "bits": case["bits"], "tqplus": case["tqplus"], "out": _results(case["nq"], case["k"])}
    index = BucketedTurboQuantIndex(case["dim"], case["bits"], BucketParams(
        n_probe=min(case["n_probe"], 64), expected_n=case["n"], rerank_k=case["rerank_k"]))
    index.add_device(rows(case["n"], 0))
    index.prepare()
    return {"kind": "learned" if case["learned"] else kind, "index": index, "queries": queries, "k": case["k"],
            "n_probe": case["n_probe"], "mlp": _probe_network(index, rows) if case["learned"] else None,
            "out": _results(case["nq"], case["k"])}


def run(state):
    kind = state["kind"]
    if kind == "host":
        res = state["index"].search(state["queries"], state["k"])
        return {"scores": res.scores, "ids": res.ids.view(np.int64)}
    if kind == "multi":
        multi = state["multi"]
        for i, q in enumerate(state["queries"]):
            multi.set_queries(i, q)
        multi.launch()
        multi.synchronize()
        torch.cuda.current_stream().synchronize()  # the launch ran there; the results are read next
        return [{"scores": s, "ids": ids.view(np.int64)}
                for s, ids in (multi.results(i) for i in range(len(state["queries"])))]
    scores, ids = state["out"]
    if kind == "flat":
        state["index"].search_device(state["queries"], state["k"], scores, ids)
    elif kind == "bucketed":
        state["index"].search_device(state["queries"], state["k"], scores, ids, n_probe=state["n_probe"])
    elif kind == "learned":
        state["index"].search_learned_device(state["queries"], state["k"], state["mlp"], scores, ids, coverage=0.9,
                                             fallback_n_probe=256)
    else:
        index = TurboQuantIndex(state["dim"], state["bits"])
        if state["tqplus"]:
            index.calibrate_device(state["rows"][:CALIBRATION_ROWS])
        index.add_device(state["rows"])
        index.prepare()
        index.search_device(state["queries"], state["k"], scores, ids)
        torch.cuda.current_stream().synchronize()  # the index goes away with this pass
        index.close()
    return {"scores": scores, "ids": ids}


def _flat_work(n, dim, bits, nq, k):
    nbg = dim // (8 // bits)
    return n * (nbg + 4) + nq * (dim * 4 + k * 12), 2.0 * nbg * n * nq


def work(case):
    """Bytes: every input once (codes, queries, rows), every result once.
    Operations: one addition per looked-up nibble; of a build, the rotation's
    butterflies and one step per quantized coordinate."""
    kind = case["kind"]
    if kind == "multi":
        parts = [_flat_work(*shape) for shape in _multi_shapes(case)]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    n, dim, nq, k = case["n"], case["dim"], case["nq"], case["k"]
    if kind == "bucketed":
        dim = -(-dim // 8) * 8
        buckets = n / 373.0
        share = min(1.0, (128 if case["learned"] else case["n_probe"]) / buckets)
        nbg = dim // (8 // case["bits"])
        touched = n * min(1.0, share * nq)
        return {"bytes": touched * (nbg + 8) + buckets * dim * 8 + nq * (dim * 4 + k * 12),
                "flops": 2.0 * nq * buckets * dim + 2.0 * nbg * n * share * nq}
    nbytes, flops = _flat_work(n, dim, case["bits"], nq, k)
    if kind == "build":
        nbytes += n * dim * 4.0
        flops += n * dim * (math.log2(dim) + 2)
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    """The 64-bit value of a case's results, where there is one. A re-ranked
    bucketed search returns inner products of unit rows, near the best of the
    whole corpus: those are given. Scores of the other searches are the
    quantized index's own (integer sums of table bytes scaled in float), fixed
    bit for bit by its codes and tables rather than by a 64-bit formula."""
    if case["kind"] != "bucketed" or not case["rerank_k"]:
        return None
    rows = _source(case, seed)
    x, q = rows(case["n"], 0).double(), rows(case["nq"], 1 << 21).double()
    x /= torch.linalg.vector_norm(x, dim=1, keepdim=True)
    q /= torch.linalg.vector_norm(q, dim=1, keepdim=True)
    step = max(1, (1 << 28) // case["n"])
    best = [torch.topk(q[at:at + step] @ x.T, case["k"], dim=1).values for at in range(0, case["nq"], step)]
    return {"scores": torch.cat(best), "ids": None}
