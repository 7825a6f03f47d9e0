"""The work this engine is asked to do, as cases that can be timed: index searches from one query to the
10,000-query batch, over every list codec, exact search, k-means training and an index build, each through
the package's public entry points (vsag_b200.index.Index for host programs, vsag_b200.engine handles for
programs that keep their vectors on the GPU).

A case is a plain dict; `kind` is one of
  "ivf"     search of a trained inverted-file index
  "bf"      exact search over all rows
  "kmeans"  Lloyd iterations of the partition trainer
  "build"   seeding, training, encoding and reading back of a whole IVF-SQ8 index
"""
import json
import math

import numpy as np
import torch

from vsag_b200 import engine
from vsag_b200.index import Index

METRICS = {"l2": engine.METRIC_L2, "ip": engine.METRIC_IP, "cosine": engine.METRIC_COSINE}
QUANTS = {"fp32": engine.QUANT_FP32, "sq8": engine.QUANT_SQ8, "rabitq": engine.QUANT_RABITQ,
          "bf16": engine.QUANT_BF16, "fp16": engine.QUANT_FP16}


def _ivf(n, dim, nlist, nprobe, nq, k, *, quant="sq8", metric="l2", components=None, sigma=0.15, deny=0.0,
         api="engine", factor=2.0, name=None):
    c = {"kind": "ivf", "quant": quant, "metric": metric, "n": n, "dim": dim, "nlist": nlist, "nprobe": nprobe,
         "nq": nq, "k": k, "components": components or nlist, "sigma": sigma, "deny": deny, "api": api,
         "factor": factor}
    return dict(c, name=name) if name else c


def _bf(n, dim, nq, k, *, quant="fp32", metric="l2", api="engine", name=None):
    c = {"kind": "bf", "quant": quant, "metric": metric, "n": n, "dim": dim, "nq": nq, "k": k, "api": api}
    return dict(c, name=name) if name else c


def _kmeans(n, dim, k, iters, *, components=None, sigma=0.1, name=None):
    c = {"kind": "kmeans", "n": n, "dim": dim, "k": k, "iters": iters, "components": components or k, "sigma": sigma}
    return dict(c, name=name) if name else c


def _build(n, dim, nlist, *, components=None, sigma=0.15, name=None):
    c = {"kind": "build", "n": n, "dim": dim, "nlist": nlist, "components": components or nlist, "sigma": sigma}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a service that answers one query at a time from host memory: the smallest call, where launches and
        # host work are the whole cost
        _ivf(100_000, 128, 256, 16, 1, 10, components=500, api="index", name="ivf_sq8_one_query"),
        # a small batch of text embeddings: wide rows, cosine, more dimensions than the other indexes have
        _ivf(300_000, 640, 1024, 32, 100, 20, metric="cosine", components=2000, sigma=0.4, name="ivf_sq8_wide_100"),
        # a tenant's search over a shared index: a tenth of the ids is filtered out, rows of 100 bytes
        _ivf(1_000_000, 100, 2048, 64, 1000, 100, metric="ip", components=1500, sigma=0.3, deny=0.1,
             name="ivf_sq8_filtered"),
        # the configuration that the headline figure is quoted on
        _ivf(10_000_000, 96, 16384, 64, 10_000, 10, name="ivf_sq8_10m"),
        # lists of the default codec
        _ivf(500_000, 128, 1024, 32, 1000, 10, quant="fp32", components=3000, sigma=0.25, name="ivf_fp32"),
        # half-precision lists, a few queries at a time, nothing a multiple of anything
        _ivf(301_003, 200, 701, 21, 33, 7, quant="bf16", metric="ip", components=997, sigma=0.3, name="ivf_bf16_ragged"),
        # one bit per dimension with the exact rerank of 4 k candidates
        _ivf(1_000_000, 960, 4096, 64, 1000, 100, quant="rabitq", sigma=0.05, factor=4.0, name="ivf_rabitq_1m"),
        # exact search for one query: one pass over the rows
        _bf(1_000_000, 128, 1, 10, name="bf_fp32_one_query"),
        # exact search for a host program's batch
        _bf(100_000, 128, 1000, 10, api="index", name="bf_fp32_100k"),
        # exact inner-product search over one GPU's share of the 50M-row base
        _bf(6_250_000, 768, 10_000, 100, quant="bf16", metric="ip", name="bf_bf16_6m"),
        # partition training
        _kmeans(1_000_000, 128, 4096, 10, name="kmeans_1m"),
        # everything between a table of vectors and an index that can be saved
        _build(250_000, 96, 1000, components=1500, sigma=0.2, name="ivf_sq8_build"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ivf", "ivf", "ivf", "rows", "rows", "rabitq", "bf", "bf", "kmeans", "build"])
    metric = rng.choice(["l2", "l2", "ip", "cosine"])
    if kind in ("ivf", "rows", "rabitq"):
        host = rng.random() < 0.25
        dim = _log(rng, 128, 960) if kind == "rabitq" else _log(rng, 32, 640)
        most = 200_000 if host else min(10_000_000, 960_000_000 // dim)
        if kind == "rows":
            most = min(most, 100_000_000 // dim)
        n = _log(rng, min(50_000, most), most)
        nlist = max(16, min(16384, int(n / rng.uniform(200, 1000))))
        nprobe = min(nlist, _log(rng, 8, 128))
        nq = _log(rng, 1, 10_000 if kind == "ivf" else 1000)
        k = _log(rng, 1, 100)
        per_list = max(1, n // nlist)
        if kind == "rows":      # a row costs 4 bytes a dimension there
            nq = max(1, min(nq, int(3.3e11 / (nprobe * per_list * dim * 2))))
        if kind == "rabitq":
            nq = max(1, min(nq, int(1.6e10 / (nprobe * per_list * dim))))
        return _ivf(n, dim, nlist, nprobe, nq, k,
                    quant={"ivf": "sq8", "rabitq": "rabitq"}.get(kind) or rng.choice(["fp32", "bf16", "fp16"]),
                    metric="l2" if kind == "rabitq" else metric,
                    components=_log(rng, max(16, nlist // 4), nlist * 2),
                    sigma=0.05 if kind == "rabitq" else round(rng.uniform(0.1, 0.4), 3),
                    deny=0.1 if not host and rng.random() < 0.2 else 0.0,
                    api="index" if host and kind != "rabitq" else "engine",
                    factor=rng.choice([2.0, 4.0]) if kind == "rabitq" else 2.0)
    if kind == "bf":
        quant = rng.choice(["fp32", "bf16"])
        host = rng.random() < 0.25
        dim = _log(rng, 32, 768)
        n = _log(rng, 10_000, 200_000 if host else 1_600_000_000 // dim // (2 if quant == "fp32" else 1))
        nq = _log(rng, 1, 10_000)
        nq = max(1, min(nq, int((1e13 if quant == "fp32" else 3e13) / (n * dim))))
        return _bf(n, dim, nq, _log(rng, 1, 100), quant=quant, metric=metric, api="index" if host else "engine")
    if kind == "kmeans":
        n, dim, iters = _log(rng, 50_000, 1_000_000), _log(rng, 32, 256), rng.randint(5, 25)
        k = min(_log(rng, 64, 4096), n // 40, int(5.2e12 / (n * dim * iters)))
        return _kmeans(n, dim, k, iters, components=_log(rng, max(16, k // 4), k * 2), sigma=round(rng.uniform(0.1, 0.3), 3))
    n = _log(rng, 30_000, 500_000)
    nlist = min(2000, max(32, int(n / rng.uniform(200, 600))))
    return _build(n, _log(rng, 32, 256), nlist, components=_log(rng, max(16, nlist // 4), nlist * 2),
                  sigma=round(rng.uniform(0.1, 0.4), 3))


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _mixture(c, n, g, centres=None):
    """n rows of a Gaussian mixture; one-bit indexes get the clipped [0, 1] kind."""
    unit = c.get("quant") == "rabitq"
    dim = c["dim"]
    if centres is None:
        centres = torch.rand((c["components"], dim), generator=g, device="cuda")
        if not unit:
            centres = centres * 2.0 - 1.0
    rows = torch.empty((n, dim), dtype=torch.float32, device="cuda")
    step = max(1, 128_000_000 // dim)
    for b in range(0, n, step):
        e = min(n, b + step)
        which = torch.randint(0, centres.shape[0], (e - b,), generator=g, device="cuda")
        rows[b:e] = centres[which] + c["sigma"] * torch.randn((e - b, dim), generator=g, device="cuda")
        if unit:
            rows[b:e].clamp_(0.0, 1.0)
    return rows, centres


def _prepare_ivf(c, g, seed):
    base, centres = _mixture(c, c["n"], g)
    queries, _ = _mixture(c, c["nq"], g, centres)
    n, dim, nlist = c["n"], c["dim"], c["nlist"]
    if c["api"] == "index":
        ix = Index("ivf", json.dumps({"dtype": "float32", "metric_type": c["metric"], "dim": dim,
                                      "index_param": {"buckets_count": nlist, "base_quantization_type": c["quant"]}}))
        ix.build(base.cpu().numpy(), np.arange(n, dtype=np.int64), n, dim)
        return {"ix": ix, "queries": queries.cpu().numpy(),
                "search": json.dumps({"ivf": {"scan_buckets_count": c["nprobe"]}})}
    ix = engine.IvfHandle(dim, METRICS[c["metric"]], nlist, QUANTS[c["quant"]], use_reorder=c["quant"] == "rabitq")
    if c["quant"] == "rabitq":
        gauss = np.random.default_rng(seed).standard_normal((dim, dim))
        ix.set_rabitq_rotation(np.ascontiguousarray(np.linalg.qr(gauss)[0], np.float32))
    # a short training run on a sample: enough for lists of the usual uneven lengths
    sample = base[:: max(1, n // (16 * nlist))][: 16 * nlist].contiguous()
    seeds = engine.kmeans_init(sample[: 4 * nlist].contiguous(), nlist, seed=47)
    ix.train(sample, iters=6, init=seeds)
    ix.add(base, torch.arange(n, dtype=torch.int64, device="cuda"))
    bits = None
    if c["deny"] > 0:
        gone = torch.rand((n + 63) // 64 * 64, generator=g, device="cuda") < c["deny"]
        bits = np.packbits(gone.cpu().numpy(), bitorder="little").view(np.uint64)
    return {"ix": ix, "queries": queries, "deny": bits}


def _prepare_bf(c, g):
    n, dim, nq = c["n"], c["dim"], c["nq"]
    unit = c["metric"] == "ip"

    def rows(m):
        if not unit:
            return torch.rand((m, dim), generator=g, device="cuda")
        x = torch.randn((m, dim), generator=g, device="cuda")
        return x.div_(x.norm(dim=1, keepdim=True))

    if c["api"] == "index":
        ix = Index("brute_force", json.dumps({"dtype": "float32", "metric_type": c["metric"], "dim": dim,
                                              "index_param": {"base_quantization_type": c["quant"]}}))
        ix.build(rows(n).cpu().numpy(), np.arange(n, dtype=np.int64), n, dim)
        return {"ix": ix, "queries": rows(nq).cpu().numpy(), "search": "{}"}
    ix = engine.BfHandle(dim, METRICS[c["metric"]], QUANTS[c["quant"]])
    base = torch.empty((n, dim), dtype=torch.bfloat16 if c["quant"] == "bf16" else torch.float32, device="cuda")
    step = max(1, 512_000_000 // dim)
    for b in range(0, n, step):
        base[b : b + step] = rows(min(step, n - b))
    ids = torch.arange(n, dtype=torch.int64, device="cuda")
    if c["quant"] == "bf16":
        ix.add_bf16(base, ids)
    else:
        ix.add(base, ids)
    return {"ix": ix, "queries": rows(nq)}


def prepare(case, seed):
    g = _generator(seed)
    if case["kind"] == "ivf":
        s = _prepare_ivf(case, g, seed)
    elif case["kind"] == "bf":
        s = _prepare_bf(case, g)
    else:
        s = {"data": _mixture(case, case["n"], g)[0]}
        if case["kind"] == "kmeans":
            s["init"] = s["data"][: case["k"]].clone()
        else:
            s["ids"] = torch.arange(case["n"], dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    return dict(s, case=case)


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(state):
    c = state["case"]
    if c["kind"] in ("ivf", "bf"):
        ix, q, k = state["ix"], state["queries"], c["k"]
        if c["api"] == "index":
            if c["nq"] == 1:
                return ix.knn_search(q[0], k, state["search"])
            return ix.knn_search_batch(q, k, state["search"])
        if c["kind"] == "bf":
            return ix.search(q, k)
        if state["deny"] is not None:
            return ix.search_filtered(q, k, c["nprobe"], factor=c["factor"], invalid_label_bits=state["deny"])
        return ix.search(q, k, c["nprobe"], factor=c["factor"])
    if c["kind"] == "kmeans":
        return engine.kmeans_train(state["data"], state["init"], c["iters"])
    ix = engine.IvfHandle(c["dim"], engine.METRIC_L2, c["nlist"], engine.QUANT_SQ8)
    sample = state["data"][: 64 * c["nlist"]]
    ix.train(sample, iters=25, init=engine.kmeans_init(sample, c["nlist"], seed=47))
    ix.add(state["data"], state["ids"])
    out = (ix.get_centroids(), *ix.get_sq8_model(), *ix.get_lists())
    ix.close()
    return out


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
_ROW_BYTES = {"fp32": lambda d: 4 * d, "bf16": lambda d: 2 * d, "fp16": lambda d: 2 * d, "sq8": lambda d: d,
              "rabitq": lambda d: (d + 31) // 32 * 4 + 8}


def work(case):
    c, dim = case, case["dim"]
    if c["kind"] == "bf":
        size = {"fp32": 4, "bf16": 2}[c["quant"]]
        return {"bytes": c["n"] * dim * size + c["nq"] * (dim * 4 + c["k"] * 12), "flops": 2.0 * c["nq"] * c["n"] * dim}
    if c["kind"] == "ivf":
        # every list that some query probes is read once; a batch spreads over the lists like random picks
        touched = c["nlist"] * (1.0 - (1.0 - c["nprobe"] / c["nlist"]) ** c["nq"])
        scored = c["nq"] * c["nprobe"] * (c["n"] / c["nlist"])
        b = touched * (c["n"] / c["nlist"]) * _ROW_BYTES[c["quant"]](dim)
        b += c["nlist"] * dim * 4 + c["nq"] * (dim * 4 + c["k"] * 12)
        f = 2.0 * dim * (c["nq"] * c["nlist"] + scored)
        if c["quant"] == "rabitq":   # the rows of the rerank and the rotation of the queries
            rows = c["nq"] * min(c["factor"] * c["k"], scored / c["nq"])
            b += min(rows, c["n"]) * dim * 4 + dim * dim * 4
            f += 2.0 * c["nq"] * dim * dim + 3.0 * rows * dim
        return {"bytes": b, "flops": f}
    if c["kind"] == "kmeans":
        return {"bytes": c["iters"] * c["n"] * dim * 4.0 + c["n"] * 4 + 2 * c["k"] * dim * 4,
                "flops": 2.0 * c["iters"] * c["n"] * c["k"] * dim}
    sample = min(c["n"], 64 * c["nlist"])
    return {"bytes": c["n"] * dim * 5.0 + c["n"] * 16 + c["nlist"] * dim * 4,
            "flops": 2.0 * dim * c["nlist"] * (26.0 * sample + c["n"])}


def tolerance(case):
    # distances and centroids are fp32 sums; an id may change where two distances tie within that rounding
    return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}
