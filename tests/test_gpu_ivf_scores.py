"""Searches that go through a score per (query, row of its lists): pair by pair when lists are probed by few queries,
as tensor-core tiles when by several.  Both must return what the batch-independent answer is: a query's result does
not depend on the batch it came in, and fp32 distances are the oracle's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_topk_equal, mixture

pytestmark = pytest.mark.gpu


def build(engine, oracle, quant, metric, n, dim, nlist, reorder=False):
    clip = quant == engine.QUANT_RABITQ
    x = mixture(dim, n, dim, nlist, 0.2, lo=0.0 if clip else -1.0, clip=clip)
    ix = engine.IvfHandle(dim, metric, nlist, quant, use_reorder=reorder)
    if clip:
        ix.set_rabitq_rotation(oracle.random_rotation(dim, seed=3))
    ix.train(x, iters=3)
    ix.add(x, np.arange(n, dtype=np.int64))
    return ix, x


@pytest.mark.parametrize("quant", ["QUANT_FP32", "QUANT_BF16", "QUANT_FP16", "QUANT_SQ8", "QUANT_RABITQ"])
@pytest.mark.parametrize("dim,n,nlist,nprobe,nq,k", [
    (1, 700, 5, 3, 40, 3),           # one dimension
    (40, 2100, 6, 3, 300, 5),        # part of a piece, more queries than an item holds
    (65, 3001, 7, 4, 90, 10),        # one past a piece, several items per list
    (128, 4096, 16, 5, 33, 33),      # whole pieces
    (200, 2500, 40, 6, 30, 7),       # items of a few queries
    (641, 1500, 6, 6, 20, 40),       # wide rows, every list probed
])
def test_tiles_equal_single_queries(engine, oracle, quant, dim, n, nlist, nprobe, nq, k):
    for metric in (0, 1):
        if quant == "QUANT_RABITQ" and metric == 1:
            continue
        ix, x = build(engine, oracle, getattr(engine, quant), metric, n, dim, nlist)
        q = mixture(dim + 1, nq, dim, nlist, 0.2, lo=0.0 if quant == "QUANT_RABITQ" else -1.0, clip=quant == "QUANT_RABITQ")
        ids, dists = ix.search(q, k, nprobe)              # as tiles
        one = [ix.search(q[i:i + 1].copy(), k, nprobe) for i in range(nq)]   # pair by pair
        one_ids, one_d = np.concatenate([o[0] for o in one]), np.concatenate([o[1] for o in one])
        assert np.array_equal(dists, one_d)
        assert_topk_equal(ids, dists, one_ids, one_d, rtol=0, atol=0)
        if quant == "QUANT_FP32" and dim < 400:
            probes, _ = oracle.route(q, ix.get_centroids(), nprobe, metric)
            sizes, codes, inner = ix.get_lists()
            off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
            want = oracle.ivf_fp32_search(x[inner], off, inner, q, probes, k, metric)
            assert np.array_equal(dists, want[1])


def test_crowded_scores_are_settled_exactly(engine, oracle):
    """Rows a thousand units from the origin and far closer to one another than the tiles' rounding: the margin check
    fails and every row of the query is scored exactly."""
    dim, n, nlist, k = 64, 2000, 4, 20
    x = (1000.0 + mixture(5, n, dim, nlist, 0.02)).astype(np.float32)
    ix = engine.IvfHandle(dim, 0, nlist, engine.QUANT_FP32)
    ix.train(x, iters=3)
    ix.add(x, np.arange(n, dtype=np.int64))
    q = (1000.0 + mixture(6, 50, dim, nlist, 0.02)).astype(np.float32)
    got = ix.search(q, k, nlist)
    want = oracle.bf_search_fp32(x, q, k)
    assert np.array_equal(got[1], want[1])
    assert_topk_equal(got[0], got[1], want[0], want[1], rtol=0, atol=0)


@pytest.mark.parametrize("n,nq,k", [(37, 1, 5), (129, 8, 40), (5000, 3, 300), (20_011, 12, 17), (70_000, 130, 100)])
@pytest.mark.parametrize("quant,dim", [("fp32", 30), ("fp32", 64), ("bf16", 33), ("bf16", 40)])
def test_exact_search_of_few_queries(engine, oracle, n, nq, k, quant, dim):
    """Up to eight queries stream the rows; more use a score matrix.  Row strides of 2, 4 and 16-byte alignment."""
    base, q = mixture(7, n, dim, 20, 0.3), mixture(8, nq, dim, 20, 0.3)
    for metric in (0, 1):
        ix = engine.BfHandle(dim, metric, engine.QUANT_FP32 if quant == "fp32" else engine.QUANT_BF16)
        ix.add(base, np.arange(n, dtype=np.int64))
        got = ix.search(q, k)
        if quant == "fp32":
            want = oracle.bf_search_fp32(base, q, k, metric)
        else:
            want = oracle.bf_search_bf16(oracle.float_to_bf16(base), q, k, metric=metric)
        assert np.array_equal(got[1], want[1])
        assert_topk_equal(got[0], got[1], want[0], want[1], rtol=0, atol=0)


@pytest.mark.parametrize("n", [8191, 8192, 8193, 20_004])
def test_selection_reads_the_passing_groups(engine, oracle, n):
    """Rows of scores around sixteen values per group, the best ones in one group of a thread and tied across many."""
    dim, nq, k = 24, 17, 20
    rng = np.random.default_rng(n)
    base = rng.integers(-3, 4, (n, dim)).astype(np.float32)
    q = rng.integers(-3, 4, (nq, dim)).astype(np.float32)
    base[5::2048] = q[0]            # many of query 0's best belong to one thread
    base[n // 2:n // 2 + 40] = q[1]  # more exact ties than results
    ix = engine.BfHandle(dim, 0, engine.QUANT_FP32)
    ix.add(base, np.arange(n, dtype=np.int64))
    got = ix.search(q, k)
    want = oracle.bf_search_fp32(base, q, k, 0)
    assert np.array_equal(got[1], want[1])
    assert_topk_equal(got[0], got[1], want[0], want[1], rtol=0, atol=0)


@pytest.mark.parametrize("n,nprobe,nq,k", [
    (20_000, 8, 1600, 3),        # around 4e6 rows: pairs or tiles below, the pruning scan above
    (200_000, 64, 800, 10),      # around 1.5e8 rows, k shallow
    (60_000, 64, 2700, 110),     # the same, k deep against lists of 940 rows
])
def test_results_do_not_depend_on_the_scan(engine, n, nprobe, nq, k):
    """A batch above the lines between the scans, the same queries in batches below them, lists pruned and not."""
    dim, nlist = 32, 64
    x, q = mixture(3, n, dim, nlist, 0.2), mixture(4, nq, dim, nlist, 0.2)
    ix = engine.IvfHandle(dim, 0, nlist, engine.QUANT_SQ8)
    ix.train(x[:20_000], iters=2)
    ix.add(x, np.arange(n, dtype=np.int64))
    want = [ix.search(q[i:i + 100].copy(), k, nprobe) for i in range(0, nq, 100)]
    want = tuple(np.concatenate(part) for part in zip(*want))
    for prune in (True, False):
        ix.set_list_pruning(prune)
        got = ix.search(q, k, nprobe)
        assert np.array_equal(got[1], want[1])
        assert_topk_equal(got[0], got[1], want[0], want[1], rtol=0, atol=0)


def test_batches_beyond_the_score_buffer(engine):
    """Scores for 2^28 (query, row) places at once: larger batches go in slices, whose results, scan time and scanned bytes
    belong together."""
    n, dim, nlist, k = 200_000, 32, 64, 7
    x, q = mixture(3, n, dim, nlist, 0.2), mixture(4, 1500, dim, nlist, 0.2)
    ix = engine.IvfHandle(dim, 0, nlist, engine.QUANT_FP32)
    ix.train(x[:20_000], iters=2)
    ix.add(x, np.arange(n, dtype=np.int64))
    one, one_ms = ix.search(q[:1200].copy(), k, nlist), ix.last_scan_ms()      # below: one slice
    one_bytes = ix.last_scanned_bytes()
    got = ix.search(q, k, nlist)
    assert np.array_equal(got[1][:1200], one[1]) and np.array_equal(got[0][:1200], one[0])
    rest = ix.search(q[1200:].copy(), k, nlist)
    assert np.array_equal(got[1][1200:], rest[1]) and np.array_equal(got[0][1200:], rest[0])
    both = []
    for _ in range(3):
        ix.search(q, k, nlist)
        both.append(ix.last_scan_ms())
    assert ix.last_scanned_bytes() * 1200 == one_bytes * 1500
    assert min(both) > 0.9 * min(one_ms, *(ix.search(q[:1200].copy(), k, nlist) and ix.last_scan_ms() for _ in range(3)))
