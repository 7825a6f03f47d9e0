"""Kernels at the edges of their tiles, pieces and buffers, and searches on both sides of the lines between their paths."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_topk_equal, mixture

pytestmark = pytest.mark.gpu


def exactly(got, want):
    assert np.array_equal(got[1], want[1])
    assert_topk_equal(got[0], got[1], want[0], want[1], rtol=0, atol=0)


# ---- exact batches that keep what passes a threshold from a sample of the rows --------------------------------
# 4 (k + 16) groups of 32 in an eighth of the rows: from 17,408 rows with k 1, 26,624 with k 10, 59,392 with k 42
@pytest.mark.parametrize("quant,metric,n,dim,nq,k", [
    ("fp32", 0, 17_280, 33, 9, 1),        # rows of 4-byte alignment
    ("fp32", 0, 17_281, 33, 9, 1),        # the last tile of the rows holds one
    ("fp32", 0, 17_407, 33, 9, 1),        # the most rows without a sample
    ("fp32", 0, 17_408, 33, 9, 1),        # the fewest with one
    ("fp32", 0, 18_433, 33, 9, 1),        # the last tile of the rows holds one
    ("fp32", 1, 26_497, 96, 129, 10),     # two row tiles of queries, six of eight k-steps
    ("fp32", 1, 26_625, 96, 129, 10),
    ("bf16", 0, 26_600, 50, 128, 10),
    ("bf16", 0, 26_700, 50, 128, 10),
    ("bf16", 1, 60_100, 200, 300, 42),
    ("fp32", 0, 70_000, 16, 1000, 10),    # a sixteenth of the rows as a sample
])
@pytest.mark.parametrize("order", ["mixed", "sorted"])
def test_exact_batches_by_threshold(engine, oracle, quant, metric, n, dim, nq, k, order):
    base, q = mixture(21, n, dim, 40, 0.25), mixture(22, nq, dim, 40, 0.25)
    if order == "sorted":      # rows of a cluster stored together: all that is nearest to a query lies in a few tiles
        base = np.ascontiguousarray(base[np.lexsort(base.T[:3])])
    ix = engine.BfHandle(dim, metric, engine.QUANT_FP32 if quant == "fp32" else engine.QUANT_BF16)
    ix.add(base, np.arange(n, dtype=np.int64))
    got = ix.search(q, k)
    some = slice(0, 64)
    if quant == "fp32":
        want = oracle.bf_search_fp32(base, q[some], k, metric)
    else:
        want = oracle.bf_search_bf16(oracle.float_to_bf16(base), q[some], k, metric=metric)
    exactly((got[0][some], got[1][some]), want)
    gone = np.full((n + 31) // 32, 0x55555555, np.uint32)      # filtered rows take the path without a sample
    left = np.flatnonzero(np.arange(n) % 2 == 1)
    few = ix.search_filtered(q, k, deny_inner_bits=gone)
    if quant == "fp32":
        want = oracle.bf_search_fp32(base[left], q[some], k, metric)
    else:
        want = oracle.bf_search_bf16(oracle.float_to_bf16(base[left]), q[some], k, metric=metric)
    exactly((few[0][some], few[1][some]), (np.where(want[0] >= 0, left[want[0]], -1), want[1]))


# the fewest rows with an eighth, a sixteenth and a thirty-second as the sample: 4 (k + 16) groups of 32 in it
@pytest.mark.parametrize("n,k", [(17_408, 1), (26_624, 10), (53_248, 10), (106_496, 10), (119_000, 42)])
@pytest.mark.parametrize("quant", ["QUANT_FP32", "QUANT_BF16"])
@pytest.mark.parametrize("metric", [0, 1])
def test_exact_batches_do_not_depend_on_the_order_of_the_rows(engine, quant, metric, n, k):
    """Rows of a cluster stored together, or clusters in turn: what the sample lets through fits as it does for mixed rows, so no
    query is left to the exact pass, which would be two launches more."""
    dim, nq, clusters = 20, 150, 96
    rng = np.random.default_rng(n)
    centres = rng.uniform(-1, 1, (clusters, dim))
    member = rng.integers(0, clusters, n)
    q = (centres[rng.integers(0, clusters, nq)] + 0.2 * rng.standard_normal((nq, dim))).astype(np.float32)
    launches = []
    for order in ("mixed", "together", "in turn"):
        which = {"mixed": member, "together": np.sort(member), "in turn": np.arange(n) % clusters}[order]
        base = (centres[which] + 0.2 * rng.standard_normal((n, dim))).astype(np.float32)
        ix = engine.BfHandle(dim, metric, getattr(engine, quant))
        ix.add(base, np.arange(n, dtype=np.int64))
        ix.search(q, k)
        before = engine.kernel_launches()
        got = ix.search(q, k)
        launches.append(engine.kernel_launches() - before)
        one = [ix.search(q[i:i + 1].copy(), k) for i in range(0, nq, 10)]
        assert np.array_equal(got[1][::10], np.concatenate([o[1] for o in one]))
    assert launches == launches[:1] * 3


@pytest.mark.parametrize("kind", ["equal", "far", "nan"])
def test_exact_batches_the_threshold_does_not_serve(engine, oracle, kind):
    """Every row within the scores' rounding of every other, many equal ones, rows that are no numbers: the results are those
    of the exact pass."""
    n, dim, nq, k = 30_000, 24, 20, 10
    base, q = mixture(23, n, dim, 30, 0.2), mixture(24, nq, dim, 30, 0.2)
    if kind == "equal":
        base[5_000:25_000] = base[7]
        q[:10] = base[7]
    elif kind == "far":
        base, q = (base * np.float32(0.01) + np.float32(80)), (q * np.float32(0.01) + np.float32(80))
    else:
        base[3::11] = np.nan
    ix = engine.BfHandle(dim, 0, engine.QUANT_FP32)
    ix.add(base, np.arange(n, dtype=np.int64))
    got = ix.search(q, k)
    one = [ix.search(q[i:i + 1].copy(), k) for i in range(nq)]      # a pass over the rows in the exact arithmetic
    assert np.array_equal(got[1], np.concatenate([o[1] for o in one]))
    if kind != "equal":
        assert np.array_equal(got[0], np.concatenate([o[0] for o in one]))


# ---- distance chains --------------------------------------------------------------------------------------------
@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("dim", [4, 31, 32, 33, 100])
@pytest.mark.parametrize("nq,nlist", [(1, 16), (15, 31), (16, 32), (17, 33), (33, 257), (640, 1000), (255, 1900)])
def test_routing_by_chains(engine, oracle, metric, dim, nq, nlist):
    nprobe = min(7, nlist)
    c, q = mixture(31, nlist, dim, 9, 0.4), mixture(32, nq, dim, 9, 0.4)
    ix = engine.IvfHandle(dim, metric, nlist, engine.QUANT_FP32)
    ix.set_centroids(c)
    got = ix.route(q, nprobe)
    got = got[0] if isinstance(got, tuple) else got
    want = oracle.route(q, c, nprobe, metric)
    want = want[0] if isinstance(want, tuple) else want
    assert np.array_equal(np.asarray(got), np.asarray(want))


# by distances and by scores, a warp a query (the first two, the last) and a CTA
@pytest.mark.parametrize("nq,nlist", [(20, 900), (300, 1000), (300, 1500), (1300, 1500), (100, 1500), (1600, 1400)])
@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("dim", [18, 32])                           # rows of 8- and of 16-byte alignment
def test_routing_with_coinciding_centroids(engine, oracle, nq, nlist, metric, dim):
    """More lists tie with the last that is wanted than a warp collects: the lowest numbers among them are probed."""
    nprobe = 40
    c, q = mixture(33, nlist, dim, 9, 0.4), mixture(34, nq, dim, 9, 0.4)
    c[100:800] = c[100]
    q[::2] = c[100]
    ix = engine.IvfHandle(dim, metric, nlist, engine.QUANT_FP32)
    ix.set_centroids(c)
    got, want = ix.route(q, nprobe), oracle.route(q, c, nprobe, metric)
    got, want = (v[0] if isinstance(v, tuple) else v for v in (got, want))
    assert np.array_equal(np.asarray(got), np.asarray(want))


# ---- k-means ----------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("n,dim", [(16, 3), (2369, 31), (5000, 32), (5001, 33), (4000, 64), (4000, 65), (4000, 80), (4001, 81), (3000, 96),
                                   (3000, 129), (148 * 512, 8), (148 * 512 + 1, 8)])   # a row per thread, and one row more
def test_seeding_by_rows_in_registers(engine, oracle, n, dim):
    x = mixture(41, n, dim, 16, 0.2)
    want_c, want_rows = oracle.kmeans_pp_init(x, 12, 47)
    got_c, got_rows = engine.kmeans_init(x, 12, 47, want_rows=True)
    assert np.array_equal(got_rows, want_rows) and np.array_equal(got_c, want_c)


@pytest.mark.parametrize("dim", [5, 32, 96, 224, 225, 300])
def test_means_of_clusters_of_all_lengths(engine, oracle, dim):
    sizes = [0, 1, 7, 8, 9, 31, 32, 33, 63, 64, 95, 96, 97, 128, 160, 1023, 1024, 1025, 1056, 2100, 0]
    labels = np.repeat(np.arange(len(sizes), dtype=np.int32), sizes)
    rng = np.random.default_rng(dim)
    rng.shuffle(labels)
    x = rng.standard_normal((labels.size, dim)).astype(np.float32)
    got = engine.kmeans_update(x, labels, len(sizes), 3)
    want = oracle.kmeans_update(x, labels, len(sizes), 3)
    got, want = (v[0] if isinstance(v, tuple) else v for v in (got, want))
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dim", [13, 61, 62, 64, 125, 126, 200])     # the three elements behind a row within, at and past a piece of 64
@pytest.mark.parametrize("offset,spread", [(0.0, 0.2), (40.0, 0.05)])
def test_training_with_the_bias_among_the_products(engine, oracle, dim, offset, spread):
    n, k, iters = 1500, 70, 3
    x = (offset + mixture(43, n, dim, 40, spread)).astype(np.float32)
    x[5] *= np.float32(30)      # one element far larger than the rest: the others keep few bits
    want_c, want_l, _, _ = oracle.kmeans_run(x, x[:k].copy(), iters)
    got_c, got_l, _ = engine.kmeans_train(x, x[:k].copy(), iters)
    assert np.array_equal(got_l, want_l) and np.array_equal(got_c, want_c)


# ---- SQ8 batches that rule lists out -----------------------------------------------------------------------------
@pytest.mark.parametrize("dim,k", [(16, 10), (96, 16), (96, 17), (112, 48), (128, 49), (130, 112), (130, 113), (256, 10), (300, 10)])
@pytest.mark.parametrize("metric,nq", [(0, 200), (1, 200), (0, 3603), (1, 3603)])      # results by a CTA, and by a warp a query
def test_pruned_batches_equal_unpruned_ones(engine, dim, k, metric, nq):
    n, nlist, nprobe, step = 40_003, 20, 12, nq // 25      # 2000 rows a list, 4.8e6 rows scanned
    x, q = mixture(51, n, dim, 60, 0.3), mixture(52, nq, dim, 60, 0.3)
    ix = engine.IvfHandle(dim, metric, nlist, engine.QUANT_SQ8)
    ix.train(x[::8].copy(), iters=2)
    ix.add(x, np.arange(n, dtype=np.int64))
    want = [ix.search(q[i:i + 1].copy(), k, nprobe) for i in range(0, nq, step)]
    got = ix.search(q, k, nprobe)
    assert np.array_equal(got[1][::step], np.concatenate([w[1] for w in want]))
    assert np.array_equal(got[0][::step], np.concatenate([w[0] for w in want]))


# ---- tiles ------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("quant", ["QUANT_FP32", "QUANT_BF16", "QUANT_SQ8", "QUANT_RABITQ"])
@pytest.mark.parametrize("dim,nq", [(16, 12), (33, 31), (64, 33), (65, 64), (128, 65), (200, 130), (520, 9)])
def test_tiles_equal_queries_one_by_one(engine, oracle, quant, dim, nq):
    """Queries per list around the eight, sixteen, thirty-two and sixty-four that warps, operands and items hold; lists of one
    row, of a tile and a row, of several segments."""
    sizes, k = [1, 129, 2200], 10
    labels = np.repeat(np.arange(3, dtype=np.int32), sizes)
    x, q = mixture(61, labels.size, dim, 3, 0.4), mixture(62, nq, dim, 3, 0.4)
    ix = engine.IvfHandle(dim, 0, 3, getattr(engine, quant))
    if quant == "QUANT_RABITQ":
        ix.set_rabitq_rotation(oracle.random_rotation(dim, seed=3))
    ix.train(x, iters=1, init=np.ascontiguousarray(x[:3]))
    ix.add(x, np.arange(labels.size, dtype=np.int64), labels=labels)
    lists = np.tile(np.arange(3, dtype=np.int32), (nq, 1))
    got = ix.search_filtered(q, k, 3, bucket_ids=lists)
    one = [ix.search_filtered(q[i:i + 1].copy(), k, 3, bucket_ids=lists[:1]) for i in range(nq)]
    exactly(got, (np.concatenate([o[0] for o in one]), np.concatenate([o[1] for o in one])))


@pytest.mark.parametrize("dim,nq", [(16, 12), (33, 31), (64, 33), (65, 64), (72, 40), (128, 65), (200, 130), (520, 9)])
@pytest.mark.parametrize("metric", [0, 1])
def test_repeated_fp32_batches_equal_the_first(engine, dim, nq, metric):
    """From the second on rows are read as two bf16 terms, a piece of 64 dimensions at a time with zeros behind the last."""
    sizes, k = [1, 129, 2200], 10
    labels = np.repeat(np.arange(3, dtype=np.int32), sizes)
    x, q = mixture(63, labels.size, dim, 3, 0.4), mixture(64, nq, dim, 3, 0.4)
    ix = engine.IvfHandle(dim, metric, 3, engine.QUANT_FP32)
    ix.train(x, iters=1, init=np.ascontiguousarray(x[:3]))
    ix.add(x, np.arange(labels.size, dtype=np.int64), labels=labels)
    lists = np.tile(np.arange(3, dtype=np.int32), (nq, 1))
    first, second = (ix.search_filtered(q, k, 3, bucket_ids=lists) for _ in range(2))
    one = [ix.search_filtered(q[i:i + 1].copy(), k, 3, bucket_ids=lists[:1]) for i in range(nq)]
    want = np.concatenate([o[0] for o in one]), np.concatenate([o[1] for o in one])
    exactly(first, want)
    exactly(second, want)


# ---- SQ8 lists that two to four queries share ---------------------------------------------------------------------
@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("dim,nq", [(16, 19), (100, 15), (130, 19), (528, 12), (2049, 10)])
def test_rows_streamed_for_several_queries(engine, dim, nq, metric):
    """Lists of one row, of 128, of an item (256 rows) and one more, of several items, with up to as many queries as come, and bytes
    enough in all (1.5e8); with and without a filter the results are those of the queries one by one."""
    sizes = [1, 5, 128, 129, 256, 257, 700] + [int(1.6e8 * 50 / (nq * 10 * dim)) // 43] * 43
    labels = np.repeat(np.arange(50, dtype=np.int32), sizes)
    n, k, nprobe = labels.size, 12, 10
    x, q = mixture(71, n, dim, 9, 0.4), mixture(72, nq, dim, 9, 0.4)
    ix = engine.IvfHandle(dim, metric, 50, engine.QUANT_SQ8)
    ix.train(x, iters=1, init=np.ascontiguousarray(x[:50]))
    ix.add(x, np.arange(n, dtype=np.int64), labels=labels)
    rng = np.random.default_rng(dim)
    lists = np.stack([rng.permutation(np.r_[np.arange(7), rng.choice(np.arange(7, 50), 3, replace=False)]) for _ in range(nq)]).astype(np.int32)
    gone = np.full((n + 31) // 32, 0x11111111, np.uint32)
    for bits in (None, gone):
        got = ix.search_filtered(q, k, nprobe, bucket_ids=lists, deny_inner_bits=bits)
        one = [ix.search_filtered(q[i:i + 1].copy(), k, nprobe, bucket_ids=lists[i:i + 1], deny_inner_bits=bits) for i in range(nq)]
        exactly(got, (np.concatenate([o[0] for o in one]), np.concatenate([o[1] for o in one])))
