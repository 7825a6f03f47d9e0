"""Searches that nominate rows by approximate scores must return the exact answer whatever the data: where the scores
cannot tell the nearest rows apart, or overflow, the exact distances decide."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_topk_equal, mixture

pytestmark = pytest.mark.gpu


def exactly(got, want):
    assert np.array_equal(got[1], want[1])
    assert_topk_equal(got[0], got[1], want[0], want[1], rtol=0, atol=0)


@pytest.mark.parametrize("quant", ["fp32", "bf16"])
@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("offset,n,dim,nq,k", [
    (50.0, 20_000, 128, 17, 10),     # scores of 3e5 with differences of 1
    (100.0, 30_011, 33, 9, 1),       # rows of 4 (fp32) and 2 (bf16) bytes alignment
    (30.0, 4_000, 24, 300, 40),      # many queries, nearly all of them undecided
    (0.0, 4_000, 24, 300, 40),       # nearly none
])
def test_exact_batches_far_from_the_origin(engine, oracle, quant, metric, offset, n, dim, nq, k):
    """The matrix of split-bf16 scores keeps k + 16 rows per query; far from the origin the true neighbours are not
    among them, and the batch has to notice."""
    base = (offset + 0.1 * mixture(3, n, dim, 30, 1.0)).astype(np.float32)
    q = (offset + 0.1 * mixture(4, nq, dim, 30, 1.0)).astype(np.float32)
    ix = engine.BfHandle(dim, metric, engine.QUANT_FP32 if quant == "fp32" else engine.QUANT_BF16)
    ix.add(base[: n // 3], np.arange(n // 3, dtype=np.int64))
    ix.add(base[n // 3:], np.arange(n // 3, n, dtype=np.int64))
    got = ix.search(q, k)
    if quant == "fp32":
        want = oracle.bf_search_fp32(base, q, k, metric)
    else:
        want = oracle.bf_search_bf16(oracle.float_to_bf16(base), q, k, metric=metric)
    exactly(got, want)
    # the same with half of the rows filtered out, and a batch whose queries come one at a time
    gone = np.zeros((n + 31) // 32, np.uint32)
    gone[:] = 0x55555555
    left = np.flatnonzero(np.arange(n) % 2 == 1)
    got = ix.search_filtered(q, k, deny_inner_bits=gone)
    if quant == "fp32":
        want = oracle.bf_search_fp32(base[left], q, k, metric)
    else:
        want = oracle.bf_search_bf16(oracle.float_to_bf16(base[left]), q, k, metric=metric)
    exactly(got, (np.where(want[0] >= 0, left[want[0]], -1), want[1]))
    one = ix.search(q[5:6].copy(), k)
    assert np.array_equal(one[1][0], ix.search(q, k)[1][5])


def test_exact_batches_with_overflowing_norms(engine, oracle):
    """Rows whose squared norm is infinite have finite distances to queries beside them."""
    n, dim, k = 1500, 16, 5
    base = mixture(5, n, dim, 10, 0.3)
    base[::7] += np.float32(3e19)
    q = np.ascontiguousarray(base[:40])
    ix = engine.BfHandle(dim, 0, engine.QUANT_FP32)
    ix.add(base, np.arange(n, dtype=np.int64))
    got = ix.search(q, k)
    exactly(got, oracle.bf_search_fp32(base, q, k, 0))


@pytest.mark.parametrize("dim,outlier,level,low,high", [
    (518, 60.0, -0.3, 0.0, 0.1),     # the widest rows whose integer sums always fit 32 bits
    (519, 60.0, -0.3, 0.0, 0.1),
    (768, 60.0, -0.2, 0.0, 0.1),
    (960, 60.0, -0.2, 0.1, 0.4),
    (2048, 120.0, -0.2, 0.1, 0.4),
    (2048, 60.0, 0.3, 0.3, 0.9),
    (2049, 60.0, 0.3, 0.3, 0.9),     # no tiled copy
])
def test_sq8_long_rows_of_extreme_codes(engine, oracle, dim, outlier, level, low, high):
    """Non-negative sparse rows (most codes are 0) against queries with one component far larger than the others: the
    second integer sum of the ranking form reaches 32 bits from 519 dimensions on, at different rows for different data."""
    n, nlist, nq, k = 1500, 4, 40, 10
    rng = np.random.default_rng(dim)
    filled = rng.random((n, dim)) < rng.uniform(low, high, (n, 1))
    x = np.where(filled, 0.5 + 0.5 * rng.random((n, dim)), 0.0).astype(np.float32)
    q = (level + 0.02 * rng.standard_normal((nq, dim))).astype(np.float32)
    q[np.arange(nq), rng.integers(0, dim, nq)] = outlier
    lower = x.min(axis=0)
    diff = x.max(axis=0) - lower
    for metric in (0, 1):
        ix = engine.IvfHandle(dim, metric, nlist, engine.QUANT_SQ8)
        ix.set_centroids(x[:nlist])
        ix.set_sq8_model(lower, diff)
        ix.add(x, np.arange(n, dtype=np.int64))
        sizes, codes, inner = ix.get_lists()
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        probes = np.tile(np.arange(nlist, dtype=np.int32), (nq, 1))
        want = oracle.ivf_sq8_search(codes, off, inner, lower, diff, q, probes, k, metric)
        exactly(ix.search(q, k, nlist), want)
        one = [ix.search(q[i:i + 1].copy(), k, nlist) for i in range(nq)]
        exactly((np.concatenate([o[0] for o in one]), np.concatenate([o[1] for o in one])), want)


@pytest.mark.parametrize("quant", ["QUANT_FP32", "QUANT_BF16"])
def test_list_batches_with_overflowing_norms(engine, oracle, quant):
    """Rows of lists whose squared norm is infinite, as tiles (a batch) and pair by pair, among them rows that are no
    numbers and rows that the filter rejects."""
    n, dim, nlist, nq, k = 2000, 40, 5, 60, 6
    base = mixture(6, n, dim, nlist, 0.3)
    base[::9] *= np.float32(3e19)
    base[7::100] = np.nan
    if quant == "QUANT_BF16":      # values the codec holds exactly, so that a row is its own query
        base = (oracle.float_to_bf16(base).astype(np.uint32) << 16).view(np.float32).reshape(n, dim)
    mine = np.flatnonzero(np.isfinite(base).all(axis=1))[:3 * nq:3]
    q = np.ascontiguousarray(base[mine])
    ix = engine.IvfHandle(dim, 0, nlist, getattr(engine, quant))
    ix.set_centroids(mixture(7, nlist, dim, nlist, 0.3))
    ix.add(base, np.arange(n, dtype=np.int64), labels=np.arange(n, dtype=np.int32) % nlist)
    gone = np.zeros((n + 31) // 32, np.uint32)
    gone[n // 64:] = 0x11111111
    lists = np.tile(np.arange(nlist, dtype=np.int32), (nq, 1))
    for bits in (None, gone):
        many = ix.search_filtered(q, k, nlist, bucket_ids=lists, deny_inner_bits=bits)
        one = [ix.search_filtered(q[i:i + 1].copy(), k, nlist, bucket_ids=lists[:1], deny_inner_bits=bits) for i in range(nq)]
        assert np.array_equal(many[1], np.concatenate([o[1] for o in one]))
        assert np.array_equal(many[0], np.concatenate([o[0] for o in one]))
        kept = np.ones(n, bool) if bits is None else (np.unpackbits(bits.view(np.uint8), bitorder="little")[:n] == 0)
        assert np.array_equal(many[0][kept[mine], 0], mine[kept[mine]]) and np.all(many[1][kept[mine], 0] == 0)


@pytest.mark.parametrize("quant", ["QUANT_SQ8", "QUANT_BF16", "QUANT_FP16", "QUANT_RABITQ"])
@pytest.mark.parametrize("offset,dim,k", [(1000.0, 64, 20), (3.0, 300, 100), (0.0, 960, 100)])
def test_crowded_scores_of_every_codec(engine, oracle, quant, offset, dim, k):
    """Rows closer to one another than the scores' rounding, from all of them to a few: batches, which go as tiles, return
    what the exact arithmetic of the codec gives."""
    n, nlist, nq = 1800, 4, 40
    clip = quant == "QUANT_RABITQ"
    spread = 0.02 if offset > 100 else 0.2
    if clip:
        x, q = (mixture(s, m, dim, nlist, 0.002 if offset else 0.05, lo=0.0, clip=True) for s, m in ((5, n), (6, nq)))
    else:
        x, q = ((offset + mixture(s, m, dim, nlist, spread)).astype(np.float32) for s, m in ((5, n), (6, nq)))
    for metric in (0,) if clip else (0, 1):
        ix = engine.IvfHandle(dim, metric, nlist, getattr(engine, quant))
        if clip:
            ix.set_rabitq_rotation(oracle.random_rotation(dim, seed=3))
        ix.train(x, iters=3)
        ix.add(x, np.arange(n, dtype=np.int64))
        got = ix.search(q, k, nlist)
        if quant == "QUANT_SQ8":
            sizes, codes, inner = ix.get_lists()
            off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
            lower, diff = ix.get_sq8_model()
            probes = np.tile(np.arange(nlist, dtype=np.int32), (nq, 1))
            exactly(got, oracle.ivf_sq8_search(codes, off, inner, lower, diff, q, probes, k, metric))
        else:     # one query goes pair by pair, which is the codec's own arithmetic
            one = [ix.search(q[i:i + 1].copy(), k, nlist) for i in range(nq)]
            exactly(got, (np.concatenate([o[0] for o in one]), np.concatenate([o[1] for o in one])))


@pytest.mark.parametrize("dim", [1024, 2048, 3000])
@pytest.mark.parametrize("value", [1.1, 0.7001, -0.3])
def test_sq8_rows_that_differ_by_less_than_the_constant_of_a_query_rounds(engine, oracle, dim, value):
    """Queries of one value throughout, so that the additions behind their constant all round the same way, and rows that differ
    from one another in two codes of opposite weight.  Each batch is routed by the engine: the constant is a warp's or a CTA's."""
    n, nlist, k = 1200, 4, 10
    rng = np.random.default_rng(dim)
    codes = np.zeros((n, dim), np.float32)
    for r, (a, b) in enumerate(rng.integers(0, dim, (n, 2))):
        codes[r, a] = rng.integers(1, 4)
        codes[r, b] = rng.integers(1, 4)
    x = codes / np.float32(255)
    lower, diff = np.zeros(dim, np.float32), np.ones(dim, np.float32)
    q = np.full((40, dim), value, np.float32)
    q[np.arange(40), np.arange(40)] += np.float32(1e-6) * np.arange(40, dtype=np.float32)
    for metric in (0, 1):
        ix = engine.IvfHandle(dim, metric, nlist, engine.QUANT_SQ8)
        ix.set_centroids(x[:nlist])
        ix.set_sq8_model(lower, diff)
        ix.add(x, np.arange(n, dtype=np.int64))
        sizes, stored, inner = ix.get_lists()
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        probes = np.tile(np.arange(nlist, dtype=np.int32), (len(q), 1))
        want = oracle.ivf_sq8_search(stored, off, inner, lower, diff, q, probes, k, metric)
        for nq in (1, 3, 40) if dim <= 2048 else (1, 3):      # (more of longer rows are grouped, which keeps k + 16 and checks nothing)
            exactly(ix.search(q[:nq].copy(), k, nlist), (want[0][:nq], want[1][:nq]))
