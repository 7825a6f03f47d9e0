"""Calls at the far ends of what the entry points take: more results than rows, very long rows, very many queries or
lists."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import assert_topk_equal, mixture

pytestmark = pytest.mark.gpu


def exactly(got, want):
    assert np.array_equal(got[1], want[1])
    assert_topk_equal(got[0], got[1], want[0], want[1], rtol=0, atol=0)


@pytest.mark.parametrize("nq", [1, 8, 9])
@pytest.mark.parametrize("n,dim,k", [
    (500, 16, 20_000),               # far more results than rows
    (1024, 16, 1025),
    (20, 45_000, 3),                 # rows too long for the kernels that keep a query in shared memory
    (20, 50_000, 30),
])
def test_exact_search_at_its_limits(engine, oracle, n, dim, k, nq):
    base, q = mixture(1, n, dim, 8, 0.3), mixture(2, nq, dim, 8, 0.3)
    for metric in (0, 1):
        ix = engine.BfHandle(dim, metric)
        ix.add(base, np.arange(n, dtype=np.int64))
        exactly(ix.search(q, k), oracle.bf_search_fp32(base, q, k, metric))


def test_more_one_bit_queries_than_a_launch_has_tiles(engine, oracle):
    """The queries' rotation is launched over tiles of up to eight queries, 65,535 at once."""
    n, dim, nlist, nq, k = 300, 32, 4, 8 * 65_535 + 9, 2
    x = mixture(1, n, dim, nlist, 0.2, lo=0.0, clip=True)
    ix = engine.IvfHandle(dim, 0, nlist, engine.QUANT_RABITQ, use_reorder=True)
    ix.set_rabitq_rotation(oracle.random_rotation(dim, seed=3))
    ix.train(x, iters=2)
    ix.add(x, np.arange(n, dtype=np.int64))
    few = mixture(2, 1000, dim, nlist, 0.2, lo=0.0, clip=True)
    want = ix.search(few, k, 2)
    q = np.ascontiguousarray(np.tile(few, (nq // 1000 + 1, 1))[:nq])
    ids, dists = ix.search(q, k, 2)
    for at in (0, 65_000, 523_000):
        assert np.array_equal(dists[at:at + 1000], want[1]) and np.array_equal(ids[at:at + 1000], want[0])
    tail = nq % 1000
    assert np.array_equal(dists[nq - tail:], want[1][:tail]) and np.array_equal(ids[nq - tail:], want[0][:tail])


@pytest.mark.parametrize("quant", ["QUANT_FP32", "QUANT_SQ8"])
def test_more_lists_than_the_finalising_kernel_has_room_for(engine, quant):
    """A caller may name as many lists as there are; two words each of shared memory are too much from 23,000 on."""
    n, dim, nlist, k = 30_000, 4, 24_000, 5
    x, q = mixture(1, n, dim, 50, 0.3), mixture(2, 3, dim, 50, 0.3)
    ix = engine.IvfHandle(dim, 0, nlist, getattr(engine, quant))
    ix.set_centroids(x[:nlist])
    if quant == "QUANT_SQ8":
        ix.set_sq8_model(x.min(axis=0), x.max(axis=0) - x.min(axis=0))
    ix.add(x, np.arange(n, dtype=np.int64))
    lists = np.tile(np.arange(nlist, dtype=np.int32), (3, 1))
    ids, dists = ix.search(q, k, nlist, bucket_ids=lists)
    some = ix.search(q, k, 900)         # the nearest of them hold the results
    assert np.array_equal(dists, some[1]) and np.array_equal(ids, some[0])
