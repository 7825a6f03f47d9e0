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
