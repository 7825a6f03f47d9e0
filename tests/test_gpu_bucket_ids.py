"""Lists that a caller names for every query (bucket_ids) instead of routing."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import mixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [3, 60])   # pair by pair, and as tiles
@pytest.mark.parametrize("quant", ["QUANT_FP32", "QUANT_FP16", "QUANT_SQ8", "QUANT_RABITQ"])
def test_a_list_named_twice_is_scanned_twice(engine, oracle, quant, nq):
    """What the general path (taken by every search with a time limit) makes of it is what every path returns: the
    longest list throughout, one repeat among distinct lists, ids that are no lists."""
    dim, n, nlist, nprobe, k = 48, 4000, 9, 6, 12
    clip = quant == "QUANT_RABITQ"
    x = mixture(1, n, dim, nlist, 0.3, lo=0.0 if clip else -1.0, clip=clip)
    q = mixture(2, nq, dim, nlist, 0.3, lo=0.0 if clip else -1.0, clip=clip)
    ix = engine.IvfHandle(dim, 0, nlist, getattr(engine, quant))
    if clip:
        ix.set_rabitq_rotation(oracle.random_rotation(dim, seed=3))
    ix.train(x, iters=3)
    ix.add(x, np.arange(n, dtype=np.int64))
    longest = int(np.argmax(ix.get_lists()[0]))
    rng = np.random.default_rng(5)
    distinct = np.stack([rng.permutation(nlist)[:nprobe] for _ in range(nq)]).astype(np.int32)
    cases = {"longest": np.full((nq, nprobe), longest, np.int32), "distinct": distinct, "one": distinct.copy(), "odd": distinct.copy()}
    cases["one"][nq - 1, nprobe - 1] = cases["one"][nq - 1, 0]
    cases["odd"][:, 1], cases["odd"][:, 2], cases["odd"][:, 4] = -1, nlist + 7, cases["odd"][:, 3]
    for name, lists in cases.items():
        want = ix.search_ex(q, k, nprobe, bucket_ids=lists, timeout_ms=1e9)
        got = ix.search(q, k, nprobe, bucket_ids=lists)
        assert np.array_equal(got[1], want[1]), name
        assert np.array_equal(got[0], want[0]), name
        again = ix.search(q, k, nprobe)       # the handle is as it was
        assert np.array_equal(again[1], ix.search_ex(q, k, nprobe, timeout_ms=1e9)[1]), name
