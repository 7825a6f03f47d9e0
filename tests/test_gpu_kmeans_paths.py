"""Training paths that ordinary data of test size do not reach: seeding from rows that the chip's shared memory cannot hold,
and assignments whose nominations decide next to nothing."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import mixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim", [(90_000, 128), (50_001, 211)])   # 46 and 42 MB; rows of 16- and 4-byte alignment
def test_seeding_streams_rows_that_do_not_fit(engine, oracle, n, dim):
    x = mixture(9, n, dim, 16, 0.2)
    want_c, want_rows = oracle.kmeans_pp_init(x, 12, 47)
    got_c, got_rows = engine.kmeans_init(x, 12, 47, want_rows=True)
    # (sums in another order: a pick differs only where the draw falls within rounding of a boundary)
    assert np.array_equal(got_rows, want_rows) and np.array_equal(got_c, want_c)


@pytest.mark.parametrize("n", [2000, 9000])   # undecided rows by CTAs of their own, and as a matrix product
def test_training_where_nominations_decide_nothing(engine, oracle, n):
    """Two far clusters with all centroids crowded into them: every row has more than four centroids within the error of
    an fp16 score, so the first iteration decides all rows over all centroids and the next ones take split terms."""
    dim, k, iters = 24, 128, 3
    rng = np.random.default_rng(n)
    x = np.where(np.arange(n)[:, None] % 2 == 0, 100.0, -100.0) + 0.01 * rng.standard_normal((n, dim))
    x = np.ascontiguousarray(x, np.float32)
    init = x[:k].copy()
    want_c, want_l, _, _ = oracle.kmeans_run(x, init, iters)
    got_c, got_l, _ = engine.kmeans_train(x, init, iters)
    assert np.array_equal(got_l, want_l) and np.array_equal(got_c, want_c)


@pytest.mark.parametrize("dim", [5, 32, 200])
@pytest.mark.parametrize("top", [1e6, 1e8, 1e9, 1e11])
def test_rows_beside_one_that_is_far_larger(engine, oracle, dim, top):
    """The scale of the fp16 operands follows the largest element: the others become subnormal, their squares vanish, and the
    margin has to say so.  Labels are the oracle's, and with centroids as near to one another as the rows (not to the large
    row) those of 64-bit distances too."""
    n, k = 3000, 70
    x = mixture(45, n, dim, 50, 0.2)
    c = np.ascontiguousarray(x[100:100 + k])
    x[5] = np.float32(top)
    got = engine.kmeans_assign(x, c)
    assert np.array_equal(got, oracle.kmeans_assign(x, c)[0])
    rest = np.r_[0:5, 6:n]
    d = ((x[rest, None, :].astype(np.float64) - c[None].astype(np.float64)) ** 2).sum(-1)
    two = np.sort(d, 1)[:, :2]
    clear = two[:, 1] - two[:, 0] > 1e-4 * (two[:, 0] + dim)      # (far above the rounding of a chain of fp32 products)
    assert clear.mean() > 0.5 and np.array_equal(got[rest][clear], d.argmin(1)[clear])
