"""Launches whose shared memory lies around what a kernel gets unasked (48 KiB, static and dynamic together).  Each in a
process of its own: a larger launch of the same kernel earlier in the process would have raised the limit already."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SEARCH = """
import sys
import numpy as np
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
from conftest import mixture
from oracle import pyoracle as O
from vsag_b200 import engine

dim, nlist, nprobe, nq, k = {dim}, {nlist}, {nprobe}, {nq}, 5
x, q = mixture(1, 3000, dim, nlist, 0.2), mixture(2, nq, dim, nlist, 0.2)
ix = engine.IvfHandle(dim, 0, nlist, engine.QUANT_SQ8)
ix.train(x, iters=2)
ix.add(x, np.arange(len(x), dtype=np.int64))
ids, dists = ix.search(q, k, nprobe)
sizes, codes, inner = ix.get_lists()
off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
lower, diff = ix.get_sq8_model()
probes, _ = O.route(q, ix.get_centroids(), nprobe)
want_ids, want = O.ivf_sq8_search(codes, off, inner, lower, diff, q, probes, k)
assert np.array_equal(dists, want), np.abs(dists - want).max()
assert np.mean(ids == want_ids) > 0.99
"""


@pytest.mark.parametrize("nq", [1, 40])   # pair by pair, and as tiles
@pytest.mark.parametrize("dim,nlist,nprobe", [(960, 128, 70), (960, 128, 80), (1000, 64, 10), (1000, 64, 32), (1000, 64, 36)])
def test_finalising_kernel_at_the_edge_of_its_shared_memory(dim, nlist, nprobe, nq):
    """Around 12 KiB of dynamic beside 37 KiB of static shared memory: (2 nprobe + 4 + 3 dim) words."""
    root = str(Path(__file__).resolve().parents[1])
    code = SEARCH.format(root=root, dim=dim, nlist=nlist, nprobe=nprobe, nq=nq)
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout + done.stderr


ADD = """
import sys
import numpy as np
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
from conftest import mixture
from vsag_b200 import engine

dim = {dim}
x = mixture(1, 400, dim, 4, 0.2)
ix = engine.IvfHandle(dim, {metric}, 4, engine.QUANT_SQ8)
ix.train(x, iters=1)
ix.add(x, np.arange(len(x), dtype=np.int64))
ids, dists = ix.search(x[:9], 1, 4)
assert np.mean(ids[:, 0] == np.arange(9)) > 0.5 or {metric} == 1, ids
"""


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("dim", [752, 767, 768, 769])
def test_adding_rows_whose_balls_fill_the_default(dim, metric):
    """Covering balls take 64 bytes of shared memory per dimension: 48 KiB at 768."""
    root = str(Path(__file__).resolve().parents[1])
    done = subprocess.run([sys.executable, "-c", ADD.format(root=root, dim=dim, metric=metric)], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout + done.stderr
