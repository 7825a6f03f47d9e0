"""A call that ends with an error leaves the handle usable: the next search returns what a fresh handle returns.  Handles
outlive the streams they were used on, and searches make do with the memory there is."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import mixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quant,reorder", [("QUANT_FP32", False), ("QUANT_SQ8", False), ("QUANT_RABITQ", True)])
@pytest.mark.parametrize("nq", [2, 90])
def test_search_after_a_filter_that_cannot_be_staged(engine, oracle, quant, reorder, nq):
    """The filter names more ids than device memory has bits for, so its copy cannot be made and the search ends after the
    pairs of every list have been counted."""
    from vsag_b200 import _capi

    dim, n, nlist, nprobe, k = 48, 4000, 9, 5, 12
    clip = quant == "QUANT_RABITQ"
    x = mixture(1, n, dim, nlist, 0.3, lo=0.0 if clip else -1.0, clip=clip)
    q = mixture(2, nq, dim, nlist, 0.3, lo=0.0 if clip else -1.0, clip=clip)
    ix = engine.IvfHandle(dim, 0, nlist, getattr(engine, quant), use_reorder=reorder)
    if clip:
        ix.set_rabitq_rotation(oracle.random_rotation(dim, seed=3))
    ix.train(x, iters=3)
    ix.add(x, np.arange(n, dtype=np.int64))
    want = ix.search(q, k, nprobe)
    lib = _capi.load()
    ids, dists = np.empty((nq, k), np.int64), np.empty((nq, k), np.float32)
    bits = np.zeros(16, np.uint32)
    for field in ("n_inner_bits", "n_label_bits"):
        f = _capi.Filter()
        f.deny_inner_bits = f.invalid_label_bits = bits.ctypes.data
        setattr(f, field, 1 << 60)
        for _ in range(2):
            status = lib.vb200_ivf_search_filtered(ix._h, q.ctypes.data_as(C.c_void_p), nq, k, nprobe, 2.0, None,
                                                   C.cast(C.byref(f), C.c_void_p), ids.ctypes.data_as(C.c_void_p),
                                                   dists.ctypes.data_as(C.c_void_p))
            assert status != 0
        got = ix.search(q, k, nprobe)
        assert np.array_equal(got[1], want[1]) and np.array_equal(got[0], want[0])


def test_a_handle_outlives_its_stream(engine):
    """Streams are the caller's: one may be destroyed before the index that was searched on it, while it is still the
    thread's current one."""
    from vsag_b200 import _capi

    _capi.load()
    rt = C.CDLL("libcudart.so.12")          # the runtime that the library is linked with
    x = mixture(1, 3000, 24, 6, 0.3)
    ids = np.arange(len(x), dtype=np.int64)
    for round_ in range(3):
        stream = C.c_void_p()
        assert rt.cudaStreamCreate(C.byref(stream)) == 0
        engine.set_stream(stream.value)
        try:
            ix = engine.IvfHandle(24, 0, 6, engine.QUANT_SQ8)
            ix.train(x, iters=2)
            ix.add(x, ids)
            bf = engine.BfHandle(24, 0)
            bf.add(x, ids)
            got, want = ix.search(x[:20].copy(), 3, 6), bf.search(x[:20].copy(), 3)
            assert np.mean(got[0][:, 0] == want[0][:, 0]) > 0.8
            assert rt.cudaStreamDestroy(stream) == 0
            ix.close()
            bf.close()
            assert _capi.load().vb200_release_workspaces() == 0
        finally:
            engine.set_stream(None)
    again = engine.BfHandle(24, 0)
    again.add(x, ids)
    assert np.array_equal(again.search(x[:20].copy(), 3)[0], want[0])


class LittleMemory:
    """All but `left` bytes of device memory taken while in scope, the library's own reserve given back first."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch

        from vsag_b200 import _capi

        _capi.load().vb200_release_workspaces()
        torch.cuda.empty_cache()
        self.taken = []
        for _ in range(3):     # (the last step may be rounded up)
            free = torch.cuda.mem_get_info()[0] - self.left
            if free > (8 << 20):
                self.taken.append(torch.empty(free >> 21 << 21, dtype=torch.uint8, device="cuda"))
        assert torch.cuda.mem_get_info()[0] <= self.left + (16 << 20)

    def __exit__(self, *exc):
        import torch

        self.taken = None
        torch.cuda.empty_cache()


def test_a_batch_whose_scores_do_not_fit(engine):
    """200,000 rows for each of 1000 queries are 800 MB of scores; the grouped scan needs a few MB."""
    n, dim, nlist, nq, k = 200_000, 32, 64, 1000, 5
    x, q = mixture(3, n, dim, nlist, 0.2), mixture(4, nq, dim, nlist, 0.2)
    ix = engine.IvfHandle(dim, 0, nlist, engine.QUANT_FP32)
    ix.train(x[:20_000], iters=2)
    ix.add(x, np.arange(n, dtype=np.int64))
    want = ix.search_ex(q, k, nlist, timeout_ms=1e9)
    with LittleMemory(400 << 20):
        got = ix.search(q, k, nlist)
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[0], want[0])
    again = ix.search(q, k, nlist)
    assert np.array_equal(again[1], want[1]) and np.array_equal(again[0], want[0])


def test_exact_search_without_room_for_a_second_copy(engine):
    """A batch of ten over rows of 563 MB (beyond the pool's largest block), whose tiled copy is as large again."""
    import torch

    n, dim, nq, k = 2_200_000, 64, 10, 4
    g = torch.Generator(device="cuda").manual_seed(1)
    base = torch.rand((n, dim), generator=g, device="cuda")
    q = base[1000:1000 + nq].cpu().numpy() + np.float32(0.01)
    ix = engine.BfHandle(dim, 0)
    ix.add(base, torch.arange(n, dtype=torch.int64, device="cuda"))
    del base
    want = [ix.search(q[i:i + 1].copy(), k) for i in range(nq)]
    with LittleMemory(300 << 20):
        got = ix.search(q, k)
    for _ in range(2):
        assert np.array_equal(got[1], np.concatenate([w[1] for w in want]))
        assert np.array_equal(got[0], np.concatenate([w[0] for w in want]))
        got = ix.search(q, k)


def test_exact_batches_with_lists_for_a_few_queries_at_a_time(engine):
    """3000 queries over 400,000 rows collect some 300 MB of candidates.  With less than that left they go in smaller parts; the
    search of more rows at a time, which a batch without any such room is left to, does not look for neighbours that the scores
    cannot tell apart, and these rows lie far from the origin."""
    import torch

    n, dim, nq, k = 400_000, 16, 3000, 100
    g = torch.Generator(device="cuda").manual_seed(8)
    base = 80 + 0.01 * torch.randn((n, dim), generator=g, device="cuda")
    q = (80 + 0.01 * torch.randn((nq, dim), generator=g, device="cuda")).cpu().numpy()
    ix = engine.BfHandle(dim, 0)
    ix.add(base, torch.arange(n, dtype=torch.int64, device="cuda"))
    del base
    ix.search(q[:9].copy(), k)                     # (the tiled copy of the rows)
    some = slice(0, nq, 100)
    one = [ix.search(v[None].copy(), k) for v in q[some]]
    with LittleMemory(160 << 20):
        got = ix.search(q, k)
    assert np.array_equal(got[1][some], np.concatenate([o[1] for o in one]))
    assert np.array_equal(got[0][some], np.concatenate([o[0] for o in one]))


def fp32_index(engine, n, dim, seed):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand((n, dim), generator=g, device="cuda")
    ix = engine.IvfHandle(dim, 0, 16, engine.QUANT_FP32)
    ix.train(x[:4000].contiguous(), iters=2, init=x[:16].contiguous())
    ix.add(x, torch.arange(n, dtype=torch.int64, device="cuda"))
    return ix, x[:200].cpu().numpy(), x[-500:].cpu().numpy()


@pytest.mark.parametrize("dim", [65, 128])
def test_only_repeated_batches_keep_a_second_copy_of_fp32_rows(engine, dim):
    """The copy is there from the second batch by tiles on, its rows no longer than the rows themselves, and goes when rows are
    added; the batches before and after it was made agree with single queries."""
    n = 50_000
    ix, q, more = fp32_index(engine, n, dim, 9)
    alone = ix.memory_usage()
    one = [ix.search(q[i:i + 1].copy(), 5, 8) for i in range(20)]
    assert ix.memory_usage() == alone
    for batch in range(3):
        got = ix.search(q, 5, 8)
        for j in (0, 1):
            assert np.array_equal(got[j][:20], np.concatenate([o[j] for o in one]))
        assert ix.memory_usage() - alone == (0 if batch == 0 else n * 4 * ((dim + 7) // 8 * 8))
    ix.add(more, np.arange(n, n + len(more), dtype=np.int64))
    assert ix.memory_usage() < alone * 1.1
    got, one = ix.search(q, 5, 8), [ix.search(q[i:i + 1].copy(), 5, 8) for i in range(20)]
    for j in (0, 1):
        assert np.array_equal(got[j][:20], np.concatenate([o[j] for o in one]))


def test_adding_to_an_index_of_more_than_a_third_of_the_memory(engine):
    """640 MB of rows, and a second copy for the tile scan as large: an add needs room for the rows beside themselves, and 400 MB
    are left."""
    n, dim = 400_000, 400
    ix, q, more = fp32_index(engine, n, dim, 10)
    want = ix.search(q, 5, 8)
    ix.search(q, 5, 8)
    with LittleMemory(400 << 20):
        ix.add(more, np.arange(n, n + len(more), dtype=np.int64))
        assert ix.num_elements() == n + len(more)
    got = ix.search(more, 2, 16)
    assert np.array_equal(np.sort(got[0], 1)[:, 1], np.arange(n, n + len(more))) and np.array_equal(got[1], np.zeros_like(got[1]))
    again = ix.search(q, 5, 8)
    assert np.all(again[1] <= want[1])


def test_a_batch_that_lacks_memory_gives_up_the_second_copy(engine):
    """A deeper batch whose scores do not fit while the copy is held."""
    n, dim = 400_000, 400
    ix, q, _ = fp32_index(engine, n, dim, 11)
    for _ in range(2):
        ix.search(q[:80].copy(), 5, 2)
    q = np.tile(q, (3, 1))
    held = ix.memory_usage()
    with LittleMemory(200 << 20):
        got = ix.search(q, 5, 16)                   # 400,000 scores a query
    assert ix.memory_usage() <= held - n * dim * 4
    one = [ix.search(q[i:i + 1].copy(), 5, 16) for i in range(20)]
    for j in (0, 1):
        assert np.array_equal(got[j][:20], np.concatenate([o[j] for o in one]))


def test_a_refused_launch_does_not_fail_the_next_call(engine):
    """A batch that is grouped over SQ8 rows of 3100 dimensions asks for more shared memory than there is and ends with an error;
    calls on other handles, and small ones on this, go on."""
    from vsag_b200 import _capi

    dim, n = 3100, 300
    x = mixture(12, n, dim, 4, 0.2)
    ix = engine.IvfHandle(dim, 0, 4, engine.QUANT_SQ8)
    ix.set_centroids(x[:4].copy())
    ix.set_sq8_model(x.min(0), x.max(0) - x.min(0))
    ix.add(x, np.arange(n, dtype=np.int64))
    want = ix.search(x[:1].copy(), 3, 4)
    with pytest.raises(_capi.VsagB200Error):
        ix.search(x[:40].copy(), 3, 4)
    bf = engine.BfHandle(24, 0)
    bf.add(x[:, :24].copy(), np.arange(n, dtype=np.int64))
    assert np.array_equal(bf.search(x[:5, :24].copy(), 1)[0][:, 0], np.arange(5))
    with pytest.raises(_capi.VsagB200Error):
        ix.search(x[:40].copy(), 3, 4)
    again = ix.search(x[:1].copy(), 3, 4)
    assert np.array_equal(again[0], want[0]) and np.array_equal(again[1], want[1])
