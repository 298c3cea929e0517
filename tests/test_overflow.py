"""Queries with more candidates than their buffers hold, rescanned by the whole
grid: more probed lists than one tile of 256, empty ones and longer ones than a
piece of 256 rows among them, more queries than CTAs, each with its own number of
lists, in one pass and in several. Bit for bit the oracle's results."""
import numpy as np
import pytest

import oracle
from _gpu import gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def data():
    rng = np.random.default_rng(7)
    nlist, dim = 530, 128
    sizes = rng.integers(0, 12, nlist).astype(np.uint32)
    sizes[[3, 255, 256, 257, 511, 529]] = 257, 256, 0, 600, 1, 255
    n = int(sizes.sum())
    x, cen = (rng.standard_normal((m, dim)).astype(np.float32) for m in (n, nlist))
    q = rng.standard_normal((700, dim)).astype(np.float32)
    return dict(centroids=cen, list_sizes=sizes, ids=rng.permutation(n).astype(np.uint32), vectors=x, rotation=None,
                head_dims=64), q


@pytest.mark.parametrize("max_batch", [4096, 300])
@pytest.mark.parametrize("budgets", [False, True])
def test_rescans_by_the_grid(data, budgets, max_batch):
    import katoann
    a, q = data
    nlist, S = len(a["list_sizes"]), 16
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], a["vectors"], head_dims=64, max_batch=max_batch)
    ref = oracle.OracleIndex(None, arrays=a)
    kw = dict(k=10, ranking="prefix", survivors=S)
    b = np.resize(np.array([1, 2, 31, 32, 33, 255, 256, 257, 511, 512, 513, nlist], np.uint32), len(q))
    if budgets:
        rid, rd = np.empty((len(q), 10), np.uint32), np.empty((len(q), 10), np.float32)
        for p in np.unique(b):
            rid[b == p], rd[b == p] = ref.search(q[b == p], nprobe=int(p), **kw)
        kw["nprobe_per_query"] = b
    else:
        rid, rd = ref.search(q, nprobe=nlist, **kw)
    try:
        assert gpu().katoann_gpu_set_candidate_cap(16) == 0
        for _ in range(2):
            ids, dists = idx.search(q, nprobe=nlist, **kw)
            assert idx.search_stats()["ranking_rescans"] > (0 if budgets else 99)  # (the last pass's)
            bad = np.nonzero((ids != rid).any(1) | (dists != rd).any(1))[0]
            assert len(bad) == 0, bad[:5]
    finally:
        assert gpu().katoann_gpu_set_candidate_cap(32768) == 0


@pytest.mark.parametrize("S", [300, 1000, 3000])
def test_rescans_with_many_survivors(data, S):
    """Survivors above the 2,048 candidates that a bound looks at otherwise, and
    counts whose eightfold lies on both sides of the buffer's size."""
    import katoann
    a, q = data
    nlist = len(a["list_sizes"])
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], a["vectors"], head_dims=64)
    kw = dict(k=10, nprobe=nlist, ranking="prefix", survivors=S)
    rid, rd = oracle.OracleIndex(None, arrays=a).search(q[:40], **kw)
    try:
        assert gpu().katoann_gpu_set_candidate_cap(max(S, 512)) == 0
        ids, dists = idx.search(q[:40], **kw)
        assert idx.search_stats()["ranking_rescans"] > 0
    finally:
        assert gpu().katoann_gpu_set_candidate_cap(32768) == 0
    assert np.array_equal(ids, rid) and np.array_equal(dists, rd)
