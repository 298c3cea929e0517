"""The ranking pass at the edges of its tiles, bit for bit against the oracle:
list lengths around its 32- and 64-row steps, query counts per list around its
groups of 8 and its items of 16, 32 and 64, prefixes of one to eight chunks,
with values that decay over the dimensions (items scored over the leading 128
alone), that do not (nearly every pair passes there) and at the ends of the
byte range (the largest sums)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZES = (0, 1, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 700)


def _arrays(dim, head, kind, nq, seed):
    rng = np.random.default_rng(seed)
    scale = np.arange(1, dim + 1) ** (-0.6 if kind == "decaying" else 0.0)
    n = sum(SIZES)
    if kind == "ends":
        x = rng.integers(0, 2, (n, dim)).astype(np.float32)
        q = rng.integers(0, 2, (nq, dim)).astype(np.float32)
        x[n // 2], q[0] = 1.0, 1.0
        x[n // 3], q[-1] = 0.0, 0.0
    else:
        x = (rng.standard_normal((n, dim)) * scale).astype(np.float32)
        q = (rng.standard_normal((nq, dim)) * scale).astype(np.float32)
    cen = (rng.standard_normal((len(SIZES), dim)) * scale).astype(np.float32)
    return dict(centroids=cen, list_sizes=np.array(SIZES, np.uint32),
                ids=np.arange(n, dtype=np.uint32), vectors=x, rotation=None, head_dims=head), q


@pytest.mark.parametrize("kind", ["decaying", "flat", "ends"])
@pytest.mark.parametrize("dim,head", [(64, 64), (128, 64), (128, 128), (192, 192), (256, 256), (320, 320),
                                      (448, 384), (1024, 1024)])
def test_ranking_tiles(dim, head, kind):
    import katoann
    a, q = _arrays(dim, head, kind, 130, dim + head)
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], a["vectors"], head_dims=head)
    ref = oracle.OracleIndex(None, arrays=a)
    for nq, nprobe, ranking in ((130, len(SIZES), "prefix"), (65, len(SIZES), "high"), (33, 9, "prefix"),
                                (9, len(SIZES), "prefix"), (1, len(SIZES), "prefix")):
        kw = dict(k=10, nprobe=nprobe, ranking=ranking, survivors=24)
        ids, dists = idx.search(q[-nq:], **kw)
        rid, rd = ref.search(q[-nq:], **kw)
        bad = np.nonzero((ids != rid).any(1) | (dists != rd).any(1))[0]
        assert len(bad) == 0, (nq, kw, bad[:5])


@pytest.mark.parametrize("kind", ["decaying", "ends"])
@pytest.mark.parametrize("S", [1, 31, 128, 129, 300, 511, 1300])
def test_seed_bounds(S, kind):
    """Survivor counts around the seed bound's own edges: all of the probed rows
    scored or a sketch's pick of 2 S, the last selection by counting (256 rows) or
    by digits, fewer rows than S, and every sketch distance in a few bins."""
    import katoann
    a, q = _arrays(128, 64, kind, 17, S)
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], a["vectors"], head_dims=64)
    ref = oracle.OracleIndex(None, arrays=a)
    for nprobe, ranking in ((len(SIZES), "prefix"), (len(SIZES), "high"), (5, "prefix"), (len(SIZES), "full")):
        kw = dict(k=min(S, 20), nprobe=nprobe, ranking=ranking, survivors=S)
        ids, dists = idx.search(q, **kw)
        rid, rd = ref.search(q, **kw)
        bad = np.nonzero((ids != rid).any(1) | (dists != rd).any(1))[0]
        assert len(bad) == 0, (kw, bad[:5])


@pytest.mark.parametrize("dim,ranking", [(192, "prefix"), (512, "high"), (576, "prefix"), (640, "high"),
                                         (832, "high"), (960, "prefix"), (1024, "prefix")])
def test_rescans_over_every_dimension(dim, ranking):
    """Candidate buffers of 16 rows: the queries are rescanned, over all of a
    prefix whose 16-byte pieces need not divide among the lanes of a row."""
    import katoann

    from _gpu import gpu
    a, q = _arrays(dim, dim, "flat", 20, dim)
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], a["vectors"], head_dims=dim)
    ref = oracle.OracleIndex(None, arrays=a)
    kw = dict(k=10, nprobe=len(SIZES), ranking=ranking, survivors=16)
    rid, rd = ref.search(q, **kw)
    try:
        assert gpu().katoann_gpu_set_candidate_cap(16) == 0
        ids, dists = idx.search(q, **kw)
        assert idx.search_stats()["ranking_rescans"] > 0
    finally:
        assert gpu().katoann_gpu_set_candidate_cap(32768) == 0
    assert np.array_equal(ids, rid) and np.array_equal(dists, rd)


def test_workspace_of_a_batch_serves_smaller_ones():
    """katoann_gpu_search_workspace grows with the batch for every ranking: a
    workspace sized for max_batch must do for any batch up to it."""
    import ctypes as C

    from _gpu import GpuIndex, gpu
    view = GpuIndex(dim=128, dc=128, nlist=4096, npts=1 << 22, head_dims=128, max_list=9000)
    for ranking in (0, 1, 2):
        for k, survivors in ((10, 32), (200, 200), (300, 600)):
            sizes = [gpu().katoann_gpu_search_workspace(C.byref(view), b, k, 512, ranking, survivors)
                     for b in (1, 2, 7, 63, 64, 500, 1000, 2000, 4096)]
            assert sizes[0] > 0 and sizes == sorted(sizes), (ranking, k, sizes)
