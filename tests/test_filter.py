"""The ranking pass's filter over the leading 128 dimensions, which rotated
indexes alone have (here the rotation is the identity, so that the dimensions are
the test's own): bit for bit the oracle's results where the values decay over the
dimensions, where they do not and nearly every pair passes, and at the ends of the
byte range. And flat values must not cost rescans: what the filter lets through
has to fit the record lists."""
import numpy as np
import pytest

import oracle
from test_rank_shapes import SIZES, _arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["decaying", "flat", "ends"])
@pytest.mark.parametrize("dim,head", [(192, 192), (256, 192), (256, 256), (320, 320), (512, 384), (1024, 512),
                                      (832, 832), (1024, 1024)])
def test_filtered_ranking(dim, head, kind):
    import katoann
    a, q = _arrays(dim, head, kind, 130, dim + head)
    a["rotation"] = np.eye(dim, dtype=np.float32)
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], a["vectors"], rotation=a["rotation"], head_dims=head)
    ref = oracle.OracleIndex(None, arrays=a)
    for nq, nprobe, ranking in ((130, len(SIZES), "prefix"), (65, len(SIZES), "high"), (33, 9, "prefix"),
                                (9, len(SIZES), "prefix"), (1, len(SIZES), "prefix")):
        kw = dict(k=10, nprobe=nprobe, ranking=ranking, survivors=24)
        ids, dists = idx.search(q[-nq:], **kw)
        rid, rd = ref.search(q[-nq:], **kw)
        bad = np.nonzero((ids != rid).any(1) | (dists != rd).any(1))[0]
        assert len(bad) == 0, (nq, kw, bad[:5])


@pytest.mark.parametrize("rotated", [True, False])
@pytest.mark.parametrize("dim", [512, 1024])
def test_flat_values_need_no_rescans(dim, rotated):
    import katoann
    rng = np.random.default_rng(dim)
    nlist, n, nq = 400, 100_000, 512
    cen = rng.standard_normal((nlist, dim)).astype(np.float32)
    of = np.sort(rng.integers(0, nlist, n))
    x = cen[of] + 0.4 * rng.standard_normal((n, dim)).astype(np.float32)
    q = cen[rng.integers(0, nlist, nq)] + 0.4 * rng.standard_normal((nq, dim)).astype(np.float32)
    rot = np.eye(dim, dtype=np.float32) if rotated else None
    a = dict(centroids=cen, list_sizes=np.bincount(of, minlength=nlist).astype(np.uint32),
             ids=np.arange(n, dtype=np.uint32), vectors=x, rotation=rot, head_dims=dim)
    idx = katoann.Index()
    idx.load_arrays(cen, a["list_sizes"], a["ids"], x, rotation=rot, head_dims=dim)
    kw = dict(k=10, nprobe=33, ranking="prefix", survivors=64)
    ids, dists = idx.search(q, **kw)
    assert idx.search_stats()["ranking_rescans"] == 0
    rid, rd = oracle.OracleIndex(None, arrays=a).search(q[:32], **kw)
    assert np.array_equal(ids[:32], rid) and np.array_equal(dists[:32], rd)
