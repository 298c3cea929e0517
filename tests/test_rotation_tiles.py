"""The query rotation of a search at the edges of its tiles, bit for bit
against the oracle: query counts around the 8- and 32-row tiles and the switch
between them, dimensions with every kind of remainder (a scalar tail, columns
beyond the last multiple of 4, a last chunk of one 16-dimension step) and rows
too wide for the few-query path's shared memory."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [16, 20, 63, 144, 203, 1040, 3728, 3744, 4096])
def test_rotation_tiles(dim):
    import katoann
    rng = np.random.default_rng(dim)
    n, nlist = 400, 5
    q, _ = np.linalg.qr(rng.standard_normal((dim, dim)))
    x = rng.standard_normal((n, dim)).astype(np.float32)
    a = dict(centroids=rng.standard_normal((nlist, dim)).astype(np.float32),
             list_sizes=np.array([100, 0, 50, 149, 101], np.uint32), ids=np.arange(n, dtype=np.uint32),
             vectors=x, rotation=np.ascontiguousarray(q, np.float32), head_dims=64)
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], x, rotation=a["rotation"], head_dims=64)
    ref = oracle.OracleIndex(None, arrays=a)
    queries = rng.standard_normal((130, dim)).astype(np.float32)
    for nq in (1, 7, 8, 9, 63, 64, 65, 130):
        kw = dict(k=10, nprobe=4, ranking="prefix", survivors=32)
        ids, dists = idx.search(queries[-nq:], **kw)
        rid, rd = ref.search(queries[-nq:], **kw)
        assert np.array_equal(ids, rid) and np.array_equal(dists, rd), nq
