"""Survivors, refinement and top-k of a query, bit for bit against the oracle:
candidate and survivor counts around the 256 that are ranked by counting, k on
both sides of a warp, fewer candidates than survivors or than k, and vectors
with many equal distances, where the results depend on the order in which the
reference's heap meets them."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _pair(kind, seed):
    import katoann
    rng = np.random.default_rng(seed)
    n, dim, nlist = 6000, 64, 6
    if kind == "ties":  # few distinct vectors: most distances tie
        x = rng.integers(0, 3, (60, dim)).astype(np.float32)[rng.integers(0, 60, n)]
        x[:, 40:] = rng.integers(0, 2, (n, dim - 40))
        q = rng.integers(0, 3, (40, dim)).astype(np.float32)
    else:
        scale = np.arange(1, dim + 1) ** -0.5
        x = (rng.standard_normal((n, dim)) * scale).astype(np.float32)
        q = (rng.standard_normal((40, dim)) * scale).astype(np.float32)
    sizes = np.array([2000, 1, 500, 0, 1499, 2000], np.uint32)
    a = dict(centroids=x[rng.choice(n, nlist, replace=False)] + 0.01, list_sizes=sizes,
             ids=np.arange(n, dtype=np.uint32), vectors=x, rotation=None, head_dims=64)
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], sizes, a["ids"], x, head_dims=64)
    return idx, oracle.OracleIndex(None, arrays=a), q


@pytest.mark.parametrize("kind", ["ties", "plain"])
@pytest.mark.parametrize("survivors", [1, 64, 255, 256, 257, 700, 2100])
def test_top_k(kind, survivors):
    idx, ref, q = _pair(kind, survivors)
    for k in (1, 10, 32, 33, 100, 300):
        for nprobe in (1, 6):
            kw = dict(k=k, nprobe=nprobe, ranking="prefix", survivors=survivors)
            ids, dists = idx.search(q, **kw)
            rid, rd = ref.search(q, **kw)
            bad = np.nonzero((ids != rid).any(1) | (dists != rd).any(1))[0]
            assert len(bad) == 0, (kw, bad[:5])
