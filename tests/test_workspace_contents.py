"""A search gives the oracle's results whatever its workspace holds before: every
word that a kernel reads was written by the search. Row widths whose padded copy
ends past the stored row (dc a multiple of 64 but not of 128, ranked over all of
it) and whole ones; bytes that are fp16 NaN and ordinary values."""
import ctypes as C

import numpy as np
import pytest

import oracle
from _gpu import check, dptr, gpu, view_of

pytestmark = pytest.mark.gpu

RANK = {"prefix": 2, "high": 1, "full": 0}
SIZES = (0, 1, 33, 64, 127, 1100)  # the longest is scored over all dimensions from the start


def _arrays(dim, nq):
    rng = np.random.default_rng(dim)
    n = sum(SIZES)
    x, q, cen = (rng.standard_normal((m, dim)).astype(np.float32) for m in (n, nq, len(SIZES)))
    return dict(centroids=cen, list_sizes=np.array(SIZES, np.uint32), ids=np.arange(n, dtype=np.uint32),
                vectors=x, rotation=None, head_dims=dim), q


@pytest.mark.parametrize("fill", [0x7F, 0x41])
@pytest.mark.parametrize("dim", [64, 192, 256, 320, 448, 832, 960, 1024])
def test_results_do_not_depend_on_the_workspace(dim, fill):
    import katoann
    import torch
    nq, k, S, p = 65, 10, 24, len(SIZES)
    a, queries = _arrays(dim, nq)
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], a["vectors"], head_dims=dim)
    ref = oracle.OracleIndex(None, arrays=a)
    v = view_of(idx)
    q = torch.from_numpy(queries).cuda()
    for ranking, code in RANK.items():
        size = gpu().katoann_gpu_search_workspace(C.addressof(v), nq, k, p, code, S)
        ws = torch.full((size,), fill, dtype=torch.uint8, device="cuda")
        ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
        dists = torch.empty((nq, k), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        check(gpu().katoann_gpu_search(C.addressof(v), dptr(q), nq, k, p, code, S, nq, dptr(ws), size,
                                       dptr(ids), dptr(dists), None))
        torch.cuda.synchronize()
        rid, rd = ref.search(queries, k=k, nprobe=p, ranking=ranking, survivors=S)
        bad = np.nonzero((ids.cpu().numpy().view(np.uint32) != rid).any(1) | (dists.cpu().numpy() != rd).any(1))[0]
        assert len(bad) == 0, (ranking, bad[:5])
