"""One pass of more queries than 65,535 tiles of 32: the same results as in
passes of 65,536, and the oracle's for the last ones."""
import ctypes as C

import numpy as np
import pytest

import oracle
from _gpu import check, dptr, gpu, view_of

pytestmark = pytest.mark.gpu


def test_two_million_rotated_queries_in_one_pass():
    import katoann
    import torch
    nq, dim, k = 65535 * 32 + 33, 16, 3
    rng = np.random.default_rng(2)
    rot = np.linalg.qr(rng.standard_normal((dim, dim)))[0].astype(np.float32)
    x = rng.standard_normal((200, dim)).astype(np.float32)
    a = dict(centroids=x[::50].copy(), list_sizes=np.array([60, 0, 99, 41], np.uint32),
             ids=np.arange(200, dtype=np.uint32), vectors=x, rotation=rot, head_dims=64)
    idx = katoann.Index()
    idx.load_arrays(a["centroids"], a["list_sizes"], a["ids"], x, rotation=rot, head_dims=64)
    v = view_of(idx)
    assert v.rotated
    q = torch.randn(nq, dim, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    got = []
    for batch in (65536, nq):
        size = gpu().katoann_gpu_search_workspace(C.addressof(v), batch, k, 2, 0, k)
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
        dists = torch.empty((nq, k), dtype=torch.float32, device="cuda")
        check(gpu().katoann_gpu_search(C.addressof(v), dptr(q), nq, k, 2, 0, k, batch, dptr(ws), size,
                                       dptr(ids), dptr(dists), None))
        torch.cuda.synchronize()
        got.append((ids, dists))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    rid, rd = oracle.OracleIndex(None, arrays=a).search(q[-40:].cpu().numpy(), k=k, nprobe=2, ranking="full")
    assert np.array_equal(got[1][0][-40:].cpu().numpy().view(np.uint32), rid)
    assert np.array_equal(got[1][1][-40:].cpu().numpy(), rd)
