"""Host searches whose queries, ids and distances are pageable or pinned, each for
itself: batches on both sides of the lines (32 KiB, 1 MiB) between the index's
own staging and copies from and to the caller's buffers."""
import itertools

import numpy as np
import pytest

import oracle
from _util import fixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("nq", [1, 34, 35, 200, 1092, 1093])  # 960 bytes each with k = 56
def test_pageable_and_pinned_buffers_give_the_same(nq, graph):
    import katoann
    import torch
    spec, z, prefix, queries = fixture("d128")
    k = 56
    assert (128 * 4 + 2 * 4 * k) * 34 < 32 << 10 < (128 * 4 + 2 * 4 * k) * 35
    assert (128 * 4 + 2 * 4 * k) * 1092 < 1 << 20 < (128 * 4 + 2 * 4 * k) * 1093
    idx = katoann.Index()
    idx.load(prefix)
    q = np.ascontiguousarray(queries[np.arange(nq) % len(queries)], np.float32)
    rid, rd = oracle.OracleIndex(prefix).search(q, k=k, nprobe=8, survivors=64)
    for pins in itertools.product([False, True], repeat=3):
        tq, ti, td = (torch.zeros(shape, dtype=t, pin_memory=pin) for shape, t, pin in
                      zip(((nq, 128), (nq, k), (nq, k)), (torch.float32, torch.int32, torch.float32), pins))
        tq.copy_(torch.from_numpy(q))
        idx.search_into(tq.data_ptr(), nq, ti.data_ptr(), td.data_ptr(), k=k, nprobe=8, survivors=64, graph=graph)
        assert np.array_equal(ti.numpy().view(np.uint32), rid) and np.array_equal(td.numpy(), rd), pins
