"""Searches between a caller's own kernels on one stream, without a host wait:
each search reads the queries that the kernel before it wrote and its results
are read, and everything it used is overwritten, by the kernels after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("nq,ranking,dim", [(1, "prefix", 128), (40, "full", 128), (300, "prefix", 130),
                                            (1500, "high", 64)])
def test_searches_between_kernels(nq, ranking, dim, captured):
    import katoann
    import torch
    rng = np.random.default_rng(nq)
    n, L, rounds, k = 6000, 40, 12, 10
    x = rng.standard_normal((n, dim)).astype(np.float32)
    rot = np.linalg.qr(rng.standard_normal((dim, dim)))[0].astype(np.float32)
    idx = katoann.Index()
    idx.load_arrays(x[:L].copy(), np.full(L, n // L, np.uint32), np.arange(n, dtype=np.uint32), x, rotation=rot,
                    head_dims=64)
    kw = dict(k=k, nprobe=9, ranking=ranking, survivors=32)
    qs = rng.standard_normal((rounds, nq, dim)).astype(np.float32)
    want = [idx.search(q, **kw) for q in qs]
    qd, ids = torch.from_numpy(qs).cuda(), torch.zeros((nq, k), dtype=torch.int32, device="cuda")
    q, d = torch.zeros((nq, dim), device="cuda"), torch.zeros((nq, k), device="cuda")
    got_i, got_d = (torch.zeros((rounds, nq, k), dtype=t, device="cuda") for t in (torch.int32, torch.float32))
    s = torch.cuda.Stream()

    def work():
        for r in range(rounds):
            q.copy_(qd[r])
            q.mul_(1.0)
            idx.search_device(q, ids, d, stream=s.cuda_stream, **kw)
            got_i[r].copy_(ids)
            got_d[r].copy_(d)
            for t in (q, ids, d):
                t.fill_(7)

    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        work()  # (sizes the workspace before a capture)
        if captured:
            s.synchronize()
            got_i.zero_()
            graph = torch.cuda.CUDAGraph()
            s.synchronize()
            with torch.cuda.graph(graph, stream=s):
                work()
            graph.replay()
        s.synchronize()
    for r in range(rounds):
        assert np.array_equal(got_i[r].cpu().numpy().astype(np.uint32), want[r][0])
        assert np.array_equal(got_d[r].cpu().numpy(), want[r][1])
