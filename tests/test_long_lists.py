"""Exact ranking over one list of more rows than 65,535 parts of 256: a flat
index of 17 million rows, through the C ABI. The expected rows come from exact
integer distances in torch, in (distance, id) order."""
import ctypes as C

import numpy as np
import pytest

from _gpu import GpuIndex, check, dptr, gpu

pytestmark = pytest.mark.gpu

ROWS = 65535 * 256 + 1
DIM = 64


@pytest.fixture(scope="module")
def flat():
    import torch
    g = torch.Generator(device="cuda").manual_seed(9)
    hi, lo = (torch.randint(0, 256, (ROWS, DIM), generator=g, device="cuda", dtype=torch.uint8) for _ in range(2))

    def norm(h, l, high_only=False):
        out = torch.empty(len(h), dtype=torch.int64, device="cuda")
        for s in range(0, len(h), 1 << 20):
            c = h[s:s + (1 << 20)].double()
            if not high_only:
                c = c * 256 + l[s:s + (1 << 20)].double()
            out[s:s + (1 << 20)] = (c * c).sum(1).long()  # below 2^53: exact
        return out

    t = dict(hi=hi, lo=lo, norm=norm(hi, lo), hinorm=norm(hi, lo, True),
             ids=torch.arange(ROWS, device="cuda", dtype=torch.int32).flip(0).contiguous(),
             off=torch.tensor([0, ROWS], device="cuda", dtype=torch.int32),
             chi=torch.zeros(1, DIM, device="cuda", dtype=torch.uint8))
    t["cnorm"] = torch.zeros(1, device="cuda", dtype=torch.int64)
    v = GpuIndex(dim=DIM, dc=DIM, nlist=1, npts=ROWS, max_list=ROWS, lo=0.0, inv_step=65535.0,
                 step_sq=1.0 / 65535.0 ** 2)
    for name, key in (("d_hi", "hi"), ("d_lo", "lo"), ("d_norm", "norm"), ("d_hinorm", "hinorm"),
                      ("d_ids", "ids"), ("d_list_off", "off"), ("d_chi", "chi"), ("d_clo", "chi"),
                      ("d_cnorm", "cnorm")):
        setattr(v, name, t[key].data_ptr())
    return v, t


def _expected(t, code, k):
    import torch
    l2 = torch.empty(ROWS, dtype=torch.int64, device="cuda")
    for s in range(0, ROWS, 1 << 20):
        d = t["hi"][s:s + (1 << 20)].double() * 256 + t["lo"][s:s + (1 << 20)].double() - code
        l2[s:s + (1 << 20)] = (d * d).sum(1).long()
    near = l2.topk(k + 64, largest=False, sorted=True)
    vals = near.values.contiguous()
    dist = torch.empty(len(vals), device="cuda", dtype=torch.float32)
    check(gpu().katoann_gpu_dist_values(dptr(vals), len(vals), 1.0 / 65535.0 ** 2, dptr(dist), None))
    torch.cuda.synchronize()
    d, ids = dist.cpu().numpy(), t["ids"][near.indices].cpu().numpy()
    order = np.lexsort((ids, d))[:k]
    return ids[order], d[order]


@pytest.mark.parametrize("k", [10, 300])
def test_exact_ranking_of_a_list_of_17_million_rows(flat, k):
    import torch
    v, t = flat
    code = torch.randint(0, 65536, (2, DIM), generator=torch.Generator(device="cuda").manual_seed(4),
                         device="cuda").double()
    q = (code / 65535.0).float().contiguous()
    size = gpu().katoann_gpu_search_workspace(C.byref(v), 2, k, 1, 0, k)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    ids = torch.empty((2, k), dtype=torch.int32, device="cuda")
    dists = torch.empty((2, k), dtype=torch.float32, device="cuda")
    check(gpu().katoann_gpu_search(C.byref(v), dptr(q), 2, k, 1, 0, k, 2, dptr(ws), size, dptr(ids),
                                   dptr(dists), None))
    torch.cuda.synchronize()
    for i in range(2):
        want_ids, want = _expected(t, code[i], k)
        assert np.array_equal(ids[i].cpu().numpy(), want_ids)
        assert np.array_equal(dists[i].cpu().numpy(), want)
