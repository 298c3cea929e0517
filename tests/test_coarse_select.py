"""The coarse selection's probes, against a sort of the distances it selects
from: list counts at the edges of its thread blocks and of the rows that stay
in registers, probe counts at the edges of its three group sizes, and distances
that are spread, ordered along the lists, or few (ties at the boundary, which
the search counts)."""
import numpy as np
import pytest

from _gpu import GpuIndex, check, dptr, gpu

pytestmark = pytest.mark.gpu

PROBES = (1, 2, 16, 42, 43, 170, 171, 384, 683, 1365, 2731, 4096, 4097)


@pytest.mark.parametrize("kind", ["spread", "ordered", "few"])
@pytest.mark.parametrize("nlist", [1, 3, 127, 512, 1023, 1024, 1025, 4096, 4098, 8192, 8193, 16384, 16385, 30001])
def test_probes_are_the_nearest_lists(nlist, kind):
    import ctypes as C

    import katoann
    import torch
    rng = np.random.default_rng(nlist)
    dim, nq = 64, 3
    cen = rng.standard_normal((nlist, dim)).astype(np.float32)
    if kind == "ordered":
        cen[:, 0] += np.linspace(0, 20, nlist, dtype=np.float32)
    elif kind == "few":
        cen = cen[rng.integers(0, min(nlist, 3), nlist)]
    q = cen[rng.integers(0, nlist, nq)] + 0.1 * rng.standard_normal((nq, dim)).astype(np.float32)
    idx = katoann.Index()
    idx.load_arrays(cen, np.ones(nlist, np.uint32), np.arange(nlist, dtype=np.uint32), cen)
    view = GpuIndex.from_address(idx.device_view)
    planes = [torch.empty((nq, view.dc), dtype=torch.uint8, device="cuda") for _ in range(2)]
    norms = [torch.empty(nq, dtype=torch.int64, device="cuda") for _ in range(3)]
    qd = torch.from_numpy(q).cuda()
    check(gpu().katoann_gpu_quantize_rows(dptr(qd), nq, dim, view.dc, view.lo, view.inv_step, 0, dptr(planes[0]),
                                          dptr(planes[1]), dptr(norms[0]), dptr(norms[1]), dptr(norms[2]), None))
    dists = torch.empty((nq, nlist), dtype=torch.float32, device="cuda")
    for p in sorted({min(p, nlist) for p in PROBES}):
        probed = torch.empty((nq, p), dtype=torch.int32, device="cuda")
        check(gpu().katoann_gpu_coarse(C.byref(view), dptr(planes[0]), dptr(planes[1]), dptr(norms[0]), nq, p,
                                       dptr(dists), dptr(probed), None))
        d, got = dists.cpu().numpy(), probed.cpu().numpy()
        want = np.argsort(d, axis=1, kind="stable")
        if p > 4096:  # a set
            got, want[:, :p] = np.sort(got, 1), np.sort(want[:, :p], 1)
        assert np.array_equal(got, want[:, :p]), p
        if p == nlist:
            continue
        idx.search(q, k=1, nprobe=p, ranking="high", survivors=1)
        s = np.sort(d, axis=1)
        assert idx.search_stats()["coarse_boundary_ties"] == int((s[:, p] == s[:, p - 1]).sum()), p
