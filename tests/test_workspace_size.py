"""Sizes of search workspaces, asked of the library without a GPU. A server sizes
its slots once, for its largest batch, k and depth: no smaller search may need
more."""
import ctypes as C

import pytest

from _gpu import GpuIndex, gpu

RANKINGS = {"full": 0, "high": 1, "prefix": 2}


def _size(dim, max_list, batch, k, nprobe, ranking, survivors):
    view = GpuIndex(dim=dim, dc=dim, nlist=4096, npts=1 << 24, head_dims=dim, max_list=max_list)
    size = gpu().katoann_gpu_search_workspace(C.byref(view), batch, k, nprobe, RANKINGS[ranking], survivors)
    assert size > 0
    return size


# ranking "high" and "prefix" over 1,152 bytes run on the CUDA cores too
@pytest.mark.parametrize("dim,ranking", [(128, "full"), (1152, "full"), (1152, "high"), (1152, "prefix"),
                                         (128, "prefix")])
@pytest.mark.parametrize("max_list", [1, 200, 256, 257, 300, 513, 9000, 200_000])
def test_workspace_grows_with_k_batch_and_probes(dim, ranking, max_list):
    ks = (1, 2, 10, 31, 100, 199, 200, 201, 255, 256, 257, 299, 300, 301, 512, 1000, 4096)
    for batch in (1, 64, 500, 4096):
        for nprobe in (1, 32, 512):
            sizes = [_size(dim, max_list, batch, k, nprobe, ranking, k) for k in ks]
            assert sizes == sorted(sizes), (batch, nprobe, sizes)
    for k in (10, 256, 300):
        sizes = [_size(dim, max_list, batch, k, 64, ranking, k) for batch in (1, 7, 64, 500, 1000, 2000, 4096)]
        assert sizes == sorted(sizes), (k, sizes)
        sizes = [_size(dim, max_list, 256, k, p, ranking, k) for p in (1, 3, 10, 64, 200, 512, 2000, 4096)]
        assert sizes == sorted(sizes), (k, sizes)


@pytest.mark.parametrize("dim,ranking", [(128, "full"), (1152, "high")])
@pytest.mark.parametrize("batch,k,nprobe", [(1, 10, 1), (4096, 10, 64), (4096, 10, 512), (4096, 100, 64), (4096, 1, 512)])
def test_splitting_lists_takes_at_most_128_mib(dim, ranking, batch, k, nprobe):
    """Lists of up to 256 rows have one part; longer ones may be split."""
    whole = _size(dim, 256, batch, k, nprobe, ranking, k)
    for max_list in (257, 6063, 30_000, 1_000_000):
        assert _size(dim, max_list, batch, k, nprobe, ranking, k) <= whole + (128 << 20), max_list


@pytest.mark.parametrize("batch,depth", [(1, 1), (64, 128), (4096, 512), (4096, 4096)])
def test_features_take_no_candidate_places(batch, depth):
    """The feature pass ends with the selected lists: its workspace does not depend
    on the lists' lengths, and is no larger than a search's of that depth."""
    gpu().katoann_gpu_probe_features_workspace.restype = C.c_size_t
    gpu().katoann_gpu_probe_features_workspace.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32]
    sizes = []
    for max_list in (1, 300, 6063, 1_000_000):
        view = GpuIndex(dim=128, dc=128, nlist=4096, npts=1 << 24, head_dims=128, max_list=max_list)
        sizes.append(gpu().katoann_gpu_probe_features_workspace(C.byref(view), batch, depth))
        assert 0 < sizes[-1] <= _size(128, max_list, batch, 1, depth, "full", 1)
    assert len(set(sizes)) == 1, sizes
    assert gpu().katoann_gpu_probe_features_workspace(C.byref(view), batch, 4097) == 0
