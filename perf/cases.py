"""The searches whose speed this framework is judged by.

Each case is a batch of queries against one index, through the module's public
entry points. Sizes are those of the benchmark's workloads (100,000 x 128,
1,000,000 x 1,024, 990,000 x 3,072, 10,000,000 x 1,024), of the server's
batches and of the tests, with odd and ragged ones among them.

Vectors: clusters whose centres and whose spread share a power-law spectrum
(eigenvalue_i ~ i^-power), unit length, as embeddings are after k-means: every
list has its own centre, several lists share a coarser component, list sizes
are skewed (log-normal). A rotated index stores the vectors reflected out of
their principal axes and holds the rotation that brings them back.
"""
from __future__ import annotations

import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "katoann-public_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import katoann  # noqa: E402

LADDER = katoann.ProbeModel.LADDER
# share of the training queries at each probe budget of the ladder
BUDGET_SHARES = (0.25, 0.12, 0.12, 0.10, 0.10, 0.09, 0.07, 0.05, 0.04, 0.03, 0.015, 0.01, 0.005)
PAD = 3.402823466e+38  # the distance of a place without a result


def _search(name, **kw):
    c = dict(name=name, n=100_000, dim=128, nlist=256, head=64, power=1.2, rotated=True,
             nq=1, k=10, nprobe=16, survivors=32, ranking="prefix", entry="device", graph=False,
             learned=False, per_query=False)
    c.update(kw)
    return c


def listed():
    return [
        # one interactive query, host arrays in and out
        _search("one_query", nq=1, survivors=64, entry="host"),
        # a handful of queries against a wide index, as a retrieval step of a
        # service issues them between its own kernels
        _search("few_queries", n=1_000_000, dim=1024, nlist=4096, head=128, nq=16, nprobe=32),
        # a server's batch under moderate load: pinned buffers, replayed graph, k = 100
        _search("server_batch", n=1_000_000, dim=1024, nlist=4096, head=256, nq=113, k=100, nprobe=64,
                survivors=128, entry="pinned", graph=True),
        # the benchmark's small workload
        _search("small_batch", nq=1024, survivors=64),
        # the benchmark's 1M x 1,024 workload
        _search("plain_batch", n=1_000_000, dim=1024, nlist=4096, head=128, nq=4096),
        # the benchmark's 990k x 3,072 workload
        _search("wide_batch", n=990_000, dim=3072, nlist=4096, head=256, power=1.0, nq=4096),
        # the benchmark's 10M x 1,024 workload: fixed probes at recall 0.99
        _search("large_fixed", n=10_000_000, dim=1024, nlist=16384, head=256, nq=4096, nprobe=72,
                survivors=64),
        # the same with the learned probe budget, host buffers, replayed graph
        _search("large_learned", n=10_000_000, dim=1024, nlist=16384, head=256, nq=4096, nprobe=512,
                survivors=64, entry="pinned", graph=True, learned=True),
        # deep probing for high recall on a mid-size index, each query its own depth
        _search("deep_budget", n=2_000_000, dim=768, nlist=5000, head=192, nq=2000, k=20, nprobe=384,
                survivors=128, per_query=True),
        # odd sizes, no rotation: ranking over all high bytes, many results
        _search("odd_high", n=300_007, dim=102, nlist=777, head=0, power=0.4, rotated=False, nq=333, k=25,
                nprobe=33, survivors=400, ranking="high", entry="host"),
        # exact distances over every probed row (labels, recall checks)
        _search("exact_rank", n=200_000, dim=128, nlist=512, head=64, nq=256, nprobe=24, ranking="full"),
    ]


def draw(rng):
    """One more case of the same ranges: dimensions 48 to 3,072, 20 thousand to
    4 million vectors, 1 to 4,096 queries, 4 to 512 probes."""

    def spread(lo, hi):  # over the logarithm
        return int(round(lo * (hi / lo) ** rng.random()))

    dim = rng.choice([rng.randint(48, 200), 64 * rng.randint(2, 16), rng.randint(200, 1100),
                      128 * rng.randint(6, 24)])
    n = spread(20_000, max(20_000, min(4_000_000, 2_500_000_000 // dim)))
    nlist = max(64, min(8192, int(n ** 0.5 * rng.uniform(0.5, 4.0))))
    ranking = rng.choice(["prefix"] * 8 + ["high", "full"])
    rotated = ranking == "prefix"
    nq = spread(1, 4096)
    nprobe = min(spread(4, 512), nlist // 2)
    if ranking == "full":
        nq, nprobe = min(nq, 256), min(nprobe, 24)
    if ranking == "high":
        nq, nprobe = min(nq, 512), min(nprobe, 64)
    k = rng.choice([1, 10, 10, 10, rng.randint(2, 100)])
    head = min(dim // 64 * 64, 64 * rng.choice([1, 2, 3, 4, 4, 6]))
    if rotated and head == 0:
        head = 64  # dimensions are stored padded to a multiple of 64
    entry = rng.choice(["host", "device", "pinned"])
    case = dict(n=n, dim=dim, nlist=nlist, head=head if rotated else 0,
                power=rng.choice([1.0, 1.1, 1.2]) if rotated else 0.4, rotated=rotated, nq=nq, k=k,
                nprobe=nprobe, survivors=rng.choice([32, 64, 128, rng.randint(16, 400)]),
                ranking=ranking, entry=entry, graph=entry != "host" and rng.random() < 0.4,
                learned=False, per_query=entry == "device" and rotated and rng.random() < 0.3)
    most = work(_search("", n=10_000_000, dim=1024, nlist=16384, head=256, nq=4096, nprobe=72, survivors=64))
    while any(work(case)[w] > most[w] for w in most):  # no more than the largest listed case
        case["nq"], case["nprobe"] = max(1, case["nq"] // 2), max(1, case["nprobe"] * 3 // 4)
    return case


# ------------------------------------------------------------------- inputs
def _gen(seed, what):
    return torch.Generator(device="cuda").manual_seed((seed * 1_000_003 + what) % (2 ** 63))


class _Vectors:
    """The distribution a seed stands for: list centres, list sizes, the
    reflection out of the principal axes, and samples of rows and queries."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        n, d, L = case["n"], case["dim"], case["nlist"]
        g = _gen(seed, 1)
        lam = torch.arange(1, d + 1, device="cuda", dtype=torch.float32) ** -case["power"]
        self.scale = torch.sqrt(lam / lam.sum())
        ncomp = max(1, L // 4)
        comp = torch.randn(ncomp, d, generator=g, device="cuda") * self.scale
        of = (torch.rand(L, generator=g, device="cuda") ** 1.5 * ncomp).long().clamp_(max=ncomp - 1)
        self.centres = comp[of] + 0.4 * torch.randn(L, d, generator=g, device="cuda") * self.scale
        weight = torch.exp(0.6 * torch.randn(L, generator=g, device="cuda"))
        cdf = torch.cumsum(weight.double() / weight.double().sum(), 0).float()
        draws = torch.rand(n, generator=g, device="cuda")
        self.list_of_id = torch.searchsorted(cdf, draws).clamp_(max=L - 1)
        self.v = torch.randn(d, generator=g, device="cuda") if case["rotated"] else None
        if self.v is not None:
            self.v /= self.v.norm()

    def sample(self, lists, g, out=None):
        """One unit vector of each given list (in the stored basis)."""
        m, d = lists.shape[0], self.case["dim"]
        x = torch.empty(m, d, device="cuda") if out is None else out
        step = max(1, (1 << 28) // d)
        for s in range(0, m, step):
            e = min(m, s + step)
            z = torch.randn(e - s, d, generator=g, device="cuda")
            z.mul_(self.scale * 0.4).add_(self.centres[lists[s:e]])
            z.div_(z.norm(dim=1, keepdim=True))
            if self.v is not None:
                z.addr_(z @ self.v, self.v, alpha=-2.0)
            x[s:e] = z
        return x

    def rows(self):
        """(ids in list order, list sizes, vectors in list order)."""
        order = torch.sort(self.list_of_id, stable=True).indices
        sizes = torch.bincount(self.list_of_id, minlength=self.case["nlist"])
        return order, sizes, self.sample(self.list_of_id[order], _gen(self.seed, 2))

    def centroids(self):
        """The lists' means: centre over the length its rows had."""
        c = self.centres / torch.sqrt((self.centres ** 2).sum(1, keepdim=True) + 0.16)
        if self.v is not None:
            c = c - 2.0 * torch.outer(c @ self.v, self.v)
        return c.contiguous()

    def queries(self, m, what=3):
        g = _gen(self.seed, what)
        at = torch.randint(0, self.case["n"], (m,), generator=g, device="cuda")
        return self.sample(self.list_of_id[at], g)

    def rotation(self):
        if self.v is None:
            return None
        d = self.case["dim"]
        return (torch.eye(d, device="cuda") - 2.0 * torch.outer(self.v, self.v)).contiguous()


def _index(case, vec):
    ids, sizes, x = vec.rows()
    index = katoann.Index()
    index.load_arrays(vec.centroids(), sizes.cpu().numpy().astype(np.uint32), ids.to(torch.int32), x,
                      rotation=vec.rotation(), head_dims=case["head"] if case["rotated"] else 0)
    return index


def _budget_model(index, vec):
    """A probe-budget model over this index: the queries whose nearest lists
    lie close together are the hard ones."""
    q = vec.queries(4096, what=5).cpu().numpy()
    z = katoann.ProbeModel.features(index, q, depth=128)
    hard = np.argsort(np.argsort(z[:, 20] - z[:, 0], kind="stable"), kind="stable")[::-1] / len(z)
    labels = np.searchsorted(np.cumsum(BUDGET_SHARES)[:-1], hard).astype(np.uint8)
    return katoann.ProbeModel.fit(z, labels, depth=128, epochs=12, batch=512)


def prepare(case, seed):
    vec = _Vectors(case, seed)
    state = dict(case=case)
    nq, k = case["nq"], case["k"]
    index = _index(case, vec)
    args = dict(k=k, nprobe=case["nprobe"], ranking=case["ranking"], survivors=case["survivors"])
    q = vec.queries(nq)
    if case["graph"]:
        args["graph"] = True
    if case["learned"]:
        args.update(budget=_budget_model(index, vec), threshold=0.5)
    if case["per_query"]:
        g = _gen(seed, 6)
        depth = torch.exp(torch.randn(nq, generator=g, device="cuda") * 0.8) * case["nprobe"] * 0.3
        args["nprobe_per_query"] = depth.clamp(1, case["nprobe"]).to(torch.int32)
    if case["entry"] == "host":
        state["q"] = q.cpu().numpy()
    else:
        pin = dict(pin_memory=True) if case["entry"] == "pinned" else dict(device="cuda")
        state["q"] = torch.empty(nq, case["dim"], **pin).copy_(q)
        state["ids"] = torch.zeros(nq, k, dtype=torch.int32, **pin)
        state["dists"] = torch.zeros(nq, k, dtype=torch.float32, **pin)
    state.update(index=index, args=args)
    torch.cuda.synchronize()
    del vec, q
    torch.cuda.empty_cache()  # the library allocates outside torch's pool
    return state


# --------------------------------------------------------------------- runs
def run(state):
    case = state["case"]
    index, q, args = state["index"], state["q"], state["args"]
    if case["entry"] == "host":
        ids, dists = index.search(q, **args)
        return dict(ids=ids.view(np.int32), dists=dists)
    ids, dists = state["ids"], state["dists"]
    if case["entry"] == "pinned":
        index.search_into(q.data_ptr(), q.shape[0], ids.data_ptr(), dists.data_ptr(), **args)
    else:
        index.search_device(q, ids, dists, stream=torch.cuda.current_stream().cuda_stream, **args)
    return dict(ids=ids, dists=dists)


def work(case):
    """Every probed list's ranking bytes once for the batch, the centroids' and
    the survivors' 16-bit codes, the rotation, the queries and the results;
    two operations per product."""
    n, d, L = case["n"], case["dim"], case["nlist"]
    nq, S = case["nq"], max(case["survivors"], case["k"])
    if case["learned"]:
        p = sum(s * b for s, b in zip(BUDGET_SHARES, LADDER))
    else:
        p = case["nprobe"] * (0.4 if case["per_query"] else 1.0)
    full = case["ranking"] == "full"
    h = 2 * d if full else (case["head"] if case["ranking"] == "prefix" else d)
    rows = n * (1.0 - (1.0 - p / L) ** nq)
    pairs = nq * p * n / L
    nbytes = 4 * nq * d + 2 * L * d + rows * h + 8 * nq * case["k"]
    flops = 2 * nq * L * d + 2 * pairs * (d if full else h)
    if case["rotated"]:
        nbytes += 4 * d * d
        flops += 2 * nq * d * d
    if not full:
        nbytes += min(n, nq * S) * 2 * d
        flops += 2 * nq * S * d
    return dict(bytes=int(nbytes), flops=int(flops))


def exact(case, seed):
    """The true squared distances of the nearest rows of each query's nearest
    lists, in 64 bits (which row is nearest has no value of its own)."""
    if case["learned"] or case["per_query"]:
        return None
    nq, k, n, p = case["nq"], case["k"], case["n"], case["nprobe"]
    if nq * n * case["dim"] > 2e11:
        return None
    vec = _Vectors(case, seed)
    _, sizes, x = vec.rows()
    q, c = vec.queries(nq).double(), vec.centroids().double()
    near = torch.cdist(q, c, compute_mode="donot_use_mm_for_euclid_dist").topk(p, largest=False).indices
    probed = torch.zeros(nq, case["nlist"], dtype=torch.bool, device="cuda")
    probed.scatter_(1, near, True)
    lists = torch.repeat_interleave(torch.arange(case["nlist"], device="cuda"), sizes)
    best = torch.full((nq, k), PAD, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // max(nq, case["dim"]))
    for s in range(0, n, step):
        xs = x[s:s + step].double()
        d2 = (q ** 2).sum(1)[:, None] + (xs ** 2).sum(1)[None, :] - 2.0 * (q @ xs.T)
        d2.masked_fill_(~probed[:, lists[s:s + step]], PAD)
        best = torch.cat([best, d2], 1).topk(k, largest=False).values
    return dict(ids=None, dists=best)
