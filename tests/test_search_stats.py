"""The diagnostics of the ranking pass name the warps it has: the scoring warps,
which wait for rows and for items, and the query staging, which waits for a free
buffer. Each first warp's total covers its waits."""
import pytest

from _util import fixture

pytestmark = pytest.mark.gpu


def test_role_cycles_of_the_ranking_pass():
    import katoann
    _, _, prefix, queries = fixture("d128")
    idx = katoann.Index()
    idx.load(prefix)
    idx.search(queries, k=10, nprobe=8, survivors=32)
    c = idx.search_stats()["ranking_role_cycles"]
    assert set(c) == {"score_wait_rows", "score_wait_items", "score_total", "stage_wait_buffer", "stage_total"}
    assert c["score_total"] > 0 and c["stage_total"] > 0
    assert c["score_wait_rows"] + c["score_wait_items"] <= c["score_total"]
    assert c["stage_wait_buffer"] <= c["stage_total"]
