"""Words of shared memory that other warps write while a warp reads them (the
error flag, the counts behind the filter) steer full-mask shuffles and votes of
the ranking kernel: every lane has to act on one and the same value. Read from
the source, as lanes that disagree would wait for one another on the GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "katoann-public_gb300", "csrc")


def _block(text: str, at: int) -> int:
    """The end of the brace block that starts at text[at]."""
    depth, e = 1, at + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[e], 0)
        e += 1
    return e


def test_ranking_kernel_reads_shared_words_as_a_warp():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "rank_tc.cu")).read())
    at = text.index("{", text.index("rank_tc_kernel(const __grid_constant__"))
    body = text[at:_block(text, at)]
    for thread in ("tid", "lane"):  # one thread's own decisions
        while (m := re.search(r"if \(" + thread + r" == 0\) \{", body)):
            body = body[:m.start()] + body[_block(body, m.end() - 1):]
    words = re.findall(r"(uint32_t |, )?\*\s*(?:static_cast<volatile uint32_t \*>\()?(err|rcount|slabs|fstaged|fpairs)\b(?!\s*=[^=])", body)
    reads = [w for declared, w in words if not declared]
    assert not reads, reads
    assert "*reinterpret_cast<volatile" not in body
    assert body.count("warp_read(err)") == 3
    assert "filt = __shfl_sync(0xffffffffu, filt, 0);" in body  # what lane 0 decided
