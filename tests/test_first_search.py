"""A host search of one pass allocates no pinned memory: the load has made its
staging and its wait count. (Pinning a page range takes longer than a search, and
the first search of every index paid for it.) Read from the sources: from outside
an allocation shows as time alone."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "katoann-public_gb300", "csrc")


def _body(text, head):
    start = text.index("{", text.index(head))
    depth, i = 1, start + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[start:i]


def test_the_load_makes_the_pinned_memory_of_one_pass_searches():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "index.cpp")).read())
    search = _body(text, "void Index::search(")
    # the buffers by their members, and a call only for the counts of more passes
    assert "cudaMallocHost" not in search and "stage()" not in search
    made = [m.group(1) for m in re.finditer(r"cudaMallocHost\(reinterpret_cast<void \*\*>\(&(\w+)\)", text)]
    assert sorted(made) == ["hstage", "hwait"]
    opened = _body(text, "void open()")
    assert "hstage" in opened and "wait_counts(1)" in opened
    # every place that makes an index's stream makes them
    assert text.count("cudaStreamCreateWithFlags(&") == 1 and "cudaStreamCreateWithFlags" in opened
    assert text.count("s.open()") == 2
