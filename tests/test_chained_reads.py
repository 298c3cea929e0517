"""Launches of a search overlap: a kernel may be resident while the one before
it still writes, and after_previous() orders ordinary accesses only. Read-only
loads (const __restrict__ parameters, __ldg) promise data that no kernel writes
meanwhile, so a chained kernel takes them for the index's arrays, the probe
model's and the caller's queries alone. Read from the sources: no run shows a
load that the compiler was merely allowed to move."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "katoann-public_gb300", "csrc")

# what no kernel of a search writes, by the names the kernels give it
CONSTANT = {"xhi", "xlo", "xnorm", "xn", "ids", "list_off", "rot", "rank"}
# the caller's queries, where a kernel reads those and never a copy of them
QUERIES = {"rotate_tma_kernel": {"in"}, "transpose_pad_kernel": {"in"}, "transpose_pad4_kernel": {"in"},
           "rotate_seq_kernel": {"in"}}


def _kernels():
    """(file, kernel, parameter list, body) of every kernel that may be chained."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void(?:\s+__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s+(\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params, j = text[m.end():i - 1], text.index("{", i)
            depth, e = 1, j + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[e], 0)
                e += 1
            body = text[j:e]
            if "after_previous()" in body:
                out.append((os.path.basename(path), m.group(1), params, body))
    return out


KERNELS = _kernels()


def test_every_launched_kernel_waits_first():
    """launch() sets the overlap: each kernel it is given is among those looked at."""
    names = {k[1] for k in KERNELS}
    assert len(names) >= 20, names
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        for name in re.findall(r"\blaunch\((\w+_kernel)\b", open(path).read()):
            assert name in names, (path, name)
    for _, name, _, body in KERNELS:
        assert body.lstrip("{ \n").startswith("after_previous();"), name


@pytest.mark.parametrize("file,name,params,body", KERNELS, ids=[k[1] for k in KERNELS])
def test_read_only_loads_of_constant_arrays(file, name, params, body):
    allowed = CONSTANT | QUERIES.get(name, set())
    promised = set(re.findall(r"__restrict__\s+(\w+)", params))
    assert promised <= allowed, (file, promised - allowed)
    # an __ldg names the array it starts from, or a row pointer made from it
    for arg in re.findall(r"__ldg\(((?:[^()]|\((?:[^()]|\([^()]*\))*\))*)\)", body):
        words = set(re.findall(r"\b[a-z]\w*\b", arg))
        assert words & (allowed | {"x"}) and not words & {"qhi", "qlo"}, (file, arg)
