"""A host search without a buffer is refused by the copy, whatever its size: in a
process of its own, as a copy by the CPU would end it."""
import subprocess
import sys

import pytest

from _util import fixture

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path[:0] = {path!r}
import numpy as np
import katoann
idx = katoann.Index()
idx.load({prefix!r})
nq, k = {nq}, 10
bufs = [np.zeros((nq, 128), np.float32), np.zeros((nq, k), np.uint32), np.zeros((nq, k), np.float32)]
ptrs = [b.ctypes.data for b in bufs]
ptrs[{null}] = 0
try:
    idx.search_into(ptrs[0], nq, ptrs[1], ptrs[2], k=k, nprobe=4)
except RuntimeError as e:
    print("refused:", e)
"""


@pytest.mark.parametrize("nq", [1, 200, 4000])
@pytest.mark.parametrize("null", [0, 1, 2])
def test_null_buffer_is_refused(null, nq):
    prefix = fixture("d128")[2]
    r = subprocess.run([sys.executable, "-c", CODE.format(path=sys.path, prefix=prefix, nq=nq, null=null)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("refused:"), (r.returncode, r.stdout, r.stderr[-500:])
