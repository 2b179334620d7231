"""A program's first transpose recorded into a CUDA graph, the library being in
use already: it needs nothing that a capture refuses, whatever form the shape
takes."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = """
import sys
sys.path.insert(0, %r)
import numpy as np
import torch
import zeknox_b200 as zk
from oracle import oracle as O
from tests.helpers import empty_dev, to_dev, to_np
lg, cols, offset = %d, %d, %d
a, b = (O.field_data(k, cols << lg) for k in (1, 2))
x, buf = to_dev(a), empty_dev((cols << lg) + offset)
out = buf[offset:]
zk.ntt_batch(0, to_dev(a[:16]), 4, 1)
torch.cuda.synchronize()
g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
with torch.cuda.graph(g, stream=s):
    zk.transpose_rev(0, out, x, lg, cols, stream=s.cuda_stream)
for data in (a, b):
    x.copy_(to_dev(data))
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(to_np(out), O.transpose_rev(data, lg, cols))
print("ok")
"""


# odd columns and an 8-byte aligned destination with 8-byte stores, the
# 16-byte form, and the register forms
@pytest.mark.parametrize("lg,cols,offset", [(18, 33, 0), (18, 7, 0), (18, 34, 1), (12, 40, 0), (5, 8, 0), (9, 5, 0)])
def test_first_transpose_in_a_capture(lg, cols, offset):
    r = subprocess.run([sys.executable, "-c", SCRIPT % (ROOT, lg, cols, offset)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["ok"], r.stderr[-2000:]
