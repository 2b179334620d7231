"""The bulk-copy transpose with 8-byte stores (odd column counts, destinations
aligned to 8 bytes alone): tile edges at 32 and 64 columns and 64 positions."""
import numpy as np
import pytest
import torch

import zeknox_b200 as zk
from oracle import oracle as O
from tests.helpers import empty_dev, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lg,cols,offset", [(18, 1, 0), (18, 7, 0), (18, 33, 0), (18, 63, 0), (17, 65, 0), (16, 135, 0),
                                            (13, 1025, 0), (6, 131073, 0), (18, 34, 1), (17, 64, 1), (18, 2, 1)])
def test_transpose_rev_eight_byte_stores(lg, cols, offset):
    n = 1 << lg
    x = O.field_data(7 * cols + lg, cols * n)
    out = empty_dev(cols * n + offset + 1)
    out.fill_(-1)
    zk.transpose_rev(0, out[offset:], to_dev(x), lg, cols)
    torch.cuda.synchronize()
    got = to_np(out)
    assert np.array_equal(got[offset:offset + cols * n], O.transpose_rev(x, lg, cols))
    assert got[-1] == np.uint64(2**64 - 1) and (offset == 0 or got[0] == np.uint64(2**64 - 1))
