"""Column transforms of up to 2^12 points, written in natural order by the one
pass itself, against the oracle; bit-exact."""
import numpy as np
import pytest

import zeknox_b200 as zk
from oracle import oracle as O
from tests.helpers import empty_dev, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lg", [1, 4, 5, 8, 11, 12, 13])
@pytest.mark.parametrize("batches", [1, 257])
@pytest.mark.parametrize("inverse,coset", [(False, False), (False, True), (True, False), (True, True)])
def test_ntt(lg, batches, inverse, coset):
    x = O.field_data(lg * 31 + batches, batches << lg)
    t = to_dev(x)
    zk.ntt_batch(0, t, lg, batches, with_coset=coset, inverse=inverse)
    assert np.array_equal(to_np(t), O.batched_ntt(x, lg, batches, inverse=inverse, with_coset=coset))


@pytest.mark.parametrize("lg,rate,cols,inverse", [(1, 1, 3, False), (4, 3, 17, False), (9, 2, 5, False), (12, 1, 3, False),
                                                  (12, 3, 2, False), (13, 1, 2, False), (9, 3, 4, True), (10, 3, 2, True)])
@pytest.mark.parametrize("shift", [None, 0, 5])
def test_lde(lg, rate, cols, inverse, shift):
    """Output apart from the input (shift None), or over it, `shift` words on."""
    n, N = 1 << lg, 1 << (lg + rate)
    x = O.field_data(lg * 7 + rate + cols, cols * n)
    want = O.batched_lde(x, lg, rate, cols, inverse=inverse)
    if shift is None:
        inp, out = to_dev(x), empty_dev(cols * N)
    else:
        buf = empty_dev(cols * N + shift)
        inp, out = buf[:cols * n], buf[shift:]
        inp.copy_(to_dev(x))
    zk.lde_batch(0, out, inp, lg, cols, rate, inverse=inverse)
    assert np.array_equal(to_np(out), want)
