"""Column transforms, written in natural order by their last pass (of up to 2^12
points: their only one), against the oracle; bit-exact."""
import os

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


@pytest.fixture
def table_after():
    zk.tune_clear()
    yield
    zk.tune_clear()
    if os.path.exists(zk.TUNE_TABLE):
        zk.tune_load(zk.TUNE_TABLE)


@pytest.mark.parametrize("split", [7, 8, 9, 10])
@pytest.mark.parametrize("lg,batches", [(8, 5), (11, 3), (14, 3), (19, 1), (20, 1)])
def test_ntt_split(split, lg, batches, table_after):
    """Every split into passes the tuning table may ask for."""
    zk.tune_set("ntt_split_logr", split)
    for inverse, coset in [(False, True), (True, True)]:
        x = O.field_data(lg * 13 + batches, batches << lg)
        t = to_dev(x)
        zk.ntt_batch(0, t, lg, batches, with_coset=coset, inverse=inverse)
        assert np.array_equal(to_np(t), O.batched_ntt(x, lg, batches, inverse=inverse, with_coset=coset))


@pytest.mark.parametrize("split,lg,rate,cols", [(0, 17, 5, 1), (0, 18, 4, 2), (9, 9, 4, 3), (9, 17, 4, 1), (10, 10, 3, 5),
                                                (10, 11, 5, 3), (10, 20, 3, 1), (7, 12, 6, 2), (8, 15, 1, 3)])
def test_lde_split(split, lg, rate, cols, table_after):
    """Extensions of several passes whose last tile holds fewer groups than a
    column has cosets, as many, and more."""
    zk.tune_set("ntt_split_logr", split)
    x = O.field_data(lg * 3 + rate, cols << lg)
    out = empty_dev(cols << (lg + rate))
    zk.lde_batch(0, out, to_dev(x), lg, cols, rate)
    assert np.array_equal(to_np(out), O.batched_lde(x, lg, rate, cols))
