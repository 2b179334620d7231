"""Poseidon-BN128 forests with five threads a state and with one, against the
oracle; bit-exact."""
import os

import numpy as np
import pytest

import zeknox_b200 as zk
from oracle import oracle as O
from tests.test_gpu_adversarial import CANON, _pick
from tests.test_gpu_merkle import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coop_leaves", [0, 1 << 40])
def test_forests_on_both_forms(coop_leaves):
    """Leaf counts around a warp's 6 groups, a block's 12 and a fold's 64; every
    remainder of the last chunk; corner values; caps == leaves."""
    shapes = [(1, 8, 0), (2, 5, 0), (4, 9, 2), (8, 20, 1), (16, 12, 4), (64, 16, 2), (128, 7, 0), (256, 8, 3)]
    shapes += [(8, 8 + r, 1) for r in range(1, 9)]
    zk.tune_set("coop_leaves.2", coop_leaves)
    try:
        for nl, ls, ch in shapes:
            leaves = O.field_data(nl * 1000 + ls, nl * ls) if ls != 8 else _pick(CANON, nl * ls, nl)
            dig, cap = run_gpu(leaves, nl, ls, ch, zk.HASH_POSEIDON_BN128)
            d2, c2 = O.merkle(leaves, ls, ch, zk.HASH_POSEIDON_BN128)
            assert np.array_equal(cap, c2), (nl, ls, ch)
            assert np.array_equal(dig, d2), (nl, ls, ch)
    finally:
        zk.tune_clear()
        if os.path.exists(zk.TUNE_TABLE):
            zk.tune_load(zk.TUNE_TABLE)
