"""Batches of tensor-core forests, whose levels are run one launch each by the
width the forests have together: against the oracle, bit-exact."""
import numpy as np
import pytest
import torch

import zeknox_b200 as zk
from oracle import oracle as O
from tests.helpers import HASHES, empty_dev, to_dev, to_np

pytestmark = pytest.mark.gpu

# (log2 leaves, leaf words, cap height): 2^11 to 2^13 nodes a level, subtrees of
# one, two and four leaves, copied leaves, one small forest beside the others
FORESTS = [(13, 9, 0), (13, 5, 13), (13, 8, 12), (13, 9, 11), (12, 3, 1), (14, 8, 3), (5, 9, 1), (13, 7, 2)]


@pytest.mark.parametrize("name", ["poseidon", "poseidon2", "monolith", "keccak"])
@pytest.mark.parametrize("times", [1, 2])  # as many forests as branches, and more
def test_forests_side_by_side(name, times):
    h = HASHES[name]
    jobs, bufs = [], []
    for k, (lg, ls, ch) in enumerate(FORESTS * times):
        leaves = O.field_data(1000 * k + lg, ls << lg)
        n_dig, n_cap = zk.merkle_sizes(1 << lg, ch)
        dev, dig, cap = to_dev(leaves), empty_dev(n_dig * 4), empty_dev(n_cap * 4)
        jobs.append(zk.merkle_job(dev, dig if n_dig else None, cap, 1 << lg, ls, ch, h))
        bufs.append((leaves, dev, dig, cap, n_dig))
    zk.merkle_batch(0, jobs)
    for (lg, ls, ch), (leaves, _, dig, cap, n_dig) in zip(FORESTS * times, bufs):
        d2, c2 = O.merkle(leaves, ls, ch, h)
        assert np.array_equal(to_np(cap).reshape(-1, 4), c2), (lg, ls, ch)
        assert np.array_equal(to_np(dig)[:4 * n_dig].reshape(-1, 4), d2), (lg, ls, ch)


@pytest.mark.parametrize("name", ["poseidon2", "poseidon"])
def test_commits_side_by_side(name):
    shapes = [(12, 1, 9, 0), (11, 2, 16, 4), (10, 3, 5, 13), (12, 2, 8, 2), (10, 1, 20, 3)]
    jobs, bufs = [], []
    for k, (lg, rate, cols, ch) in enumerate(shapes):
        c = O.field_data(50 + k, cols << lg)
        N = 1 << (lg + rate)
        n_dig, n_cap = zk.merkle_sizes(N, ch)
        dev, leaves, dig, cap = to_dev(c), empty_dev(N * cols), empty_dev(n_dig * 4), empty_dev(n_cap * 4)
        jobs.append(zk.commit_job(lg, rate, cols, ch, HASHES[name], dev, leaves, dig, cap))
        bufs.append((c, dev, leaves, dig, cap, n_dig))
    zk.commit_batch(0, jobs)
    torch.cuda.synchronize()
    for (lg, rate, cols, ch), (c, _, leaves, dig, cap, n_dig) in zip(shapes, bufs):
        rows = O.lde_rows(c, lg, rate, cols)
        d2, c2 = O.merkle(rows, cols, ch, HASHES[name])
        assert np.array_equal(to_np(leaves), rows)
        assert np.array_equal(to_np(cap).reshape(-1, 4), c2), (lg, rate, cols, ch)
        assert np.array_equal(to_np(dig)[:4 * n_dig].reshape(-1, 4), d2), (lg, rate, cols, ch)
