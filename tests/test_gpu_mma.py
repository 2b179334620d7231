"""The tensor-core permutations (hash_mma.cuh) in both forms -- 32 and 8 states
per warp -- and the forests built with them, against the oracle; bit-exact."""
import ctypes

import numpy as np
import pytest

import zeknox_b200 as zk
from oracle import oracle as O
from tests.helpers import HASHES, to_dev, to_np
from tests.test_gpu_adversarial import CANON, P, _corner_states, _pick
from tests.test_gpu_merkle import run_gpu

pytestmark = pytest.mark.gpu

WIDE, NARROW = 2, 3  # zeknox_permute's `cooperative`: 32 or 8 states per warp


@pytest.mark.parametrize("form", [WIDE, NARROW])
@pytest.mark.parametrize("name", ["poseidon", "poseidon2"])
def test_permutation_on_corner_states(name, form):
    h = HASHES[name]
    states = _corner_states(12, 930 + h, canonical=False)
    canon = np.where(states >= np.uint64(P), states - np.uint64(P), states)
    want = np.stack([O.permute(h, c) for c in canon])
    for n in (1, 7, 8, 9, 31, 32, 33, 129, len(states)):  # partial quads, tiles, warps and blocks
        t = to_dev(states[:n].reshape(-1))
        zk._check(zk.load().zeknox_permute(0, ctypes.c_void_p(t.data_ptr()), n, h, form, None))
        got = to_np(t).reshape(-1, 12)
        bad = np.flatnonzero((got != want[:n]).any(axis=1))
        assert not len(bad), (name, form, n, bad[:4])


@pytest.mark.parametrize("states_per_warp", [8, 16, 32])
@pytest.mark.parametrize("name", ["poseidon", "poseidon2", "monolith"])
def test_forests_on_every_form(name, states_per_warp):
    """Leaf counts around a warp's 8, 16 and 32 rows and a block's 128; every
    remainder of the last chunk of a row (its lanes 1..7 kept from the chunk
    before); caps == leaves and two-leaf subtrees."""
    h = HASHES[name]
    shapes = [(1, 8, 0), (1024, 8, 4), (2, 5, 0), (8, 9, 3), (16, 20, 1), (32, 31, 5), (64, 16, 5), (128, 7, 2), (256, 135, 0)]
    shapes += [(64, 8 + r, 3) for r in range(1, 9)]
    zk.tune_set("wide_level_nodes.%d" % h, 16)
    try:
        for nl, ls, ch in shapes:
            # up to coop_leaves leaves 8 per warp, up to four times as many 16
            zk.tune_set("coop_leaves.%d" % h, {8: nl, 16: (nl + 3) // 4, 32: 0}[states_per_warp])
            leaves = O.field_data(nl * 1000 + ls, nl * ls)
            if ls == 8:  # corner values: one permutation per leaf
                leaves = _pick(CANON, nl * ls, nl)
            dig, cap = run_gpu(leaves, nl, ls, ch, h)
            d2, c2 = O.merkle(leaves, ls, ch, h)
            assert np.array_equal(cap, c2), (nl, ls, ch)
            assert np.array_equal(dig, d2), (nl, ls, ch)
    finally:
        zk.tune_clear()
        if zk.os.path.exists(zk.TUNE_TABLE):
            zk.tune_load(zk.TUNE_TABLE)


@pytest.mark.parametrize("threads", [32, 64, 128])
@pytest.mark.parametrize("states_per_warp", [8, 16, 32])
@pytest.mark.parametrize("name", ["poseidon", "poseidon2", "monolith"])
def test_forests_with_every_block_size(name, states_per_warp, threads):
    """Every number of leaves per warp in blocks of one, two and four warps (each
    its own register budget and shared-memory slices): a block not full, one
    full, several."""
    h = HASHES[name]
    zk.tune_set("leaf_threads.%d" % h, threads)
    try:
        for nl, ls, ch in [(2, 9, 0), (32, 12, 1), (128, 20, 2), (512, 17, 3), (2048, 8, 0)]:
            zk.tune_set("coop_leaves.%d" % h, {8: nl, 16: (nl + 3) // 4, 32: 0}[states_per_warp])
            leaves = O.field_data(nl * 77 + ls, nl * ls) if ls != 8 else _pick(CANON, nl * ls, nl + threads)
            dig, cap = run_gpu(leaves, nl, ls, ch, h)
            d2, c2 = O.merkle(leaves, ls, ch, h)
            assert np.array_equal(cap, c2), (nl, ls, ch)
            assert np.array_equal(dig, d2), (nl, ls, ch)
    finally:
        zk.tune_clear()
        if zk.os.path.exists(zk.TUNE_TABLE):
            zk.tune_load(zk.TUNE_TABLE)


@pytest.mark.parametrize("name,lg", [("poseidon", 17), ("poseidon2", 17), ("monolith", 17), ("monolith", 18)])
def test_large_forests_as_built_in(name, lg):
    """The forms chosen above 2^16 leaves: 32 per warp in blocks of two warps,
    Monolith's 16 and 32 per warp in blocks of four."""
    h, nl, ls = HASHES[name], 1 << lg, 9
    zk.tune_clear()
    try:
        leaves = O.field_data(lg + h, nl * ls)
        dig, cap = run_gpu(leaves, nl, ls, 4, h)
    finally:
        if zk.os.path.exists(zk.TUNE_TABLE):
            zk.tune_load(zk.TUNE_TABLE)
    d2, c2 = O.merkle(leaves, ls, 4, h)
    assert np.array_equal(cap, c2)
    assert np.array_equal(dig, d2)
