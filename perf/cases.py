"""The work that programs have this library do, as cases that can be timed and compared.

A case is one call (or one batch call) of the public Python API, which is the C ABI under the same
names: fused commits, Merkle forests, transforms, the leaf transpose and a graph-captured batch.
Sizes are those of the benchmark, the tests and the reference comparison, or lie between them.
"""
import random

import numpy as np
import torch

import zeknox_b200 as zk

HASHES = {"poseidon": zk.HASH_POSEIDON, "keccak": zk.HASH_KECCAK, "poseidon_bn128": zk.HASH_POSEIDON_BN128,
          "poseidon2": zk.HASH_POSEIDON2, "monolith": zk.HASH_MONOLITH}
# 64 x 64-bit field products of one permutation (S-boxes and dense layers); Monolith's and Keccak-f's
# small-constant and bit operations, and a 256-bit product of Poseidon-BN128, counted as as many products of that size
PRODUCTS = {"poseidon": 1077, "keccak": 200, "poseidon_bn128": 16800, "poseidon2": 736, "monolith": 300}


def listed():
    return [
        # the benchmark's commit: 256 columns of 2^15 coefficients, blowup 8, resident on the GPU
        {"name": "commit_poseidon2", "kind": "commit", "lg": 15, "rate": 3, "cols": 256, "cap": 4, "hash": "poseidon2",
         "values": False, "host": False},
        # a prover's wire commit: 135 columns given as evaluations in pinned host memory, the default hash
        {"name": "commit_wires_host", "kind": "commit", "lg": 14, "rate": 3, "cols": 135, "cap": 4, "hash": "poseidon",
         "values": True, "host": True},
        # a small request of a proving service, where launches and narrow tree levels count
        {"name": "commit_small", "kind": "commit", "lg": 10, "rate": 3, "cols": 20, "cap": 4, "hash": "poseidon",
         "values": False, "host": False},
        # the reference's own Merkle benchmark: 8192 leaves x 84, one root
        {"name": "forest_poseidon", "kind": "forest", "lg": 13, "cols": 84, "cap": 0, "hash": "poseidon"},
        # the alternative hashes at scale, on leaf rows of 135 elements
        {"name": "forest_monolith", "kind": "forest", "lg": 20, "cols": 135, "cap": 4, "hash": "monolith"},
        {"name": "forest_keccak", "kind": "forest", "lg": 20, "cols": 135, "cap": 4, "hash": "keccak"},
        {"name": "forest_bn128", "kind": "forest", "lg": 14, "cols": 135, "cap": 2, "hash": "poseidon_bn128"},
        # a handful of short columns: the smallest transform call
        {"name": "ntt_small", "kind": "ntt", "lg": 10, "cols": 16, "inverse": False, "coset": False},
        # coset evaluations back to coefficients, a whole trace
        {"name": "intt_coset", "kind": "ntt", "lg": 18, "cols": 135, "inverse": True, "coset": True},
        # the extension alone, columns in and natural-order columns out
        {"name": "lde_columns", "kind": "lde", "lg": 16, "rate": 2, "cols": 84, "inverse": False},
        # columns to bit-reversed leaf rows, an odd number of columns
        {"name": "transpose_odd", "kind": "transpose", "lg": 18, "cols": 135},
        # commits of uneven sizes submitted together (one captured graph)
        {"name": "batch_uneven", "kind": "batch", "jobs": 12, "lg_min": 10, "lg_max": 15, "cols_max": 200,
         "hash": "poseidon", "mix": 7},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["commit", "commit", "forest", "forest", "ntt", "lde", "transpose", "batch"])
    if kind == "commit":
        name = rng.choice(["poseidon", "poseidon2", "poseidon", "poseidon2", "monolith", "keccak"])
        lg, rate = rng.randint(10, 15), rng.randint(1, 3)
        values = rng.random() < 0.3
        return {"kind": kind, "lg": lg, "rate": rate, "cols": _log_uniform(rng, 8, 240), "cap": rng.randint(0, 6),
                "hash": name, "values": values, "host": rng.random() < 0.3}
    if kind == "forest":
        name = rng.choice(["poseidon", "poseidon2", "monolith", "keccak", "poseidon_bn128"])
        top = {"poseidon": 19, "poseidon2": 19, "monolith": 20, "keccak": 20, "poseidon_bn128": 13}[name]
        return {"kind": kind, "lg": rng.randint(8, top), "cols": _log_uniform(rng, 5, 135), "cap": rng.randint(0, 6),
                "hash": name}
    lg = rng.randint(8, 20)
    most = max(1, min(4096, (1 << 25) >> lg))
    if kind == "ntt":
        return {"kind": kind, "lg": lg, "cols": _log_uniform(rng, 1, most), "inverse": rng.random() < 0.5,
                "coset": rng.random() < 0.5}
    if kind == "lde":
        lg = min(lg, 17)
        rate = rng.randint(1, 3)
        return {"kind": kind, "lg": lg, "rate": rate, "cols": _log_uniform(rng, 1, max(1, min(400, (1 << 25) >> (lg + rate)))),
                "inverse": rng.random() < 0.2}
    if kind == "transpose":
        return {"kind": kind, "lg": lg, "cols": _log_uniform(rng, 1, min(400, most))}
    return {"kind": kind, "jobs": rng.randint(3, 12), "lg_min": 10, "lg_max": rng.randint(12, 14),
            "cols_max": _log_uniform(rng, 16, 200), "hash": rng.choice(["poseidon", "poseidon2"]),
            "mix": rng.randrange(1 << 20)}


# ------------------------------------------------------------------ inputs

def _jobs(case):
    r = random.Random(case["mix"])
    return [{"lg": r.randint(case["lg_min"], case["lg_max"]), "rate": r.randint(1, 3),
             "cols": r.randint(8, case["cols_max"]), "cap": 4, "hash": case["hash"]} for _ in range(case["jobs"])]


def _field(n, gen):
    """n words uniform in [0, p), as int64 bit patterns (words of [p, 2^64) folded by -p)."""
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), dtype=torch.int64, device="cuda", generator=gen)
    eps = (1 << 32) - 1
    return torch.where((x < 0) & (x >= -eps), x + eps, x)


def _forest_buffers(n_leaves, cap):
    n_dig, n_caps = zk.merkle_sizes(n_leaves, min(cap, n_leaves.bit_length() - 1))
    return (torch.zeros(max(n_dig, 1) * 4, dtype=torch.int64, device="cuda"),
            torch.zeros(n_caps * 4, dtype=torch.int64, device="cuda"))


def _commit_state(case, gen):
    lg, rate, cols = case["lg"], case["rate"], case["cols"]
    inp = _field(cols << lg, gen)
    if case.get("host"):
        inp = inp.cpu().pin_memory()
    leaves = torch.empty(cols << (lg + rate), dtype=torch.int64, device="cuda")
    digests, caps = _forest_buffers(1 << (lg + rate), case["cap"])
    job = zk.commit_job(lg, rate, cols, case["cap"], HASHES[case["hash"]], inp, leaves, digests, caps,
                        input_is_values=case.get("values", False))
    return {"job": job, "inp": inp, "out": [leaves, digests, caps]}


def prepare(case, seed):
    zk.load()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "commit":
        state = _commit_state(case, gen)
    elif kind == "batch":
        state = {"jobs": [_commit_state(j, gen) for j in _jobs(case)]}
    elif kind == "forest":
        state = {"leaves": _field(case["cols"] << case["lg"], gen)}
        state["digests"], state["caps"] = _forest_buffers(1 << case["lg"], case["cap"])
    else:
        state = {"x": _field(case["cols"] << case["lg"], gen)}
        if kind != "ntt":
            state["out"] = torch.empty(case["cols"] << (case["lg"] + case.get("rate", 0)), dtype=torch.int64, device="cuda")
    state["case"] = case
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "commit":
        zk.commit(0, state["job"])
        return state["out"]
    if kind == "batch":
        zk.commit_batch(0, [j["job"] for j in state["jobs"]])
        return [j["out"] for j in state["jobs"]]
    if kind == "forest":
        zk.fill_digests_buf_linear_gpu(state["digests"], state["caps"], state["leaves"], 1 << case["lg"], case["cols"],
                                       case["cap"], HASHES[case["hash"]])
        return [state["digests"], state["caps"]]
    if kind == "ntt":
        return zk.ntt_batch(0, state["x"], case["lg"], case["cols"], with_coset=case["coset"], inverse=case["inverse"])
    if kind == "lde":
        return zk.lde_batch(0, state["out"], state["x"], case["lg"], case["cols"], case["rate"], inverse=case["inverse"])
    return zk.transpose_rev_batch(0, state["out"], state["x"], case["lg"], case["cols"])


# -------------------------------------------------------------------- work

def _forest_work(lg, cols, cap, name):
    leaves = 1 << lg
    rate = 17 if name == "keccak" else 8
    per_leaf = 0 if cols <= 4 else (cols // 17 + 1 if name == "keccak" else -(-cols // rate))
    nodes = leaves - (1 << cap)
    return {"bytes": 8.0 * leaves * cols + 32.0 * (2 * leaves - (1 << cap)),
            "flops": 2.0 * PRODUCTS[name] * (leaves * per_leaf + nodes)}


def _transform_work(lg, columns, in_words, out_words):
    return {"bytes": 8.0 * (in_words + out_words), "flops": 2.0 * columns * (lg << lg) / 2}


def _commit_work(case):
    lg, rate, cols = case["lg"], case["rate"], case["cols"]
    tree = _forest_work(lg + rate, cols, case["cap"], case["hash"])
    lde = _transform_work(lg, cols * ((1 << rate) + bool(case.get("values"))), cols << lg, 0)
    # the leaves are an output, written once and hashed from where they are: _forest_work counts them once
    return {"bytes": tree["bytes"] + lde["bytes"], "flops": tree["flops"] + lde["flops"]}


def work(case):
    kind = case["kind"]
    if kind == "commit":
        return _commit_work(case)
    if kind == "batch":
        parts = [_commit_work(j) for j in _jobs(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "forest":
        return _forest_work(case["lg"], case["cols"], case["cap"], case["hash"])
    words = case["cols"] << case["lg"]
    if kind == "ntt":
        return _transform_work(case["lg"], case["cols"], words, words)
    if kind == "lde":
        return _transform_work(case["lg"], case["cols"] << case["rate"], words, words << case["rate"])
    return {"bytes": 16.0 * words, "flops": 0.0}


def tolerance(case):
    """Field elements and digest bytes: whole numbers, the same in every correct implementation."""
    return "exact"


# -------------------------------------- the transforms in plain numpy (64-bit words)

_P, _EPS, _M = np.uint64(0xFFFFFFFF00000001), np.uint64(0xFFFFFFFF), np.uint64(0xFFFFFFFF)
_ROOT_2_32, _SHIFT, _PI = 0x185629DCDA58878C, 7, 0xFFFFFFFF00000001
_32 = np.uint64(32)


def _mul(a, b):
    a0, a1, b0, b1 = a & _M, a >> _32, b & _M, b >> _32
    low = a0 * b0
    mid = a0 * b1 + (low >> _32)
    mid2 = a1 * b0 + (mid & _M)
    hi = a1 * b1 + (mid >> _32) + (mid2 >> _32)
    lo = (mid2 << _32) | (low & _M)
    t = lo - (hi >> _32)
    t = t - np.where(lo < (hi >> _32), _EPS, np.uint64(0))
    e = (hi & _M) * _EPS
    s = t + e
    s = s + np.where(s < e, _EPS, np.uint64(0))
    return np.where(s >= _P, s - _P, s)


def _add(a, b):
    s = a + b
    return np.where((s < a) | (s >= _P), s - _P, s)


def _sub(a, b):
    return np.where(a < b, a - b + _P, a - b)


def _powers(w, n):
    t = np.ones(1, dtype=np.uint64)
    while t.size < n:
        t = np.concatenate([t, _mul(t, np.uint64(pow(w, t.size, _PI)))])
    return t[:n]


def _dft(x, lg, inverse):
    """Natural-order transform of each row of x, by decimation in time."""
    w = pow(_ROOT_2_32, 1 << (32 - lg), _PI)
    if inverse:
        w = pow(w, _PI - 2, _PI)
    order = np.zeros(1 << lg, dtype=np.int64)
    for b in range(lg):
        order = (order << 1) | ((np.arange(1 << lg) >> b) & 1)
    x = x[:, order]
    for s in range(1, lg + 1):
        half = 1 << (s - 1)
        tw = _powers(pow(w, 1 << (lg - s), _PI), half)
        y = x.reshape(x.shape[0], -1, 2, half)
        u, v = y[:, :, 0, :], _mul(y[:, :, 1, :], tw)
        x = np.stack([_add(u, v), _sub(u, v)], axis=2).reshape(x.shape[0], -1)
    return x


def _reversed_rows(cols, lg):
    order = np.zeros(1 << lg, dtype=np.int64)
    for b in range(lg):
        order = (order << 1) | ((np.arange(1 << lg) >> b) & 1)
    return cols.T[order].reshape(-1)


def _out(a):
    return np.ascontiguousarray(a).reshape(-1).view(np.int64)


def exact(case, seed):
    """Transforms, leaf rows and transposes computed again with numpy's 64-bit words; None in the place of digests and
    caps, and for the cases that would take too long (and for batches and forests, whose outputs are digests)."""
    kind = case["kind"]
    if kind in ("forest", "batch"):
        return None
    lg, rate, cols = case["lg"], case.get("rate", 0), case["cols"]
    if kind != "transpose" and (cols << (lg + rate)) > (1 << 22):
        return None
    state = prepare(case, seed)
    x = (state["inp"] if kind == "commit" else state["x"]).cpu().numpy().view(np.uint64).reshape(cols, 1 << lg)
    if kind == "transpose":
        return _out(_reversed_rows(x, lg))
    n_inv = lambda k: np.uint64(pow(1 << k, _PI - 2, _PI))  # noqa: E731
    if kind == "ntt":
        shift = _powers(_SHIFT, 1 << lg) if case["coset"] else np.ones(1 << lg, dtype=np.uint64)
        if case["inverse"]:
            # the reference multiplies by the forward powers of the shift here, before 1/n
            return _out(_mul(_mul(_dft(x, lg, True), shift), n_inv(lg)))
        return _out(_dft(_mul(x, shift), lg, False))
    if kind == "commit" and case["values"]:
        x = _mul(_dft(x, lg, True), n_inv(lg))
    big = lg + rate
    wide = np.zeros((cols, 1 << big), dtype=np.uint64)
    wide[:, :1 << lg] = x
    if case.get("inverse"):
        return _out(_mul(_mul(_dft(wide, big, True), _powers(_SHIFT, 1 << big)), n_inv(big)))
    wide[:, :1 << lg] = _mul(x, _powers(_SHIFT, 1 << lg))
    y = _dft(wide, big, False)
    return _out(y) if kind == "lde" else [_out(_reversed_rows(y, big)), None, None]
