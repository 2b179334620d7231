"""Tuning table (zeknox_tune_*): host-side behaviour, no GPU needed.

The knobs only choose launch shapes; that results do not depend on them is
checked on the GPU in test_gpu_tune.py.
"""
import os
import subprocess
import sys

import pytest

import zeknox_b200 as zk
from zeknox_b200 import autotune

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KNOBS = {"leaf_threads": {32, 64, 128, 256}, "lde_chunk_mib": None, "lde_last_logr": set(range(1, 9)),
         "wide_level_nodes": None, "coop_leaves": None, "lde_host_chunk_mib": None,
         "ntt_split_logr": {0, 7, 8, 9, 10}, "transpose_bulk": set(range(10))}


@pytest.fixture
def clean_table():
    zk.load()
    zk.tune_clear()
    yield
    zk.tune_clear()
    if os.path.exists(zk.TUNE_TABLE):
        zk.tune_load(zk.TUNE_TABLE)


def test_set_get_and_size_fallback(clean_table):
    assert zk.tune_get("lde_chunk_mib", 18, 64) == 64
    zk.tune_set("lde_chunk_mib", 32)  # every size
    assert zk.tune_get("lde_chunk_mib", 18, 64) == 32
    zk.tune_set("lde_chunk_mib", 96, lg=18)  # this size wins over the size-free entry
    assert zk.tune_get("lde_chunk_mib", 18, 64) == 96
    assert zk.tune_get("lde_chunk_mib", 17, 64) == 32
    assert zk.tune_get("lde_chunk_mib", None, 64) == 32
    zk.tune_clear()
    assert zk.tune_get("lde_chunk_mib", 18, 64) == 64


def test_load_table_with_comments_and_blank_lines(clean_table, tmp_path):
    p = tmp_path / "t.txt"
    p.write_text("# header\n\nleaf_threads.3 18 128   # per size\n  lde_last_logr * 8\n\t\nwide_level_nodes.0 20 8192\n")
    zk.tune_load(p)
    assert zk.tune_get("leaf_threads.3", 18, 256) == 128
    assert zk.tune_get("leaf_threads.3", 17, 256) == 256
    assert zk.tune_get("lde_last_logr", 15, 9) == 8
    assert zk.tune_get("wide_level_nodes.0", 20, 1 << 15) == 8192


@pytest.mark.parametrize("bad", ["lde_chunk_mib 18\n", "lde_chunk_mib x 32\n", "lde_chunk_mib 18 32 7\n",
                                 "lde_chunk_mib 18 -\n", "lde_chunk_mib 999 32\n"])
def test_malformed_table_changes_nothing(clean_table, tmp_path, bad):
    p = tmp_path / "t.txt"
    p.write_text("leaf_threads.3 18 64\n" + bad)
    with pytest.raises(zk.ZeknoxError) as e:
        zk.tune_load(p)
    assert ":2:" in str(e.value)
    assert zk.tune_get("leaf_threads.3", 18, 256) == 256  # the good first line was not applied


def test_missing_table_is_an_error(clean_table, tmp_path):
    with pytest.raises(zk.ZeknoxError):
        zk.tune_load(tmp_path / "absent.txt")


def test_env_table_read_by_the_c_library(tmp_path):
    # a C-ABI consumer (no Python) gets the table through ZEKNOX_TUNE_FILE
    p = tmp_path / "t.txt"
    p.write_text("lde_chunk_mib * 48\n")
    code = ("import ctypes; L = ctypes.CDLL(%r); L.zeknox_tune_get.restype = ctypes.c_uint64;"
            "L.zeknox_tune_get.argtypes = [ctypes.c_char_p, ctypes.c_uint32, ctypes.c_uint64];"
            "print(L.zeknox_tune_get(b'lde_chunk_mib', 18, 64))" % zk.LIB_PATH)
    env = dict(os.environ, ZEKNOX_TUNE_FILE=str(p))
    out = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, check=True)
    assert out.stdout.strip() == "48"
    env["ZEKNOX_TUNE_FILE"] = "none"
    out = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, check=True)
    assert out.stdout.strip() == "64"


def test_committed_table_is_well_formed():
    if not os.path.exists(zk.TUNE_TABLE):
        pytest.skip("no tuning table committed")
    for ln, line in enumerate(open(zk.TUNE_TABLE), 1):
        body = line.split("#", 1)[0].split()
        if not body:
            continue
        name, lg, value = body
        base = name.split(".")[0]
        assert base in KNOBS, (ln, name)
        if "." in name:
            assert int(name.split(".")[1]) in autotune.HASH_NAMES, (ln, name)
        assert lg == "*" or 0 <= int(lg) <= 32, (ln, lg)
        allowed = KNOBS[base]
        assert allowed is None or int(value) in allowed, (ln, value)
        assert int(value) > 0 or (allowed is not None and 0 in allowed), (ln, value)


def test_autotune_partial_run_keeps_other_knobs(tmp_path):
    """A run of some searches only (--only) keeps the other knobs' lines."""
    p = tmp_path / "t.txt"
    p.write_text("# header\nleaf_threads.3 18 128   # ms\nntt_split_logr 20 9 # ms\n"
                 "transpose_bulk 18 3\nlde_last_logr 13 8\n")
    kept = autotune.kept_table_lines(str(p), {"ntt_split_logr", "transpose_bulk"})
    assert [k.split()[0] for k in kept] == ["leaf_threads.3", "lde_last_logr"]
    assert autotune.kept_table_lines(str(tmp_path / "missing.txt"), {"lde_last_logr"}) == []


def test_autotune_candidates_include_the_defaults():
    for knob, dflt in autotune.DEFAULTS.items():
        assert autotune.CANDIDATES[knob][0] == dflt
        assert all(v in KNOBS[knob] for v in autotune.CANDIDATES[knob]) if KNOBS[knob] else True
    for lg, cols in autotune.lde_shapes(False):
        assert cols >= 16 and (cols << (lg + autotune.RATE)) <= 1 << 27


@pytest.mark.parametrize("quick", [True, False])
def test_autotune_shapes(quick):
    for shapes in (autotune.lde_shapes, autotune.ntt_shapes, autotune.transpose_shapes):
        assert all(lg >= 1 and cols >= 1 for lg, cols in shapes(quick))
    for h, lg, leaf in autotune.merkle_shapes(quick):
        threads = autotune.leaf_threads(h, lg)
        assert h in autotune.HASH_NAMES and leaf > 4 and set(threads) <= KNOBS["leaf_threads"]
        assert len(set(threads)) == len(threads)


@pytest.mark.parametrize("argv", [[], ["--quick"], ["--only", "merkle"]])
def test_autotune_run_writes_its_table(clean_table, tmp_path, monkeypatch, capsys, argv):
    """A whole run with the GPU's part faked: every search at every shape, the
    table, and the closing count."""
    import torch

    class FakeTimer:
        def __init__(self, *a):
            pass

        def on(self, stream):
            return self

        def __call__(self, fn):  # one candidate of leaf_threads is clearly faster, the rest are even
            return 0.5 if zk.tune_get("leaf_threads.3", 18) == 128 else 1.0

    def merkle(z, t, timer, h, lg, leaf, margin, log):
        threads = autotune.leaf_threads(h, lg)
        args = (lambda: None, lambda k, v: None, margin, log)
        autotune.search(z, timer, "leaf_threads.%d" % h, lg, threads, threads[0], *args)
        if (h, lg) == (3, 18):
            z.tune_set("leaf_threads.3", threads[0], lg=18)  # the other searches at even times
        for knob in ("wide_level_nodes", "coop_leaves"):
            autotune.search(z, timer, "%s.%d" % (knob, h), lg, autotune.CANDIDATES[knob], autotune.DEFAULTS[knob], *args)

    def other(*knobs):
        def tune(z, t, timer, *a):
            lg, margin, log = a[-4], a[-2], a[-1]
            for k in knobs:
                autotune.search(z, timer, k, lg, autotune.CANDIDATES[k], autotune.DEFAULTS[k], lambda: None,
                                lambda *_: None, margin, log)
        return tune

    monkeypatch.setenv("ZEKNOX_TUNE_FILE", "none")
    for name, value in {"is_available": lambda: True, "set_device": lambda d: None, "Stream": lambda: None,
                        "default_stream": lambda: None, "empty_cache": lambda: None,
                        "get_device_name": lambda d: "a GPU"}.items():
        monkeypatch.setattr(torch.cuda, name, value)
    monkeypatch.setattr(autotune, "Timer", FakeTimer)
    monkeypatch.setattr(autotune, "tune_merkle", merkle)
    monkeypatch.setattr(autotune, "tune_lde", other("lde_last_logr", "lde_chunk_mib"))
    monkeypatch.setattr(autotune, "tune_ntt", other("ntt_split_logr"))
    monkeypatch.setattr(autotune, "tune_transpose", other("transpose_bulk"))
    out = tmp_path / "t.txt"
    autotune.main(argv + ["--out", str(out)])
    assert capsys.readouterr().out.rstrip().endswith("1 differ from the built-in defaults")
    zk.tune_clear()
    zk.tune_load(out)  # what it wrote is a table the library reads
    assert zk.tune_get("leaf_threads.3", 18) == 128
    monkeypatch.setattr(zk, "TUNE_TABLE", str(out))
    test_committed_table_is_well_formed()
