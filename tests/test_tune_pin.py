"""A call reads one version of the tuning table from its first knob to its last
launch, whatever other threads set meanwhile (host check, no GPU)."""
import os
import subprocess

import zeknox_b200 as zk

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_pinned_table(tmp_path):
    table = tmp_path / "t.txt"
    table.write_text("ntt_split_logr 12 10\n")
    exe = tmp_path / "tune_pin"
    lib = os.path.dirname(zk.LIB_PATH)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "zeknox_b200", "csrc"), "-I",
                        os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "c", "tune_pin.cpp"), "-o", str(exe),
                        zk.LIB_PATH, "-Wl,-rpath," + lib, "-lpthread", "-ldl"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(exe), str(table)], capture_output=True, text=True, env=dict(os.environ, ZEKNOX_TUNE_FILE="none"))
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
