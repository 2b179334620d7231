"""The tables of the tensor-core permutations (zeknox_b200/csrc/mma_tables.h):
the permutations computed from them on the host, every byte-column sum as the
tensor core takes it and the sums recombined in 32-bit words, equal the plain
ones on corner and random states; no sum exceeds the generator's worst one, and
the limit it holds that to is the recombination's."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_permutations_from_the_tables(tmp_path):
    exe = tmp_path / "mma_perm"
    r = subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(ROOT, "tests", "c", "mma_perm.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.split() == ["108", "states"]
