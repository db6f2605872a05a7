"""quot_rn (ddc-svd_gb300/csrc/fp64.cuh) against the division operator, bit for
bit: divisors next to powers of two, quotients next to the midpoint of two
doubles, the ends of its range and special values, random pairs.  The stages
that keep the plain formulas' bits rely on it."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_quotients_equal_the_operators(lib, cuda, tmp_path):
    from ddcsvd import build as b
    exe = str(tmp_path / "quotient_check")
    subprocess.run([b._nvcc(), *b.ARCH, "-O3", "-std=c++17", "-I", b.CSRC, os.path.join(HERE, "c", "quotient_check.cu"),
                    "-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = {n: (float(c), int(d)) for n, c, d in (line.split() for line in r.stdout.splitlines())}
    assert {n: d for n, (_, d) in rows.items() if d} == {}
    assert rows["seed_log2"][0] <= -19.9 and rows["midpoints_large_divisors"][0] == 400000 and "done" in rows
