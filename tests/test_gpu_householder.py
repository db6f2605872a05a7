"""The cluster tail's short form of a reflector and its compensated sums
(ddc-svd_gb300/csrc/common.cuh, householder_fast, ff_acc) against FP64."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_reflector_and_sums(lib, cuda, tmp_path):
    from ddcsvd import build as b
    exe = str(tmp_path / "householder_check")
    subprocess.run([b._nvcc(), *b.ARCH, "-O3", "-std=c++17", "-I", b.CSRC, os.path.join(HERE, "c", "householder_check.cu"),
                    "-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    v = {n: float(x) for n, x in (line.split() for line in r.stdout.splitlines())}
    # one rounding of alpha; of tau and of the reciprocal in it; of the denominator, of
    # alpha in it and of the quotient
    assert v["alpha"] <= 1.01 and v["tau"] <= 2.01 and v["scale"] <= 3.01, v
    # a compensated sum of up to 768 squares: its tails' roundings
    assert v["sum"] <= 4.0 and v["zero"] == 0.0, v
