"""The short form of the secular roots (ddc-svd_gb300/csrc/dc.cu, sec_root of
single SVDs) on problems of any magnitude: its FP32 phase has FP32's exponent
range, and where that does not hold a root the FP64 iteration takes over."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_roots_at_any_scale(lib, cuda, tmp_path):
    from ddcsvd import build as b
    exe, libdir = str(tmp_path / "secular_check"), os.path.dirname(b.LIB_PATH)
    subprocess.run([b._nvcc(), *b.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", b.CSRC, "-I", b.INCLUDE,
                    os.path.join(HERE, "c", "secular_check.cu"), "-o", exe, f"-L{libdir}", "-lddcsvd", "-Xlinker",
                    f"-rpath={libdir}"], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [tuple(float(x) for x in line.split()) for line in r.stdout.splitlines()]
    assert len(rows) == 15
    # both stop where f is below its rounding, eps (8 (1 + |psi| + |phi|) + |tau| f'): the
    # plain form's roots at other scales differ by some 35 units, and twice that is allowed
    plain = max(p for _, _, p in rows)
    assert plain <= 64.0, rows
    assert all(s <= 2.0 * plain for _, s, _ in rows), rows
