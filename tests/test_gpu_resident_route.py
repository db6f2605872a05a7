"""Square and nearly square matrices just beyond the cluster tail's 512 columns
go from the grid-resident columns to the tail without a panel: the reset and
scan kernels, two launches for the columns, and the scaling back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(513, 513), (514, 513), (545, 544), (600, 600), (632, 632), (700, 560), (760, 520)])
def test_no_panel_beyond_the_tail(lib, cuda, m, n):
    A = np.random.default_rng(m).standard_normal((m, n)).astype(np.float32)
    before = lib.launch_count()
    _, d, e, _, _ = lib.bidiag_device(cuda.from_numpy(A).cuda(), mode="tf32x6")
    # status, scan, scaling, columns, tail, scaling back (a panel adds four and more)
    assert lib.launch_count() - before <= 6
    B = np.diag(d.double().cpu().numpy()) + np.diag(e.double().cpu().numpy(), 1)
    want = np.linalg.svd(A.astype(np.float64), compute_uv=False)
    got = np.linalg.svd(B, compute_uv=False)
    # backward error of n FP32 reflections on each side, as in the tail's and the columns' tests
    assert np.max(np.abs(got - want)) <= 4 * 2.0 ** -24 * np.sqrt(n + 8) * np.linalg.norm(A)
