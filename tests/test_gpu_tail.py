"""The register-resident cluster tail of the bidiagonalisation at the edges of
its tiles: slices of 32 columns, 8 C R rows (C CTAs, R rows per warp), one
column, square blocks (whose last reflector has one element)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (2, 1), (2, 2), (5, 3), (31, 31), (33, 32), (33, 33), (64, 33), (65, 64),
                                 (129, 65), (128, 128), (257, 96), (300, 129), (256, 256), (513, 257), (512, 512),
                                 (1024, 512), (1025, 512), (1536, 512), (1537, 400), (2048, 384), (2048, 256),
                                 (2049, 256), (3072, 250), (3073, 256), (1700, 100), (3000, 40)])
@pytest.mark.parametrize("kind", ["normal", "rank"])
def test_tail_tile_edges(lib, cuda, m, n, kind):
    rng = np.random.default_rng(m * 7 + n)
    A = rng.standard_normal((m, n))
    if kind == "rank":  # zero rows, columns and reflectors on the way
        r = max(1, n // 3)
        A = A[:, :r] @ rng.standard_normal((r, n))
        A[:, n // 2] = 0.0
        A[0, :] = 0.0
    A = A.astype(np.float32)
    W, d, e, tq, tp = lib.bidiag_device(cuda.from_numpy(A).cuda(), mode="tf32x6")
    B = np.diag(d.double().cpu().numpy()) + (np.diag(e.double().cpu().numpy(), 1) if n > 1 else 0.0)
    want = np.linalg.svd(A.astype(np.float64), compute_uv=False)
    got = np.linalg.svd(B, compute_uv=False)
    # backward error of n FP32 reflections on each side
    assert np.max(np.abs(got - want)) <= 4 * 2.0 ** -24 * np.sqrt(n + 8) * max(np.linalg.norm(A), 1e-30)
    # the stored reflectors: H = I - tau u u^T with ||u||^2 = 2 / tau wherever tau is not zero
    Wm = W.double().cpu().numpy().T[:m]
    tq, tp = tq.double().cpu().numpy(), tp.double().cpu().numpy()
    for i in range(n):
        u = np.r_[1.0, Wm[i + 1:, i]]
        assert tq[i] == 0.0 or abs(tq[i] * (u @ u) - 2.0) <= 1e-4
        if i + 1 < n:
            v = np.r_[1.0, Wm[i, i + 2:]]
            assert tp[i] == 0.0 or abs(tp[i] * (v @ v) - 2.0) <= 1e-4
