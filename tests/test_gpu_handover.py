"""The hand-over from the bidiagonal reduction to the singular-value stage: the
layout made ahead for one unreduced block, the one made anew when the bidiagonal
splits, and the range scale taken back between them, alternating on one handle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (2, 1), (2, 2), (33, 32), (65, 65), (200, 90), (513, 300), (1500, 257), (300, 1030)]


def _check(sig, U, V, A):
    """FP32 factors against the FP64 matrix, relative to its largest value."""
    top = np.linalg.norm(A, 2)
    ref = np.linalg.svd(A, compute_uv=False)
    assert np.abs(np.sort(sig)[::-1] - ref).max() <= 1e-5 * top
    assert np.linalg.norm((U * (sig / top)) @ V.T - A / top) <= 1e-5 * np.linalg.norm(A / top)


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("scale", [1.0, 1e-33, 1e33])
def test_split_and_unreduced_alternate(lib, cuda, m, n, scale):
    torch = cuda
    k = min(m, n)
    rng = np.random.default_rng(m + 3 * n)
    full = rng.standard_normal((m, n))
    block = full.copy()  # two independent parts: the bidiagonal of the whole splits
    block[: k // 2, n // 2 :] = 0.0
    block[k // 2 :, : n // 2] = 0.0
    diag = np.zeros((m, n))
    diag[np.arange(k), np.arange(k)] = 1.0 + np.arange(k) % 3
    h = lib.Handle()
    for A in (full, diag, full, block):
        A32 = (A * scale).astype(np.float32)
        s, U, V = lib.svd_device(torch.from_numpy(A32).cuda(), handle=h)
        _check(s.double().cpu().numpy(), U.double().cpu().numpy(), V.double().cpu().numpy(), A32.astype(np.float64))
