"""Stage 2 as a single SVD runs it (the third-order secular step, the
separate products of z-hat, the pairwise FP32 phase): the SVD of an FP32 upper
bidiagonal, which the FP32 reduction passes through with sign flips only, so
sigma must be the bidiagonal's to the rounding of the FP32 output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bidiagonal(n, kind):
    rng = np.random.default_rng(n + 31 * len(kind))
    b = rng.uniform(0.5, 1.5, max(n - 1, 0))
    if kind == "uniform":
        a = rng.uniform(0.5, 1.5, n)
    elif kind == "signed":
        a = rng.uniform(0.5, 1.5, n) * np.where(rng.random(n) < 0.5, -1.0, 1.0)
    else:  # peaks at both ends: values that coincide to working precision
        a, b = np.abs(np.arange(n) - n // 2) + 1.0, np.ones(max(n - 1, 0))
    return a.astype(np.float32), b.astype(np.float32)


@pytest.mark.parametrize("kind", ["uniform", "signed", "pairs"])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 33, 64, 65, 130, 257, 700])
def test_sigma_of_a_bidiagonal(lib, cuda, n, kind):
    a, b = _bidiagonal(n, kind)
    B = np.diag(a.astype(np.float64)) + (np.diag(b.astype(np.float64), 1) if n > 1 else 0.0)
    want = np.sort(np.linalg.svd(B, compute_uv=False))
    s, _, _ = lib.svd_device(cuda.from_numpy(B.astype(np.float32)).cuda())
    s = s.double().cpu().numpy()
    assert np.all(np.abs(s - want) <= 2.0 ** -23 * want + 1e-12 * want[-1])
