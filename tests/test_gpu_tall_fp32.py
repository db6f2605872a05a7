"""Tall blocks beyond the cluster tail's 3072 rows whose columns are FP32
throughout: the tensor-core modes give the bidiagonal of the CUDA-core mode."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(3100, 40), (4000, 128), (5000, 64), (6000, 48), (8000, 16)])
def test_tall_blocks_stay_fp32(lib, cuda, m, n):
    A = cuda.from_numpy(np.random.default_rng(m + n).standard_normal((m, n)).astype(np.float32)).cuda()
    _, d, e, tq, tp = lib.bidiag_device(A, mode="blocked")
    for mode in ("tf32x3", "tf32x6"):
        got = lib.bidiag_device(A, mode=mode)[1:]
        assert all(cuda.equal(x, y) for x, y in zip(got, (d, e, tq, tp))), mode
