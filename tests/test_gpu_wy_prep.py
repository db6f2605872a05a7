"""The WY preparation of the tensor-core back-transformation at the edges of its
blocks (128 reflectors, pairs of them, a last pair with one block or a part of
one) and of its row chunks (128 rows, 512 where the blocks alone fill the GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(513, 513), (640, 640), (641, 641), (769, 768), (1100, 897), (1030, 1025), (2100, 520),
                                 (1500, 1001), (2700, 2560), (3100, 2945)])
def test_wy_preparation(lib, cuda, m, n):
    torch = cuda
    rng = np.random.default_rng(3 * m + n)
    A = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32)).cuda()
    s, U, V = lib.svd_device(A, mode="tf32x6")
    Ad, Ud, Vd, sd = A.double(), U.double(), V.double(), s.double()
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    assert float(torch.linalg.norm(Ad - (Ud * sd) @ Vd.T) / torch.linalg.norm(Ad)) <= 1e-5
    assert float(torch.linalg.norm(Ud.T @ Ud - eye)) / n ** 0.5 <= 1e-5
    assert float(torch.linalg.norm(Vd.T @ Vd - eye)) / n ** 0.5 <= 1e-5
