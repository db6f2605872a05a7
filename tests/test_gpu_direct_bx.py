"""The register back-transformation of small problems at the edges of its
tiles (128 rows per register, four reflectors per group, four columns per
CTA), on tight and on padded, unaligned outputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (2, 1), (2, 2), (3, 3), (4, 4), (6, 5), (64, 64), (65, 33), (128, 97), (129, 128), (256, 256),
          (257, 255), (257, 257), (512, 31), (513, 300), (1024, 260), (1025, 200), (2048, 512), (2049, 512), (600, 513)]


@pytest.mark.parametrize("m,n", SHAPES)
@pytest.mark.parametrize("pad", [0, 3])
def test_direct_back_transformation(lib, cuda, m, n, pad):
    torch = cuda
    rng = np.random.default_rng(m + 5 * n)
    A = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32)).cuda()
    Ac = A.t().contiguous()
    s = torch.empty(n, device="cuda")
    U = torch.full((n, m + pad), 7.0, device="cuda")
    V = torch.full((n, n + pad), 7.0, device="cuda")
    h = lib.Handle()
    lib.check(lib.load().ddcsvd_svd_f32_device(h.ptr, m, n, Ac.data_ptr(), m, s.data_ptr(), U.data_ptr(), m + pad,
                                               V.data_ptr(), n + pad, lib.MODES["tf32x6"]), "svd")
    assert bool((U[:, m:] == 7.0).all()) and bool((V[:, n:] == 7.0).all())  # padding is the caller's
    Ud, Vd, sd = U[:, :m].t().double(), V[:, :n].t().double(), s.double()
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    assert float(torch.linalg.norm(A.double() - (Ud * sd) @ Vd.T) / torch.linalg.norm(A.double())) <= 1e-5
    assert float(torch.linalg.norm(Ud.T @ Ud - eye)) / n ** 0.5 <= 1e-5
    assert float(torch.linalg.norm(Vd.T @ Vd - eye)) / n ** 0.5 <= 1e-5
