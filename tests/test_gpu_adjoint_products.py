"""The adjoint's batched products at the edges of their tiles (64 x 64, K in
slabs of 32 and exact chunks of 128) and on matrices of any layout, against
the formula in FP64; Inf and NaN still come through where the derivative does
not exist."""
import pytest

pytestmark = pytest.mark.gpu


def problem(torch, B, m, n, dtype, layout, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(m * 100 + n)
    r = lambda *s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    U, V = torch.linalg.qr(r(B, m, n))[0], torch.linalg.qr(r(B, n, n))[0]
    S = (1.0 + torch.arange(n, device="cuda", dtype=torch.float64) / n).repeat(B, 1)
    mats = [U, V, scale * r(B, m, n), r(B, n, n)]
    if layout == "t":  # column-major matrices
        mats = [x.transpose(1, 2).contiguous().transpose(1, 2) for x in mats]
    elif layout == "cut":  # rows and columns of a larger tensor, batch not outermost
        out = []
        for x in mats:
            w = torch.zeros((x.shape[1] + 1, B, x.shape[2] + 3), device="cuda", dtype=torch.float64)
            w[1:, :, 2:-1] = x.transpose(0, 1)
            out.append(w[1:, :, 2:-1].transpose(0, 1))
        mats = out
    gS = r(B, n)
    return [x.to(dtype) for x in (mats[0], S, mats[1], mats[2], gS, mats[3])]


def formula(torch, U, S, V, gU, gS, gV):
    U, S, V, gU, gS, gV = (x.double() for x in (U, S, V, gU, gS, gV))
    eye = torch.eye(S.shape[1], device="cuda", dtype=torch.bool)
    sj, si = S[:, None, :], S[:, :, None]
    F = torch.where(eye, 0.0, 1.0 / torch.where(eye, 1.0, (sj - si) * (sj + si)))
    J, K = U.mT @ gU, V.mT @ gV
    M = torch.diag_embed(gS) + F * (J - J.mT) * sj + si * (F * (K - K.mT)) - J / sj
    return (U @ M + gU / sj) @ V.mT


@pytest.mark.parametrize("layout", ["rows", "t", "cut"])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("m,n", [(1, 1), (5, 3), (31, 31), (64, 33), (65, 64), (129, 65), (257, 97), (300, 130)])
def test_products_against_formula(lib, cuda, m, n, dtype, layout):
    args = problem(cuda, 3, m, n, getattr(cuda, dtype), layout)
    ref = formula(cuda, *args)
    got = lib.svd_backward_device(*args).double()
    err = float(cuda.linalg.norm(got - ref) / cuda.linalg.norm(ref))
    assert err <= (1e-14 if dtype == "float64" else 4e-6), err


@pytest.mark.parametrize("scale", [1e-200, 1e200])
def test_fp64_range(lib, cuda, scale):
    """Rows are scaled by their own largest entry: gradients of any magnitude."""
    args = problem(cuda, 2, 70, 40, cuda.float64, "rows", scale)
    args[4], args[5] = args[4] * scale, args[5] * scale
    ref = formula(cuda, *args)
    got = lib.svd_backward_device(*args)
    assert float(cuda.linalg.norm((got - ref) / scale) / cuda.linalg.norm(ref / scale)) <= 1e-14


def test_coinciding_values_stay_nonfinite(lib, cuda):
    args = problem(cuda, 2, 70, 40, cuda.float64, "rows")
    args[1][0, 7] = args[1][0, 8]
    got = lib.svd_backward_device(*args)
    assert not bool(cuda.isfinite(got[0]).all()) and bool(cuda.isfinite(got[1]).all())
