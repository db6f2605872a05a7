"""The one-launch FP32 adjoint on both sides of its rule for the CTA's threads
(512 from 512 tiles of 4 x 4 in an m x n matrix on, 256 below), with and
without each gradient, against the formula in FP64."""
import pytest
from test_gpu_adjoint_products import formula, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(128, 60), (125, 61), (128, 64), (129, 64), (256, 32), (172, 48), (253, 29), (200, 75)])
@pytest.mark.parametrize("given", ["all", "U", "V"])
def test_thread_rule(lib, cuda, m, n, given):
    U, S, V, gU, gS, gV = problem(cuda, 3, m, n, cuda.float32, "rows")
    zero = cuda.zeros_like
    ref = formula(cuda, U, S, V, zero(gU) if given == "V" else gU, gS, zero(gV) if given == "U" else gV)
    got = lib.svd_backward_device(U, S, V, None if given == "V" else gU, gS, None if given == "U" else gV).double()
    # FP32 sums of at most m products, F's denominators of neighbouring values: as for the products' test
    err = float(cuda.linalg.norm(got - ref) / cuda.linalg.norm(ref))
    assert err <= 4e-6, err
