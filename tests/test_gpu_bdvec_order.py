"""bdvec_device keeps the order of the ascending values that it is given, also of
negative ones (which enter the vectors through their squares)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 300])
def test_order_of_negative_values(lib, cuda, n):
    rng = np.random.default_rng(n)
    a, b = (cuda.from_numpy(rng.uniform(0.5, 2.0, n)).cuda() for _ in range(2))
    b[-1] = 0.0
    s = lib.bdsdc_sigma_device(a, b)
    X, Y = lib.bdvec_device(a, b, s)
    X2, Y2 = lib.bdvec_device(a, b, -s.flip(0))
    assert cuda.equal(X2, X.flip(1)) and cuda.equal(Y2, Y.flip(1))
