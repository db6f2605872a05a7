"""Device-side waits of the bidiagonalisation that run out: a record that never
comes ends every wait at the handle's limit, the call returns
DDCSVD_ERR_TIMEOUT promptly and the handle works again afterwards."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run_out(lib, cuda, m, n, extra, mode="tf32x6"):
    A = cuda.from_numpy(np.random.default_rng(m + n).standard_normal((m, n)).astype(np.float32)).cuda()
    h = lib.Handle()
    want = lib.svd_device(A, mode=mode, handle=h)[0].cpu().numpy()
    keep = h.limits
    h.limits = {"wait_us": 2000, "barrier_extra_arrivals": extra}
    t0 = time.perf_counter()
    with pytest.raises(lib.DdcsvdError) as ei:
        lib.svd_device(A, mode=mode, handle=h)
    elapsed = time.perf_counter() - t0
    assert ei.value.status == 5
    assert elapsed < 0.5, elapsed  # (the default limit is seconds)
    h.limits = keep
    assert np.array_equal(lib.svd_device(A, mode=mode, handle=h)[0].cpu().numpy(), want)


@pytest.mark.parametrize("m,n", [(24, 16), (64, 48), (300, 129), (512, 256), (1500, 512)])
def test_cluster_tail(lib, cuda, m, n):
    """Clusters of 1 to 16 CTAs, with and without slices of their own."""
    run_out(lib, cuda, m, n, 1)


@pytest.mark.parametrize("m,n", [(4500, 300), (8190, 200)])
def test_column_ring(lib, cuda, m, n):
    """A column that is never asked for, with several slots of the ring's own and with one."""
    run_out(lib, cuda, m, n, 1024)
