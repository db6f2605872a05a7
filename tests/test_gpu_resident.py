"""The grid-resident columns of the bidiagonalisation at the edges of their
configurations (8, 12, 16, 20 or 24 rows per CTA, columns in registers and in shared
memory, hand-over to the cluster tail), and next to shapes that start in the
panels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(513, 513), (514, 513), (545, 544), (1216, 520), (1217, 1024), (1024, 1024),
                                 (1025, 1025), (1216, 1216), (1300, 1217), (1824, 600), (1825, 1025), (2432, 700), (2433, 540), (2048, 2048),
                                 (2049, 2049), (2500, 1800), (3648, 900), (3649, 600), (2700, 2600), (3040, 560), (3041, 580)])
@pytest.mark.parametrize("kind", ["normal", "rank"])
def test_resident_edges(lib, cuda, m, n, kind):
    rng = np.random.default_rng(m * 7 + n)
    A = rng.standard_normal((m, n))
    if kind == "rank":  # zero rows, columns and reflectors on the way
        r = max(1, n // 3)
        A = A[:, :r] @ rng.standard_normal((r, n))
        A[:, n // 2] = 0.0
        A[0, :] = 0.0
    A = A.astype(np.float32)
    W, d, e, tq, tp = lib.bidiag_device(cuda.from_numpy(A).cuda(), mode="tf32x6")
    B = np.diag(d.double().cpu().numpy()) + np.diag(e.double().cpu().numpy(), 1)
    want = cuda.linalg.svdvals(cuda.from_numpy(A).double()).numpy()
    got = cuda.linalg.svdvals(cuda.from_numpy(B)).numpy()
    # backward error of n FP32 reflections on each side
    assert np.max(np.abs(got - want)) <= 4 * 2.0 ** -24 * np.sqrt(n + 8) * np.linalg.norm(A)
    # the stored reflectors: H = I - tau u u^T with ||u||^2 = 2 / tau wherever tau is not zero
    Wm = W.double().cpu().numpy().T[:m]
    tq, tp = tq.double().cpu().numpy(), tp.double().cpu().numpy()
    for i in range(n):
        u = np.r_[1.0, Wm[i + 1:, i]]
        assert tq[i] == 0.0 or abs(tq[i] * (u @ u) - 2.0) <= 1e-4
        if i + 1 < n:
            v = np.r_[1.0, Wm[i, i + 2:]]
            assert tp[i] == 0.0 or abs(tp[i] * (v @ v) - 2.0) <= 1e-4


@pytest.mark.parametrize("m,n", [(900, 700), (2600, 2500)])  # polled words; grid barriers
def test_waits_that_run_out_end_with_a_status(lib, cuda, m, n):
    """One CTA's arrival is missing: every wait ends at the 2 ms limit, the call
    returns DDCSVD_ERR_TIMEOUT and the handle works again afterwards."""
    rng = np.random.default_rng(3)
    A = cuda.from_numpy(rng.standard_normal((m, n)).astype(np.float32)).cuda()
    h = lib.Handle()
    want = lib.svd_device(A, handle=h)[0].cpu().numpy()
    keep = h.limits
    h.limits = {"wait_us": 2000, "barrier_extra_arrivals": 1}
    with pytest.raises(lib.DdcsvdError) as ei:
        lib.svd_device(A, handle=h)
    assert ei.value.status == 5
    h.limits = keep
    assert np.array_equal(lib.svd_device(A, handle=h)[0].cpu().numpy(), want)
