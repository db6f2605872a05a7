"""Two handles in two host threads (the cooperative kernels on one stream, so that
they follow one another): a call whose kernel needs much shared memory is not refused because
the other thread has just launched the same kernel with less."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def together(*calls):
    """Each call repeatedly in a thread of its own; the first error is raised."""
    errors = []

    def loop(f, count):
        try:
            for _ in range(count):
                if errors:
                    return
                f()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=loop, args=c) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_fp32_adjoint(lib, cuda):
    """Each thread on a stream of its own, through the C ABI: little else between the calls."""
    fn = lib.load().ddcsvd_svd_backward_f32_device

    def call(m, n):
        g = cuda.Generator(device="cuda").manual_seed(m)
        r = lambda *s: cuda.randn(s, generator=g, device="cuda")  # noqa: E731
        ten = [r(n, m), 1.0 + cuda.arange(n, device="cuda") / n, r(n, n), r(n, m), r(n), r(n, n), r(n, m)]
        h = lib.Handle(stream=cuda.cuda.Stream())
        cuda.cuda.synchronize()
        args = (h.ptr, 1, m, n, *(t.data_ptr() for t in ten))

        def f():
            lib.check(fn(*args), "svd_backward")

        f.keep = (h, ten)
        return f

    together((call(128, 64), 6000), (call(40, 24), 6000))


def test_batch(lib, cuda):
    def call(shapes):
        h = lib.Handle()
        rng = np.random.default_rng(len(shapes))
        mats = [cuda.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda() for s in shapes]
        want = [o[0].clone() for o in lib.svd_batched_device(mats, handle=h)]

        def f():
            got = lib.svd_batched_device(mats, handle=h)
            assert all(cuda.equal(g[0], w) for g, w in zip(got, want))

        return f

    together((call([(200, 100)] * 3), 60), (call([(16, 8)] * 3), 150))


def test_resident_columns(lib, cuda):
    def call(m, n):
        h = lib.Handle()
        A = cuda.from_numpy(np.random.default_rng(n).standard_normal((m, n)).astype(np.float32)).cuda()
        want = lib.svd_device(A, handle=h)[0].clone()

        def f():
            assert cuda.equal(lib.svd_device(A, handle=h)[0], want)

        return f

    together((call(2500, 1750), 6), (call(2500, 1580), 6))
