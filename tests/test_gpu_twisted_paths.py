"""The vectors of a bidiagonal do not depend on the path of the twisted
transforms: a block whose warps hold it alone (whole batches of steps in short
form) and the same block next to others (lane by lane) give equal bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chi(rng, n):
    i = np.arange(n)
    return np.sqrt(rng.chisquare(int(1.5 * n) - i)), np.append(np.sqrt(rng.chisquare(n - 1 - i[:-1])), 0.0)


@pytest.mark.parametrize("n", [17, 100, 301])
def test_block_alone_and_among_others(lib, cuda, n):
    rng = np.random.default_rng(n)
    a, b = chi(rng, n)
    dev = lambda x: cuda.from_numpy(x).cuda()  # noqa: E731
    s = lib.bdsdc_sigma_device(dev(a), dev(b))
    X, Y = lib.bdvec_device(dev(a), dev(b), s)
    # blocks of 5 before and between: no warp holds one block only, and their values lie apart
    parts, big, lo, at = [], 1e3, 0, []
    for _ in range(3):
        a5, b5 = chi(rng, 5)
        parts.append((a5 * big, b5 * big))
        big *= 1e3
        at.append(lo + 5)
        parts.append((a, b))
        lo += 5 + n
    A, B = (np.concatenate([p[k] for p in parts]) for k in (0, 1))
    S = lib.bdsdc_sigma_device(dev(A), dev(B))
    X2, Y2 = lib.bdvec_device(dev(A), dev(B), S)
    for r0 in at:
        cols = (X2[r0:r0 + n].abs().sum(0) > 0).nonzero().flatten()
        assert cols.numel() == n
        assert cuda.equal(X2[r0:r0 + n][:, cols], X) and cuda.equal(Y2[r0:r0 + n][:, cols], Y)
