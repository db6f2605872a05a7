"""The FP64 adjoint of unevenly scaled problems: every column and every row of
the gradient as close to extended precision as FP64 sums of the same formula
come, where the matrices' entries differ by many orders of magnitude within a
row or column (V or U near the identity, graded singular values)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


def haar(rng, m, n):
    q, r = np.linalg.qr(rng.standard_normal((m, n)))
    return q * np.sign(np.diag(r))


def jacobi(A):
    """One-sided Jacobi SVD: small entries of V relatively accurate.  Ascending."""
    A, n = A.copy(), A.shape[1]
    V = np.eye(n)
    for _ in range(20):
        off = 0.0
        for p in range(n - 1):
            for q in range(p + 1, n):
                al, be, ga = A[:, p] @ A[:, p], A[:, q] @ A[:, q], A[:, p] @ A[:, q]
                off = max(off, abs(ga) / np.sqrt(al * be))
                if ga == 0.0:
                    continue
                z = (be - al) / (2 * ga)
                t = 1 / (abs(z) + np.sqrt(1 + z * z)) * (1 if z >= 0 else -1)
                c = 1 / np.sqrt(1 + t * t)
                for M in (A, V):
                    M[:, p], M[:, q] = c * M[:, p] - c * t * M[:, q], c * t * M[:, p] + c * M[:, q]
        if off < 1e-15:
            break
    s = np.sqrt((A * A).sum(0))
    o = np.argsort(s)
    return (A / s)[:, o], s[o], V[:, o]


def factors(rng, kind, m, n):
    i = np.arange(n)
    up = lambda x: x[::-1].copy()  # noqa: E731
    if kind == "even":
        return haar(rng, m, n), 1.0 + i / n, haar(rng, n, n)
    if kind == "graded":
        return haar(rng, m, n), up(10.0 ** (-8.0 * i / (n - 1))), haar(rng, n, n)
    if kind == "v_identity":
        return haar(rng, m, n), up(2.0 ** (-60.0 * i / (n - 1))), np.eye(n)
    if kind == "u_identity":
        return np.eye(m, n), up(2.0 ** (-60.0 * i / (n - 1))), haar(rng, n, n)
    X = rng.standard_normal((m, n))
    if kind == "columns":  # V graded towards the identity
        return jacobi(X * 2.0 ** (-60.0 * i / (n - 1)))
    if kind == "one_column":
        X[:, 0] *= 2.0 ** 40
        return jacobi(X)
    assert kind == "rows"
    return jacobi(X * (10.0 ** (-8.0 * np.arange(m) / (m - 1)))[:, None])


def formula(U, s, V, gU, gS, gV, t):
    U, s, V = (x.astype(t) for x in (U, s, V))
    n = len(s)
    eye = np.eye(n, dtype=bool)
    sj, si = s[None, :], s[:, None]
    F = np.where(eye, t(0), t(1) / np.where(eye, t(1), (sj - si) * (sj + si)))
    M = np.zeros((n, n), t)
    if gS is not None:
        M += np.diag(gS.astype(t))
    if gU is not None:
        J = U.T @ gU.astype(t)
        M += F * (J - J.T) * sj - J / sj
    if gV is not None:
        K = V.T @ gV.astype(t)
        M += si * (F * (K - K.T))
    P = U @ M
    if gU is not None:
        P = P + gU.astype(t) / sj
    return P @ V.T


def worst(G, R):
    """Largest relative error of a column and of a row (of those that are not zero)."""
    out = []
    for ax in (0, 1):
        e, r = (np.sqrt((x * x).sum(ax)) for x in (G.astype(LD) - R, R))
        out.append(float((e[r > 0] / r[r > 0]).max()))
    return out


@pytest.mark.parametrize("m,n", [(70, 40), (129, 65), (20, 7)])
@pytest.mark.parametrize("kind", ["even", "graded", "v_identity", "u_identity", "columns", "one_column", "rows"])
@pytest.mark.parametrize("loss", ["all", "S", "logdet", "U", "V"])
def test_columns_and_rows(lib, cuda, kind, loss, m, n):
    assert np.finfo(LD).eps < 2e-19
    rng = np.random.default_rng(m + n)
    U, s, V = factors(rng, kind, m, n)
    gU = rng.standard_normal((m, n)) if loss in ("all", "U") else None
    gV = rng.standard_normal((n, n)) if loss in ("all", "V") else None
    gS = 1.0 / s if loss == "logdet" else rng.standard_normal(n) if loss in ("all", "S") else None
    exact = formula(U, s, V, gU, gS, gV, LD)
    sums = worst(formula(U, s, V, gU, gS, gV, np.float64), exact)
    dev = [None if x is None else cuda.from_numpy(x[None]).cuda() for x in (U, s, V, gU, gS, gV)]
    got = worst(lib.svd_backward_device(*dev)[0].cpu().numpy(), exact)
    # rounding errors of the same size in another order: a factor of 4, and four
    # roundings of the result where the FP64 sums happen to be nearly exact
    for g, w in zip(got, sums):
        assert g <= 4.0 * w + 4.0 * 2.0 ** -53, (got, sums)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -300, 2.0 ** -520])
def test_quotients_are_rounded_once(lib, cuda, scale):
    """U = [I; 0], V = I and gU in U's complement: the gradient is gU / s, and each entry the
    quotient that a division gives (operands within and beyond the range of the short form)."""
    rng = np.random.default_rng(5)
    B, n = 16, 40
    U, V = np.zeros((B, 2 * n, n)), np.broadcast_to(np.eye(n), (B, n, n)).copy()
    U[:, :n] = np.eye(n)
    s = np.sort(rng.uniform(1.0, 3.0, (B, n)), axis=1)
    gU = np.zeros((B, 2 * n, n))
    gU[:, n:] = rng.uniform(0.5, 1.0, (B, n, n)) * scale
    got = lib.svd_backward_device(*(cuda.from_numpy(x).cuda() for x in (U, s, V, gU)), None, None).cpu().numpy()
    assert np.array_equal(got, gU / s[:, None, :])
