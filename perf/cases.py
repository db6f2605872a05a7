"""Performance cases of the SVD library: what a program calls, over the sizes that it calls it with.

Seven kinds of work, each through the package's public entry points:

  factors   svd_device on a matrix with separated singular values; sigma, U and V come back with the usual
            sign convention (the entries of each right vector sum to a non-negative number)
  host      the same through the host-buffer call `svd` (numpy in and out)
  shrink    singular value thresholding, U max(sigma - tau, 0) V^T: the proximal step of matrix completion
            and robust PCA (svd_device, then the library's GEMM)
  polar     the orthogonal polar factor U V^T: Procrustes problems, orthogonalised updates
  batch     a BatchPlan of uneven problems; its flat sigma, U and V
  denoise   a BatchPlan of equal patches, each thresholded: locally low-rank denoising
  adjoint   svd_backward_device: the backward pass of a batch of thin SVDs
  bdsvd     the SVD of a bidiagonal: bdsdc_sigma_device, then bdvec_device

Large single SVDs return sigma and the matrix formed from all of U, sigma and V rather than the vectors
themselves: the vectors of neighbouring singular values of a large FP32 matrix are not determined by it
(they turn by rounding / gap), the matrices that programs form from them are.
"""
import concurrent.futures
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ddc-svd_gb300"))
import ddcsvd  # noqa: E402


def listed():
    return [
        # the smallest single call: a small least-squares or alignment problem, all launches and latency
        dict(name="factors_64x48", kind="factors", m=64, n=48, mode="auto"),
        # the plain configuration: one 512 x 256 matrix, entries uniform in [-1, 1)
        dict(name="shrink_512x256", kind="shrink", m=512, n=256, values="uniform", mode="auto"),
        # a wide matrix (decomposed through its transpose), as data with more features than samples
        dict(name="polar_300x1100", kind="polar", m=300, n=1100, values="normal", mode="auto"),
        # odd sizes; low rank plus noise, as in matrix completion
        dict(name="shrink_1500x1001", kind="shrink", m=1500, n=1001, values="lowrank", mode="auto"),
        # the precision configuration: 4096^2, graded spectrum with condition 1e6
        dict(name="shrink_4096x4096", kind="shrink", m=4096, n=4096, values="graded", mode="tf32x3"),
        # the tall configuration (QR first), the largest single matrix
        dict(name="polar_16384x8192", kind="polar", m=16384, n=8192, values="normal", mode="tf32x3"),
        # host buffers in and out, as the reference's callers have them
        dict(name="host_900x250", kind="host", m=900, n=250, mode="auto"),
        # the batched configuration: 2048 problems, m in [16, 256], n in [8, m], entries uniform in [-1, 1)
        dict(name="batch_2048", kind="batch", count=2048, m_max=256, shapes=3),
        # a small batch of equal patches
        dict(name="denoise_400x96x36", kind="denoise", count=400, m=96, n=36),
        # the differentiation configuration in FP64, and ragged sizes in FP32
        dict(name="adjoint_f64_256x128x64", kind="adjoint", count=256, m=128, n=64, dtype="float64"),
        dict(name="adjoint_f32_300x97x41", kind="adjoint", count=300, m=97, n=41, dtype="float32"),
        # stages 2-4 alone, on the bidiagonal of a Gaussian matrix
        dict(name="bdsvd_3000", kind="bdsvd", n=3000),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["factors", "host", "shrink", "shrink", "polar", "batch", "denoise", "adjoint", "adjoint",
                       "bdsvd"])
    mode = rng.choice(["auto", "auto", "tf32x3"])
    if kind in ("factors", "host"):
        n = _log_int(rng, 8, 256)
        return dict(kind=kind, m=_log_int(rng, n, 4 * n), n=n, mode=mode)
    if kind == "shrink":
        values = rng.choice(["uniform", "lowrank", "graded"])
        m, n = _log_int(rng, 32, 4096), _log_int(rng, 32, 4096)
        return dict(kind=kind, m=m, n=n, values=values, mode=mode)
    if kind == "polar":
        k, f = _log_int(rng, 16, 2048), rng.uniform(2.0, 6.0)
        m, n = int(k * f), k
        if rng.random() < 0.3:
            m, n = n, m
        return dict(kind=kind, m=m, n=n, values="normal", mode=mode)
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 4, 2048), m_max=_log_int(rng, 24, 256), shapes=rng.randrange(1000))
    if kind == "denoise":
        m = _log_int(rng, 16, 256)
        return dict(kind=kind, count=_log_int(rng, 16, 1024), m=m, n=rng.randint(8, max(8, m // 2)))
    if kind == "adjoint":
        m = _log_int(rng, 16, 256)
        return dict(kind=kind, count=_log_int(rng, 8, 400), m=m, n=rng.randint(max(4, m // 4), m),
                    dtype=rng.choice(["float64", "float32"]))
    return dict(kind="bdsvd", n=_log_int(rng, 32, 4096))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, dtype=torch.float32):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def _matrix(case, seed):
    """A float32 CUDA matrix of the case's kind, and its threshold for `shrink`."""
    m, n, g = case["m"], case["n"], _gen(seed)
    k = min(m, n)
    values = case.get("values", "linear")
    if values == "uniform":
        A = torch.rand((m, n), generator=g, device="cuda") * 2 - 1
        return A, 0.5 * (math.sqrt(m) + math.sqrt(n)) / math.sqrt(3.0)
    if values == "normal":
        return _randn(g, m, n), 0.0
    if values == "lowrank":  # rank k/10 with values of order 1, plus noise of 1%
        r = max(1, k // 10)
        noise = 0.01 / math.sqrt(max(m, n))
        A = (_randn(g, m, r) / math.sqrt(m)) @ (_randn(g, r, n) / math.sqrt(n)) + noise * _randn(g, m, n)
        return A, 1.5 * noise * (math.sqrt(m) + math.sqrt(n))
    Q1 = torch.linalg.qr(_randn(g, m, k))[0]
    Q2 = torch.linalg.qr(_randn(g, n, k))[0]
    i = torch.arange(k, device="cuda", dtype=torch.float64)
    s = 10.0 ** (-6.0 * i / max(k - 1, 1)) if values == "graded" else 1.0 - i / (k + 1)
    return (Q1 * s.float()) @ Q2.T, 0.01


def _shapes(case):
    """The uneven batch's sizes: m in [16, m_max], n in [8, m]."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for _ in range(case["count"]):
        m = int(rng.integers(16, case["m_max"] + 1))
        out.append((m, int(rng.integers(8, m + 1))))
    return out


def prepare(case, seed):
    kind, st = case["kind"], {"case": dict(case)}
    if kind in ("factors", "shrink", "polar"):
        st["A"], st["tau"] = _matrix(case, seed)
    elif kind == "host":
        st["A"] = np.asfortranarray(_matrix(case, seed)[0].cpu().numpy())
    elif kind == "batch":
        st["plan"] = ddcsvd.BatchPlan(_shapes(case))
        st["plan"].A.uniform_(-1.0, 1.0, generator=_gen(seed))
    elif kind == "denoise":  # patches of rank n/4 plus noise of 10%
        g, B, m, n = _gen(seed), case["count"], case["m"], case["n"]
        r = max(1, n // 4)
        noise = 0.1 / math.sqrt(m)
        P = (_randn(g, B, m, r) / math.sqrt(m)) @ (_randn(g, B, r, n) / math.sqrt(n)) + noise * _randn(g, B, m, n)
        st["P"], st["tau"] = P, noise * (math.sqrt(m) + math.sqrt(n))
        st["plan"] = ddcsvd.BatchPlan([(m, n)] * B)
    elif kind == "adjoint":
        g, B, m, n = _gen(seed), case["count"], case["m"], case["n"]
        dt = getattr(torch, case["dtype"])
        st["U"] = torch.linalg.qr(_randn(g, B, m, n, dtype=torch.float64))[0].to(dt)
        st["V"] = torch.linalg.qr(_randn(g, B, n, n, dtype=torch.float64))[0].to(dt)
        s = 1.0 + torch.arange(n, device="cuda", dtype=torch.float64) / n
        st["S"] = (s * (0.5 + torch.rand((B, 1), generator=g, device="cuda", dtype=torch.float64))).to(dt)
        st["gU"], st["gS"], st["gV"] = (_randn(g, *sh, dtype=torch.float64).to(dt)
                                        for sh in ((B, m, n), (B, n), (B, n, n)))
    else:  # bdsvd: the bidiagonal of a 1.5 n x n Gaussian matrix has independent chi entries
        n, rng = case["n"], np.random.default_rng(seed)
        i = np.arange(n)
        a = np.sqrt(rng.chisquare(int(1.5 * n) - i))
        b = np.append(np.sqrt(rng.chisquare(n - 1 - i[:-1])), 0.0)
        st["a"], st["b"] = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    return st


# ---------------------------------------------------------------- one pass
def _signed(U, V):
    sg = torch.where(V.sum(0) < 0, -1.0, 1.0)
    return U * sg, V * sg


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "factors":
        s, U, V = ddcsvd.svd_device(st["A"], mode=case["mode"])
        return (s, *_signed(U, V))
    if kind == "host":
        s, U, V = ddcsvd.svd(st["A"], mode=case["mode"])
        sg = np.where(V.sum(0) < 0, np.float32(-1.0), np.float32(1.0))
        return s, U * sg, V * sg
    if kind in ("shrink", "polar"):
        s, U, V = ddcsvd.svd_device(st["A"], mode=case["mode"])
        if kind == "shrink":
            U = U * torch.clamp(s - st["tau"], min=0.0)
        # the GEMM reads rows with K contiguous; its tensor-core modes want K in whole 16-byte units
        tc = "tf32x6" if case["mode"] == "auto" else case["mode"]
        return s, ddcsvd.gemm_nt_device(U.contiguous(), V.contiguous(), mode=tc if s.shape[0] % 4 == 0 else "blocked")
    if kind == "batch":
        p = st["plan"]
        p.run()
        return p.S, p.U, p.V
    if kind == "denoise":
        p, B, m, n = st["plan"], case["count"], case["m"], case["n"]
        p.A.view(B, n, m).copy_(st["P"].transpose(1, 2))
        p.run()
        w = torch.clamp(p.S.view(B, n, 1) - st["tau"], min=0.0)
        return p.S, torch.bmm(p.U.view(B, n, m).transpose(1, 2), w * p.V.view(B, n, n))
    if kind == "adjoint":
        return (ddcsvd.svd_backward_device(*(st[k] for k in ("U", "S", "V", "gU", "gS", "gV"))),)
    s = ddcsvd.bdsdc_sigma_device(st["a"], st["b"])
    return (s, *ddcsvd.bdvec_device(st["a"], st["b"], s))


# ---------------------------------------------------------------- what a pass cannot do without
def _svd_work(m, n):
    m, n = max(m, n), min(m, n)
    return 4 * (2 * m * n + n * n + n), 8.0 * m * n * n - 4.0 / 3.0 * n ** 3


def work(case):
    kind = case["kind"]
    if kind in ("factors", "host"):
        by, fl = _svd_work(case["m"], case["n"])
    elif kind in ("shrink", "polar"):  # the product replaces the factors as the output
        m, n = case["m"], case["n"]
        by, fl = 4 * (2 * m * n + min(m, n)), _svd_work(m, n)[1] + 2.0 * m * n * min(m, n)
    elif kind == "batch":
        by, fl = (sum(x) for x in zip(*(_svd_work(m, n) for m, n in _shapes(case))))
    elif kind == "denoise":
        B, m, n = case["count"], case["m"], case["n"]
        by, fl = 4 * B * (2 * m * n + n), B * (_svd_work(m, n)[1] + 2.0 * m * n * n)
    elif kind == "adjoint":
        B, m, n, e = case["count"], case["m"], case["n"], 8 if case["dtype"] == "float64" else 4
        by, fl = e * B * (3 * m * n + 2 * n * n + 2 * n), B * (6.0 * m * n * n + 2.0 * n ** 3)
    else:  # secular sums and products over the merge tree, then two qd sweeps and two solves per vector
        n = case["n"]
        by, fl = 8 * n * n + 24 * n, 60.0 * n * n
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------- the same in 64 bits, by torch and numpy
def _exact_matrix(case, seed):
    """sigma and V f(sigma) of the Gram matrix of A (its eigenvalues are far above 64-bit rounding)."""
    A, tau = _matrix(case, seed)
    A = A.double()
    wide = A.shape[0] < A.shape[1]
    if wide:
        A = A.T
    w, V = torch.linalg.eigh(A.T @ A)
    s = torch.sqrt(torch.clamp(w, min=0.0))
    f = torch.clamp(1.0 - tau / torch.clamp(s, min=1e-300), min=0.0) if case["kind"] == "shrink" else 1.0 / s
    P = A @ ((V * f) @ V.T)
    return s, P.T if wide else P


def exact(case, seed):
    kind = case["kind"]
    if kind in ("factors", "host"):
        A = _matrix(case, seed)[0].double()
        U, s, Vh = torch.linalg.svd(A, full_matrices=False)
        return (s.flip(0), *_signed(U.flip(1), Vh.T.flip(1)))
    if kind in ("shrink", "polar"):
        if min(case["m"], case["n"]) > 4096:
            return None  # an eigendecomposition of this size takes too long in 64 bits
        return _exact_matrix(case, seed)
    if kind == "batch":
        st = prepare(case, seed)
        p = st["plan"]
        flat = p.A.double().cpu().numpy()

        def values(b):
            m, n, o = int(p.ms[b]), int(p.ns[b]), int(p.offA[b])
            return np.linalg.svd(flat[o:o + m * n].reshape(n, m), compute_uv=False)[::-1]

        with concurrent.futures.ThreadPoolExecutor(8) as ex:
            s = np.concatenate(list(ex.map(values, range(len(p.ms)))))
        return s, None, None  # vectors of close values are not determined by an FP32 problem
    if kind == "denoise":
        st = prepare(case, seed)
        U, s, Vh = np.linalg.svd(st["P"].double().cpu().numpy(), full_matrices=False)
        P = np.matmul(U * np.maximum(s - st["tau"], 0.0)[:, None, :], Vh)
        return np.ascontiguousarray(s[:, ::-1]).reshape(-1), P
    if kind == "adjoint":
        st = prepare(case, seed)
        U, S, V, gU, gS, gV = (st[k].double() for k in ("U", "S", "V", "gU", "gS", "gV"))
        n = case["n"]
        eye = torch.eye(n, device="cuda", dtype=torch.bool)
        sj, si = S[:, None, :], S[:, :, None]
        F = torch.where(eye, 0.0, 1.0 / torch.where(eye, 1.0, (sj - si) * (sj + si)))
        J, K = U.mT @ gU, V.mT @ gV
        M = torch.diag_embed(gS) + F * (J - J.mT) * sj + si * (F * (K - K.mT)) - J / sj
        return ((U @ M + gU / sj) @ V.mT,)
    st, n = prepare(case, seed), case["n"]
    off = torch.stack([st["a"], st["b"]], 1).reshape(-1)[:-1]  # the Golub-Kahan tridiagonal of the bidiagonal
    T = torch.diag(off, 1) + torch.diag(off, -1)
    return torch.linalg.eigvalsh(T)[n:], None, None
