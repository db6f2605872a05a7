"""CPU check of the secular solver's FP32 phase on poles kept as float pairs
(ddc-svd_gb300/csrc/dc.cu, sec_mid32 and pair_diff): the midpoint sign agrees
with FP64 whenever |f32| clears twice its bound, and a pole difference from
the pairs keeps FP32's relative accuracy where the heads alone lose it."""
import numpy as np
import pytest

from test_secular_bound import E32, mid64, poles

F = np.float32


def split(d):
    hi = d.astype(F)
    return hi, (d - hi.astype(np.float64)).astype(F)


def diff(a, b):
    return F((a[0] - b[0]) + (a[1] - b[1])) if np.isscalar(a[0]) else (a[0] - b[0]) + (a[1] - b[1])


def mid32(d, z, i):
    """f at the midpoint of (d_i, d_i+1) and its bound, as sec_mid32 computes them."""
    hi, lo = split(d)
    zf = z.astype(F)
    with np.errstate(all="ignore"):
        tau = F(0.5) * F(F((hi[i + 1] - hi[i]) + (lo[i + 1] - lo[i])) * F(hi[i + 1] + hi[i]))
        dif = (hi - hi[i]) + (lo - lo[i])
        dl = dif * (hi + hi[i]) - tau
        ir = F(1.0) / dl
        tt = zf * zf * ir
        ad = np.abs(hi) + np.abs(hi[i])
        ed = F(4.0) * E32 * (np.abs(dif) * ad + np.abs(tau)) + F(2.0 ** -44) * ad * ad
        adl = np.abs(dl)
        ok = (ed < F(0.5) * adl) & (adl >= F(2.0 ** -100)) & (adl <= F(2.0 ** 100))
        at = np.abs(tt)
        ea = np.where(ok, at * (F(2.5) * ed * np.abs(ir) + F(6.0) * E32), F(np.inf))
        s = sa = e = F(0.0)
        for j in range(len(d)):
            s, sa, e = F(s + tt[j]), F(sa + at[j]), F(e + ea[j])
        return F(1.0) + s, e + F(len(d) + 2) * E32 * (F(1.0) + sa)


@pytest.mark.parametrize("kind", ["uniform", "graded", "cluster9", "cluster12", "tiny", "huge"])
def test_midpoint_sign_from_pairs_matches_fp64_when_bound_clears(kind):
    rng = np.random.default_rng(100 + len(kind))
    used = total = 0
    for _ in range(12):
        d = poles(rng, kind, int(rng.integers(3, 120)))
        if len(d) < 3:
            continue
        z = rng.standard_normal(len(d)) * np.abs(d).max() * 10.0 ** rng.uniform(-3, 0, len(d))
        z[rng.random(len(d)) < 0.1] *= 1e-6
        for i in range(len(d) - 1):
            f32, err = mid32(d, z, i)
            total += 1
            if np.isfinite(f32) and abs(f32) > 2 * err:
                used += 1
                assert (f32 >= 0) == (mid64(d, z, i) >= 0), (kind, i, float(f32), float(err))
    assert total > 0
    if kind in ("uniform", "graded"):
        assert used > 0.5 * total


@pytest.mark.parametrize("gap", [1e-2, 1e-4, 1e-6])
def test_pair_difference_keeps_relative_accuracy(gap):
    rng = np.random.default_rng(7)
    a = rng.uniform(0.5, 2.0, 2000)
    b = a * (1.0 + gap * rng.uniform(0.5, 1.0, 2000))
    (ah, al), (bh, bl) = split(a), split(b)
    got = ((bh - ah) + (bl - al)).astype(np.float64)
    # one rounding of each part (2^-24), plus 2^-48 |a| from each pair
    assert np.max(np.abs(got - (b - a)) / (b - a)) <= 2.0 ** -23 + 2.0 ** -45 / gap
