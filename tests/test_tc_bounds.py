"""Bounds behind the 64-bit integer sums of the FP64 tensor-core contraction.

legendre_fp64_tc.cu sizes its integer unit from sum over north rings of |lambda_lm| (spin 2:
|lambda1| + |lambda2|) < 0.85 nside, and from sum over the l of one parity of |lambda_lm| 2^-EA(l)
< 0.4 (lmax/2 + 1), 2^EA(l) the power of two above sqrt((2l+1)/4pi).  Every l, m and ring of a
few plans with lmax = 4 nside, lambda by the plain recursion with scaled seeds.
"""
import numpy as np
import pytest


def _sums(ns):
    lmax, nn = 4 * ns, 2 * ns
    i = np.arange(nn) + 1
    z = np.where(i < ns, 1 - i * i / (3.0 * ns * ns), (2 * ns - i) * 2 / (3.0 * ns))
    s = np.sqrt((1 - z) * (1 + z))
    m = np.arange(lmax + 1)[:, None].astype(float)
    k = np.arange(1, lmax + 1)
    lg = np.concatenate([[0], np.cumsum(np.log2((2 * k + 1) / (2 * k)))])[:, None]
    lg = 0.5 * (lg - np.log2(4 * np.pi)) + m * np.log2(s)[None]
    e = np.minimum(0, np.ceil((lg - 300) / 600))
    seed = np.exp2(lg - 600 * e)
    cur, prev = np.zeros((2, lmax + 1, nn))
    rings = np.zeros(2)                       # spin 0, spin 2
    cols = np.zeros((2, 2, lmax + 1, nn))
    for l in range(lmax + 1):
        with np.errstate(all="ignore"):
            a = np.nan_to_num(np.where(l > m, np.sqrt((4.0 * l * l - 1) / (l * l - m * m)), 0))
            b = np.nan_to_num(np.where(
                l > m, np.sqrt(((l - 1) ** 2 - m * m) / (4.0 * (l - 1) ** 2 - 1)) * a, 0))
        nx = a * z * cur - b * prev
        nx[l] = seed[l]
        prev, cur = cur, nx
        up = (np.abs(cur) > 2.0 ** 300) & (e < 0)
        cur, prev = np.where(up, cur * 2.0 ** -600, cur), np.where(up, prev * 2.0 ** -600, prev)
        e = e + up
        lam, lp = np.where(e >= 0, cur, 0)[:l + 1], np.where(e >= 0, prev, 0)[:l + 1]
        ea = np.exp2(np.floor(np.log2(np.sqrt((2 * l + 1) / (4 * np.pi)))) + 1)
        rings[0] = max(rings[0], np.abs(lam).sum(1).max())
        cols[0, l & 1, :l + 1] += np.abs(lam) / ea
        if l >= 2:
            mm = m[:l + 1]
            nl = 1 / np.sqrt((l + 2.0) * (l + 1.0) * l * (l - 1.0))
            lf = 2 * np.sqrt((2 * l + 1.0) / (2 * l - 1.0) * (l * l - mm * mm))
            l1 = (lp * lf * z / s ** 2 - lam * (2 * (l - mm * mm) / s ** 2 + l * (l - 1.0))) * nl
            l2 = (lp * lf - lam * 2 * z * (l - 1.0)) * mm / s ** 2 * nl
            rings[1] = max(rings[1], (np.abs(l1) + np.abs(l2)).sum(1).max())
            cols[1, l & 1, :l + 1] += np.abs(l1) / ea
            cols[1, 1 - (l & 1), :l + 1] += np.abs(l2) / ea
    return rings / ns, cols.max((1, 2, 3)) / (lmax // 2 + 1)


@pytest.mark.parametrize("ns", [1, 2, 8, 32, 64])
def test_sums_stay_below_the_integer_units(ns):
    rings, cols = _sums(ns)
    assert rings.max() <= 0.85
    assert cols.max() <= 0.4 or ns < 8        # (the contraction takes nside >= 32)
