"""CPU model of the split X-stage's epilogue: the register sums W[s1][s2] of every stream pair go into two halves of the
staging area, [baseline x product][channels], and the output is the mean of W[s1][s2] and conj(W[s2][s1]).  Each value of
each half is written exactly once, and the means are the Gram sums of every baseline and product."""
import numpy as np
import pytest


def _baseline(j, k, nant):
    """Output row of antennas j <= k: crosses first, then the autocorrelations (baseline_index of csrc/gxc_internal.h)."""
    return nant * (nant - 1) // 2 + j if j == k else j * nant - j * (j + 1) // 2 + (k - j - 1)


@pytest.mark.parametrize("autos", [True, False])
@pytest.mark.parametrize("nant", list(range(1, 33)))
def test_halves_hold_every_pair_once(nant, autos):
    n = 2 * nant
    nbl = nant * (nant - 1) // 2 + (nant if autos else 0)
    nent = nbl * 4
    R = 16
    while R < 2 * n:
        R *= 2
    CS = 2 * (128 // R)                           # channels of a CTA: two groups of 128 / R
    assert 2 * nent * CS * 8 <= 2 * 65536         # the operand ring: two stages of 64 KiB
    rng = np.random.default_rng(nant)
    D = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))  # not symmetric, as hi.hi + 2 lo.hi
    staged = np.full(2 * nent, np.nan, complex)
    writes = np.zeros(2 * nent, int)
    for s1 in range(n):
        for s2 in range(n):
            j, l, k, m = s1 >> 1, s1 & 1, s2 >> 1, s2 & 1
            if j == k and not autos:
                continue
            bl4 = 4 * _baseline(min(j, k), max(j, k), nant)
            at = [(0 if j <= k else nent) + bl4 + (2 * l + m if j <= k else 2 * m + l)]
            if j == k:
                at.append(nent + bl4 + 2 * m + l)
            for a in at:
                staged[a] = D[s1, s2]
                writes[a] += 1
    assert (writes == 1).all()
    for j in range(nant):
        for k in range(j if autos else j + 1, nant):
            for l in range(2):
                for m in range(2):
                    e = _baseline(j, k, nant) * 4 + 2 * l + m
                    g = 0.5 * staged[e] + 0.5 * np.conj(staged[nent + e])
                    assert abs(g - (D[2 * j + l, 2 * k + m] + np.conj(D[2 * k + m, 2 * j + l])) / 2) < 1e-15
