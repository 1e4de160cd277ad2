"""The emulated form rounds every f once, whatever the slices and the width of the contraction (B200 only).

Inputs under which a record's emp5i is one f: J has one row b, in the block of the largest i alone, T2 one row c in each
block, t1v and dintx one entry, and the denominator is -1/2, so that emp5i = -1/2 (-2 f1n(b, c)) and every other term is
an exact zero.  The last element of each T2 row makes the sum cancel to 2^-12 of its size: then a sum of levels
that is rounded before the last addition shows in the result.  The expected value is the kept digit products added up in
Python's integers and rounded once."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

B, C = 1, 3


def _digits(x, slices):
    """Base-128 digits of a row and its exponent: x = 2^e sum_p d_p 128^-(p+1), |d_p| <= 64."""
    e = int(np.frexp(np.max(np.abs(x)))[1]) + 1
    x = np.ldexp(x, -e)
    out = []
    for _ in range(slices):
        d = np.rint(x * 128.0)
        x = x * 128.0 - d
        out.append(d.astype(np.int64))
    return out, e


def _expected(a, b, slices):
    da, ea = _digits(a, slices)
    db, eb = _digits(b, slices)
    total = 0
    for p in range(slices):
        for q in range(slices - p):
            total += int(np.dot(da[p], db[q])) * 128 ** (slices - 1 - p - q)
    return float(Fraction(total, 128 ** (slices + 1)) * Fraction(2) ** (ea + eb))  # one rounding


def _system(T, nocc, nvir, rng):
    s = T.synth_system(nocc, nvir, seed=1)
    for name in ("jvv", "kvv", "t2", "tov", "xov", "jov", "kov", "dintc", "dintx", "t1v", "eorb"):
        s.arrays[name] = np.zeros_like(s.arrays[name])
    ar, i, vv = s.arrays, nocc - 1, nvir * nvir
    ar["eorb"][s.ncor + nocc:] = 0.5
    ar["eorb"][s.a - 1] = 1.0
    assert s.a - 1 - s.ncor - nocc not in (B, C)
    ar["t1v"][i * nvir + B] = 1.0
    ar["dintx"][i * nvir + C] = 1.0
    row = rng.uniform(-1.0, 1.0, nvir)
    row[C] = 0.0
    row[nvir - 1] = 0.9
    ar["jvv"][i * vv + B:(i + 1) * vv:nvir] = row
    cols = {}
    for j in range(nocc):
        for k in range(nocc - 1):
            t = rng.uniform(-1.0, 1.0, nvir)
            t[nvir - 1] -= (1.0 - 2.0 ** -12) * float(np.dot(row, t)) / row[nvir - 1]
            ar["t2"][(j * nocc + k) * vv + C:(j * nocc + k + 1) * vv:nvir] = t
            cols[j, k] = t
    return s, row, cols


# 7 slices: all levels joined in one integer up to a width of 504, beyond and with 8 slices in two groups
@pytest.mark.parametrize("slices,nocc,nvir", [(4, 6, 50), (5, 6, 51), (7, 6, 50), (7, 4, 476), (7, 4, 477), (7, 3, 797),
                                              (7, 3, 829), (8, 6, 50), (8, 6, 51), (8, 4, 572), (8, 4, 573), (8, 5, 700)])
def test_every_f_is_rounded_once(T, slices, nocc, nvir):
    rng = np.random.default_rng(1000 * slices + nvir)
    s, row, cols = _system(T, nocc, nvir, rng)
    with T.Plan([s], mode=T.MODE_EMULATED, slices=slices) as p:
        p.upload()
        p.execute()
        rec, ijk = p.triple_energies(0), p.triples(0)
    n = 0
    for t, (i, j, k) in enumerate(ijk):
        if i != nocc or k == nocc:
            continue
        assert rec[t, 1] == _expected(row, cols[j - 1, k - 1], slices), (i, j, k)
        n += 1
    assert n == nocc * (nocc - 1)
