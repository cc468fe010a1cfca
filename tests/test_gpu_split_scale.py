"""The split trailing update on rows whose largest entry lies just below a
power of two: their scale is one bit larger than that of other rows, and their
small entries keep the bits that 16 slices promise all the same.

One or two columns, random significands (so that every digit counts), and C the
dd product itself, so that what is left is the split's own error.  Bound in
units of 2^(E_i+E_j), max|row| < 2^E, scale 2^(E+2) or 2^(E+1) (a factor of at
most 16), a column: diagonals past the 16th, 14 products of two digits up to
128, 14 2^14 2^-136 (1 + 2^-8) = 2^-118.2; the operands' truncation at 2^-120 in
each half, 2 (1/4) 2^-119 = 2^-120; two roundings by 2^-53 of the small groups,
at most 9.04 2^14 2^24 2^-104 = 2^-62.8: 2^-114.8.  Together below 16 2^-114.6 <
2^-110.5; then the dd rounding, 2^-103 of the result."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from conftest import DD, load_pkg

pytestmark = pytest.mark.gpu


def _frac(x):
    return Fraction(float(x["hi"])) + Fraction(float(x["lo"]))


def _dd(f):
    hi = float(f)
    return hi, float(f - Fraction(hi))


@pytest.mark.parametrize("k", [1, 2])
@pytest.mark.parametrize("top", [0.99, 0.9961, 0.998, 0.9999999])
def test_rows_below_a_power_of_two(top, k):
    import torch
    sddd = load_pkg()
    n = 140
    rng = np.random.default_rng(int(top * 1e7) + k)
    P = np.zeros((n, k), DD)
    P["hi"] = rng.uniform(-1, 1, (n, k)) * 0.9
    # every significand random to its last bit, the largest entry of a row just above `top`
    P["hi"][:, 0] = rng.choice([-1.0, 1.0], n) * rng.uniform(top, top + 0.01 * (1 - top), n) * np.exp2(rng.integers(-3, 4, n))
    if k == 2:
        P["hi"][:, 1] *= P["hi"][:, 0] * np.exp2(-rng.integers(0, 40, n))
    P["lo"] = P["hi"] * rng.uniform(-1, 1, (n, k)) * 2.0 ** -54
    Pf = [[_frac(P[i, q]) for q in range(k)] for i in range(n)]
    E = [int(np.frexp(np.abs(P["hi"][i]).max())[1]) for i in range(n)]
    prod = [[sum(a * b for a, b in zip(Pf[i], Pf[j])) for j in range(i + 1)] for i in range(n)]
    C = np.zeros((n, n), DD)
    for i in range(n):
        for j in range(i + 1):
            C[i, j] = _dd(prod[i][j])
    dP = torch.from_numpy(np.ascontiguousarray(P.T).view(np.float64).copy()).cuda()
    dC = torch.from_numpy(np.ascontiguousarray(C.T).view(np.float64).copy()).cuda()
    with sddd.Context(0) as c:
        assert c.L.sddd_Rsyrk_tc(c.h, n, k, ctypes.c_void_p(dP.data_ptr()), n, ctypes.c_void_p(dC.data_ptr()), n, 16) == 0
    got = dC.cpu().numpy().view(DD).reshape(n, n).T
    for i in range(n):
        for j in range(i + 1):
            want = _frac(C[i, j]) - prod[i][j]
            err = abs(_frac(got[i, j]) - want)
            unit = Fraction(2) ** (E[i] + E[j])
            assert err <= k * unit * Fraction(3, 2 ** 112) + abs(want) / 2 ** 103, (i, j, float(err / unit) * 2.0 ** 111)
