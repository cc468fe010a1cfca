"""The digits of the split trailing update, sddd_Rsyrk_tc, against exact
integer arithmetic where they can go wrong: orders around the 16- and 128-row
tiles, every slice count, row maxima at both sides of the exponent's step
(0.996 of a power of two) and of equal magnitude and sign in every column (the
largest diagonals), entries down to the digits' last bit, and row scales whose
products lie at the ends of the exponent range.

Bound for S slices carried by B = ceil(7S/8) base-256 digits, M the row
maxima: |P| 2^-e <= 1/2 and M 2^-e > 0.249, so in units of M_i M_j (16.2 of
2^(e_i+e_j)): the operands' remainders 2 (1/2) 2^-(8B+1) (1 + 2^-6) a term, the
dropped diagonals (B-1) 2^14 2^-8(B+2) / (1 - 2^-8) a term: k 2^-8B
16.2 (0.51 + (B-1)/3.98) < k 2^-(8B-6).  Beyond that the dd rounding: 2^-103
of the result, 2^-107 of M_i M_j for the small groups' sum, and half an ulp of
a subnormal.
"""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from conftest import DD, load_pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    sddd = load_pkg()
    c = sddd.Context(0)
    yield c
    c.close()


def ints(a, scale):
    """dd array -> integers (value * 2^scale)"""
    out = np.empty(a.shape, dtype=object)
    for q in np.ndindex(a.shape):
        f = Fraction(float(a[q]["hi"])) + Fraction(float(a[q]["lo"]))
        f *= Fraction(2) ** scale
        assert f.denominator == 1
        out[q] = f.numerator
    return out


def run(ctx, P, C, slices):
    import torch
    n, k = P.shape
    dP = torch.from_numpy(np.ascontiguousarray(P.T).view(np.float64).copy()).cuda()
    dC = torch.from_numpy(np.ascontiguousarray(C.T).view(np.float64).copy()).cuda()
    rc = ctx.L.sddd_Rsyrk_tc(ctx.h, n, k, ctypes.c_void_p(dP.data_ptr()), n, ctypes.c_void_p(dC.data_ptr()), n, slices)
    assert rc == 0, ctx.L.sddd_last_error(ctx.h)
    return dC.cpu().numpy().view(DD).reshape(n, n).T.copy()


def check(P, C, got, slices, scale):
    n, k = P.shape
    B = (7 * slices + 7) // 8
    Pi, Ci, Gi = ints(P, scale), ints(C, scale), ints(got, scale)
    M = [max(abs(x) for x in Pi[i]) for i in range(n)]
    for i in range(n):
        for j in range(n):
            if i < j:
                assert got[i, j] == C[i, j], (i, j)
                continue
            want = Ci[i, j] * 2 ** scale - sum(a * b for a, b in zip(Pi[i], Pi[j]))
            err = abs(Gi[i, j] * 2 ** scale - want)
            mm = M[i] * M[j]
            bound = Fraction(mm) * (Fraction(k, 2 ** (8 * B - 6)) + Fraction(1, 2 ** 107)) + Fraction(abs(want), 2 ** 103) + 2 * Fraction(2) ** (
                2 * scale - 1075)
            assert err <= bound, (i, j, float(Fraction(err) / bound))


def make(rng, n, k, kind):
    P = np.zeros((n, k), DD)
    if kind == "step":  # row maxima around 0.996 of a power of two
        hi = rng.uniform(-0.9, 0.9, (n, k))
        hi[np.arange(n), rng.integers(0, k, n)] = rng.choice([0.9955, 0.99599, 0.99601, 0.9999999, 1.0, -0.99601, -1.0, np.nextafter(1.0, 0)], n)
    elif kind == "flat":  # one magnitude and sign: every product adds up
        hi = np.full((n, k), -0.9959)
    else:
        hi = rng.standard_normal((n, k)) * np.exp2(-rng.integers(0, 100, (n, k)))
    P["hi"] = hi
    P["lo"] = hi * rng.uniform(-1, 1, (n, k)) * 1e-17
    C = np.zeros((n, n), DD)
    C["hi"] = rng.standard_normal((n, n))
    C["lo"] = C["hi"] * rng.uniform(-1, 1, (n, n)) * 1e-17
    return P, C


@pytest.mark.parametrize("n,k", [(1, 1), (15, 64), (16, 3), (17, 64), (127, 5), (128, 64), (129, 17), (145, 64), (257, 16)])
def test_orders(ctx, n, k):
    P, C = make(np.random.default_rng(n), n, k, "spread")
    check(P, C, run(ctx, P, C, 16), 16, 340)


@pytest.mark.parametrize("slices", range(8, 17))
@pytest.mark.parametrize("kind", ["step", "flat", "spread"])
def test_slice_counts(ctx, slices, kind):
    P, C = make(np.random.default_rng(slices), 40, 64, kind)
    check(P, C, run(ctx, P, C, slices), slices, 340)


@pytest.mark.parametrize("shift", [-530, -470, -455, 380, 490, 504])
def test_exponent_range(ctx, shift):
    """Products near 2^(2 shift): the scaled form's limits and beyond them."""
    P, C = make(np.random.default_rng(5), 33, 4, "step")
    for x, s in ((P, shift), (C, 2 * shift)):
        x["hi"] = np.ldexp(x["hi"], s)
        x["lo"] = np.ldexp(x["lo"], s)
    got = run(ctx, P, C, 16)
    check(P, C, got, 16, 1140)
