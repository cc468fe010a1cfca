"""Forward triangular solves whose zero entries of x start and end inside the
64-entry blocks and change from one block to the next, against the oracle's
loop, bit for bit.  The loop skips the column of a zero entry altogether, so
those columns hold NaN below the diagonal: a step that is not skipped, or a
skip that belongs to another block, shows."""
import ctypes

import numpy as np
import pytest

from conftest import as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu

L_ = ctypes.c_long


def _zero_rows(rng, n, pattern):
    """Rows of the solution that are zero."""
    i = np.arange(n)
    if pattern == "blocks":  # every other block
        return (i // 64) % 2 == 0
    if pattern == "halves":  # the other half in the next block
        return (i // 32) % 4 < 2
    if pattern == "first":  # a unit vector
        return i < n - 5
    z = np.zeros(n, bool)  # runs of odd lengths
    at = 0
    while at < n:
        run = int(rng.integers(1, 70))
        z[at:at + run] = rng.random() < 0.5
        at += run
    return z


def _factor(rng, n, zero):
    """Lower triangle whose rows couple only to rows of the same kind, so that
    the rows marked zero stay zero for a right-hand side that is zero there."""
    M = rng.standard_normal((n, n)) / n
    M[zero[:, None] != zero[None, :]] = 0.0
    M = np.tril(M, -1) + np.diag(rng.uniform(0.5, 2.0, n))
    L = as_dd(M.T.ravel())
    L["lo"] = L["hi"] * 2.0 ** -55
    return L


@pytest.mark.parametrize("pattern", ["blocks", "halves", "first", "runs"])
@pytest.mark.parametrize("n", [64, 100, 330, 1327])
def test_forward_solve_skips_zero_entries(oracle_lib, n, pattern):
    import torch
    sddd = load_pkg()
    rng = np.random.default_rng(n + len(pattern))
    zero = _zero_rows(rng, n, pattern)
    L = _factor(rng, n, zero)
    x0 = as_dd(np.where(zero, 0.0, rng.standard_normal(n)))
    want = x0.copy()
    oracle_lib.o_trsv(ctypes.c_char(b"N"), L_(n), ptr(L), L_(n), ptr(want))
    assert np.array_equal(want["hi"] == 0.0, zero)
    both = want.copy()
    oracle_lib.o_trsv(ctypes.c_char(b"T"), L_(n), ptr(L), L_(n), ptr(both))
    planted = L.reshape(n, n).copy()  # planted[j, i] = L(i, j)
    planted["hi"][zero[:, None] & (np.arange(n)[None, :] > np.arange(n)[:, None])] = np.nan
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.float64).reshape(-1, 2).copy()).cuda()
    host = lambda t: t.cpu().numpy().view(x0.dtype).reshape(-1)
    dL, dP = dev(L), dev(planted)
    with sddd.Context(0) as c:
        for _ in range(10):
            x = dev(x0)
            c.call("sddd_Rtrsv", b"L", b"N", b"N", n, dP.data_ptr(), n, x.data_ptr(), 1)
            assert np.array_equal(host(x), want)
        # right-hand sides side by side, each with its own zeros
        B = np.stack([x0, as_dd(rng.standard_normal(n)), x0])
        sol = np.stack([both, B[1], both])
        for trans in (b"N", b"T"):
            r = np.ascontiguousarray(sol[1])
            oracle_lib.o_trsv(ctypes.c_char(trans), L_(n), ptr(L), L_(n), ptr(r))
            sol[1] = r
        dB = dev(B)
        c.call("sddd_Rpotrs", b"L", n, 3, dL.data_ptr(), n, dB.data_ptr(), n)
        assert np.array_equal(host(dB).reshape(3, n), sol)
