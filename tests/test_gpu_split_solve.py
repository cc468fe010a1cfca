"""The split form's blocked solves (sddd_Rpotrs with the split on): orders at
the edges of the 64-blocks, several right-hand sides side by side and in groups.

Every column is bit for bit the same solve alone, and lies within the
componentwise bound of a substitution from the plain form's: each of the two
triangular solves has |dx| <= c n u |L^-1| |L| |x| (u = 2^-104 for dd products
and sums, c = 4 for both forms' sums and the refined diagonal blocks together),
so with y = L^T x the difference is at most
4 n u (|L^-T| |L^T| |x| + |L^-T| |L^-1| |L| |y|)."""
import numpy as np
import pytest

from conftest import DD, load_pkg

pytestmark = pytest.mark.gpu


def solve(c, L, B, slices):
    import torch
    n, k = B.shape
    assert c.L.sddd_set_tc_split(c.h, slices) == 0
    dL = torch.from_numpy(np.ascontiguousarray(L.T).view(np.float64).copy()).cuda()
    dB = torch.from_numpy(np.ascontiguousarray(B.T).view(np.float64).copy()).cuda()
    c.call("sddd_Rpotrs", b"L", n, k, dL.data_ptr(), n, dB.data_ptr(), n)
    return dB.cpu().numpy().view(DD).reshape(k, n).T.copy()


@pytest.mark.parametrize("n,nrhs", [(1, 1), (1, 5), (63, 2), (64, 4), (65, 3), (129, 9), (500, 2), (1000, 4), (9500, 1)])
def test_columns(n, nrhs):
    rng = np.random.default_rng(n + nrhs)
    L, B = np.zeros((n, n), DD), np.zeros((n, nrhs), DD)
    for a in (L, B):
        a["hi"] = rng.uniform(-1, 1, a.shape)
    L["hi"] = np.tril(L["hi"], -1) / np.sqrt(n) + np.diag(rng.uniform(1, 2, n))
    for a in (L, B):
        a["lo"] = a["hi"] * 2.0 ** -54 * rng.uniform(-1, 1, a.shape)
    sddd = load_pkg()
    with sddd.Context(0) as c:
        got = solve(c, L, B, 16)
        if nrhs > 1:
            for j in range(nrhs):
                assert np.array_equal(solve(c, L, B[:, j:j + 1], 16)[:, 0], got[:, j])
        if n > 1000:  # the bound's inverse is too much work: residual of the double parts
            x = got["hi"][:, 0]
            assert np.abs(L["hi"] @ (L["hi"].T @ x) - B["hi"][:, 0]).max() < 1e-10
            return
        want = solve(c, L, B, 0)
    A = np.abs(L["hi"])
    I = np.abs(np.linalg.inv(L["hi"]))
    x = np.abs(want["hi"])
    y = np.abs(L["hi"].T @ want["hi"])
    bound = 4 * n * 2.0 ** -104 * (I.T @ (A.T @ x) + I.T @ (I @ (A @ y)))
    diff = np.abs((got["hi"] - want["hi"]) + (got["lo"] - want["lo"]))
    assert (diff <= bound).all(), (diff / bound).max()
