"""The step-length eigenvalue (eig.cu) at the edges of its forms: the Lanczos
kernel's 8-row chunks and cluster sizes against the oracle's Lanczos, and the
small blocks' tridiagonal solver against mpmath, with decoupled rows.

Tolerance, both: 1e-25 of the spectrum's scale, the bar of the reference
comparisons (the sums of n <= 520 dd products of the five chains carry about
n 2^-104 = 3e-29 of the scale)."""
import ctypes

import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu


def _min_eig(n, L, D):
    import torch
    lib = load_pkg().lib()
    t = [torch.from_numpy(np.ascontiguousarray(a).view(np.float64).copy()).cuda() for a in (L, D)]
    out = torch.full((2,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.sddd_min_eig_noalloc(None, n, t[0].data_ptr(), t[1].data_ptr(), out.data_ptr()) == 0
    torch.cuda.synchronize()
    return tuple(out.cpu().numpy())


def _pair(rng, n):
    A = rng.standard_normal((n, n))
    L = np.linalg.cholesky(A @ A.T / n + 0.1 * np.eye(n))
    S = rng.standard_normal((n, n))
    D = as_dd((S + S.T).ravel())
    lo = rng.uniform(-0.5, 0.5, (n, n)) * 2.0 ** -53
    D["lo"] = D["hi"] * (np.triu(lo) + np.triu(lo, 1).T).ravel()
    return as_dd(L.T.ravel()), D


@pytest.mark.parametrize("n", [21, 24, 25, 32, 33, 64, 65, 97, 128, 129, 192, 193, 520])
def test_lanczos_matches_oracle(oracle_lib, n):
    class ODD(ctypes.Structure):
        _fields_ = [("hi", ctypes.c_double), ("lo", ctypes.c_double)]
    oracle_lib.o_lanczos_min_eig.restype = ODD
    L, D = _pair(np.random.default_rng(100 + n), n)
    want = oracle_lib.o_lanczos_min_eig(ctypes.c_long(n), ptr(L), ptr(D))
    got = _min_eig(n, L, D)
    assert abs((got[0] - want.hi) + (got[1] - want.lo)) <= 1e-25 * abs(want.hi), (got, want.hi, want.lo)


@pytest.mark.parametrize("kind", ["dense", "diagonal", "blocks", "ties"])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 19, 20])
def test_small_block_matches_mpmath(n, kind):
    import mpmath
    rng = np.random.default_rng(7 * n + len(kind))
    S = rng.standard_normal((n, n))
    S = S + S.T
    if kind == "diagonal":
        S = np.diag(np.diag(S))
    elif kind == "blocks":
        S[: n // 2, n // 2:] = 0.0
        S[n // 2:, : n // 2] = 0.0
    elif kind == "ties":
        S = np.ones((n, n)) - 2.0 * np.eye(n)
    L = np.zeros(n * n, DD)
    L["hi"][:: n + 1] = 1.0
    got = _min_eig(n, L, as_dd(S.ravel()))
    with mpmath.workdps(60):
        E = mpmath.eigsy(mpmath.matrix(S.tolist()), eigvals_only=True)
        scale = max(abs(x) for x in E)
        assert abs(mpmath.mpf(float(got[0])) + mpmath.mpf(float(got[1])) - min(E)) <= mpmath.mpf(10) ** -25 * scale, (got, min(E))
