"""The forms of the small dd products (tile16.cuh: 16 steps a chunk; the
pipelined loop up to 296 tiles, the unrolled one above; all four transposes) and
of the stacked F and G products (tiles of 40 to 64 columns), against the
oracle's loops, bit for bit."""
import ctypes

import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu

L_ = ctypes.c_long


def _full(rng, size):
    out = as_dd(rng.standard_normal(size))
    out["lo"] = out["hi"] * rng.uniform(-1, 1, size) * 2.0 ** -54
    return out


def _device(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.float64).reshape(-1, 2).copy()).cuda()


# 33 x 20: 6 tiles; 270 x 271: 289 tiles, pipelined; 275 x 276: 324 tiles, unrolled; 1200 x 7: thin, 75 tiles
@pytest.mark.parametrize("ta,tb", ["NN", "TN", "NT", "TT"])
@pytest.mark.parametrize("m,n", [(33, 20), (270, 271), (275, 276), (1200, 7), (4801, 9)])
@pytest.mark.parametrize("k", [1, 15, 16, 17, 33])
def test_rgemm_forms(oracle_lib, m, n, k, ta, tb):
    sddd = load_pkg()
    rng = np.random.default_rng(m + 100 * n + 10000 * k)
    A, B = _full(rng, m * k), _full(rng, k * n)
    lda, ldb = (m if ta == "N" else k), (k if tb == "N" else n)
    want = np.zeros(m * n, DD)
    # the oracle's loop has no "TT": the same terms in the same order as "TN" with B transposed
    Bo, to, ldo = (np.ascontiguousarray(B.reshape(k, n).T), "N", k) if ta + tb == "TT" else (B, tb, ldb)
    oracle_lib.o_gemm(ctypes.c_char(ta.encode()), ctypes.c_char(to.encode()), L_(m), L_(n), L_(k), ptr(A), L_(lda), ptr(Bo), L_(ldo), ptr(want), L_(m))
    dA, dB, dC = _device(A), _device(B), _device(_full(rng, m * n))
    with sddd.Context(0) as ctx:
        ctx.call("sddd_Rgemm", ta.encode(), tb.encode(), m, n, k, sddd.SdddDD(1.0, 0.0), dA.data_ptr(), lda, dB.data_ptr(), ldb, sddd.SdddDD(0.0, 0.0),
                 dC.data_ptr(), m)
    assert np.array_equal(dC.cpu().numpy().view(DD).reshape(-1), want)


@pytest.mark.parametrize("n,m", [(32, 310), (41, 240), (48, 210), (57, 170), (64, 150), (65, 80)])
def test_stacked_products(oracle_lib, workdir, n, m):
    import importlib
    sddd = load_pkg()
    P = importlib.import_module("sdpa_dd_b200.problems")
    import sdpa_problem
    text = P.dense_random(n=n, m=m, seed=n)
    path = workdir / f"stack_{n}_{m}.dat-s"
    path.write_text(text)
    rng = np.random.default_rng(n + m)

    def spd():
        G = rng.standard_normal((n, n))
        out = as_dd((G @ G.T / n + np.eye(n)).ravel())
        lo = rng.uniform(-0.5, 0.5, (n, n)) * 2.0 ** -53
        out["lo"] = out["hi"] * (np.triu(lo) + np.triu(lo, 1).T).ravel()
        return out
    X, Z = spd(), spd()
    with sddd.Context(0) as ctx:
        ctx.read_problem(path)
        assert (ctx.formula() != 2).all()
        assert ctx.set_point(X, as_dd(np.zeros(m)), Z) == 0
        ctx.call("sddd_schur_build")
        B, Zi = ctx.get("B"), ctx.get("invZ")
    want = sdpa_problem.schur(sdpa_problem.Problem(oracle_lib, text), [X], [Zi])
    assert np.array_equal(B.view(np.float64).ravel() + 0.0, want.view(np.float64).ravel() + 0.0)
