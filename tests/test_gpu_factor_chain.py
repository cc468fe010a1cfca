"""The factorisations' and solves' latency chains (the diagonal block's pivot
warp and helpers, the corrected quotients of fastdiv.cuh) against the oracle's
plain loops, bit for bit: orders at the edges of the helpers' columns and of
the 64-blocks, values inside and outside the corrected quotients' range,
failing pivots."""
import ctypes

import numpy as np
import pytest

from conftest import as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu

L_ = ctypes.c_long


@pytest.fixture(scope="module")
def ctx():
    with load_pkg().Context(0) as c:
        yield c


def _spd(rng, n, spread):
    """Column-major dd SPD matrix; row and column i scaled by 2^s_i,
    |s_i| <= spread, s_i an integer."""
    G = rng.standard_normal((n, n))
    A = G @ G.T / n + 0.05 * np.eye(n)
    s = 2.0 ** rng.integers(-spread, spread + 1, n)
    A = A * s[:, None] * s[None, :]
    out = as_dd(A.T.ravel())
    lo = rng.uniform(-0.5, 0.5, (n, n)) * 2.0 ** -53
    out["lo"] = out["hi"] * (np.triu(lo) + np.triu(lo, 1).T).ravel()
    return out


def _device(a):
    import torch
    return torch.from_numpy(a.view(np.float64).reshape(-1, 2).copy()).cuda()


def _host(t, like):
    return t.cpu().numpy().view(like.dtype).reshape(like.shape)


def _lower(a, n):
    return a.reshape(n, n).T[np.tril_indices(n)]


@pytest.mark.parametrize("spread", [0, 150, 230])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 25, 26, 27, 31, 32, 33, 49, 50, 51, 63, 64, 65, 130])
def test_potrf_bits(ctx, oracle_lib, n, spread):
    rng = np.random.default_rng(1000 * n + spread)
    A = _spd(rng, n, spread)
    want = A.copy()
    oracle_lib.o_potrf.restype = L_
    assert oracle_lib.o_potrf(L_(n), ptr(want), L_(n)) == 0
    d = _device(A)
    assert ctx.call("sddd_Rpotrf", b"L", n, d.data_ptr(), n) == 0
    assert np.array_equal(_lower(_host(d, A), n), _lower(want, n))


@pytest.mark.parametrize("n,col", [(1, 0), (5, 1), (40, 26), (64, 2), (64, 63), (70, 64), (130, 70)])
@pytest.mark.parametrize("bad", [-1.0, 0.0, float("nan")])
def test_potrf_failing_column(ctx, n, col, bad):
    A = as_dd(np.eye(n).ravel())
    A["hi"][col * (n + 1)] = bad
    d = _device(A)
    assert ctx.call("sddd_Rpotrf", b"L", n, d.data_ptr(), n) == col + 1


@pytest.mark.parametrize("n", [1, 20, 33, 64])
def test_batched_blocks_bits(oracle_lib, n):
    """Equal blocks factored one CTA each (the inverses of X and Z)."""
    sddd = load_pkg()
    rng = np.random.default_rng(n)
    blocks = [_spd(rng, n, 3) for _ in range(5)]
    with sddd.Context(0) as c:
        c.upload(1, [n] * 5, as_dd(np.ones(1)), [1], [1], [1], [1], as_dd(np.ones(1)))
        X = np.concatenate(blocks)
        assert c.set_point(X, as_dd(np.zeros(1)), X) == 0
        got = c.get("invCholX").reshape(5, n * n)
    for A, g in zip(blocks, got):
        L, inv = A.copy(), np.zeros_like(A)
        oracle_lib.o_potrf.restype = L_
        assert oracle_lib.o_potrf(L_(n), ptr(L), L_(n)) == 0
        oracle_lib.o_inv_lower(L_(n), ptr(L), L_(n), ptr(inv), L_(n))
        assert np.array_equal(_lower(g, n), _lower(inv, n))


def _factor(oracle_lib, rng, n, spread):
    L = _spd(rng, n, spread)
    oracle_lib.o_potrf.restype = L_
    assert oracle_lib.o_potrf(L_(n), ptr(L), L_(n)) == 0
    return L


@pytest.mark.parametrize("spread", [0, 200])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 330])
def test_trsv_bits(ctx, oracle_lib, n, spread):
    """Entries of x that are zero and stay zero among the others: the forward
    solve skips them."""
    rng = np.random.default_rng(7000 + n + spread)
    L = _factor(oracle_lib, rng, n, spread)
    x0 = as_dd(rng.standard_normal(n))
    x0["lo"] = x0["hi"] * 2.0 ** -55
    x0[: n // 3] = (0.0, 0.0)
    d = _device(L)
    for trans in "NT":
        want = x0.copy()
        oracle_lib.o_trsv(ctypes.c_char(trans.encode()), L_(n), ptr(L), L_(n), ptr(want))
        x = _device(x0)
        ctx.call("sddd_Rtrsv", b"L", trans.encode(), b"N", n, d.data_ptr(), n, x.data_ptr(), 1)
        assert np.array_equal(_host(x, x0), want), trans


@pytest.mark.parametrize("n,nrhs", [(1, 1), (64, 2), (65, 3), (200, 8), (130, 9)])
def test_potrs_bits(ctx, oracle_lib, n, nrhs):
    """Right-hand sides in groups side by side, their columns ldb apart."""
    rng = np.random.default_rng(n * nrhs)
    L = _factor(oracle_lib, rng, n, 0)
    ldb = n + 3
    B = as_dd(rng.standard_normal((nrhs, ldb)))
    want = B.copy()
    for r in range(nrhs):
        x = np.ascontiguousarray(want[r, :n])
        for trans in (b"N", b"T"):
            oracle_lib.o_trsv(ctypes.c_char(trans), L_(n), ptr(L), L_(n), ptr(x))
        want[r, :n] = x
    dL, dB = _device(L), _device(B)
    ctx.call("sddd_Rpotrs", b"L", n, nrhs, dL.data_ptr(), n, dB.data_ptr(), ldb)
    assert np.array_equal(_host(dB, B), want)
