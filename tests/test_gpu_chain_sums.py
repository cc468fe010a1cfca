"""The ordered sums formed by one CTA (devops.cuh cta_chain) at the edges of
their chunks: C.X over a sparse C and over small dense C's, and b.y, against
the same "+=" chains of the host's dd arithmetic, bit for bit."""
import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu


def _op(lib, op, a, b):
    out = np.zeros(len(a), DD)
    assert lib.sddd_host_dd_op(op, len(a), ptr(a), ptr(b), ptr(out)) == 0
    return out


def _chain(lib, terms):
    acc = np.zeros(1, DD)
    for t in range(len(terms)):
        acc = _op(lib, 1, acc, terms[t:t + 1])
    return acc


def _full(rng, shape):
    hi = rng.standard_normal(shape)
    out = as_dd(hi)
    out["lo"] = hi * rng.uniform(-1, 1, shape) * 2.0 ** -54
    return out


def _solver(sddd, n, m, ci, cj, cv, b, rng):
    """One block of order n: C entries (ci <= cj), constraint k = one entry."""
    ctx = sddd.Context(0)
    d = np.arange(m) % n
    k = np.concatenate([np.zeros(len(ci), int), 1 + np.arange(m)])
    i, j = np.concatenate([ci, d]) + 1, np.concatenate([cj, d]) + 1
    ctx.upload(m, [n], b, k, np.ones(len(k), int), i, j, np.concatenate([cv, as_dd(np.ones(m))]))
    X = _full(rng, (n, n))
    y = _full(rng, m)
    ctx.set("X", X.T.ravel())
    ctx.set("y", y)
    return ctx, X, y


@pytest.mark.parametrize("nnz", [1, 3, 4, 7, 2044, 2047, 2048, 2052, 4101])
def test_sparse_c_product(nnz):
    sddd = load_pkg()
    rng = np.random.default_rng(nnz)
    n = 150
    iu, ju = np.triu_indices(n)
    at = rng.permutation(len(iu))[:nnz]  # any order: the sum follows the input's
    ci, cj, cv = iu[at], ju[at], _full(rng, nnz)
    ctx, X, _ = _solver(sddd, n, 2, ci, cj, cv, as_dd(np.ones(2)), rng)
    with ctx:
        got = ctx.dd_scalar("sddd_inner", 0)
        lib = ctx.L
        v = _op(lib, 14, cv, cv)  # C = -F_0
        off = _op(lib, 4, v, _op(lib, 0, X[ci, cj], X[cj, ci]))
        t = np.where(ci == cj, _op(lib, 4, v, X[ci, ci]), off)
        r, g = nnz % 4, t[nnz % 4:].reshape(-1, 4)
        groups = _op(lib, 0, _op(lib, 0, _op(lib, 0, *(np.ascontiguousarray(g[:, c]) for c in (0, 1))), np.ascontiguousarray(g[:, 2])),
                     np.ascontiguousarray(g[:, 3])) if len(g) else np.zeros(0, DD)
        want = _chain(lib, np.concatenate([t[:r], groups]))[0]
    assert got == (want["hi"], want["lo"]), (got, want)


@pytest.mark.parametrize("n", [1, 5, 22, 23, 32])
def test_dense_c_product(n):
    sddd = load_pkg()
    rng = np.random.default_rng(n)
    ci, cj = np.triu_indices(n)
    cv = _full(rng, len(ci))
    ctx, X, _ = _solver(sddd, n, 2, ci, cj, cv, as_dd(np.ones(2)), rng)
    with ctx:
        got = ctx.dd_scalar("sddd_inner", 0)
        lib = ctx.L
        C = np.zeros((n, n), DD)
        C[ci, cj] = C[cj, ci] = _op(lib, 14, cv, cv)
        want = _chain(lib, _op(lib, 4, np.ascontiguousarray(C.T.ravel()), np.ascontiguousarray(X.T.ravel())))[0]
    assert got == (want["hi"], want["lo"]), (got, want)


@pytest.mark.parametrize("m", [1, 8, 511, 512, 513, 1023, 1024])
def test_vector_dot(m):
    sddd = load_pkg()
    rng = np.random.default_rng(m)
    b = _full(rng, m)
    ctx, _, y = _solver(sddd, 30, m, np.array([0]), np.array([0]), as_dd(np.ones(1)), b, rng)
    with ctx:
        got = ctx.dd_scalar("sddd_inner", 1)
        want = _chain(ctx.L, _op(ctx.L, 4, b, y))[0]
    assert got == (want["hi"], want["lo"]), (got, want)
