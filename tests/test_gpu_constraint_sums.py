"""The sums over the constraints' matrices (newton.cu) at the edges of their
tasks and chunks: A_k . M (dense matrices by groups of 32, 32 terms at a time;
sparse ones by task or by thread) and sum_k y_k A_k, through the residuals,
against the same chains of the host's dd arithmetic, bit for bit."""
import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu


def _op(lib, op, a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    out = np.zeros(a.shape, DD)
    assert lib.sddd_host_dd_op(op, a.size, ptr(a), ptr(b), ptr(out)) == 0
    return out


def _fold(lib, terms):
    """Rows of terms summed along the first axis in order, with "+="."""
    acc = np.zeros(terms.shape[1:], DD)
    for t in terms:
        acc = _op(lib, 1, acc, t)
    return acc


def _full(rng, shape):
    out = as_dd(rng.standard_normal(shape))
    out["lo"] = out["hi"] * rng.uniform(-1, 1, shape) * 2.0 ** -54
    return out


def _sym(rng, n):
    S = _full(rng, (n, n))
    iu = np.triu_indices(n, 1)
    S.T[iu] = S[iu]
    return S


def _residuals(ctx, sizes, m, mats, X, y, Z, rng):
    """Uploads constraints mats[k] = {block: (kind, matrix or (i, j, v))}."""
    cols = [[], [], [], [], []]
    for k, bs in enumerate(mats):
        for l, (kind, d) in sorted(bs.items()):
            i, j, v = d if kind == "sparse" else (*np.triu_indices(sizes[l]), d[np.triu_indices(sizes[l])])
            for c, a in zip(cols, (np.full(len(i), k + 1), np.full(len(i), l + 1), i + 1, j + 1, v)):
                c.append(a)
    b = _full(rng, m)
    ctx.upload(m, sizes, b, *(np.concatenate(c) for c in cols))
    ctx.set("X", np.concatenate([x.T.ravel() for x in X]))
    ctx.set("Z", np.concatenate([z.T.ravel() for z in Z]))
    ctx.set("y", y)
    import ctypes
    p, d = load_pkg().SdddDD(), load_pkg().SdddDD()
    ctx.call("sddd_residuals", ctypes.byref(p), ctypes.byref(d))
    return b, ctx.get("primalVec"), ctx.get("dualMat")


def _sparse_dot(lib, i, j, v, M):
    t = _op(lib, 4, v, _op(lib, 0, M[i, j], M[j, i]))
    t = np.where(i == j, _op(lib, 4, v, M[i, j]), t)
    r, g = len(t) % 4, t[len(t) % 4:].reshape(-1, 4)
    groups = _op(lib, 0, _op(lib, 0, _op(lib, 0, g[:, 0], g[:, 1]), g[:, 2]), g[:, 3]) if len(g) else g[:, 0]
    return _fold(lib, np.concatenate([t[:r], groups])[:, None])[0]


@pytest.mark.parametrize("sizes,m", [([1], 1), ([4], 3), ([5], 31), ([6], 32), ([8], 33), ([9, 11], 40), ([17], 65), ([3, 16, 3], 20)])
def test_dense_constraints(sizes, m):
    sddd = load_pkg()
    rng = np.random.default_rng(m)
    mats = [{l: ("dense", _sym(rng, n)) for l, n in enumerate(sizes)} for _ in range(m)]
    X, Z, y = [_sym(rng, n) for n in sizes], [_sym(rng, n) for n in sizes], _full(rng, m)
    with sddd.Context(0) as ctx:
        b, prim, dual = _residuals(ctx, sizes, m, mats, X, y, Z, rng)
        lib = ctx.L
        one, mone = as_dd(np.ones(m)), as_dd(-np.ones(m))
        ret = np.zeros(m, DD)
        for l, n in enumerate(sizes):
            A = np.stack([mats[k][l][1].T.ravel() for k in range(m)], axis=1)  # n^2 x m
            x = np.broadcast_to(X[l].T.ravel()[:, None], A.shape)
            ret = _op(lib, 1, ret, _op(lib, 1, np.zeros(m, DD), _fold(lib, _op(lib, 4, A, x))))
        want = _op(lib, 1, _op(lib, 4, mone, ret), _op(lib, 4, one, b))
        assert np.array_equal(prim, want)
        off = 0
        for l, n in enumerate(sizes):
            A = np.stack([mats[k][l][1].T.ravel() for k in range(m)])
            acc = _fold(lib, _op(lib, 4, A, np.broadcast_to(y[:, None], A.shape)))
            r = _op(lib, 4, as_dd(-np.ones(n * n)), acc)
            r = _op(lib, 1, r, _op(lib, 4, as_dd(-np.ones(n * n)), Z[l].T.ravel()))
            assert np.array_equal(dual[off:off + n * n], r), l
            off += n * n


@pytest.mark.parametrize("m", [3, 300])
def test_sparse_constraints(m):
    """Sums of 1 to 43 steps; 300 long ones are more than the tasks take."""
    sddd = load_pkg()
    rng = np.random.default_rng(m)
    n = 40
    iu, ju = np.triu_indices(n)
    X, Z, y = [_sym(rng, n)], [_sym(rng, n)], _full(rng, m)
    mats = []
    for k in range(m):
        nnz = int(rng.integers(30, 160)) if m > 100 else [1, 31, 159][k]
        at = np.sort(rng.permutation(len(iu))[:nnz])
        mats.append({0: ("sparse", (iu[at], ju[at], _full(rng, nnz)))})
    with sddd.Context(0) as ctx:
        b, prim, _ = _residuals(ctx, [n], m, mats, X, y, Z, rng)
        lib = ctx.L
        ret = np.array([_op(lib, 1, np.zeros(1, DD), _sparse_dot(lib, *mats[k][0][1], X[0])[None])[0] for k in range(m)], DD)
        want = _op(lib, 1, _op(lib, 4, as_dd(-np.ones(m)), ret), _op(lib, 4, as_dd(np.ones(m)), b))
    assert np.array_equal(prim, want)
