"""The sparse factor and solves (sparse_chol.cu) against the plain loops of
Lal::getCholesky and Lal::solveSystems (sdpa_linear.cpp:353-395, 654-810) in
the host's dd arithmetic, bit for bit: orders at the edges of the 64-blocks,
structures from near-diagonal to dense, a negative pivot."""
import numpy as np
import pytest

from conftest import DD, load_pkg, ptr

pytestmark = pytest.mark.gpu


def _structure(rng, m, density):
    """Rows of struct(b), b first, ascending, closed under elimination."""
    rows = [set() for _ in range(m)]
    for b in range(m):
        later = np.arange(b + 1, m)
        rows[b].update(later[rng.random(len(later)) < density].tolist())
        if b + 1 < m and rng.random() < 0.8:
            rows[b].add(min(m - 1, b + 1 + int(rng.integers(0, 3))))
    for b in range(m):
        s = sorted(rows[b])
        if len(s) > 1:
            rows[s[0]].update(s[1:])
    di, ci = [0], []
    for b in range(m):
        ci += [b] + sorted(rows[b])
        di.append(len(ci))
    return np.array(di, np.int32), np.array(ci, np.int32)


def _op(lib, op, a, b):
    a, b = (np.ascontiguousarray(np.broadcast_to(x, np.broadcast(a, b).shape)) for x in (a, b))
    out = np.zeros(a.shape, DD)
    assert lib.sddd_host_dd_op(op, a.size, ptr(a), ptr(b), ptr(out)) == 0
    return out


ONE = np.array([(1.0, 0.0)], DD)


def _factor(lib, m, di, ci, v):
    v = v.copy()
    for b in range(m):
        p, e = di[b], di[b + 1]
        d = v[p:p + 1]
        inv = np.zeros(1, DD) if d["hi"][0] < 0 else _op(lib, 6, ONE, _op(lib, 7, d, d))
        v[p] = inv[0]
        if e - p > 1:
            v[p + 1:e] = _op(lib, 5, v[p + 1:e], inv)
        for q in range(p + 1, e):
            r = ci[q]
            at = di[r] + np.searchsorted(ci[di[r]:di[r + 1]], ci[q:e])
            v[at] = _op(lib, 2, v[at], _op(lib, 4, v[q:q + 1], v[q:e]))
    return v


def _solve(lib, m, di, ci, v, x):
    x = x.copy()
    for b in range(m):
        p, e = di[b], di[b + 1]
        x[b:b + 1] = _op(lib, 5, x[b:b + 1], v[p:p + 1])
        if e - p > 1:
            a = ci[p + 1:e]
            x[a] = _op(lib, 2, x[a], _op(lib, 4, v[p + 1:e], x[b:b + 1]))
    for b in range(m - 1, -1, -1):
        p, e = di[b], di[b + 1]
        for q in range(e - 1, p, -1):
            x[b:b + 1] = _op(lib, 2, x[b:b + 1], _op(lib, 4, v[q:q + 1], x[ci[q]:ci[q] + 1]))
        x[b:b + 1] = _op(lib, 5, x[b:b + 1], v[p:p + 1])
    return x


@pytest.mark.parametrize("m,density,negative", [(1, 0.0, None), (2, 1.0, None), (40, 0.3, None), (63, 0.02, None), (64, 1.0, None), (65, 0.05, 3),
                                                (130, 0.01, None), (130, 1.0, None), (200, 0.02, 70), (330, 0.004, None)])
def test_factor_and_solve(m, density, negative):
    import torch
    sddd = load_pkg()
    rng = np.random.default_rng(m + int(1000 * density))
    di, ci = _structure(rng, m, density)
    v = np.zeros(di[m], DD)
    v["hi"] = rng.standard_normal(di[m]) * 0.1
    v["lo"] = v["hi"] * 2.0 ** -55 * rng.uniform(-1, 1, di[m])
    v["hi"][di[:-1]] = 4.0 + 10.0 * rng.random(m)
    v["lo"][di[:-1]] = 0.0
    if negative is not None:
        v["hi"][di[negative]] = -1.0
    x = np.zeros(m, DD)
    x["hi"] = rng.standard_normal(m)
    x["lo"] = x["hi"] * 2.0 ** -56

    def dev(a):
        return torch.from_numpy(a.view(np.float64).copy()).cuda()
    with sddd.Context(0) as ctx:
        dv, dx = dev(v), dev(x)
        ctx.call("sddd_sparse_getCholesky", m, ptr(di), ptr(ci), dv.data_ptr())
        got = dv.cpu().numpy().view(DD)
        want = _factor(ctx.L, m, di, ci, v)
        assert np.array_equal(got, want)
        ctx.call("sddd_sparse_solveSystems", m, ptr(di), ptr(ci), dv.data_ptr(), dx.data_ptr())
        assert np.array_equal(dx.cpu().numpy().view(DD), _solve(ctx.L, m, di, ci, want, x))
