"""The step-length eigenvalue of large blocks: vectors in global memory (orders
of about 4000 and more), and a large block among many small ones, where a CTA's
own rows ask for a larger cluster than the number of blocks.  L and D hold a few
bands, some far from the diagonal, so that the Lanczos loop of the reference
(sdpa_linear.cpp:27-122) can be written down on n-vectors here, in dd; the loop
itself is checked against the oracle's at a small order.

Tolerance 1e-25 of the value, the bar of the reference comparisons (a product
with a band has a handful of terms, the dot products n = 6500: 1e4 2^-104 =
5e-28)."""
import ctypes

import mpmath
import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg, ptr


# ---- dd on numpy vectors (pairs of high and low parts)
def _two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def _split(a):
    t = 134217729.0 * a
    h = t - (t - a)
    return h, a - h


def _add(a, b):
    s, e = _two_sum(a[0], b[0])
    t, f = _two_sum(a[1], b[1])
    s, e = _two_sum(s, e + t)
    return _two_sum(s, e + f)


def _mul(a, b):
    p = a[0] * b[0]
    (ah, al), (bh, bl) = _split(a[0]), _split(b[0])
    e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    return _two_sum(p, e + (a[0] * b[1] + a[1] * b[0]))


def _dot(a, b):
    s = _mul(a, b)
    while len(s[0]) > 1:
        if len(s[0]) % 2:
            s = tuple(np.append(x, 0.0) for x in s)
        s = _add(tuple(x[::2] for x in s), tuple(x[1::2] for x in s))
    return mpmath.mpf(float(s[0][0])) + mpmath.mpf(float(s[1][0]))


def _scalar(x):
    h = float(x)
    return np.float64(h), np.float64(float(x - mpmath.mpf(h)))


# ---- banded matrices: {s: (hi, lo)}, entry (j + s, j) at place j
def _bands(rng, n, shifts, diag):
    out = {}
    for s in shifts:
        h = diag(n) if s == 0 else 0.2 * rng.standard_normal(n - s)
        out[s] = (h, h * rng.uniform(-1, 1, n - s) * 2.0 ** -54)
    return out


def _apply(M, x, lower, upper):
    """The product with M's lower triangle, its transpose's, or both."""
    n = len(x[0])
    y = (np.zeros(n), np.zeros(n))
    for s, c in M.items():
        for down in ([True] if lower else []) + ([False] if upper and (s > 0 or not lower) else []):
            t = _mul(c, tuple(v[: n - s] if down else v[s:] for v in x))
            at = slice(s, n) if down else slice(0, n - s)
            r = _add(tuple(v[at] for v in y), t)
            for v, w in zip(y, r):
                v[at] = w
    return y


def _dense(M, n, symmetric):
    """Column-major n x n dd."""
    out = np.zeros((n, n), DD)
    j = np.arange(n)
    for s, (h, l) in M.items():
        for a, b in [(j[: n - s], j[s:])] + ([(j[s:], j[: n - s])] if symmetric and s else []):
            out["hi"][a, b], out["lo"][a, b] = h, l
    return out.reshape(-1)


def _tri_min(d, e):
    """Smallest eigenvalue of the tridiagonal (d, e) and the last component of
    its unit eigenvector: Newton's method on the leading minors from below."""
    with mpmath.workdps(200):
        k = len(d)
        if k == 1:
            return d[0], mpmath.mpf(1)
        T = np.diag([float(x) for x in d]) + np.diag([float(x) for x in e[: k - 1]], 1)
        w = np.linalg.eigvalsh(T + np.triu(T, 1).T)
        x = mpmath.mpf(float(w[0])) - mpmath.mpf(1e-12) * max(abs(w[0]), abs(w[-1]))
        for _ in range(60):
            p0, q0, p1, q1 = mpmath.mpf(1), mpmath.mpf(0), d[0] - x, mpmath.mpf(-1)
            for i in range(1, k):
                p2 = (d[i] - x) * p1 - e[i - 1] ** 2 * p0
                q2 = (d[i] - x) * q1 - p1 - e[i - 1] ** 2 * q0
                p0, q0, p1, q1 = p1, q1, p2, q2
            step = p1 / q1
            x -= step
            if abs(step) < mpmath.mpf(10) ** -120 * abs(x):
                break
        z = [mpmath.mpf(1)]
        for i in range(k - 1):
            z.append(((x - d[i]) * z[i] - (e[i - 1] * z[i - 1] if i else 0)) / e[i])
        return x, z[-1] / mpmath.sqrt(sum(v * v for v in z))


def _lanczos(n, L, D):
    mpmath.mp.dps = 40
    mn, old, err = mpmath.mpf("1e51"), mpmath.mpf("1e52"), mpmath.mpf("1e10")
    q, r = (np.zeros(n), np.zeros(n)), (np.ones(n), np.zeros(n))
    beta = mpmath.sqrt(n)
    d, e, k, kk = [], [], 0, 0
    while k < n and k < mpmath.sqrt(n) + 10 and beta > 1e-16 and (
            abs(mn - old) > abs(mn) * 1.0e-5 + 1.0e-8 or abs(err * beta) > abs(mn) * 1.0e-2 + 1.0e-4):
        qold, q = q, _mul(r, _scalar(1 / beta))
        w = _apply(L, _apply(D, _apply(L, q, False, True), True, True), True, False)
        alpha = _dot(q, w)
        r = _add(_add(w, _mul(q, _scalar(-alpha))), _mul(qold, _scalar(-beta)))
        d.append(alpha)
        if k <= kk * kk or k == n - 1 or k > mpmath.sqrt(n + 9):
            kk = 0
            old = mn
            mn, err = _tri_min(d, e)
        beta = mpmath.sqrt(_dot(r, r))
        e.append(beta)
        k, kk = k + 1, kk + 1
    return mn - abs(err * beta), k


def _pair(rng, n, shifts):
    # the lowest end of the spectrum stands out, so that the loop settles
    L = _bands(rng, n, shifts, lambda m: rng.uniform(0.8, 1.2, m))
    D = _bands(rng, n, [s + 2 if s else 0 for s in shifts], lambda m: rng.uniform(0.5, 1.5, m) - 3.0 * (np.arange(m) == m // 3))
    return L, D


def _close(got, want):
    return abs(mpmath.mpf(float(got[0])) + mpmath.mpf(float(got[1])) - want) <= mpmath.mpf(10) ** -25 * abs(want)


@pytest.mark.parametrize("n", [30, 101])
def test_band_lanczos_is_the_oracles(oracle_lib, n):
    class ODD(ctypes.Structure):
        _fields_ = [("hi", ctypes.c_double), ("lo", ctypes.c_double)]
    oracle_lib.o_lanczos_min_eig.restype = ODD
    L, D = _pair(np.random.default_rng(n), n, [0, 1, 7, 19])
    A, B = _dense(L, n, False), _dense(D, n, True)
    want, k = _lanczos(n, L, D)
    got = oracle_lib.o_lanczos_min_eig(ctypes.c_long(n), ptr(A), ptr(B))
    assert k > 4
    assert _close((got.hi, got.lo), want), (got.hi, got.lo, want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3840, 4001, 4089, 4096])
def test_one_large_block(n):
    import torch
    L, D = _pair(np.random.default_rng(n), n, [0, 1, 37, 2051, n - 5])
    want, k = _lanczos(n, L, D)
    assert k > 4
    t = [torch.from_numpy(_dense(M, n, sym).view(np.float64)).cuda() for M, sym in ((L, False), (D, True))]
    out = torch.full((2,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert load_pkg().lib().sddd_min_eig_noalloc(None, n, t[0].data_ptr(), t[1].data_ptr(), out.data_ptr()) == 0
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert _close(got, want), (tuple(got), want, k)


@pytest.mark.gpu
def test_large_block_among_many_small_ones():
    """148 clusters or more want one CTA each; a block of 6500 rows does not
    fit one."""
    sddd = load_pkg()
    n, small, count = 6500, 21, 75
    L, D = _pair(np.random.default_rng(n), n, [0, 1, 37, 2051, n - 5])
    want, k = _lanczos(n, L, D)
    assert k > 4 and want < 1
    blk = np.arange(1, count + 2)
    one = np.ones(count + 1, np.int32)
    eye = np.zeros(small * small, DD)
    eye["hi"][:: small + 1] = 1.0
    five = eye.copy()
    five["hi"] *= 5.0
    with sddd.Context(0) as c:
        c.upload(1, [n] + [small] * count, as_dd(np.ones(1)), np.repeat([0, 1], count + 1), np.tile(blk, 2), np.tile(one, 2), np.tile(one, 2),
                 as_dd(np.ones(2 * (count + 1))))
        assert c.sizes == [n] + [small] * count
        c.set("invCholX", np.concatenate([_dense(L, n, False)] + [eye] * count))
        c.set("Dx", np.concatenate([_dense(D, n, True)] + [five] * count))
        got = c.dd_scalar("sddd_min_eig", 0)
    assert _close(got, want), (got, want, k)
