"""The inverse of a Cholesky factor, column by column in registers
(inv_lower_rows_kernel), against the oracle's plain loops, bit for bit: orders
at the edges of the kernel's forms, a factor with zero entries (steps that are
skipped), values outside the corrected quotients' range."""
import ctypes

import numpy as np
import pytest

from conftest import as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu

L_ = ctypes.c_long


@pytest.mark.parametrize("n,spread,zeros", [(1, 0, False), (2, 0, False), (33, 230, False), (95, 0, True), (96, 0, False), (97, 230, False), (128, 0, True),
                                            (129, 0, False), (256, 230, True), (257, 0, False), (512, 0, True), (513, 230, False), (1025, 0, True)])
def test_inverse_bits(oracle_lib, n, spread, zeros):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n))
    A = G @ G.T / n + 0.05 * np.eye(n)
    if zeros:  # blocks of a third, apart from one column
        b = np.arange(n) * 3 // n
        A *= b[:, None] == b[None, :]
    s = 2.0 ** rng.integers(-spread, spread + 1, n)
    A = A * s[:, None] * s[None, :]
    X = as_dd(A.T.ravel())
    with load_pkg().Context(0) as c:
        c.upload(1, [n], as_dd(np.ones(1)), [1], [1], [1], [1], as_dd(np.ones(1)))
        assert c.set_point(X, as_dd(np.zeros(1)), X) == 0
        got = c.get("invCholX").reshape(n, n).T
    L, inv = X.copy(), np.zeros_like(X)
    oracle_lib.o_potrf.restype = L_
    assert oracle_lib.o_potrf(L_(n), ptr(L), L_(n)) == 0
    oracle_lib.o_inv_lower(L_(n), ptr(L), L_(n), ptr(inv), L_(n))
    low = np.tril_indices(n)
    assert np.array_equal(got[low], inv.reshape(n, n).T[low])
