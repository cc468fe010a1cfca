"""Products with more rows than a launch has 16-row tiles down (65,535), and at
that edge, against the oracle's triple loop, bit for bit."""
import ctypes

import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu

L_ = ctypes.c_long


@pytest.mark.parametrize("ta,tb", ["NN", "TT"])
@pytest.mark.parametrize("m,n,k", [(1_048_560, 1, 1), (1_048_561, 1, 1), (1_100_000, 8, 8)])
def test_tall_product(oracle_lib, m, n, k, ta, tb):
    import torch
    sddd = load_pkg()
    rng = np.random.default_rng(m + n)
    A, B = as_dd(rng.standard_normal(m * k)), as_dd(rng.standard_normal(k * n))
    A["lo"] = A["hi"] * 2.0 ** -55
    lda, ldb = (m if ta == "N" else k), (k if tb == "N" else n)
    want = np.zeros(m * n, DD)
    # the oracle's loop has no "TT": the same terms in the same order as "TN" with B transposed
    Bo = np.ascontiguousarray(B.reshape(k, n).T) if ta + tb == "TT" else B
    oracle_lib.o_gemm(ctypes.c_char(ta.encode()), ctypes.c_char(b"N"), L_(m), L_(n), L_(k), ptr(A), L_(lda), ptr(Bo), L_(k), ptr(want), L_(m))
    dA, dB = (torch.from_numpy(a.view(np.float64).reshape(-1, 2)).cuda() for a in (A, B))
    dC = torch.full((m * n, 2), float("nan"), dtype=torch.float64, device="cuda")
    with sddd.Context(0) as ctx:
        ctx.call("sddd_Rgemm", ta.encode(), tb.encode(), m, n, k, sddd.SdddDD(1.0, 0.0), dA.data_ptr(), lda, dB.data_ptr(), ldb, sddd.SdddDD(0.0, 0.0),
                 dC.data_ptr(), m)
    assert np.array_equal(dC.cpu().numpy().view(DD).reshape(-1), want)
