"""Small products (tile16.cuh) at the edges of their 16 x 16 tiles and 32-step
chunks, against the oracle's triple loop, bit for bit."""
import ctypes

import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu

L_ = ctypes.c_long


def _full(rng, shape):
    out = as_dd(rng.standard_normal(shape))
    out["lo"] = out["hi"] * rng.uniform(-1, 1, shape) * 2.0 ** -54
    return out


def _device(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).view(np.float64).reshape(-1, 2).copy()).cuda()


@pytest.mark.parametrize("ta,tb", ["NN", "TN", "NT"])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (16, 16, 32), (17, 15, 33), (8, 9, 64), (9, 8, 2), (31, 33, 31), (100, 7, 95), (3, 130, 1)])
def test_rgemm_small(oracle_lib, m, n, k, ta, tb):
    sddd = load_pkg()
    rng = np.random.default_rng(m + 100 * n + 10000 * k)
    A = _full(rng, (m if ta == "N" else k) * (k if ta == "N" else m))
    B = _full(rng, k * n)
    lda, ldb = (m if ta == "N" else k), (k if tb == "N" else n)
    want = np.zeros(m * n, DD)
    oracle_lib.o_gemm(ctypes.c_char(ta.encode()), ctypes.c_char(tb.encode()), L_(m), L_(n), L_(k), ptr(A), L_(lda), ptr(B), L_(ldb), ptr(want), L_(m))
    dA, dB, dC = _device(A), _device(B), _device(_full(rng, m * n))
    with sddd.Context(0) as ctx:
        ctx.call("sddd_Rgemm", ta.encode(), tb.encode(), m, n, k, sddd.SdddDD(1.0, 0.0), dA.data_ptr(), lda, dB.data_ptr(), ldb, sddd.SdddDD(0.0, 0.0),
                 dC.data_ptr(), m)
    assert np.array_equal(dC.cpu().numpy().view(DD).reshape(-1), want)
