"""Equal blocks whose Cholesky factors are one launch with one failure word,
some of them not positive definite: the launch ends, the failure is reported,
and the same context takes the next point (orders around the diagonal block's
columns in one and two lanes, and more blocks than run at once)."""
import numpy as np
import pytest

from conftest import DD, load_pkg

pytestmark = pytest.mark.gpu


def _blocks(rng, n, count):
    """Positive definite blocks, column-major, one after the other."""
    A = rng.standard_normal((count, n, n))
    S = A @ A.transpose(0, 2, 1) / n + np.eye(n)
    out = np.zeros(count * n * n, DD)
    out["hi"] = S.ravel()
    return out


@pytest.mark.parametrize("n,count", [(1, 400), (2, 400), (3, 400), (20, 300), (33, 300), (64, 300)])
def test_indefinite_blocks_among_many(n, count):
    sddd = load_pkg()
    rng = np.random.default_rng(100 * n + count)
    k = np.concatenate([np.full(count, q) for q in range(2)])
    blk = np.tile(np.arange(1, count + 1), 2)
    one = np.ones(2 * count, np.int32)
    val = np.zeros(2 * count, DD)
    val["hi"] = 1.0
    b = np.zeros(1, DD)
    b["hi"] = 1.0
    with sddd.Context(0) as c:
        c.upload(1, [n] * count, b, k, blk, one, one, val)
        y = np.zeros(1, DD)
        good = [_blocks(rng, n, count) for _ in range(2)]
        for where in ([count // 2], [0], [count - 1], list(range(0, count, 7)), list(range(count))):
            for side in range(2):
                bad = good[side].copy()
                for t in where:  # a negative pivot in a column of its own
                    j = int(rng.integers(n))
                    bad["hi"][t * n * n + j * (n + 1)] = -1.0
                pair = [bad, good[1]] if side == 0 else [good[0], bad]
                assert c.set_point(pair[0], y, pair[1]) == 1, (where[:3], side)
        assert c.set_point(good[0], y, good[1]) == 0
        # L^-1 of X's blocks, as of no failed point before it
        Linv = c.get("invCholX")["hi"].reshape(count, n, n).transpose(0, 2, 1)
        X = good[0]["hi"].reshape(count, n, n)
        got = Linv @ X @ Linv.transpose(0, 2, 1)
        # the high parts' products: n^2 terms of at most cond(X) < 1e4 in double
        assert np.abs(got - np.eye(n)).max() < 1e-9
