"""The Schur matrix of one dense block (F1 owners) at the shapes where its
products change form: stacked tiles of 36, 40 and 52 or 56 columns, 16 x 16
tiles, ragged last tiles; against the oracle, bit for bit."""
import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(5, 3), (16, 16), (17, 33), (20, 60), (33, 300), (40, 250), (50, 200), (76, 130)])
def test_dense_block(oracle_lib, workdir, n, m):
    import importlib
    sddd = load_pkg()
    P = importlib.import_module("sdpa_dd_b200.problems")
    import sdpa_problem
    text = P.dense_random(n=n, m=m, seed=n)
    path = workdir / f"shape_{n}_{m}.dat-s"
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
    a, b = B.view(np.float64) + 0.0, want.view(np.float64) + 0.0
    assert np.array_equal(a.ravel(), b.ravel())
