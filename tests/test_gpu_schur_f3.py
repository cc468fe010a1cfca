"""The Schur matrix's F3 owners (a few entries a constraint, 32 x 32 pairs a
CTA) against the oracle, bit for bit: numbers of constraints at the tile's
edges, diagonal and off-diagonal entries, and dense constraints among them (so
that the owners' positions have gaps)."""
import numpy as np
import pytest

from conftest import as_dd, load_pkg

pytestmark = pytest.mark.gpu


def _text(rng, n, m, dense):
    lines = [str(m), "1", str(n), " ".join(repr(float(v)) for v in rng.standard_normal(m))]
    lines += [f"0 1 {i + 1} {i + 1} {1.0 + i / n!r}" for i in range(n)]
    for k in range(m):
        count = n * n // 3 if k in dense else int(rng.integers(1, 4))
        seen = set()
        while len(seen) < count:
            i, j = sorted(rng.integers(1, n + 1, 2).tolist())
            seen.add((i, j))
            if len(seen) >= n * (n + 1) // 2:
                break
        lines += [f"{k + 1} 1 {i} {j} {rng.standard_normal()!r}" for i, j in sorted(seen)]
    return "\n".join(lines) + "\n"


@pytest.mark.parametrize("n,m,dense", [(30, 1, ()), (40, 31, ()), (40, 32, ()), (40, 33, ()), (60, 65, (3, 40)), (60, 130, (0, 64, 129))])
def test_f3_owners(oracle_lib, workdir, n, m, dense):
    import sdpa_problem
    rng = np.random.default_rng(n + m)
    text = _text(rng, n, m, set(dense))
    path = workdir / f"f3_{n}_{m}.dat-s"
    path.write_text(text)

    def spd():
        G = rng.standard_normal((n, n))
        out = as_dd((G @ G.T / n + np.eye(n)).ravel())
        lo = rng.uniform(-0.5, 0.5, (n, n)) * 2.0 ** -53
        out["lo"] = out["hi"] * (np.triu(lo) + np.triu(lo, 1).T).ravel()
        return out
    X, Z = spd(), spd()
    with load_pkg().Context(0) as ctx:
        ctx.read_problem(path)
        assert (ctx.formula() == 2).sum() >= m - len(dense) - 1
        assert ctx.set_point(X, as_dd(np.zeros(m)), Z) == 0
        ctx.call("sddd_schur_build")
        B, Zi = ctx.get("B"), ctx.get("invZ")
    want = sdpa_problem.schur(sdpa_problem.Problem(oracle_lib, text), [X], [Zi])
    a, b = B.view(np.float64) + 0.0, want.view(np.float64) + 0.0
    assert np.array_equal(a.ravel(), b.ravel())
