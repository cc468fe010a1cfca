"""The step-length eigenvalue of one space and of both side by side: a solver's
step (both spaces in one launch) is, bit for bit, the step that sddd_min_eig's
values give a program that makes the pass itself.  Blocks whose clusters fill
the GPU differently for one space and for two."""
import ctypes

import numpy as np
import pytest

from conftest import DD, as_dd, load_pkg, ptr

pytestmark = pytest.mark.gpu


def _problem(rng, n, blocks, m):
    k, b, i, j, v = [], [], [], [], []
    for con in range(m + 1):
        for blk in range(1, blocks + 1):
            a, c = rng.integers(1, n + 1, 60), rng.integers(1, n + 1, 60)
            pairs = sorted({(min(x, y), max(x, y)) for x, y in zip(a, c)})
            k += [con] * len(pairs)
            b += [blk] * len(pairs)
            i += [x for x, _ in pairs]
            j += [y for _, y in pairs]
            v += list(rng.standard_normal(len(pairs)) * (1000.0 if con == 0 else 1.0))  # (an F_0 that holds the step back)
    return k, b, i, j, as_dd(np.array(v))


def _dd(sddd, op, a, b):
    x, y, out = as_dd(np.zeros(1)), as_dd(np.zeros(1)), as_dd(np.zeros(1))
    x[0], y[0] = a, b
    assert sddd.lib().sddd_host_dd_op(op, 1, ptr(x), ptr(y), ptr(out)) == 0
    return float(out[0]["hi"]), float(out[0]["lo"])


@pytest.mark.parametrize("n,blocks", [(21, 40), (64, 50), (97, 10), (150, 5), (200, 7)])
def test_solver_step_is_the_step_of_single_eigenvalues(n, blocks):
    sddd = load_pkg()
    m = 30
    rng = np.random.default_rng(n)
    k, blk, i, j, val = _problem(rng, n, blocks, m)
    par = sddd.param()
    b = as_dd(rng.standard_normal(m))
    with sddd.Context(0) as c, sddd.Context(0) as u:
        for x in (c, u):
            x.upload(m, [n] * blocks, b, k, blk, i, j, val)
        c.call("sddd_solver_start", ctypes.byref(par))
        assert c.call("sddd_iterate") == 0
        u.call("sddd_init_point", sddd.SdddDD(par.lambdaStar, 0.0))
        for what in ("Dx", "Dy", "Dz"):
            u.set(what, c.get(what))
        step = []
        for which in range(2):
            e = u.dd_scalar("sddd_min_eig", which)
            a = _dd(sddd, 6, (-1.0, 0.0), e) if e[0] < -0.01 else (100.0, 0.0)
            step.append(min(_dd(sddd, 8, a, (par.gammaStar, 0.0)), (1.0, 0.0)))
        assert min(step)[0] < 1.0, step
        u.call("sddd_update", *[sddd.SdddDD(*a) for a in step])
        for what in ("X", "Z", "y"):
            assert np.array_equal(u.get(what), c.get(what)), what
