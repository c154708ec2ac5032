"""The kernels' quotients, reciprocals and roots against the built-in operations (GPU).

Bounds: the last step of each adds a correction to a value that is off by at most a few units in the
last place, from a remainder known to 2^-38 or better, so results are half a unit and 2^-20 off at
most: the correctly rounded value or its neighbour. Below 2^-1000 the remainder itself may be
rounded away, which leaves the uncorrected product: two units. The pivot reciprocal's last Newton step
does the same to a value that is off by 2^-36 at most.

Subnormal divisors count as zeros and those above 2^1022 as infinities; the root of a subnormal is
the subnormal itself. Everything else, zeros, infinities, NaN and overflow included, is as built in."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF, NAN, TINY = np.inf, np.nan, 2.0**-1022
SPECIAL = [0.0, INF, NAN, 5e-324, 2.0**-1040, TINY - 5e-324, TINY, 1.5 * TINY, 2.0**-1021, 2.0**-700,
           0.1, 1.0, 3.0, 2.0**700, 2.0**1020, 1e308, 2.0**1021, 1.7 * 2.0**1021, 1.3 * 2.0**1022,
           2.0**1023, np.finfo(float).max]


def _operands(kind):
    if kind == "special":
        s = np.array([v * sign for v in SPECIAL for sign in (1.0, -1.0)])
        a, b = np.meshgrid(s, s)
        return a.ravel(), b.ravel()
    rng = np.random.default_rng(11)
    n = 1 << 21
    top = {"ordinary": 30, "wide": 1074}[kind]
    draw = lambda: np.ldexp(  # noqa: E731
        rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n), rng.integers(-top, min(top, 1023), n))
    return draw(), draw()


@pytest.mark.parametrize("kind", ["ordinary", "wide", "special"])
def test_against_built_in(cuda, kind):
    from pyeulerale_b200 import _lib

    a, b = _operands(kind)
    n = a.size
    size = np.abs(b)
    normal = (size >= TINY) & (size < 2.0**1022)
    counted = np.where(size < TINY, np.copysign(0.0, b),
                       np.where(size > 2.0**1022, np.copysign(INF, b), b))
    da, db, dc = (cuda.from_numpy(v).cuda() for v in (a, b, counted))
    out = cuda.empty((4, n), dtype=cuda.float64, device="cuda")
    _lib.call("eb_scalar_probe", n, da.data_ptr(), db.data_ptr(), out.data_ptr(), None)
    one = cuda.ones_like(db)
    want = [da / dc, one / dc, cuda.where((db > 0.0) & (db < TINY), db, cuda.sqrt(db)), one / db]
    got = out.cpu().numpy()
    want = [w.cpu().numpy() for w in want]
    for name, g, w, where in zip(["quotient", "reciprocal", "root", "pivot reciprocal"], got, want,
                                 [slice(None)] * 3 + [normal]):
        g, w = g[where], w[where]
        exact = ~np.isfinite(w) | (w == 0.0)
        np.testing.assert_array_equal(g[exact], w[exact], err_msg=name)
        np.testing.assert_array_equal(np.signbit(g[w == 0.0]), np.signbit(w[w == 0.0]), err_msg=name)
        g, w = g[~exact], w[~exact]
        units = np.abs(g - w) / np.spacing(np.abs(w))
        small = np.abs(a[where][~exact]) < 2.0**-1000 if name == "quotient" else 0.0 * units > 0.0
        worst = np.argmax(units)
        assert units[~small].max(initial=0.0) <= 1.0, (name, units[worst], w[worst])
        assert units.max(initial=0.0) <= 2.0, (name, units[worst], w[worst])
