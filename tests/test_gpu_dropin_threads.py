"""Threads that apply products of one drop-in solver get what one thread gets (GPU)."""

from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from helpers import crandn

pytestmark = pytest.mark.gpu


def test_concurrent_products(cuda):
    from pyeulerale_b200 import SpatialDiscretization
    from pyeulerale_b200 import grid as G

    M = N = 96
    solver = SpatialDiscretization(G.naca_ogrid(M + 1, N + 1, 0.12, 1.0, 20.0, 0.01))
    rng = np.random.default_rng(5)
    solver.states[:] = G.perturbed_states(M, N, 0.5, 1.25, 0.01, rng)
    solver.linearize()
    inputs = [crandn(rng, (4, M, N)) for _ in range(16)]
    want = [(solver.apply_odes_wrt_states_fwd(w), solver.apply_odes_wrt_states_rev(w))
            for w in inputs]

    def work(k):
        for _ in range(12):
            got = (solver.apply_odes_wrt_states_fwd(inputs[k]),
                   solver.apply_odes_wrt_states_rev(inputs[k]))
            if not all(np.array_equal(a, b) for a, b in zip(got, want[k])):
                return False
        return True

    with ThreadPoolExecutor(8) as pool:
        assert all(pool.map(work, range(16)))
