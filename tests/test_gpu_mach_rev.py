"""apply_odes_wrt_mach_rev over batches: instances with a cluster of CTAs each, with a CTA each, and
both in one call (GPU).

Tolerance: both sides add the same products in another order, so they differ by a few units of the sum
of their absolute values: 1e-13 of it is left for up to 20,000 cells of four terms."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BATCHES = [[(4, 5, 1)], [(16, 32, 1)], [(16, 33, 1)], [(128, 128, 1)], [(4, 5, 9)], [(64, 64, 3)],
           [(45, 45, 16)], [(32, 32, 40)], [(5, 6, 600)], [(7, 200, 50)], [(128, 128, 2), (5, 6, 30)],
           [(5, 6, 700), (100, 150, 1)], [(4, 9, 515), (120, 130, 2), (6, 7, 20), (128, 100, 1)]]


@pytest.mark.parametrize("sizes", BATCHES, ids=lambda s: ",".join("%dx%d*%d" % q for q in s))
def test_sums(cuda, sizes):
    from pyeulerale_b200 import grid as G
    from pyeulerale_b200.batch import InstanceSet, InstanceSpec

    specs, cells = [], []
    for M, N, count in sizes:
        X = G.naca_ogrid(M + 1, N + 1, 0.12, 1.0, 20.0, 0.02)
        specs += [InstanceSpec(X, 0.5, 1.25)] * count
        cells += [M * N] * count
    inst = InstanceSet(specs)
    rng = np.random.default_rng(len(cells))
    J = rng.standard_normal((inst.n_cells, 4))
    w = rng.standard_normal((inst.n_cells, 4)) + 1j * rng.standard_normal((inst.n_cells, 4))
    out = cuda.full((2 * len(cells),), float("nan"), dtype=cuda.float64, device="cuda")
    inst.call("eb_apply_odes_wrt_mach_rev", cuda.from_numpy(J.ravel()).cuda(),
              cuda.from_numpy(w.ravel().view(np.float64)).cuda(), out)
    got = out.cpu().numpy().view(complex)
    starts = np.concatenate([[0], np.cumsum(cells)[:-1]])
    terms = np.sum(J * w, axis=1)
    want = np.add.reduceat(terms, starts)
    size = np.add.reduceat(np.sum(np.abs(J * w), axis=1), starts)
    assert np.all(np.abs(got - want) <= 1e-13 * size)
