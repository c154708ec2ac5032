"""The blocked inversion over ring sizes and shift counts: 64- and 128-column blocks, last blocks of
every remainder, both sides of the line to the cooperative form, halves of unequal size (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import crandn, rel_err
from test_gpu_ringlu_sizes import _setup

pytestmark = pytest.mark.gpu

# (N, shifts): the blocked form begins with the second cooperative launch, up to N = 64 with the third
# (148 SMs hold 27, 12 and 9 blocks at N = 32, 48 and 64, 3 at 79, 2 at 100 to 144, then one)
SIZES = [(32, 54), (32, 55), (33, 35), (48, 24), (48, 25), (50, 23), (52, 24), (61, 19), (64, 18),
         (64, 19), (79, 4), (82, 5), (100, 2), (100, 24), (126, 3), (128, 3), (129, 3), (131, 3),
         (135, 4), (144, 3), (161, 2), (200, 3), (253, 2)]


@pytest.mark.parametrize("N,count", SIZES)
def test_blocked_matches_single(cuda, N, count):
    """Each shift of the call against a factorisation of its own (in the cooperative form): relative
    residuals of 1e-10, and without refinement no worse than a hundred times the single shift's (both
    invert by partial pivoting, in another order of sums)."""
    from pyeulerale_b200 import solver

    M = 4
    gpu, J, rng = _setup(cuda, M, N, N)
    shifts = [1j * k for k in np.logspace(-2, 1, count - 1)] + [1.5 - 0.25j]
    rhs = [gpu.dev(crandn(rng, (4, M, N))) for _ in shifts]
    many = solver.RingLUMany(gpu.batch, capacity=count, tol=1e-10)
    one = solver.RingLU(gpu.batch, tol=1e-10)
    many.factor(J, shifts)
    for adjoint in (False, True):
        xs, rels = many.solve(rhs, adjoint=adjoint)
        assert max(rels) <= 1e-10, rels
        for k in sorted({0, (count - 1) // 2, (count + 1) // 2, count - 1}):
            one.factor(J, shifts[k])
            x, _ = one.solve(rhs[k], adjoint=adjoint)
            assert rel_err(xs[k].cpu().numpy(), x.cpu().numpy()) <= 1e-9, (k, adjoint)
            many.tol = one.tol = 1e30  # the factors as they are
            many.max_refine = one.max_refine = 0
            raw, single = many.solve(rhs, adjoint=adjoint)[1][k], one.solve(rhs[k], adjoint=adjoint)[1]
            many.tol = one.tol = 1e-10
            many.max_refine = one.max_refine = 4
            assert raw <= 100.0 * max(single, 1e-14), (k, adjoint, raw, single)
