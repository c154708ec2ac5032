"""The ring LU over ring sizes: each variant of the cooperative inversion at its limits (K = 4 N
unknowns per ring: 16 real or 8 complex columns per CTA, one to four rows per thread), partial
column groups, and few or many rings (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import Gpu, crandn

pytestmark = pytest.mark.gpu


def _setup(cuda, M, N, seed):
    from pyeulerale_b200 import grid as G

    rng = np.random.default_rng(seed)
    X = G.naca_ogrid(M + 1, N + 1, 0.12, 1.0, 20.0, 0.02)
    case = dict(X=X, V=np.zeros_like(X), U=G.perturbed_states(M, N, 0.5, 1.25, 0.01, rng),
                mach=0.5, aoa=1.25)
    gpu = Gpu(cuda, case)
    J = gpu.empty(144 * M * N)
    gpu.call("eb_compute_odes_wrt_states", gpu.X, gpu.V, gpu.U, J)
    return gpu, J, rng


@pytest.mark.parametrize("shift", [0.0, 0.2 + 0.4j])
@pytest.mark.parametrize("M,N", [(4, 5), (5, 7), (6, 32), (7, 33), (9, 64), (4, 65), (8, 96),
                                 (5, 128), (5, 129), (4, 192), (4, 193), (5, 256)])
def test_ringlu_sizes(cuda, M, N, shift):
    """The solves of one factorisation (both directions, refined as by default) reach a relative
    residual of 1e-10, measured against the Jacobian itself."""
    from pyeulerale_b200 import solver

    gpu, J, rng = _setup(cuda, M, N, M + N)
    lu = solver.RingLU(gpu.batch, tol=1e-10)
    for _ in range(2):  # launched, then captured
        lu.factor(J, shift)
    for adjoint in (False, True):
        _, rel = lu.solve(gpu.dev(crandn(rng, (4, M, N))), adjoint=adjoint)
        assert rel <= 1e-10, (M, N, shift, adjoint, rel)


@pytest.mark.parametrize("shifts", [[0.1j, 2.0, 0.3 - 1j], [0.0, 0.5, 2.0]])
def test_ringlu_few_shifts(cuda, shifts):
    """Several shifts below the blocked form's count, more systems than fit the GPU at once."""
    from pyeulerale_b200 import solver

    M, N = 6, 129
    gpu, J, rng = _setup(cuda, M, N, 3)
    lu = solver.RingLUMany(gpu.batch, capacity=len(shifts), tol=1e-10)
    lu.factor(J, shifts)
    for adjoint in (False, True):
        rhs = [gpu.dev(crandn(rng, (4, M, N))) for _ in shifts]
        _, rels = lu.solve(rhs, adjoint=adjoint)
        assert max(rels) <= 1e-10, (adjoint, rels)


def test_ringlu_singular_block(cuda):
    """A singular ring block (a zero Jacobian) ends the factorisation with EB_ERR_NAN, and the
    workspace serves the next one."""
    from pyeulerale_b200 import _lib, solver

    M, N = 5, 40
    gpu, J, rng = _setup(cuda, M, N, 4)
    lu = solver.RingLU(gpu.batch, tol=1e-10)
    for shift in (0.0, 0.5j):
        bad = J.clone()
        bad[:16 * 3] = float("nan")
        for Jx, s in ((gpu.empty(144 * M * N), 0.0), (bad, shift)):
            with pytest.raises(_lib.EulerB200Error) as e:
                lu.factor(Jx, s)
            assert e.value.code == _lib.EB_ERR_NAN
        lu.factor(J, shift)
        _, rel = lu.solve(gpu.dev(crandn(rng, (4, M, N))))
        assert rel <= 1e-10
