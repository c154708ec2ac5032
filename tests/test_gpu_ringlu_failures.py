"""Failing factorisations of the ring LU: zero pivots at any step of any CTA's columns, a wait that runs
out, and threads that factor grids of different sizes (GPU)."""

from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor

import pytest

from helpers import crandn
from test_gpu_ringlu_sizes import _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [0, 3, 4, 5, 6, 9, 14, 15, 16, 22, 63, 110, 159])
@pytest.mark.parametrize("shift", [0.0, 0.5j])
def test_zero_pivot(cuda, step, shift):
    """The first ring's block is the identity but for a zero pivot at one step: a zero column, or at a
    complex shift i w the second column of [[0, -w], [w, 0]]. The failing step is published, so the
    status is that of a singular block, not that of a wait that ran out."""
    from pyeulerale_b200 import _lib, solver

    M, N = 4, 40
    if shift and step % 4 == 0:
        step += 1  # the pair's two columns are in one cell
    gpu, J, rng = _setup(cuda, M, N, 4)
    bad = cuda.zeros_like(J)
    own = bad[:16 * M * N].reshape(N, M, 4, 4)  # [cell, ring, column, row] of the own-cell blocks
    own[:] = cuda.eye(4, dtype=cuda.float64, device="cuda")
    n, k = divmod(step, 4)
    own[n, 0, k] = 0.0
    if shift:
        w = shift.imag
        own[n, 0, k - 1] = 0.0
        own[n, 0, k, k - 1], own[n, 0, k - 1, k] = -w, w
    lu = solver.RingLU(gpu.batch, tol=1e-10)
    with pytest.raises(_lib.EulerB200Error) as e:
        lu.factor(bad, shift)
    assert e.value.code == _lib.EB_ERR_NAN
    lu.factor(J, shift)
    _, rel = lu.solve(gpu.dev(crandn(rng, (4, M, N))))
    assert rel <= 1e-10


def test_wait_runs_out(cuda):
    from pyeulerale_b200 import _lib

    scratch = cuda.zeros(2, dtype=cuda.int64, device="cuda")
    with pytest.raises(_lib.EulerB200Error) as e:
        _lib.call("eb_ringlu_wait_probe", 1000, scratch.data_ptr(), None)
    assert e.value.code == _lib.EB_ERR_CUDA and "ran out" in str(e.value)
    cuda.cuda.synchronize()


def test_threads_of_different_sizes(cuda, monkeypatch):
    """Two kernels serve ranges of sizes: neither thread's factorisations and sweeps are refused because
    of the other's smaller ones."""
    from pyeulerale_b200 import solver

    monkeypatch.setenv("EB_RINGLU_GRAPHS", "0")
    jobs = []
    for N in (66, 128, 70, 120):
        gpu, J, rng = _setup(cuda, 5, N, N)
        jobs.append((solver.RingLU(gpu.batch, tol=1e-10), J, gpu.dev(crandn(rng, (4, 5, N)))))

    def work(job):
        lu, J, rhs = job
        worst = 0.0
        for k in range(40):
            lu.factor(J, 0.3j)
            worst = max(worst, lu.solve(rhs)[1])
        return worst

    with ThreadPoolExecutor(len(jobs)) as pool:
        assert max(pool.map(work, jobs)) <= 1e-10
