"""Which failed factorisations the batched drivers retry one at a time: those of a singular or
non-converging system, not failures of the device (CPU, with a stand-in for the solver)."""

from __future__ import annotations

from types import SimpleNamespace

import pytest

from pyeulerale_b200 import _lib, drivers, solver


class _Solver:
    code = 0
    calls: list = []

    def __init__(self, batch, capacity, tol, workspace):
        pass

    def factor(self, J, shifts):
        self.calls.append(len(J))
        if shifts[-1] == "bad":
            raise _lib.EulerB200Error("eb_ringlu_factor_many", self.code, "")

    def solve(self, rhs, adjoint=False):
        return rhs, [0.0] * len(rhs)


@pytest.mark.parametrize("code,retried", [(_lib.EB_ERR_NAN, True), (_lib.EB_ERR_NOCONV, True),
                                          (_lib.EB_ERR_CUDA, False), (_lib.EB_ERR_ARG, False)])
def test_only_numerical_failures_are_retried(monkeypatch, code, retried):
    monkeypatch.setattr(solver, "RingLUMany", _Solver)
    monkeypatch.setattr(solver, "ringlu_workspace_bytes", lambda M, N: 256)
    monkeypatch.setattr(drivers, "_shape_groups", lambda instances: {(4, 5): [0, 1, 2]})
    _Solver.code, _Solver.calls = code, []
    done, failed = [], []
    args = (SimpleNamespace(cell_offsets=[0, 20, 40]), [0] * 8640, {0: 0.0, 1: 1.0, 2: "bad"},
            lambda i: i, lambda i, x: done.append(i), False,
            SimpleNamespace(numel=lambda: 1024), 1e-10)
    if retried:
        drivers._batched_solves(*args, on_fail=failed.append)
        assert done == [0, 1] and failed == [2] and _Solver.calls == [3, 1, 1, 1]
    else:
        with pytest.raises(_lib.EulerB200Error):
            drivers._batched_solves(*args, on_fail=failed.append)
        assert not done and not failed
