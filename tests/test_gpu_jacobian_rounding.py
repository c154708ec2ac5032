"""Rounding of d(odes)/d(velocities) against extended precision (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import Gpu

pytestmark = pytest.mark.gpu


def _interior(X, U, dtype):
    """d(odes)/d(velocities) of the cells off the boundary rows: a face's flux moves with the velocities
    of its two corners by minus half the mean of its states times its normal, and a cell's odes are
    minus the sum over its faces, divided by the area."""
    X, U = X.astype(dtype), U.astype(dtype)
    c = [X[:, 1:-2, :-1], X[:, 1:-2, 1:], X[:, 2:-1, 1:], X[:, 2:-1, :-1]]  # the cells' corners
    normal = lambda a, b: np.stack([b[1] - a[1], a[0] - b[0]])  # noqa: E731
    own, M = U[:, 1:-1], U.shape[1]
    other = [U[:, :M - 2], np.roll(own, -1, axis=2), U[:, 2:], np.roll(own, 1, axis=2)]
    # faces i, f, o, b between corners 0-1, 1-2, 2-3, 3-0: (4 states, 2 components, cells)
    faces = [((own + r) / 2)[:, None] * (normal(c[q], c[(q + 1) % 4]) / 2)[None]
             for q, r in enumerate(other)]
    d, e = c[2] - c[0], c[3] - c[1]
    area = np.abs(d[0] * e[1] - d[1] * e[0]) / 2
    return np.stack([(faces[k] + faces[k - 1]) / area for k in range(4)], axis=-1)


def test_velocities_no_worse_than_plain(cuda):
    """The root-mean-square error over some 20,000 cells is that of the plain evaluation in doubles, or
    less. (Its spread from one such set of cells to another is below 1 %: 3 % are allowed.)"""
    from pyeulerale_b200 import grid as G

    sums = np.zeros(2)
    for k, (M, N, t) in enumerate([(64, 64, 0.12), (33, 47, 0.04), (60, 41, 0.12), (96, 121, 0.04)]):
        rng = np.random.default_rng(k)
        X = G.naca_ogrid(M + 1, N + 1, t, 1.0, 20.0, 0.01)
        U = G.perturbed_states(M, N, 0.4 + 0.1 * k, 1.0, 0.01, rng)
        gpu = Gpu(cuda, dict(X=X, V=G.smooth_velocities(X, rng), U=U, mach=0.4 + 0.1 * k, aoa=1.0))
        J = gpu.empty(32 * M * N)
        gpu.call("eb_compute_odes_wrt_velocities", gpu.X, gpu.V, gpu.U, J)
        got = gpu.host(J, (4, 2, M, N, 4))[:, :, 1:-1]
        exact = _interior(X, U, np.longdouble)
        scale = np.sqrt(np.mean(exact.astype(float)**2))
        assert np.max(np.abs(got - exact)) <= 1e-12 * np.max(np.abs(exact))
        for i, v in enumerate([got, _interior(X, U, float)]):
            sums[i] += np.sum(((v - exact) / scale).astype(float)**2)
    assert sums[0] <= 1.03**2 * sums[1], np.sqrt(sums)
