"""Boundary rows whose ghost state has no real speed of sound: the faces next to the boundaries carry
no dissipation, so their fluxes and derivatives stay finite whatever the ghost's pressure (GPU).

The far-field ghost is 2 U_inf - U: a boundary cell at 2.5 times the free stream's pressure gives it a
negative pressure, one at 2.5 times its density a negative density. A wall that moves at twice the
speed of sound gives the wall ghost a negative pressure."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import Gpu, oracle_eval, rel_err
from test_gpu_jacobian_sizes import KEYS

pytestmark = pytest.mark.gpu

KINDS = ["pressure", "density", "wall"]
STEP = 1e-6


def _case(kind, M=7, N=9):
    from pyeulerale_b200 import grid as G

    rng = np.random.default_rng(31)
    X = G.naca_ogrid(M + 1, N + 1, 0.12, 1.0, 20.0, 0.02)
    U = G.perturbed_states(M, N, 0.5, 1.25, 0.01, rng)
    V = np.zeros_like(X)
    cells = [2, 5]  # of the far-field row
    if kind == "pressure":
        U[3, -1, cells] += 1.5 / 0.4
    elif kind == "density":
        U[:, -1, cells] *= 2.5
        U[3, -1, cells] -= 1.5 / 0.4  # at the free stream's pressure
    else:
        edge = X[:, 0, 1:] - X[:, 0, :-1]
        normal = np.stack([edge[1], -edge[0]]) / np.hypot(*edge)
        V[:, 0, :-1] = 2.0 * np.sqrt(1.4) * normal
        V[:, 0, -1] = V[:, 0, 0]
    return dict(X=X, V=V, U=np.asfortranarray(U), mach=0.5, aoa=1.25)


def _ghost_pressures(case, kind):
    """Pressure over density of the ghosts of the boundary row in question."""
    U, X, V = case["U"], case["X"], case["V"]
    if kind == "wall":
        n = np.stack([X[1, 0, 1:] - X[1, 0, :-1], X[0, 0, :-1] - X[0, 0, 1:]])
        g = 0.5 * (V[:, 0, 1:] + V[:, 0, :-1])
        u = U[:, 0]
        proj = np.sum(n * (u[1:3] - g * u[0]), axis=0) / np.sum(n * n, axis=0)
        ghost = np.stack([u[0], *(u[1:3] - 2.0 * n * proj), u[3]])
    else:
        speed = case["mach"] * np.sqrt(1.4)
        a = np.deg2rad(case["aoa"])
        free = np.array([1.0, speed * np.cos(a), speed * np.sin(a), 2.5 + 0.5 * speed**2])
        ghost = 2.0 * free[:, None] - U[:, -1]
    return 0.4 * (ghost[3] - 0.5 * (ghost[1]**2 + ghost[2]**2) / ghost[0]) / ghost[0]


@pytest.mark.parametrize("kind", KINDS)
def test_jacobians_match_oracle(cuda, oracle, kind):
    case = _case(kind)
    assert (_ghost_pressures(case, kind) < 0.0).any()
    got, ref = Gpu(cuda, case).evaluate(), oracle_eval(oracle, case)
    assert np.isfinite(ref["R"]).all() and rel_err(got["R"], ref["R"]) <= 1e-12
    for k in KEYS:
        assert np.isfinite(ref[k]).all() and np.isfinite(got[k]).all(), k
        assert rel_err(got[k], ref[k]) <= 1e-10, (k, rel_err(got[k], ref[k]))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dir_kind,key,scale", [(0, "U", 1.0), (1, "X", 0.01), (2, "V", 1.0)])
def test_directions_match_differences(cuda, kind, dir_kind, key, scale):
    """Tolerance as in test_gpu_second_order_sizes.py: 1e-5 of the largest entry."""
    case = _case(kind)
    gpu = Gpu(cuda, case)
    base = {"U": gpu.U, "X": gpu.X, "V": gpu.V}
    rng = np.random.default_rng(7 + dir_kind)
    part = cuda.from_numpy(scale * rng.uniform(-1.0, 1.0, base[key].numel())).cuda()
    d = cuda.stack([part, -part], dim=1).reshape(-1).contiguous()
    for entry, per_cell in {"states": 144, "vertices": 32}.items():
        size = per_cell * gpu.M * gpu.N
        got = [gpu.empty(size) for _ in range(2)]
        gpu.call(f"eb_odes_wrt_{entry}_dir", base["X"], base["V"], base["U"], dir_kind, d, *got)
        sides = []
        for sign in (1.0, -1.0):
            at = dict(base)
            at[key] = (base[key] + sign * STEP * part).contiguous()
            J = gpu.empty(size)
            gpu.call(f"eb_compute_odes_wrt_{entry}", at["X"], at["V"], at["U"], J)
            sides.append(J)
        diff = (sides[0] - sides[1]) / (2.0 * STEP)
        bound = 1e-5 * max(diff.abs().max().item(), 1e-3)
        assert (got[0] - diff).abs().max().item() <= bound, entry
        assert (got[1] + diff).abs().max().item() <= bound, entry
