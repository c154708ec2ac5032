"""The closed-form Jacobian kernels over odd sizes: partial warps at the end of an instance, the
smallest grid, boundary rows in every lane position, and several sizes in one launch (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import Gpu, oracle_eval, rel_err

pytestmark = pytest.mark.gpu

SIZES = [(4, 5), (5, 7), (7, 9), (9, 37), (31, 33), (33, 6)]
KEYS = {"J_u": ("eb_compute_odes_wrt_states", 144), "J_x": ("eb_compute_odes_wrt_vertices", 32),
        "J_v": ("eb_compute_odes_wrt_velocities", 32), "J_ma": ("eb_compute_odes_wrt_mach", 4)}


def _case(M, N):
    from pyeulerale_b200 import grid as G

    rng = np.random.default_rng(100 * M + N)
    X = G.naca_ogrid(M + 1, N + 1, 0.12, 1.0, 20.0, 0.02)
    return dict(X=X, V=G.smooth_velocities(X, rng),
                U=G.perturbed_states(M, N, 0.6, 2.0, 0.01, rng), mach=0.6, aoa=2.0)


@pytest.mark.parametrize("M,N", SIZES)
def test_jacobians_match_oracle(cuda, oracle, M, N):
    case = _case(M, N)
    got, ref = Gpu(cuda, case).evaluate(), oracle_eval(oracle, case)
    for k in KEYS:
        assert rel_err(got[k], ref[k]) <= 1e-10, (k, rel_err(got[k], ref[k]))


def test_batch_equals_single_launches(cuda):
    """One launch over all sizes writes what one launch per instance writes, bit for bit."""
    from pyeulerale_b200.batch import InstanceSet, InstanceSpec

    cases = [_case(M, N) for M, N in SIZES]
    inst = InstanceSet([InstanceSpec(c["X"], c["mach"], c["aoa"]) for c in cases])
    pack = lambda k: cuda.from_numpy(  # noqa: E731
        np.concatenate([np.asarray(c[k]).ravel(order="F") for c in cases])).cuda()
    X, V, U = pack("X"), pack("V"), pack("U")
    for name, per_cell in KEYS.values():
        J = cuda.full((per_cell * inst.n_cells,), float("nan"), dtype=cuda.float64, device="cuda")
        inst.call(name, X, V, U, J)
        parts = []
        for c in cases:
            gpu = Gpu(cuda, c)
            one = gpu.empty(per_cell * gpu.M * gpu.N)
            gpu.call(name, gpu.X, gpu.V, gpu.U, one)
            parts.append(one)
        np.testing.assert_array_equal(J.cpu().numpy(), cuda.cat(parts).cpu().numpy())


@pytest.mark.parametrize("count", [2, 33, 128, 129])
def test_many_uneven_instances(cuda, count):
    """Batches below, at and above the rounds of the flat range's search: every cell is written with
    what its own launch writes."""
    from pyeulerale_b200.batch import InstanceSet, InstanceSpec

    kinds = [_case(M, N) for M, N in SIZES[:3] + SIZES[4:]]
    cases = [kinds[(7 * k) % 5 if k else 3] for k in range(count)]
    inst = InstanceSet([InstanceSpec(c["X"], c["mach"], c["aoa"]) for c in cases])
    pack = lambda k: cuda.from_numpy(  # noqa: E731
        np.concatenate([np.asarray(c[k]).ravel(order="F") for c in cases])).cuda()
    X, V, U = pack("X"), pack("V"), pack("U")
    for name, per_cell in KEYS.values():
        J = cuda.full((per_cell * inst.n_cells,), float("nan"), dtype=cuda.float64, device="cuda")
        inst.call(name, X, V, U, J)
        parts = {}
        for c in kinds:
            gpu = Gpu(cuda, c)
            parts[id(c)] = gpu.empty(per_cell * gpu.M * gpu.N)
            gpu.call(name, gpu.X, gpu.V, gpu.U, parts[id(c)])
        assert cuda.equal(J, cuda.cat([parts[id(c)] for c in cases]))
