"""Directional derivatives of the Jacobians over odd sizes, every direction kind, against central
differences of the first-order Jacobian kernels (GPU).

Tolerance: with steps of 1e-6 of directions that move states by about 1 and vertices by about a
hundredth, the quotient carries the Jacobians' rounding (about 1e-13 of their largest entry, so
1e-7 after the division) and a truncation of order 1e-10; 1e-5 of the largest entry leaves room for
derivatives smaller than the Jacobians themselves."""

from __future__ import annotations

import numpy as np
import pytest

from helpers import Gpu
from test_gpu_jacobian_sizes import _case

pytestmark = pytest.mark.gpu

SIZES = [(4, 5), (5, 7), (9, 37), (33, 6)]
ENTRIES = {"states": 144, "vertices": 32}
STEP = 1e-6


@pytest.mark.parametrize("kind,key,scale", [(0, "U", 1.0), (1, "X", 0.01), (2, "V", 1.0)])
@pytest.mark.parametrize("M,N", SIZES)
def test_directions_match_differences(cuda, M, N, kind, key, scale):
    case = _case(M, N)
    gpu = Gpu(cuda, case)
    base = {"U": gpu.U, "X": gpu.X, "V": gpu.V}
    rng = np.random.default_rng(17 * M + N + kind)
    n = base[key].numel()
    parts = [cuda.from_numpy(scale * rng.uniform(-1.0, 1.0, n)).cuda() for _ in range(2)]
    d = cuda.stack(parts, dim=1).reshape(-1).contiguous()
    for entry, per_cell in ENTRIES.items():
        size = per_cell * M * N
        got = [cuda.full((size,), float("nan"), dtype=cuda.float64, device="cuda")
               for _ in range(2)]
        gpu.call(f"eb_odes_wrt_{entry}_dir", base["X"], base["V"], base["U"], kind, d, *got)
        for part, exact in zip(parts, got):
            sides = []
            for sign in (1.0, -1.0):
                at = dict(base)
                at[key] = (base[key].reshape(-1) + sign * STEP * part).contiguous()
                J = gpu.empty(size)
                gpu.call(f"eb_compute_odes_wrt_{entry}", at["X"], at["V"], at["U"], J)
                sides.append(J.reshape(-1))
            diff = (sides[0] - sides[1]) / (2.0 * STEP)
            scale_of = max(diff.abs().max().item(), 1e-3)
            assert (exact - diff).abs().max().item() <= 1e-5 * scale_of, entry
