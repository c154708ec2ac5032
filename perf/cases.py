"""What is measured: the work that programs built on this package have it do.

A case names one kind of call and its sizes (cells, not points: M radial, N angular). The kinds:

* ``residual``: R(U, X, V) of packed instances on the device (a serving loop, an explicit
  integrator); from one small grid, where the launch counts, to a batch that fills the GPU.
* ``gradient``: R and the gradients of <w, R> with respect to U, X, V and the Mach numbers
  through autograd (training and inverse design; forward and backward).
* ``tangent``: the matrix-free product of all four derivatives with a complex direction.
* ``linearize``: all six Jacobians of a batch of uneven grids.
* ``products``: forward and reverse products with stored Jacobians (Krylov methods, adjoints).
* ``dropin``: the drop-in class with host arrays: residual, forces, linearization and products, the
  calls with which the reference's response example prepares a right-hand side.
* ``second_order``: three second-order gradients of the drop-in class (the gain example's terms).
* ``resolvent``: factor J - s I, then one forward and one adjoint solve; s = 0 is the adjoint
  gradient's and the static gain's shift, s imaginary a reduced frequency's.
* ``ptc``: steps of the pseudo-transient continuation to the steady state on the device.
* ``response``: a pitch frequency sweep with the adjoint lift gradient (the response example's
  sweep with many shifts at once).

Grids are NACA O-grids of this package with a seeded thickness, states a seeded smooth flow with a
little noise, vertex velocities seeded smooth fields, as in the tests. ``exact`` evaluates the
same operators cell by cell in float64 torch (forward- and reverse-mode derivatives, block
elimination for the solves).
"""

from __future__ import annotations

import math

import numpy as np
import torch

from pyeulerale_b200 import SpatialDiscretization, drivers, solver
from pyeulerale_b200.autograd import residual
from pyeulerale_b200.batch import InstanceSet, InstanceSpec
from pyeulerale_b200.grid import naca_ogrid

F64 = torch.float64
C128 = torch.complex128


def listed() -> list[dict]:
    return [
        # one small grid per call: launch and dispatch cost
        {"name": "residual_33", "kind": "residual", "sizes": "32x32"},
        # the bench's batch of 129x129 grids
        {"name": "residual_129_x256", "kind": "residual", "sizes": "128x128*256"},
        # value and gradients of a batch
        {"name": "gradient_129_x64", "kind": "gradient", "sizes": "128x128*64"},
        # one direction on the largest grids of the tests, beside odd ones
        {"name": "tangent_257", "kind": "tangent", "sizes": "256x256*4,512x256*2,131x97*8"},
        # uneven grids, the sizes of the uneven batch and odd ones
        {"name": "linearize_uneven", "kind": "linearize",
         "sizes": "64x64*6,128x128*6,256x256*2,33x47*4,101x75*3"},
        # a batch of stored Jacobians
        {"name": "products_129_x48", "kind": "products", "sizes": "128x128*48"},
        # host arrays in and out, one grid
        {"name": "dropin_129", "kind": "dropin", "sizes": "128x128"},
        {"name": "second_order_129", "kind": "second_order", "sizes": "128x128"},
        # the 33x33 grid of the tests at a complex shift, and the 129x129 adjoint's shift 0
        {"name": "resolvent_33", "kind": "resolvent", "sizes": "32x32", "re": 0.3, "im": 0.7},
        {"name": "resolvent_129_adjoint", "kind": "resolvent", "sizes": "128x128", "re": 0.0,
         "im": 0.0},
        # four steps on a 65x65 grid
        {"name": "ptc_65", "kind": "ptc", "sizes": "64x64", "steps": 4},
        # the sweep of the 129x129 pitch response, with the lift gradient
        {"name": "response_129_64", "kind": "response", "sizes": "128x128", "shifts": 64,
         "kmin": 0.01, "kmax": 3.0},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["residual", "residual", "gradient", "gradient", "tangent", "linearize",
                       "linearize", "products", "dropin", "second_order", "resolvent",
                       "resolvent", "ptc", "response"])
    if kind in ("residual", "gradient", "tangent", "linearize", "products"):
        cells = {"residual": 4_000_000, "gradient": 1_000_000, "tangent": 600_000,
                 "linearize": 280_000, "products": 780_000}[kind]
        groups, left = [], _log_int(rng, 64, cells)
        for _ in range(rng.randint(1, 4)):
            M, N = _log_int(rng, 4, 512), _log_int(rng, 5, 256)
            count = min(left // (M * N), 256)
            if count >= 1:
                count = _log_int(rng, 1, count)
                groups.append(f"{M}x{N}*{count}")
                left -= count * M * N
        if not groups:
            groups = [f"{_log_int(rng, 4, 64)}x{_log_int(rng, 5, 64)}"]
        return {"kind": kind, "sizes": ",".join(groups)}
    if kind in ("dropin", "second_order"):
        return {"kind": kind, "sizes": f"{_log_int(rng, 8, 128)}x{_log_int(rng, 8, 128)}"}
    if kind == "resolvent":
        M, N = _log_int(rng, 8, 128), _log_int(rng, 8, 128)
        im = rng.choice([0.0, math.exp(rng.uniform(-5.0, 1.0))])
        re = rng.choice([0.0, math.exp(rng.uniform(-5.0, 2.0))])
        return {"kind": kind, "sizes": f"{M}x{N}", "re": re, "im": im}
    if kind == "ptc":
        return {"kind": kind, "sizes": f"{_log_int(rng, 8, 64)}x{_log_int(rng, 8, 64)}",
                "steps": rng.randint(2, 5)}
    return {"kind": kind, "sizes": f"{_log_int(rng, 8, 64)}x{_log_int(rng, 8, 64)}",
            "shifts": _log_int(rng, 4, 48), "kmin": 0.01, "kmax": math.exp(rng.uniform(-1.0, 1.5))}


def _sizes(case: dict) -> list[tuple[int, int]]:
    out = []
    for group in case["sizes"].split(","):
        size, _, count = group.partition("*")
        M, N = size.split("x")
        out += [(int(M), int(N))] * int(count or 1)
    return out


# ---- inputs ------------------------------------------------------------------------------------

def _free_stream(mach, aoa_deg: float):
    a = math.radians(aoa_deg)
    speed = mach * math.sqrt(1.4)
    return 1.0, speed * math.cos(a), speed * math.sin(a)


def _smooth(gen, M: int, N: int, modes: int = 6) -> torch.Tensor:
    """A smooth field (M, N), periodic in the second index and decaying along the first."""
    th = torch.arange(N, dtype=F64, device="cuda") * (2.0 * math.pi / N)
    r = torch.arange(M, dtype=F64, device="cuda") / M
    f = torch.zeros(M, N, dtype=F64, device="cuda")
    ab = torch.randn(modes, 2, dtype=F64, device="cuda", generator=gen)
    for k in range(1, modes + 1):
        a = (ab[k - 1, 0] * torch.cos(k * th) + ab[k - 1, 1] * torch.sin(k * th)) / k
        f += a[None, :] * torch.exp(-(2.0 + k) * r)[:, None]
    return f


def _flat(a: torch.Tensor) -> torch.Tensor:
    """(var, M, N) -> the package's packed layout (var fastest, then M, then N)."""
    return a.permute(2, 1, 0).contiguous().reshape(-1)


def _inputs(case: dict, seed: int) -> list[dict]:
    """Per instance: vertices, velocities (2, M+1, N+1), states (4, M, N), Mach, angle."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    steady = case["kind"] in ("ptc", "response")
    amp, noise = (0.01, 1e-5) if steady else (0.03, 2e-3)
    grids: dict = {}
    out = []
    for M, N in _sizes(case):
        if (M, N) not in grids:
            X = naca_ogrid(M + 1, N + 1, thickness=float(rng.uniform(0.08, 0.14)), chord=1.0,
                           far_radius=20.0, first_spacing=0.01)
            grids[M, N] = (X, torch.from_numpy(np.ascontiguousarray(X)).cuda())
        X, dX = grids[M, N]
        mach, aoa = float(rng.uniform(0.3, 0.6)), float(rng.uniform(-2.0, 3.0))
        rho0, u0, w0 = _free_stream(mach, aoa)
        # primitive variables around the free stream
        rho = rho0 * (1.0 + amp * _smooth(gen, M, N))
        u = u0 + amp * _smooth(gen, M, N)
        w = w0 + amp * _smooth(gen, M, N)
        p = 1.0 + amp * _smooth(gen, M, N)
        U = torch.stack([rho, rho * u, rho * w, p / 0.4 + rho * (u * u + w * w) / 2.0])
        U = U * (1.0 + noise * torch.randn(U.shape, dtype=F64, device="cuda", generator=gen))
        V = torch.zeros(2, M + 1, N + 1, dtype=F64, device="cuda")
        if not steady:
            for d in range(2):
                V[d, :, :N] = 0.05 * _smooth(gen, M + 1, N)
            V[:, :, N] = V[:, :, 0]
        out.append(dict(M=M, N=N, X=X, dX=dX, V=V, U=U, mach=mach, aoa=aoa))
    return out


def _randn(gen, n: int) -> torch.Tensor:
    return torch.randn(n, dtype=F64, device="cuda", generator=gen)


def _extra(case: dict, inputs: list[dict], seed: int) -> dict:
    """The seeded directions and cotangents of a case (packed device vectors)."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 1_000_003)
    nc = sum(i["M"] * i["N"] for i in inputs)
    nv = sum((i["M"] + 1) * (i["N"] + 1) for i in inputs)
    kind = case["kind"]
    if kind == "gradient":
        return {"w": _randn(gen, 4 * nc)}
    if kind in ("tangent", "products"):
        return {"dU": _randn(gen, 8 * nc), "dX": _randn(gen, 4 * nv), "dV": _randn(gen, 4 * nv),
                "dMa": _randn(gen, 2 * len(inputs)), "w": _randn(gen, 8 * nc)}
    if kind == "resolvent":
        return {"b": _randn(gen, 8 * nc), "c": _randn(gen, 8 * nc)}
    if kind in ("dropin", "second_order"):
        M, N = inputs[0]["M"], inputs[0]["N"]
        d = {"w": (4, M, N), "dU": (4, M, N), "dX": (2, M + 1, N + 1)}
        return {k: torch.view_as_complex(_randn(gen, 2 * math.prod(s)).view(-1, 2)).reshape(s)
                for k, s in d.items()}
    return {}


def _host(a: torch.Tensor, dtype=float) -> np.ndarray:
    return np.asfortranarray(a.cpu().numpy(), dtype=dtype)


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    inputs = _inputs(case, seed)
    extra = _extra(case, inputs, seed)
    one = inputs[0]
    if kind in ("dropin", "second_order", "response"):
        s = SpatialDiscretization(one["X"], mach_number=one["mach"], angle_of_attack=one["aoa"],
                                  coefficient_center=(0.25, 0.0))
        s.states[:] = _host(one["U"])
        s.velocities[:] = _host(one["V"])
        if kind == "response":  # the sweep starts from a linearized solver
            s.compute_odes()
            s.linearize()
            s.compute_forces()
        return {"kind": kind, "solver": s, "case": case,
                **{k: _host(v, complex) for k, v in extra.items()}}
    inst = InstanceSet([InstanceSpec(i["X"], i["mach"], i["aoa"]) for i in inputs])
    st = {"kind": kind, "inst": inst, "case": case, **extra,
          "X": torch.cat([_flat(i["dX"]) for i in inputs]),
          "V": torch.cat([_flat(i["V"]) for i in inputs]),
          "U": torch.cat([_flat(i["U"]) for i in inputs])}
    nc, nv = inst.n_cells, inst.n_verts
    new = lambda n: torch.zeros(n, dtype=F64, device="cuda")  # noqa: E731
    if kind in ("residual", "tangent"):
        st["R"] = new((4 if kind == "residual" else 8) * nc)
    elif kind == "gradient":
        st["mach"] = torch.tensor([i["mach"] for i in inputs], dtype=F64)
        for k in ("U", "X", "V", "mach"):
            st[k].requires_grad_()
    elif kind in ("linearize", "products"):
        st["J"] = {"mach": new(4 * nc), "states": new(144 * nc), "vertices": new(32 * nc),
                   "velocities": new(32 * nc), "forces_states": new(8 * inst.n_wall),
                   "forces_vertices": new(8 * inst.n_wall)}
        if kind == "products":
            _linearize(st)
            st["out"] = {"mach_fwd": new(8 * nc), "states_fwd": new(8 * nc),
                         "vertices_fwd": new(8 * nc), "velocities_fwd": new(8 * nc),
                         "mach_rev": new(2 * len(inst)), "states_rev": new(8 * nc),
                         "vertices_rev": new(4 * nv), "velocities_rev": new(4 * nv)}
    elif kind == "resolvent":
        J = new(144 * nc)
        inst.call("eb_compute_odes_wrt_states", st["X"], st["V"], st["U"], J, stream=_stream())
        st["J"], st["lu"] = J, solver.RingLU(inst.batch)
    elif kind == "ptc":
        st.update(U0=st["U"].clone(), R=new(4 * nc), J=new(144 * nc))
        need = solver._bind_ptc().eb_ptc_workspace_bytes(one["M"], one["N"], case["steps"])
        st["workspace"] = torch.empty(int(need), dtype=torch.uint8, device="cuda")
    return st


def _linearize(st: dict) -> None:
    inst, X, V, U, J, s = st["inst"], st["X"], st["V"], st["U"], st["J"], _stream()
    inst.call("eb_compute_odes_wrt_mach", X, V, U, J["mach"], stream=s)
    inst.call("eb_compute_odes_wrt_states", X, V, U, J["states"], stream=s)
    inst.call("eb_compute_odes_wrt_vertices", X, V, U, J["vertices"], stream=s)
    inst.call("eb_compute_odes_wrt_velocities", X, V, U, J["velocities"], stream=s)
    inst.call("eb_compute_forces_wrt_states", X, U, J["forces_states"], stream=s)
    inst.call("eb_compute_forces_wrt_vertices", X, U, J["forces_vertices"], stream=s)


def run(st: dict):
    kind = st["kind"]
    if kind in ("dropin", "second_order", "response"):
        return _run_class(kind, st)
    inst, X, V, U, s = st["inst"], st["X"], st["V"], st["U"], _stream()
    if kind == "residual":
        inst.call("eb_compute_odes", X, V, U, st["R"], stream=s)
        return st["R"]
    if kind == "gradient":
        R = residual(U, X, V, st["mach"], inst)
        return [R.detach(), *torch.autograd.grad(R, (U, X, V, st["mach"]), st["w"])]
    if kind == "tangent":
        inst.call("eb_apply_odes_tangent", X, V, U, st["dU"], st["dX"], st["dV"], st["dMa"],
                  st["R"], None, stream=s)
        return st["R"]
    if kind == "linearize":
        _linearize(st)
        return st["J"]
    if kind == "products":
        J, o = st["J"], st["out"]
        inst.call("eb_apply_odes_wrt_mach_fwd", J["mach"], st["dMa"], o["mach_fwd"], stream=s)
        inst.call("eb_apply_odes_wrt_states_fwd", J["states"], st["dU"], o["states_fwd"], stream=s)
        inst.call("eb_apply_odes_wrt_vertices_fwd", J["vertices"], st["dX"], o["vertices_fwd"],
                  stream=s)
        inst.call("eb_apply_odes_wrt_vertices_fwd", J["velocities"], st["dV"],
                  o["velocities_fwd"], stream=s)
        inst.call("eb_apply_odes_wrt_mach_rev", J["mach"], st["w"], o["mach_rev"], stream=s)
        inst.call("eb_apply_odes_wrt_states_rev", J["states"], st["w"], o["states_rev"], stream=s)
        inst.call("eb_apply_odes_wrt_vertices_rev", J["vertices"], st["w"], o["vertices_rev"],
                  stream=s)
        inst.call("eb_apply_odes_wrt_vertices_rev", J["velocities"], st["w"],
                  o["velocities_rev"], stream=s)
        return o
    if kind == "resolvent":
        lu = st["lu"]
        lu.factor(st["J"], complex(st["case"]["re"], st["case"]["im"]))
        x, _ = lu.solve(st["b"])
        y, _ = lu.solve(st["c"], adjoint=True)
        return [x, y]
    if kind == "ptc":
        U.copy_(st["U0"])
        norms, rels, _ = solver.ptc_run(inst.batch, X, V, U, st["R"], st["J"], rtol=1e-10,
                                        max_steps=st["case"]["steps"], workspace=st["workspace"])
        return {"U": U, "R": st["R"], "J": st["J"], "norms": norms, "rel_norms": rels}
    raise ValueError(kind)


def _run_class(kind: str, st: dict):
    s = st["solver"]
    if kind == "dropin":
        s.compute_odes()
        s.compute_forces()
        s.linearize()
        rhs = (s.apply_odes_wrt_vertices_fwd(st["dX"])
               + s.apply_odes_wrt_velocities_fwd(0.1j * st["dX"]))
        dF = s.apply_forces_wrt_vertices_fwd(st["dX"]) + s.apply_forces_wrt_states_fwd(st["dU"])
        return {"odes": s.odes, "forces": s.forces, "rhs": rhs, "d_forces": dF,
                "rev": s.apply_odes_wrt_states_rev(st["w"]),
                "rev_x": s.apply_odes_wrt_vertices_rev(st["w"])}
    if kind == "second_order":
        return {"uu": s.compute_odes_wrt_states_inner_product_wrt_states(st["w"], st["dU"]),
                "um": s.compute_odes_wrt_states_inner_product_wrt_mach(st["w"], st["dU"]),
                "ux": s.compute_odes_wrt_states_inner_product_wrt_vertices(st["w"], st["dU"])}
    ks = _reduced_frequencies(st["case"])
    cl, cm, grad = drivers.frequency_response_batched(s, 1.0, 0.25, ks, method="anchored",
                                                      lift_gradient=True)
    return {"cl": cl, "cm": cm, "grad": grad}


def _reduced_frequencies(case: dict) -> np.ndarray:
    return np.geomspace(case["kmin"], case["kmax"], case["shifts"])


def work(case: dict) -> dict:
    """Bytes that a pass has to move, and the operations of the solves (the block elimination's;
    the stencil's few hundred operations per cell are not counted)."""
    sizes = _sizes(case)
    nc = sum(M * N for M, N in sizes)
    nv = sum((M + 1) * (N + 1) for M, N in sizes)
    kind = case["kind"]
    state = 32 * nc + 32 * nv                        # U, X and V
    jac = (1152 + 256 + 256 + 32) * nc
    if kind == "residual":
        return {"bytes": state + 32 * nc, "flops": 0}
    if kind == "gradient":                           # R, w and the four gradients
        return {"bytes": state + 32 * nc * 3 + 32 * nv, "flops": 0}
    if kind == "tangent":
        return {"bytes": state + 64 * nc * 2 + 64 * nv, "flops": 0}
    if kind == "linearize":
        return {"bytes": state + jac, "flops": 0}
    if kind == "products":
        return {"bytes": 2 * jac + 64 * nc * 7 + 64 * nv * 2, "flops": 0}
    if kind == "dropin":
        return {"bytes": state + 32 * nc + 2 * jac + 64 * nc * 3 + 64 * nv, "flops": 0}
    if kind == "second_order":
        return {"bytes": state + 64 * nc * 3 + 32 * nv, "flops": 0}
    M, N = sizes[0]
    # one inversion and three products of order 4N per ring, real or complex multiply-adds
    real = 2 * 4 * (4 * N) ** 3 * M
    if kind == "resolvent":
        return {"bytes": 1152 * nc + 4 * 64 * nc, "flops": real * (1 if case["im"] == 0.0 else 4)}
    if kind == "ptc":
        return {"bytes": case["steps"] * (state + 2 * 1152 * nc),
                "flops": real * (case["steps"] - 1)}
    anchors = -(-case["shifts"] // 3)
    return {"bytes": 1152 * nc + case["shifts"] * 64 * nc, "flops": real * (4 * anchors + 1)}


# ---- the same operators in float64 torch ---------------------------------------------------------

SLOTS = ((0, 0), (0, -1), (0, -2), (0, 1), (0, 2), (-1, 0), (-2, 0), (1, 0), (2, 0))


def _abs(x):
    return torch.where(x < 0, -x, x)


def _max(x, y):
    return torch.where(x > y + 1e-8, x, y)


def _pressure(s):
    return 0.4 * (s[3] - (s[1] ** 2 + s[2] ** 2) / s[0] / 2.0)


def _flux(ll, l, r, rr, nx, nz, gx, gz, jst):
    """JST face flux with its ALE term; where ``jst`` is False the dissipation is off."""
    out = []
    phys, lam = [], []
    for s in (l, r):
        vn, p = (nx * s[1] + nz * s[2]) / s[0], _pressure(s)
        phys.append((s[0] * vn, s[1] * vn + nx * p, s[2] * vn + nz * p, (s[3] + p) * vn))
        lam.append(_abs(vn) + torch.sqrt(1.4 * p / s[0]) * torch.sqrt(nx * nx + nz * nz))
    lam = _max(lam[0], lam[1])
    pll, pl, pr, prr = _pressure(ll), _pressure(l), _pressure(r), _pressure(rr)
    sens = _max(_abs(pll - 2 * pl + pr) / (pll + 2 * pl + pr),
                _abs(pl - 2 * pr + prr) / (pl + 2 * pr + prr))
    c2 = sens * lam
    c4 = lam / 32.0 - 2.0 * c2
    c4 = torch.where(c4 < -1e-8, torch.zeros_like(c4), c4)
    for k in range(4):
        d = c2 * (r[k] - l[k]) - c4 * (rr[k] - 3 * r[k] + 3 * l[k] - ll[k])
        f = (phys[0][k] + phys[1][k]) / 2 - torch.where(jst, d, torch.zeros_like(d))
        out.append(f - (l[k] + r[k]) / 2 * (gx * nx + gz * nz))
    return torch.stack(out)


def _ode(u, x, w, mach, aoa):
    """R of every cell of a group of G equal grids from its nine states u (9, 4, M, G, N) and its
    corners x, w (4, 2, M, G, N); mach and aoa (radian) have G values."""
    M = u.shape[2]
    m = torch.arange(M, device=u.device)[:, None, None].expand(u.shape[2:])
    c, b, bb, f, ff, i, ii, o, oo = u

    def edge(p, q):
        a, e = x[p], x[q]
        return e[1] - a[1], a[0] - e[0], (w[p][0] + w[q][0]) / 2, (w[p][1] + w[q][1]) / 2

    n_i, n_f, n_o, n_b = edge(0, 1), edge(1, 2), edge(2, 3), edge(3, 0)
    d1, d2 = x[2] - x[0], x[3] - x[1]
    area = _abs(d1[0] * d2[1] - d1[1] * d2[0]) / 2
    nx, nz, gx, gz = n_i
    proj = (nx * (c[1] - gx * c[0]) + nz * (c[2] - gz * c[0])) / (nx * nx + nz * nz)
    wall = torch.stack([c[0], c[1] - 2 * nx * proj, c[2] - 2 * nz * proj, c[3]])
    speed = mach[:, None] * math.sqrt(1.4)
    one = torch.ones_like(c[0])
    far = 2 * torch.stack([one, one * speed * torch.cos(aoa)[:, None],
                           one * speed * torch.sin(aoa)[:, None],
                           one * (2.5 + speed * speed / 2)]) - c
    i = torch.where(m == 0, wall, i)
    o = torch.where(m == M - 1, far, o)
    ii = torch.where(m < 2, c, ii)
    oo = torch.where(m > M - 3, c, oo)
    yes = torch.ones_like(m, dtype=torch.bool)
    total = _flux(f, c, b, bb, *n_b, yes) + _flux(b, c, f, ff, *n_f, yes)
    total = total + _flux(o, c, i, ii, *n_i, m >= 2) + _flux(i, c, o, oo, *n_o, m <= M - 3)
    return -total / area


def _stencil(U):
    """(4, M, G, N) -> (9, 4, M, G, N); rows past the radial ends hold the end's state."""
    M = U.shape[1]
    at = torch.arange(M, device=U.device)
    return torch.stack([torch.roll(U[:, (at + dm).clamp(0, M - 1)], -dn, 3) for dm, dn in SLOTS])


def _corners(X):
    return torch.stack([X[:, :-1, :, :-1], X[:, :-1, :, 1:], X[:, 1:, :, 1:], X[:, 1:, :, :-1]])


def _forces(U, X):
    p = _pressure(U[:, 0])
    a, b = X[:, 0, :, :-1], X[:, 0, :, 1:]
    return torch.stack([p * (b[1] - a[1]), p * (a[0] - b[0])])


def _groups(inputs: list[dict]) -> list[dict]:
    """The instances of each grid size together: arrays (var, M, G, N), offsets of the parts."""
    found: dict = {}
    cells = verts = 0
    for k, one in enumerate(inputs):
        g = found.setdefault((one["M"], one["N"]), {"ids": [], "cells": [], "verts": []})
        g["ids"].append(k)
        g["cells"].append(4 * cells)
        g["verts"].append(2 * verts)
        cells += one["M"] * one["N"]
        verts += (one["M"] + 1) * (one["N"] + 1)
    out = []
    for (M, N), g in found.items():
        part = [inputs[k] for k in g["ids"]]
        vec = lambda v: torch.tensor(v, dtype=F64, device="cuda")  # noqa: E731
        aoa = vec([math.radians(i["aoa"]) for i in part])
        args = (*(torch.stack([i[k] for i in part], 2) for k in ("U", "dX", "V")),
                vec([i["mach"] for i in part]))
        f = lambda U, X, V, mach, aoa=aoa: _ode(  # noqa: E731
            _stencil(U), _corners(X), _corners(V), mach, aoa)
        out.append(dict(g, M=M, N=N, aoa=aoa, args=args, f=f))
    return out


def _unpack(v, offsets, shape, per_complex: bool = True):
    """The group's parts of a packed vector as (var, M, G, N), complex where interleaved."""
    n = math.prod(shape)
    if per_complex:
        v = torch.view_as_complex(v.view(-1, 2))
    return torch.stack([v[o:o + n].reshape(*reversed(shape)).permute(2, 1, 0) for o in offsets], 2)


def _real_imag(fn, d):
    """A linear real map of a complex argument."""
    return torch.complex(fn(d.real.contiguous()), fn(d.imag.contiguous()))


def _packed(a) -> torch.Tensor:
    """One instance's array in the package's layout (first index fastest), interleaved."""
    a = a.permute(*reversed(range(a.ndim))).contiguous().reshape(-1)
    return torch.view_as_real(a).reshape(-1) if a.is_complex() else a


def _each(a, dim: int) -> list:
    """A group's array as one packed vector per instance (the group's dimension is `dim`)."""
    return [_packed(a.select(dim, g)) for g in range(a.shape[dim])]


def _jacobians(group, U=None):
    """The six Jacobians per instance of the group, and d(odes)/d(states) as (4,4,M,G,N,9)."""
    U, X, V, mach = (group["args"][0] if U is None else U), *group["args"][1:]
    aoa, M = group["aoa"], group["M"]
    u, x, w = _stencil(U), _corners(X), _corners(V)

    def columns(fn, at, var):
        cols = []
        for j in range(var):
            for s in range(at.shape[0]):
                t = torch.zeros_like(at)
                t[s, j] = 1.0
                cols.append(torch.func.jvp(fn, (at,), (t,))[1])
        # (var * slots, 4, M, G, N) -> (4, var, M, G, N, slots)
        c = torch.stack(cols)
        return c.reshape(var, at.shape[0], *c.shape[1:]).permute(2, 0, 3, 4, 5, 1)

    Ju = columns(lambda t: _ode(t, x, w, mach, aoa), u, 4)
    rows = torch.arange(M, device=U.device)
    for s, (dm, _) in enumerate(SLOTS):
        Ju[:, :, (rows + dm < 0) | (rows + dm >= M), :, :, s] = 0.0
    Jx = columns(lambda t: _ode(u, t, w, mach, aoa), x, 2)
    Jv = columns(lambda t: _ode(u, x, t, mach, aoa), w, 2)
    Jm = torch.func.jvp(lambda t: _ode(u, x, w, t, aoa), (mach,), (torch.ones_like(mach),))[1]
    ends = torch.stack([X[:, 0, :, :-1], X[:, 0, :, 1:]])              # (2 ends, 2, G, N)
    wall = U[:, 0]

    def force(s, e):
        p = _pressure(s)
        return torch.stack([p * (e[1][1] - e[0][1]), p * (e[0][0] - e[1][0])])

    def unit(a, *at):
        t = torch.zeros_like(a)
        t[at] = 1.0
        return t

    JFu = torch.stack([torch.func.jvp(lambda t: force(t, ends), (wall,), (unit(wall, k),))[1]
                       for k in range(4)], 1)                           # (2, 4, G, N)
    JFx = torch.stack([torch.stack([torch.func.jvp(lambda t: force(wall, t), (ends,),
                                                   (unit(ends, e, k),))[1] for k in range(2)], 1)
                       for e in range(2)], -1)                          # (2, 2, G, N, ends)
    return {"mach": _each(Jm, 2), "states": _each(Ju, 3), "vertices": _each(Jx, 3),
            "velocities": _each(Jv, 3), "forces_states": _each(JFu, 2),
            "forces_vertices": _each(JFx, 2)}, Ju


class _Elimination:
    """(J - s I) or its Hermitian adjoint as a block tridiagonal system over pairs of rings."""

    def __init__(self, Ju, shift: complex, adjoint: bool, dtype=C128):
        _, _, M, N, _ = Ju.shape
        self.M, self.N, self.K, self.P = M, N, 4 * N, (M + 1) // 2
        K, P = self.K, self.P
        n = torch.arange(N, device=Ju.device)
        blocks = {}
        for s, (dm, dn) in enumerate(SLOTS):  # all rings' blocks of one offset at a time
            B = blocks.setdefault(dm, torch.zeros(M, N, 4, N, 4, dtype=dtype, device=Ju.device))
            B[:, n, :, (n + dn) % N, :] += Ju[..., s].permute(3, 2, 0, 1).to(dtype)
        eye = torch.eye(K, dtype=dtype, device=Ju.device)
        get = {}
        for dm, B in blocks.items():
            B = B.reshape(M, K, K)
            if dm == 0:
                B = B - (shift if dtype == C128 else shift.real) * eye
            for m in range(max(0, -dm), min(M, M - dm)):
                get[(m + dm, m) if adjoint else (m, m + dm)] = B[m].conj().T if adjoint else B[m]
        zero = torch.zeros(K, K, dtype=dtype, device=Ju.device)

        def pair(p, q):
            def of(a, b):
                if a >= M or b >= M:
                    return eye if a == b else zero
                return get.get((a, b), zero)
            return torch.cat([torch.cat([of(2 * p, 2 * q), of(2 * p, 2 * q + 1)], 1),
                              torch.cat([of(2 * p + 1, 2 * q), of(2 * p + 1, 2 * q + 1)], 1)])

        self.A = [[pair(p, q) if 0 <= q < P else None for q in (p - 1, p, p + 1)]
                  for p in range(P)]
        self.lu, self.up = [], []
        for p in range(P):
            D = self.A[p][1]
            if p:
                D = D - self.A[p][0] @ self.up[-1]
            self.lu.append(torch.linalg.lu_factor(D))
            if p + 1 < P:
                self.up.append(torch.linalg.lu_solve(*self.lu[-1], self.A[p][2]))

    def _times(self, x):
        out = []
        for p in range(self.P):
            v = self.A[p][1] @ x[p]
            if p:
                v = v + self.A[p][0] @ x[p - 1]
            if p + 1 < self.P:
                v = v + self.A[p][2] @ x[p + 1]
            out.append(v)
        return torch.stack(out)

    def _solve(self, b):
        z = []
        for p in range(self.P):
            r = b[p] - self.A[p][0] @ z[-1] if p else b[p]
            z.append(torch.linalg.lu_solve(*self.lu[p], r))
        for p in range(self.P - 2, -1, -1):
            z[p] = z[p] - self.up[p] @ z[p + 1]
        return torch.stack(z)

    def solve(self, rhs):
        """rhs (4, M, N) -> the solution in the same layout, refined once."""
        v = rhs.permute(1, 2, 0).reshape(self.M, self.K)
        if 2 * self.P > self.M:
            v = torch.cat([v, torch.zeros_like(v[:1])])
        v = v.reshape(self.P, 2 * self.K, 1)
        x = self._solve(v)
        x = x + self._solve(v - self._times(x))
        return x.reshape(-1, self.N, 4)[:self.M].permute(2, 0, 1)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("resolvent", "ptc", "response"):
        M, N = _sizes(case)[0]
        runs = {"resolvent": 2, "ptc": case.get("steps", 0), "response": case.get("shifts", 0) + 1}
        if runs[kind] * M * (2e9 + (8 * N) ** 3) > 1e12:  # over some 15 seconds of eliminations
            return None
    inputs = _inputs(case, seed)
    extra = _extra(case, inputs, seed)
    groups = _groups(inputs)
    if kind in ("dropin", "second_order", "response"):
        parts = {"dropin": _exact_dropin, "second_order": _exact_second_order,
                 "response": _exact_response}[kind](case, groups[0], extra)
        return {k: v.cpu().numpy() for k, v in parts.items()}
    if kind == "ptc":
        return _exact_ptc(case, groups[0])
    if kind == "resolvent":
        return _exact_resolvent(case, groups[0], extra)
    outputs: dict = {}
    for g in groups:  # the instances' parts in their order
        for key, parts in _exact_group(kind, g, extra).items():
            outputs.setdefault(key, [None] * len(inputs))
            for k, part in zip(g["ids"], parts):
                outputs[key][k] = part
    out = {k: torch.cat(v) for k, v in outputs.items()}
    if kind in ("residual", "tangent"):
        return out["R"]
    if kind == "gradient":
        return [out["R"], out["U"], out["X"], out["V"], out["mach"].cpu()]
    return out


def _pullback(f, args, w):
    """The four reverse products with a complex cotangent."""
    pull = torch.func.vjp(f, *args)[1]
    return [torch.complex(a, b) for a, b in zip(pull(w.real.contiguous()),
                                                pull(w.imag.contiguous()))]


def _exact_group(kind, g, extra) -> dict:
    f, args, M, N = g["f"], g["args"], g["M"], g["N"]
    su, sx = (4, M, N), (2, M + 1, N + 1)
    if kind == "residual":
        return {"R": _each(f(*args), 2)}
    if kind == "gradient":
        R, pull = torch.func.vjp(f, *args)
        d = pull(_unpack(extra["w"], g["cells"], su, False))
        return {"R": _each(R, 2), "U": _each(d[0], 2), "X": _each(d[1], 2), "V": _each(d[2], 2),
                "mach": list(d[3].reshape(-1, 1))}
    if kind == "linearize":
        return _jacobians(g)[0]
    d = (_unpack(extra["dU"], g["cells"], su), _unpack(extra["dX"], g["verts"], sx),
         _unpack(extra["dV"], g["verts"], sx),
         torch.view_as_complex(extra["dMa"].view(-1, 2))[g["ids"]])
    along = lambda *t: torch.func.jvp(f, args, t)[1]  # noqa: E731
    if kind == "tangent":
        return {"R": _each(torch.complex(along(*(v.real.contiguous() for v in d)),
                                         along(*(v.imag.contiguous() for v in d))), 2)}
    zero = [torch.zeros_like(a) for a in args]
    names = ("states", "vertices", "velocities", "mach")
    out = {}
    for k, name in enumerate(names):
        one = lambda t, k=k: along(*zero[:k], t, *zero[k + 1:])  # noqa: E731
        out[f"{name}_fwd"] = _each(_real_imag(one, d[k]), 2)
    rev = _pullback(f, args, _unpack(extra["w"], g["cells"], su))
    for name, v in zip(names[:3], rev):
        out[f"{name}_rev"] = _each(v, 2)
    out["mach_rev"] = list(torch.view_as_real(rev[3]))
    return out


def _exact_dropin(case, g, extra) -> dict:
    f, args = g["f"], g["args"]
    U, X, V, mach = args
    w, dU, dX = (extra[k][:, :, None] for k in ("w", "dU", "dX"))
    zU, zX, zm = torch.zeros_like(U), torch.zeros_like(X), torch.zeros_like(mach)
    rhs = (_real_imag(lambda t: torch.func.jvp(f, args, (zU, t, zX, zm))[1], dX)
           + _real_imag(lambda t: torch.func.jvp(f, args, (zU, zX, t, zm))[1], 0.1j * dX))
    dF = (_real_imag(lambda t: torch.func.jvp(_forces, (U, X), (zU, t))[1], dX)
          + _real_imag(lambda t: torch.func.jvp(_forces, (U, X), (t, zX))[1], dU))
    rev = _pullback(f, args, w)
    return {"odes": f(*args)[:, :, 0], "forces": _forces(U, X)[:, 0], "rhs": rhs[:, :, 0],
            "d_forces": dF[:, 0], "rev": rev[0][:, :, 0], "rev_x": rev[1][:, :, 0]}


def _exact_second_order(case, g, extra) -> dict:
    f, (U, X, V, mach) = g["f"], g["args"]
    w, dU = extra["w"][:, :, None], extra["dU"][:, :, None]

    def inner(wr, d):
        """The gradients of <wr, dR/dU d> with respect to U, the Mach number and X."""
        def scalar(U, X, mach):
            return (wr * torch.func.jvp(lambda t: f(t, X, V, mach), (U,), (d,))[1]).sum()
        return torch.func.grad(scalar, argnums=(0, 2, 1))(U, X, mach)

    wr, wi = w.real.contiguous(), -w.imag.contiguous()  # the cotangent enters conjugated
    dr, di = dU.real.contiguous(), dU.imag.contiguous()
    rr, ri, ir, ii = inner(wr, dr), inner(wr, di), inner(wi, dr), inner(wi, di)
    uu, um, ux = (torch.complex(rr[k] - ii[k], ri[k] + ir[k]) for k in range(3))
    return {"uu": uu[:, :, 0], "um": um, "ux": ux[:, :, 0]}


def _exact_resolvent(case, g, extra) -> list:
    Ju = _jacobians(g)[1][:, :, :, 0]
    s, shape = complex(case["re"], case["im"]), (4, g["M"], g["N"])
    x = _Elimination(Ju, s, False).solve(_unpack(extra["b"], [0], shape)[:, :, 0])
    y = _Elimination(Ju, s, True).solve(_unpack(extra["c"], [0], shape)[:, :, 0])
    return [_packed(x), _packed(y)]


def _exact_ptc(case, g) -> dict:
    U, X, V, mach = g["args"]
    norms, rels = [], []
    for _ in range(case["steps"]):
        R = g["f"](U, X, V, mach)
        norms.append(float(R.abs().max()))
        rels.append(norms[-1] / norms[0])
        J, Ju = _jacobians(g, U)
        dU = _Elimination(Ju[:, :, :, 0], complex(rels[-1] / 0.1), False, F64).solve(-R[:, :, 0])
        U = U + dU[:, :, None]
    return {"U": _packed(U[:, :, 0]), "R": _packed(R[:, :, 0]), "J": J["states"][0],
            "norms": norms, "rel_norms": rels}


def _exact_response(case, g, extra) -> dict:
    f, args = g["f"], g["args"]
    U, X, V, mach = args
    Ju = _jacobians(g)[1][:, :, :, 0]
    ma = float(mach)
    q = ma**2 * 1.4 / 2
    dX = torch.stack([X[1], -(X[0] - 0.25)])
    zU, zX, zm = torch.zeros_like(U), torch.zeros_like(X), torch.zeros_like(mach)
    rx = torch.func.jvp(f, args, (zU, dX, zX, zm))[1][:, :, 0].to(C128)
    rv = torch.func.jvp(f, args, (zU, zX, dX, zm))[1][:, :, 0].to(C128)
    F = _forces(U, X)
    dFx = torch.func.jvp(_forces, (U, X), (zU, dX))[1].to(C128)
    along = lambda t: torch.func.jvp(_forces, (U, X), (t, zX))[1]  # noqa: E731
    px = (X[0, 0, :, :-1] + X[0, 0, :, 1:]) / 2 - 0.25
    pz = (X[1, 0, :, :-1] + X[1, 0, :, 1:]) / 2
    mid = (dX[:, 0, :, :-1] + dX[:, 0, :, 1:]) / 2
    cm_x = ((F[0] * mid[1] - F[1] * mid[0]) / q).sum()  # the arm's change at fixed forces
    cl, cm = [], []
    for k in _reduced_frequencies(case):
        s = 1j * k * ma * math.sqrt(1.4) / 0.5
        dU = -_Elimination(Ju, s, False).solve(rx + s * rv)
        dF = dFx + _real_imag(along, dU[:, :, None])
        cl.append((dF[1] / q).sum())
        cm.append(((pz * dF[0] - px * dF[1]) / q).sum() + cm_x)
    gU, gX = torch.func.vjp(_forces, U, X)[1](
        torch.stack([torch.zeros_like(F[0]), torch.full_like(F[1], 1.0 / q)]))
    lam = _Elimination(Ju, 0j, True, F64).solve(gU[:, :, 0])
    grad = gX - torch.func.vjp(f, *args)[1](lam[:, :, None])[1]
    return {"cl": torch.stack(cl), "cm": torch.stack(cm), "grad": grad[:, :, 0]}
