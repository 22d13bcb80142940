"""The work a user of the SIMP library has it do, as timed cases.

Every case is one call (or the two or three calls of one step) through the
public Python entry points of ``sparlab_gb300``:

* ``iterate``: one SIMP iteration of a resident problem -- the design set,
  filter, SIMP law, assembly, AMG reuse setup, one PCG solve per load case,
  sensitivities, OC update -- and the new design copied back;
* ``evaluate``: the two halves of the iteration as ``ComplianceObjective`` and
  ``optimality_criteria_update`` callers use them, with every output array
  (densities, gradients, energies, displacements) copied to the host;
* ``batch``: one SIMP iteration of several uneven independent instances with
  their solves advanced together;
* ``solve``: the drop-in linear solver alone: factorize a host CSR matrix
  whose pattern is known (aggregates reused) and solve it;
* ``forward`` / ``gradient``: the displacement surrogate's inference and one
  training example's forward and backward pass.

Sizes, radii, volume fractions, tolerances and load counts are those of the
workloads, benchmark decks and tests of this repository, or lie between them.
Designs are seeded fields with the densities of a run's early iterations
(dense flanges and members in a grey field); problems are created, and their hierarchy is
built on the uniform start design, in ``prepare``, as a run's first iteration
does.  Solves start from zero (``warm_start = 0``): a pass is then the same
work however often it is repeated.
"""
import math
import random

import numpy as np
import torch

from sparlab_gb300 import problems as P
from sparlab_gb300.linear_solver import GpuAmgCgSolver
from sparlab_gb300.surrogate import LAYERS, Surrogate
from sparlab_gb300.topopt import GpuSimpProblem, iterate_batch

EMIN, PENALTY, MOVE, POISSON = 1e-9, 3.0, 0.2, 0.3


def _simp(name, op, nx, ny, nz, precision, loads=1, radius=1.5, vf=0.3, rtol=1e-8, projection=False):
    return {"name": name, "op": op, "nx": nx, "ny": ny, "nz": nz, "precision": precision, "loads": loads,
            "radius": radius, "vf": vf, "rtol": rtol, "projection": projection}


def listed():
    return [
        # interactive 2-D studies and continuation loops: the smallest workload,
        # a call's latency and its launches
        _simp("q4_120x40", "iterate", 120, 40, 0, "mixed", vf=0.5),
        # the default precision on the 2-D benchmark grid with a wide filter
        # (radius 4.5 cells), gradients and displacements read back
        _simp("q4_180x60_fp64_arrays", "evaluate", 180, 60, 0, "fp64", radius=4.5, vf=0.5, rtol=1e-10),
        # the fine 2-D workload: three load cases solved at the same time
        _simp("q4_600x200_3loads", "iterate", 600, 200, 0, "mixed", loads=3, radius=3.0, vf=0.35),
        # the small 3-D benchmark bracket: two load cases, plain FP64
        _simp("hex8_32x16x8_fp64", "iterate", 32, 16, 8, "fp64", loads=2, rtol=1e-10),
        # a part with odd, unequal edges in plain FP64
        _simp("hex8_61x37x29_fp64", "iterate", 61, 37, 29, "fp64", vf=0.25),
        # the large bracket: Heaviside projection, two load cases, gradients read back
        _simp("hex8_96x48x24_projected", "evaluate", 96, 48, 24, "mixed", loads=2, rtol=1e-10, projection=True),
        # the middle 3-D workload
        _simp("hex8_96x48x48", "iterate", 96, 48, 48, "mixed", vf=0.2),
        # the headline workload: 1.77 M elements, 5.4 M unknowns
        _simp("hex8_192x96x96", "iterate", 192, 96, 96, "mixed", vf=0.15),
        # a parameter sweep: uneven small instances advanced together
        {"name": "batch_12_uneven", "op": "batch", "q4": 8, "hex8": 4, "precision": "mixed", "rtol": 1e-8},
        # a finite-element code that calls the linear solver alone (host matrix)
        {"name": "solve_48x24x12", "op": "solve", "nx": 48, "ny": 24, "nz": 12, "precision": "fp64", "vf": 0.3,
         "rtol": 1e-10},
        # the learned start's inference at the headline workload's nodes
        {"name": "surrogate_forward_193x97x97", "op": "forward", "nx": 193, "ny": 97, "nz": 97},
        # its training step's forward and backward pass on the larger training grid
        {"name": "surrogate_gradient_97x49x49", "op": "gradient", "nx": 97, "ny": 49, "nz": 49},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["iterate", "iterate", "iterate", "iterate", "evaluate", "evaluate", "batch", "solve", "forward",
                     "gradient"])
    if op == "batch":
        return {"op": op, "q4": rng.randint(2, 10), "hex8": rng.randint(1, 5),
                "precision": rng.choice(["mixed", "fp64"]), "rtol": 1e-8}
    if op in ("forward", "gradient"):
        # the network's grids halve three times: any node counts from 17
        big = 193 if op == "forward" else 97
        return {"op": op, "nx": _log(rng, 33, big), "ny": _log(rng, 17, big // 2), "nz": _log(rng, 17, big // 2)}
    if op == "solve":
        if rng.random() < 0.4:
            return {"op": op, "nx": _log(rng, 60, 400), "ny": _log(rng, 30, 150), "nz": 0, "precision": "fp64",
                    "vf": rng.uniform(0.2, 0.5), "rtol": 1e-10}
        return {"op": op, "nx": _log(rng, 20, 64), "ny": _log(rng, 10, 32), "nz": _log(rng, 6, 24),
                "precision": rng.choice(["fp64", "mixed"]), "vf": rng.uniform(0.2, 0.5), "rtol": 1e-10}
    precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
    if rng.random() < 0.35:
        nx = _log(rng, 64, 600)
        ny = max(24, min(200, int(nx * rng.uniform(0.25, 0.6))))
        nz, radius = 0, rng.choice([1.5, 2.0, 3.0, 4.5])
    else:
        top = 150 if precision == "mixed" else 72
        nx = _log(rng, 20, top)
        ny, nz = (max(6, int(nx * rng.uniform(0.25, 0.6))) for _ in range(2))
        radius = rng.choice([1.5, 1.5, 2.0])
    case = _simp("", op, nx, ny, nz, precision, loads=rng.choice([1, 1, 2, 3]), radius=radius,
                 vf=round(rng.uniform(0.15, 0.5), 3), rtol=rng.choice([1e-8, 1e-10]),
                 projection=op == "evaluate" and rng.random() < 0.5)
    del case["name"]
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _design(nx, ny, nz, vf, seed):
    """Element densities of a run's early iterations, x fastest: dense flanges
    and seeded members growing out of a grey field, mean vf."""
    r = random.Random(seed)
    shape = (max(nz, 1), ny, nx)
    x = torch.arange(nx, dtype=torch.float64).add(0.5).div(nx).view(1, 1, nx)
    y = torch.arange(ny, dtype=torch.float64).add(0.5).div(ny).view(1, ny, 1)
    z = torch.arange(shape[0], dtype=torch.float64).add(0.5).div(shape[0]).view(-1, 1, 1)
    h = z if nz else y     # the bending direction
    f = 1.2 * (2.0 * h - 1.0).abs().pow(2) * (1.0 - 0.3 * x) + torch.zeros(shape, dtype=torch.float64)
    for _ in range(8):
        k = [r.uniform(-5.0, 5.0), r.uniform(-3.0, 3.0), r.uniform(-3.0, 3.0) if nz else 0.0]
        f = f + 0.22 * torch.cos(2.0 * math.pi * (k[0] * x + k[1] * y + k[2] * z) + r.uniform(0.0, 6.28))
    f = f.reshape(-1)
    lo, hi = -4.0, 4.0
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        d = 0.03 + 0.97 * torch.sigmoid(2.5 * (f - mid))
        if float(d.mean()) > vf:
            lo = mid
        else:
            hi = mid
    return (0.03 + 0.97 * torch.sigmoid(2.5 * (f - hi))).numpy()


def _spec(nx, ny, nz, seed, loads, radius, vf, rtol, projection=False):
    """A cantilever of unit cells, x = 0 clamped, with seeded loads spread over
    short runs of nodes on the far face."""
    dim = 3 if nz else 2
    spec = P.ProblemSpec(dim=dim, nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=float(nz), poisson=POISSON,
                         filter_radius=radius, volume_fraction=vf, rtol=rtol, warm_start=0, projection=projection,
                         penalty=PENALTY, emin_ratio=EMIN, move_limit=MOVE)
    spec.fixed = P.clamp_left(spec)
    r = random.Random(seed * 7919 + 17)
    cases = []
    for _ in range(loads):
        j0 = r.randint(0, ny - 1)
        js = range(j0, min(ny, j0 + max(1, ny // 8)) + 1)
        k = r.randint(0, nz) if nz else 0
        t = r.uniform(-0.6, 0.6)
        force = (math.sin(t), -math.cos(t)) if dim == 2 else (0.3 * math.sin(3 * t), math.sin(t), -math.cos(t))
        cases.append(P.point_load(spec, [spec.node_index(nx, j, k) for j in js], force))
    spec.loads = np.stack(cases)
    spec.weights = np.array([1.0 / (1 + k) for k in range(loads)])
    return spec


def _simp_spec(case, seed):
    return _spec(case["nx"], case["ny"], case["nz"], seed, case["loads"], case["radius"], case["vf"], case["rtol"],
                 case["projection"])


def _batch_specs(case, seed):
    r = random.Random(seed * 104729 + 5)
    out = []
    for q in range(case["q4"] + case["hex8"]):
        # instance sizes are the case's, not the seed's: the work stays the same
        s = random.Random(1000 * case["q4"] + 10 * case["hex8"] + q)
        if q < case["q4"]:
            n = (s.randint(64, 256), s.randint(32, 128), 0)
        else:
            n = (s.randint(16, 40), s.randint(16, 40), s.randint(16, 40))
        out.append((_spec(*n, r.randint(0, 1 << 30), s.randint(1, 3), 1.5, s.uniform(0.2, 0.5), case["rtol"]), n))
    return out


def _network_tensors(case, seed):
    g = torch.Generator().manual_seed(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x = torch.zeros((nz, ny, nx, 16))
    x[..., 0] = torch.rand((nz, ny, nx), generator=g)                 # density
    x[nz // 2, :, -1, 3] = -torch.rand((ny,), generator=g)           # a tip edge load
    target = torch.rand((nz, ny, nx, 3), generator=g) * 2.0 - 1.0
    mask = torch.full((nz, ny, nx), 7, dtype=torch.uint8)
    mask[:, :, 0] = 0
    params = []
    for cins, cout in LAYERS:
        cin = sum(cins)
        params.append(torch.randn(27 * cout * cin, generator=g) * math.sqrt(2.0 / (27 * cin)))
        params.append(torch.randn(cout, generator=g) * 0.01)
    return x.to(torch.bfloat16), target.to(torch.bfloat16), mask, torch.cat(params)


def prepare(case, seed):
    op = case["op"]
    if op in ("iterate", "evaluate"):
        prob = GpuSimpProblem(_simp_spec(case, seed), precision=case["precision"])
        prob.evaluate(arrays=False)          # the first iteration's hierarchy, at the uniform design
        return {"op": op, "prob": prob, "x": _design(case["nx"], case["ny"], case["nz"], case["vf"], seed)}
    if op == "batch":
        probs, xs = [], []
        for k, (spec, n) in enumerate(_batch_specs(case, seed)):
            probs.append(GpuSimpProblem(spec, precision=case["precision"]))
            probs[-1].evaluate(arrays=False)
            xs.append(_design(*n, spec.volume_fraction, seed * 31 + k))
        return {"op": op, "probs": probs, "xs": xs}
    if op == "solve":
        spec = _spec(case["nx"], case["ny"], case["nz"], seed, 1, 0.0, case["vf"], case["rtol"])
        prob = GpuSimpProblem(spec)
        x = _design(case["nx"], case["ny"], case["nz"], case["vf"], seed)
        ptr, col, start = prob.kff(np.full(x.size, case["vf"] ** PENALTY))
        _, _, values = prob.kff(EMIN + x ** PENALTY * (1.0 - EMIN))
        prob.close()
        solver = GpuAmgCgSolver(iterative_tolerance=case["rtol"], precision=case["precision"])
        free = spec.free_dofs()
        solver.set_layout(spec.dim, spec.node_coords(), free)
        solver.factorize(ptr, col, start)
        return {"op": op, "solver": solver, "matrix": (ptr, col, values), "b": spec.loads[0][free]}
    x, target, mask, params = _network_tensors(case, seed)
    sur = Surrogate(seed=7)
    sur.set_params(params.numpy())
    dims = (case["nx"], case["ny"], case["nz"])
    state = {"op": op, "sur": sur, "dims": dims, "x": x.cuda()}
    if op == "forward":
        state["out"] = torch.zeros((dims[2], dims[1], dims[0], 3), device="cuda")
    else:
        state["target"], state["mask"] = target.cuda(), mask.cuda()
        state["count"] = 3 * int((mask > 0).sum())
    torch.cuda.synchronize()
    return state


def _step(rec, x):
    return {"compliance": rec.compliance, "volume_fraction": rec.volume_fraction, "max_change": rec.max_change,
            "gray_level": rec.gray_level, "x": x}


def run(state):
    op = state["op"]
    if op == "iterate":
        prob = state["prob"]
        prob.set_design(state["x"])
        return _step(prob.iterate(), prob.design())
    if op == "evaluate":
        prob = state["prob"]
        prob.set_design(state["x"])
        ev = prob.evaluate(arrays=True, displacements=True)
        step = prob.oc_update(apply=False)
        return {"compliance": ev.compliance, "volume": ev.volume, "rho": ev.physical_density,
                "dc_dphysical": ev.dc_dphysical, "dc_dx": ev.dc_dx, "dv_dx": ev.dv_dx,
                "energy": ev.element_strain_energy, "u": ev.displacements, "x": step.x}
    if op == "batch":
        for prob, x in zip(state["probs"], state["xs"]):
            prob.set_design(x)
        recs = iterate_batch(state["probs"])
        return [_step(r, p.design()) for r, p in zip(recs, state["probs"])]
    if op == "solve":
        state["solver"].factorize(*state["matrix"])
        return {"u": state["solver"].solve(state["b"])}
    if op == "forward":
        state["sur"].forward(*state["dims"], state["x"].data_ptr(), state["out"].data_ptr())
        return {"out": state["out"]}
    loss, grad = state["sur"].loss_gradient(*state["dims"], state["x"].data_ptr(), state["target"].data_ptr(),
                                            state["mask"].data_ptr(), state["count"])
    return {"loss": loss, "gradient": grad}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _solve_flops(cells, dim, solves):
    """Twenty products with K per solve (a V-cycle's and the CG's of a few
    iterations), element by element."""
    ed = 24 if dim == 3 else 8
    return 20.0 * solves * 2.0 * ed * ed * cells


def work(case):
    op = case["op"]
    if op in ("forward", "gradient"):
        flops, grid = 0.0, float(case["nx"]) * case["ny"] * case["nz"]
        level = [0, 0, 1, 1, 2, 2, 3, 3, 2, 1, 0, 0]
        for (cins, cout), l in zip(LAYERS, level):
            flops += 2.0 * 27 * sum(cins) * cout * grid / 8 ** l
        params = sum(27 * sum(c) * n + n for c, n in LAYERS)
        if op == "forward":
            return {"bytes": grid * (32 + 12) + 2 * params, "flops": flops}
        return {"bytes": grid * (32 + 6 + 1) + 6 * params, "flops": 3 * flops}
    if op == "batch":
        by = fl = 0.0
        for spec, n in _batch_specs(case, 0):
            cells = spec.num_elements
            by += 8.0 * (2 * cells + len(spec.weights) * spec.num_dofs)
            fl += _solve_flops(cells, spec.dim, len(spec.weights))
        return {"bytes": by, "flops": fl}
    dim = 3 if case["nz"] else 2
    cells = float(case["nx"]) * case["ny"] * max(case["nz"], 1)
    dofs = dim * (case["nx"] + 1.0) * (case["ny"] + 1) * (case["nz"] + 1)
    if op == "solve":
        nnz = dofs * dim * (27 if dim == 3 else 9)
        return {"bytes": 12.0 * nnz + 16.0 * dofs, "flops": _solve_flops(cells, dim, 1)}
    arrays = 7 if op == "evaluate" else 2
    return {"bytes": 8.0 * (arrays * cells + case["loads"] * dofs), "flops": _solve_flops(cells, dim, case["loads"])}


# ---------------------------------------------------------------------------
# 64-bit values without the library
# ---------------------------------------------------------------------------
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
MOST_DENSE = 24000      # unknowns of a dense factorisation


def _element_matrix(dim):
    """Stiffness of a unit cell (E = 1, thickness 1) by 2-point quadrature."""
    g = 1.0 / math.sqrt(3.0)
    corner = CORNERS[: 2 ** dim]
    ke = np.zeros((dim * len(corner),) * 2)
    if dim == 2:
        f = 1.0 / (1.0 - POISSON ** 2)
        d = f * np.array([[1, POISSON, 0], [POISSON, 1, 0], [0, 0, 0.5 * (1 - POISSON)]])
    else:
        lam = POISSON / ((1 + POISSON) * (1 - 2 * POISSON))
        mu = 0.5 / (1 + POISSON)
        d = np.diag([lam + 2 * mu] * 3 + [mu] * 3)
        d[:3, :3] += lam * (1 - np.eye(3))
    points = np.stack(np.meshgrid(*[[-g, g]] * dim, indexing="ij"), -1).reshape(-1, dim)
    for p in points:
        b = np.zeros((len(d), len(ke)))
        for a, c in enumerate(corner):
            s = [2 * c[k] - 1 for k in range(dim)]
            v = [0.5 * (1 + s[k] * p[k]) for k in range(dim)]
            gr = [s[k] * np.prod([v[o] for o in range(dim) if o != k]) for k in range(dim)]
            for k in range(dim):
                b[k, dim * a + k] = gr[k]
            pairs = [(0, 1)] if dim == 2 else [(0, 1), (1, 2), (2, 0)]
            for q, (i, j) in enumerate(pairs):
                b[dim + q, dim * a + i] = gr[j]
                b[dim + q, dim * a + j] = gr[i]
        ke += 0.5 ** dim * b.T @ d @ b
    return 0.5 * (ke + ke.T)


def _element_dofs(spec):
    dim, nx, ny = spec.dim, spec.nx, spec.ny
    nz = max(spec.nz, 1)
    ez, ey, ex = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    dofs = []
    for cx, cy, cz in CORNERS[: 2 ** dim]:
        node = ((ez + cz) * (ny + 1) + ey + cy) * (nx + 1) + ex + cx
        dofs += [(dim * node + k).ravel() for k in range(dim)]
    return np.stack(dofs, 1)


def _solve_dense(spec, scale, loads):
    """Displacements (loads x dofs) by a dense Cholesky factorisation with
    two steps of iterative refinement."""
    ke, ed = torch.from_numpy(_element_matrix(spec.dim)).cuda(), torch.from_numpy(_element_dofs(spec)).cuda()
    free = torch.from_numpy(spec.free_dofs().astype(np.int64)).cuda()
    place = torch.full((spec.num_dofs,), -1, dtype=torch.int64, device="cuda")
    place[free] = torch.arange(free.numel(), device="cuda")
    n = free.numel()
    local = place[ed]
    k = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    s = torch.from_numpy(scale).cuda()
    for a in range(ed.shape[1]):
        for b in range(ed.shape[1]):
            ok = (local[:, a] >= 0) & (local[:, b] >= 0)
            k.index_add_(0, (local[:, a] * n + local[:, b])[ok], (s * ke[a, b])[ok])
    k = k.view(n, n)
    rhs = torch.from_numpy(loads).cuda()[:, free].t().contiguous()
    chol = torch.linalg.cholesky(k)
    u = torch.cholesky_solve(rhs, chol)
    for _ in range(2):
        u = u + torch.cholesky_solve(rhs - k @ u, chol)
    full = torch.zeros((loads.shape[0], spec.num_dofs), dtype=torch.float64, device="cuda")
    full[:, free] = u.t()
    ue = full[:, ed]                                        # loads x elements x ed
    energy = torch.einsum("lea,ab,leb->le", ue, ke, ue)     # u_e^T K_e u_e
    return full.cpu().numpy(), energy.cpu().numpy()


class _Filter:
    """Cone weights r - distance, rows normalised (unit cells)."""

    def __init__(self, spec):
        self.shape = (max(spec.nz, 1), spec.ny, spec.nx)
        reach = int(math.ceil(spec.filter_radius))
        zs = range(-reach, reach + 1) if spec.dim == 3 else [0]
        self.taps = []
        for dz in zs:
            for dy in range(-reach, reach + 1):
                for dx in range(-reach, reach + 1):
                    w = spec.filter_radius - math.sqrt(dx * dx + dy * dy + dz * dz)
                    if w > 0.0:
                        self.taps.append(((dz, dy, dx), w))
        self.rows = self._sum(np.ones(self.shape))

    def _sum(self, a):
        out = np.zeros(self.shape)
        for off, w in self.taps:
            to = tuple(slice(max(0, -o), min(n, n - o)) for o, n in zip(off, self.shape))
            at = tuple(slice(max(0, o), min(n, n + o)) for o, n in zip(off, self.shape))
            if all(s.stop > s.start for s in to):
                out[to] += w * a[at]
        return out

    def forward(self, x):
        return (self._sum(x.reshape(self.shape)) / self.rows).ravel()

    def adjoint(self, v):
        return self._sum(v.reshape(self.shape) / self.rows).ravel()


def _exact_step(spec, x):
    """Evaluation and optimality-criteria step in 64 bits."""
    flt = _Filter(spec)
    filtered = np.clip(flt.forward(x), 0.0, 1.0)
    if spec.projection:
        beta, eta = spec.beta_start, spec.eta
        den = math.tanh(beta * eta) + math.tanh(beta * (1.0 - eta))
        project = lambda v: (math.tanh(beta * eta) + np.tanh(beta * (v - eta))) / den  # noqa: E731
        slope = beta * (1.0 - np.tanh(beta * (filtered - eta)) ** 2) / den
    else:
        project, slope = lambda v: v, np.ones_like(filtered)  # noqa: E731
    rho = project(filtered)
    scale = EMIN + (1.0 - EMIN) * rho ** PENALTY
    u, quad = _solve_dense(spec, scale, spec.loads)
    w = spec.weights / spec.weights.sum()
    c = float((w * (u * spec.loads).sum(axis=1)).sum())
    dcp = -PENALTY * (1.0 - EMIN) * rho ** (PENALTY - 1.0) * (w @ quad)
    dcx, dvx = flt.adjoint(dcp * slope), flt.adjoint(slope)
    target = spec.volume_fraction * x.size
    g = x * np.sqrt(np.maximum(0.0, -dcx / dvx))
    low, high = np.maximum(0.0, x - MOVE), np.minimum(1.0, x + MOVE)
    lo, hi = -60.0, 60.0
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        xn = np.clip(g * math.exp(-0.5 * mid), low, high)
        if project(np.clip(flt.forward(xn), 0.0, 1.0)).sum() > target:
            lo = mid
        else:
            hi = mid
    return {"compliance": c, "rho": rho, "dcp": dcp, "dcx": dcx, "dvx": dvx, "energy": 0.5 * scale * (w @ quad), "u": u,
            "x": xn}


def _exact_iterate(spec, x):
    e = _exact_step(spec, x)
    return {"compliance": e["compliance"], "volume_fraction": float(e["rho"].mean()),
            "max_change": float(np.abs(e["x"] - x).max()),
            "gray_level": float(4.0 * (e["rho"] * (1.0 - e["rho"])).mean()), "x": e["x"]}


def exact(case, seed):
    op = case["op"]
    if op in ("forward", "gradient"):
        return None      # every layer rounds to 16 bits: no 64-bit value of the whole network
    if op == "batch":
        got = [None if s.free_dofs().size > 8000 else _exact_iterate(s, _design(*n, s.volume_fraction, seed * 31 + k))
               for k, (s, n) in enumerate(_batch_specs(case, seed))]
        return got if any(g is not None for g in got) else None
    dim = 3 if case["nz"] else 2
    if dim * case["nx"] * (case["ny"] + 1) * (case["nz"] + 1) > MOST_DENSE:
        return None
    x = _design(case["nx"], case["ny"], case["nz"], case["vf"], seed)
    if op == "solve":
        spec = _spec(case["nx"], case["ny"], case["nz"], seed, 1, 0.0, case["vf"], case["rtol"])
        u, _ = _solve_dense(spec, EMIN + x ** PENALTY * (1.0 - EMIN), spec.loads)
        return {"u": u[0][spec.free_dofs()]}
    spec = _simp_spec(case, seed)
    if op == "iterate":
        return _exact_iterate(spec, x)
    e = _exact_step(spec, x)
    return {"compliance": e["compliance"], "volume": float(e["rho"].sum()), "rho": e["rho"], "dc_dphysical": e["dcp"],
            "dc_dx": e["dcx"], "dv_dx": e["dvx"], "energy": e["energy"], "u": e["u"], "x": e["x"]}
