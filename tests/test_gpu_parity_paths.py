"""Callers of the parity operator above its sizes (20,000 grid nodes for the CG
product, 150,000 for the FP32 cycle): supports on other faces and inside the
grid, one smoothing step a sweep, the FP32 CG operator, modal and buckling
analyses with their own stiffness factors, and roller supports, which keep the
general kernels.

Bounds: products as in test_gpu_parity.py (1e-11 and 1e-5 of max |K x|);
compliances and eigenvalues the 1e-6 that mixed precision is held to."""
import numpy as np
import pytest

from sparlab_gb300 import problems as P
from sparlab_gb300.topopt import GpuSimpProblem

pytestmark = pytest.mark.gpu

BIG = (61, 47, 52)  # 157,728 nodes


def clamp(spec, nodes, components=(0, 1, 2)):
    for k in components:
        spec.fixed[np.asarray(nodes) * 3 + k] = 1


def supported(n, kind):
    spec = P.hex8_cantilever(*n, 0.3, "paths")
    nx, ny, nz = n
    if kind == "faces":       # no node of x = 0, all of y = 0 and of z = nz
        spec.fixed[:] = 0
        clamp(spec, P.box_nodes(spec, ymax=0.0))
        clamp(spec, P.box_nodes(spec, zmin=float(nz)))
    elif kind == "inside":    # single nodes and a block of them
        clamp(spec, np.random.default_rng(1).choice((nx + 1) * (ny + 1) * (nz + 1), 300, replace=False))
        clamp(spec, P.box_nodes(spec, 29.0, 33.0, 6.0, 9.0, 10.0, 12.0))
    elif kind == "roller":    # y alone on one face
        clamp(spec, P.box_nodes(spec, ymax=0.0), (1,))
    spec.loads = spec.loads * (1 - spec.fixed)
    return spec


def products(spec):
    import torch
    x = P.seeded_density(spec, 11, 0.0, 1.0)
    v = torch.from_numpy(np.random.default_rng(5).standard_normal(len(spec.free_dofs()))).cuda()
    out = []
    for precision in ("fp64", "mixed"):
        prob = GpuSimpProblem(spec, precision=precision)
        prob.set_design(x)
        prob.evaluate(arrays=False)
        y, y0 = torch.zeros_like(v), torch.zeros_like(v)
        prob.apply_operator(v.data_ptr(), y.data_ptr())
        prob.apply_level0(v.data_ptr(), y0.data_ptr())
        torch.cuda.synchronize()
        out.append((y, y0))
        prob.close()
    (ref, _), (cg, cycle) = out
    return float((cg - ref).abs().max() / ref.abs().max()), float((cycle - ref).abs().max() / ref.abs().max())


@pytest.mark.parametrize("kind", ["faces", "inside", "roller"])
def test_products_with_other_supports(kind):
    cg, cycle = products(supported(BIG, kind))
    assert cg <= 1e-11 and cycle <= 1e-5, (cg, cycle)


def solved(spec, precision, **options):
    prob = GpuSimpProblem(spec, precision=precision, **options)
    prob.set_design(P.seeded_density(spec, 4, 0.2, 1.0))
    spec_ev = [prob.evaluate(arrays=False) for _ in range(2)]  # the first setup and a reuse
    prob.close()
    return [(e.compliance, e.linear_iterations) for e in spec_ev]


@pytest.mark.parametrize("options", [dict(smoother_degree=1), dict(matrix_free=2),
                                     dict(matrix_free=2, smoother_degree=1)])
def test_solves_with_vectors_in_planes(options):
    spec = P.hex8_cantilever(*BIG, 0.3, "paths")
    spec.warm_start = 0
    got = solved(spec, "mixed", **options)
    ref = solved(spec, "fp64", **{k: v for k, v in options.items() if k != "matrix_free"})
    for (c, it), (cr, itr) in zip(got, ref):
        assert abs(c / cr - 1) <= 1e-6
        if "matrix_free" not in options:  # (its restarts add iterations)
            assert abs(it - itr) <= 2


@pytest.mark.parametrize("nx,ny,nz", [(52, 20, 19), (61, 47, 52)])  # 22,260 nodes; cycle vectors in planes too
def test_modal(nx, ny, nz):
    spec = P.hex8_cantilever(nx, ny, nz, 0.3, "paths")
    spec.density = 7.8
    ks = 1e-3 + P.SplitMix64(8).uniform_array(spec.num_elements, 0.05, 1.0) ** 3
    values = {}
    for precision in ("fp64", "mixed"):
        prob = GpuSimpProblem(spec, precision=precision)
        m = prob.modal(num_modes=3, stiffness_scale=ks, tolerance=1e-9, mode_shapes=False)
        assert m.converged
        values[precision] = m.eigenvalues
        prob.close()
    np.testing.assert_allclose(values["mixed"], values["fp64"], rtol=1e-6)


def test_buckling():
    spec = P.column(3, 90, 15, 15, height=0.12, width=0.12)  # 23,296 nodes
    ks = 0.5 + P.SplitMix64(9).uniform_array(spec.num_elements, 0.0, 1.0)
    factors = {}
    for precision in ("fp64", "mixed"):
        prob = GpuSimpProblem(spec, precision=precision)
        b = prob.buckling(num_modes=2, stiffness_scale=ks, mode_shapes=False)
        assert b.converged
        factors[precision] = b.load_factors
        prob.close()
    np.testing.assert_allclose(factors["mixed"], factors["fp64"], rtol=1e-6)
