"""The level-0 operator in the cell's parity basis (double-float CG product and
FP32 cycle product of mixed precision) against the FP64 assembled product,
at grids around the edges of its blocks: 31 node columns a warp, 8 (FP32) or 4
(double-float) node rows a block, chunks of node layers, and around the
sizes from which it is used.  Element matrices without the box cell's
symmetry keep the general kernels.

Bounds, of max |K x| for x of unit normal entries: the double-float product
1e-11 (the bound of the CG operator's own test); the FP32 product rounds each
of at most 8 x 24 terms and the vectors to 2^-24, 1e-5."""
import numpy as np
import pytest

from sparlab_gb300 import problems as P
from sparlab_gb300.topopt import GpuSimpProblem, element_stiffness

pytestmark = pytest.mark.gpu


def products(spec, element_matrix=None):
    import torch
    x = P.seeded_density(spec, 11, 0.0, 1.0)
    v = torch.from_numpy(np.random.default_rng(5).standard_normal(len(spec.free_dofs()))).cuda()
    out = []
    for precision in ("fp64", "mixed"):
        prob = GpuSimpProblem(spec, precision=precision, element_matrix=element_matrix)
        prob.set_design(x)
        prob.evaluate(arrays=False)
        y, y0 = torch.zeros_like(v), torch.zeros_like(v)
        prob.apply_operator(v.data_ptr(), y.data_ptr())
        prob.apply_level0(v.data_ptr(), y0.data_ptr())
        torch.cuda.synchronize()
        out.append((y.cpu().numpy(), y0.cpu().numpy()))
        prob.close()
    (ref, _), (cg, cycle) = out
    scale = np.abs(ref).max()
    return np.abs(cg - ref).max() / scale, np.abs(cycle - ref).max() / scale


@pytest.mark.parametrize("n", [
    (61, 47, 52),     # 62 = 2 x 31 columns, 48 = 6 x 8 rows, 157 k nodes: both products
    (62, 48, 49),     # one column and one row more
    (30, 30, 156),    # a single block column, long march, 150,877 nodes
    (60, 46, 50),     # 146 k nodes: the CG product alone
    (31, 11, 52),     # 20,352 nodes: just above the CG product's size
    (92, 2, 71),      # fewer rows than a block
    (200, 99, 1),     # one cell layer
])
def test_products_match_fp64(n):
    cg, cycle = products(P.hex8_cantilever(*n, 0.3, "parity"))
    assert cg <= 1e-11, cg
    assert cycle <= 1e-5, cycle


def test_unequal_edges_and_element_without_the_symmetry():
    spec = P.hex8_cantilever(40, 30, 20, 0.3, "parity")
    spec.lx, spec.ly, spec.lz = 40.0, 21.0, 33.0
    spec.fixed = P.clamp_left(spec)
    cg, cycle = products(spec)
    assert cg <= 1e-11 and cycle <= 1e-5, (cg, cycle)
    # a symmetric term that couples the parities: the general kernels
    ke = element_stiffness(3, 1.0, 0.7, 1.65, 1.0, 0.3)
    w = ke @ np.random.default_rng(2).standard_normal(24)
    cg, cycle = products(spec, ke + 0.05 * np.outer(w, w))
    assert cg <= 1e-11 and cycle <= 1e-5, (cg, cycle)
