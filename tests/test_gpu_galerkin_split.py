"""Galerkin products of the exact FP64 setup with a node's rows split among
warps and half warps, at node counts on both sides of the rules (2432 fine
nodes; 608 and 9728 coarse ones) and with one and several levels of 2-D and
3-D blocks: the reference's order of rounded products, to the 1e-12 of the
largest entry that the level operators are held to."""
import numpy as np
import pytest

import oracle
from sparlab_gb300 import problems as P
from sparlab_gb300.linear_solver import GpuAmgCgSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nx,ny,nz", [(3, 5, 4, 3), (3, 19, 11, 9), (3, 34, 23, 21), (2, 13, 9, 0),
                                          (2, 61, 41, 0), (2, 191, 83, 0), (2, 401, 233, 0)])
def test_level_operators(dim, nx, ny, nz):
    spec = P.bench_model(dim, nx, ny, nz)
    rho = P.SplitMix64(7).uniform_array(spec.num_elements, 0.01, 1.0)
    pr = oracle.Problem(spec)
    ptr, col, val = pr.kff(1e-9 + (1 - 1e-9) * rho ** 3)
    ref = oracle.Solver(rtol=1e-12, coarse_size=60)
    ref.factorize(ptr, col, val, dim, pr.coords(), pr.free_dofs())
    gpu = GpuAmgCgSolver(coarse_size=60)
    gpu.set_layout(dim, pr.coords(), pr.free_dofs())
    gpu.factorize(ptr, col, val)
    assert gpu.amg_stats()["num_levels"] == ref.num_levels() >= 2
    for lvl in range(1, ref.num_levels()):
        gp, gc, gv = gpu.level_matrix(lvl)
        rp, rc, rv = ref.level_matrix(lvl)
        np.testing.assert_array_equal(gp, rp)
        np.testing.assert_array_equal(gc, rc)
        assert np.abs(gv - rv).max() <= 1e-12 * np.abs(rv).max()
