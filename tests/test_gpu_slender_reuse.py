"""Reuse setups of slender beams in mixed precision, whose coarse operators lose
their definiteness to FP32 Galerkin products: every evaluation solves, to the
FP64 loop's compliance within the 1e-6 that mixed precision is held to.  A matrix
that is indefinite in FP64 too stays refused, and the one after it is taken
again."""
import numpy as np
import pytest

import oracle
from sparlab_gb300 import problems as P
from sparlab_gb300._lib import SolverError
from sparlab_gb300.linear_solver import GpuAmgCgSolver
from sparlab_gb300.topopt import GpuSimpProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,solid", [((140, 4, 4), True), ((260, 4, 4), False), ((300, 8, 8), True), ((460, 8, 8), True),
                                     ((700, 15, 15), True)])  # level-0 vectors in planes
def test_evaluations_after_the_first(n, solid):
    spec = P.hex8_cantilever(*n, 0.3, "slender")
    spec.warm_start = 0
    x = np.ones(spec.num_elements) if solid else P.seeded_density(spec, 4, 0.2, 1.0)
    got = {}
    for precision in ("fp64", "mixed"):
        prob = GpuSimpProblem(spec, precision=precision)
        prob.set_design(x)
        evs = [prob.evaluate(arrays=False) for _ in range(3)]
        got[precision] = [e.compliance for e in evs]
        prob.close()
    np.testing.assert_allclose(got["mixed"], got["fp64"], rtol=1e-6)


def test_drop_in_solver_and_an_indefinite_matrix():
    spec = P.hex8_cantilever(140, 4, 4, 0.3, "slender")
    pr = oracle.Problem(spec)
    ptr, col, val = pr.kff(None)
    f = spec.loads[0][pr.free_dofs()]
    gpu = GpuAmgCgSolver(precision="mixed", iterative_tolerance=1e-8, coarse_size=200)
    gpu.set_layout(3, pr.coords(), pr.free_dofs())
    gpu.factorize(ptr, col, val)
    first = gpu.solve(f)
    gpu.factorize(ptr, col, val)
    again = gpu.solve(f)
    assert abs((f @ again) / (f @ first) - 1) <= 1e-6
    shifted = val.copy()
    rows = np.repeat(np.arange(len(ptr) - 1), np.diff(ptr))
    shifted[rows == col] -= 0.1 * val[rows == col].min()
    with pytest.raises(SolverError, match="under-constrained|positive"):
        gpu.factorize(ptr, col, shifted)
    gpu.factorize(ptr, col, val)
    assert abs((f @ gpu.solve(f)) / (f @ first) - 1) <= 1e-6
