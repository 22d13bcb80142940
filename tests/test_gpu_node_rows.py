"""The FP32 products of the 3-D coarse levels by a warp a node, at node counts
around the eight nodes of a block and row lengths around the 64 columns of a
step, through what the FP32 reuse setup and the solve make of them.  The
spectral estimate: twelve Lanczos steps with FP32 rows of n <= 1000 products on
FP32 values move an eigenvalue by at most the norm of their rounding, 12
sqrt(n) 2^-24 = 2.3e-5 of it (1e-4 taken).  The iteration count: a
preconditioner whose levels are good to 1e-3 converges as the FP64 one does,
to one iteration."""
import numpy as np
import pytest

import oracle
from sparlab_gb300 import problems as P
from sparlab_gb300.linear_solver import GpuAmgCgSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(5, 4, 3), (9, 7, 5), (16, 8, 8), (23, 13, 11), (40, 18, 15)])
def test_estimates_and_iterations(nx, ny, nz):
    spec = P.bench_model(3, nx, ny, nz)
    pr = oracle.Problem(spec)
    matrix = pr.kff(None)
    f = spec.loads[0][pr.free_dofs()]
    got = {}
    for precision in ("fp64", "mixed"):
        gpu = GpuAmgCgSolver(precision=precision, coarse_size=60, iterative_tolerance=1e-8)
        gpu.set_layout(3, pr.coords(), pr.free_dofs())
        gpu.factorize(*matrix)
        gpu.factorize(*matrix)  # the reuse setup, FP32 in mixed precision
        gpu.solve(f)
        got[precision] = ([lv["lambda_max"] for lv in gpu.amg_stats()["levels"]], gpu.last_iterations())
    assert len(got["fp64"][0]) == len(got["mixed"][0]) >= 2
    np.testing.assert_allclose(got["mixed"][0], got["fp64"][0], rtol=1e-4)
    assert abs(got["mixed"][1] - got["fp64"][1]) <= 1
