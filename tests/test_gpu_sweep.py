"""The dense sweep of the coarse solve on whole matrices (one level), at sizes
around its 32-wide pivot blocks and 16-row update tiles: with the inverse
exact to cond * 2^-53 (below 1e-6 here) the second CG iteration is at the
1e-12 tolerance, and the pivots' ratio is that of the Cholesky factor's
squared diagonal to cond * 2^-53 (below 1e-6)."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle
from sparlab_gb300 import problems as P
from sparlab_gb300.linear_solver import GpuAmgCgSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nx,ny,nz,n", [(2, 1, 1, 0, 4), (2, 8, 1, 0, 32), (2, 17, 1, 0, 68), (3, 4, 1, 1, 48),
                                            (3, 8, 1, 1, 96), (2, 5, 12, 0, 130), (3, 6, 6, 6, 882),
                                            (2, 25, 29, 0, 1500)])
def test_inverse_and_pivots(dim, nx, ny, nz, n):
    spec = P.bench_model(dim, nx, ny, nz)
    pr = oracle.Problem(spec)
    ptr, col, val = pr.kff(None)
    assert len(ptr) - 1 == n
    gpu = GpuAmgCgSolver(iterative_tolerance=1e-12)
    gpu.set_layout(spec.dim, pr.coords(), pr.free_dofs())
    gpu.factorize(ptr, col, val)
    st = gpu.amg_stats()
    assert st["num_levels"] == 1
    k = sp.csr_matrix((val, col, ptr), shape=(n, n)).toarray()
    d = np.diag(np.linalg.cholesky(k)) ** 2
    assert abs(st["coarse_pivot_ratio"] / (d.min() / d.max()) - 1) <= 1e-6
    b = np.random.default_rng(n).standard_normal(n)
    x = gpu.solve(b)
    assert gpu.last_iterations() <= 2
    assert np.linalg.norm(k @ x - b) <= 1e-11 * np.linalg.norm(b)
