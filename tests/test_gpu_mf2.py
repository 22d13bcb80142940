"""The matrix-free Q4 operator of the FP32 cycle against the FP64 assembled
product, at grids around its 32 x 4 node blocks.  FP32 sums of at most 4 x 8
products of numbers rounded to 2^-24: below 1e-5 of max |K x| for x of unit
normal entries."""
import numpy as np
import pytest

from sparlab_gb300 import problems as P
from sparlab_gb300.topopt import GpuSimpProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (31, 3), (32, 4), (63, 8), (7, 61), (130, 45)])
def test_level0_product(nx, ny):
    import torch
    spec = P.ProblemSpec(dim=2, nx=nx, ny=ny, nz=0, lx=float(nx), ly=1.3 * ny, lz=0.0)
    spec.fixed = P.clamp_left(spec)
    spec.loads = P.point_load(spec, [spec.node_index(nx, ny // 2)], (0.3, -1.0))[None, :]
    spec.weights = np.ones(1)
    x = P.seeded_density(spec, 4, 0.0, 1.0)
    v = torch.from_numpy(np.random.default_rng(nx).standard_normal(len(spec.free_dofs()))).cuda()
    got = {}
    for precision in ("fp64", "mixed"):
        prob = GpuSimpProblem(spec, precision=precision)
        prob.set_design(x)
        prob.evaluate(arrays=False)
        got[precision] = torch.zeros_like(v)
        prob.apply_level0(v.data_ptr(), got[precision].data_ptr())
        torch.cuda.synchronize()
        prob.close()
    assert (got["mixed"] - got["fp64"]).abs().max() <= 1e-5 * got["fp64"].abs().max()
