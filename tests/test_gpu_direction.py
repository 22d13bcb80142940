"""The CG direction update with four values a thread (1.25 M unknowns and more;
neither count is a multiple of the 1024 values of a block): a lost or repeated
value would end the mixed-precision solve short of its tolerance.  Compliance
against the FP64 solve within the 1e-6 that mixed precision is held to."""
import numpy as np
import pytest

from sparlab_gb300 import problems as P
from sparlab_gb300.topopt import GpuSimpProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(760, 818), (800, 800)])  # 1,244,880 and 1,281,600 unknowns: both sides
def test_large_solve(nx, ny):
    spec = P.ProblemSpec(dim=2, nx=nx, ny=ny, nz=0, lx=float(nx), ly=float(ny), lz=0.0)
    spec.fixed = P.clamp_left(spec)
    spec.loads = P.point_load(spec, [spec.node_index(nx, ny // 2)], (0.0, -1.0))[None, :]
    spec.weights = np.ones(1)
    x = P.seeded_density(spec, 4, 0.3, 1.0)
    compliance = {}
    for precision in ("fp64", "mixed"):
        prob = GpuSimpProblem(spec, precision=precision)
        prob.set_design(x)
        ev = prob.evaluate(arrays=False)
        compliance[precision] = ev.compliance
        prob.close()
    assert abs(compliance["mixed"] / compliance["fp64"] - 1) <= 1e-6
