"""The multi-RHS CG operator (one launch over a shared assembled K_ff above 128
MiB of value pairs for up to four load cases): problems whose CG operator is
assembled -- Hex8 with matrix_free=0, Q4 -- advanced in one graph compute what
their load cases compute one after another, bit for bit.  Five load cases are
two launches, three are one."""
import numpy as np
import pytest

from sparlab_gb300 import problems as P
from sparlab_gb300.topopt import GpuSimpProblem

pytestmark = pytest.mark.gpu


def hex8():
    spec = P.hex8_cantilever(64, 36, 36, 0.3, "fused")
    loads = []
    for i in range(5):
        rng = P.SplitMix64(9, i)
        node = spec.node_index(64, int(rng.uniform(0.0, 36.99)), int(rng.uniform(0.0, 36.99)))
        t = np.radians(rng.uniform(-90.0, 90.0))
        loads.append(P.point_load(spec, [node], (0.0, np.sin(t), -np.cos(t))))
    spec.loads = np.stack(loads)
    return spec, dict(matrix_free=0)


def q4():
    n = 700
    spec = P.ProblemSpec(dim=2, nx=n, ny=n, nz=0, lx=float(n), ly=float(n), lz=0.0)
    spec.fixed = P.clamp_left(spec)
    spec.loads = np.stack([P.point_load(spec, [spec.node_index(n, j)], (0.3, -1.0)) for j in (10, 350, 600)])
    return spec, {}


@pytest.mark.parametrize("make", [hex8, q4])
def test_load_cases_share_a_launch(make):
    spec, options = make()
    spec.weights = np.full(len(spec.loads), 1.0 / len(spec.loads))
    spec.rtol = 1e-10
    out = {}
    for mode in (False, "graph"):
        prob = GpuSimpProblem(spec, precision="mixed", block_pcg=mode, **options)
        assert prob.nnz * 8 >= 128 * 1024 * 1024
        recs = [prob.iterate() for _ in range(3)]
        out[mode] = [(r.compliance, r.linear_iterations, r.lam, r.bisections) for r in recs]
        prob.close()
    assert out["graph"] == out[False]
