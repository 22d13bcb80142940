"""The OC update's volumes, posted by the kernels that sum them, against the
one-by-one bisection in numpy, at element counts around the 256-element
blocks, the 8 x 32 partials of the last block's first pass and the 1024-block
grid.  Sums of n <= 3e5 positive FP64 terms differ by at most n 2^-53 = 4e-11
of themselves, a bisection ends at 1e-10 of the target: the multiplier agrees
to a few 1e-10 (1e-8 taken) unless a volume lies within 4e-11 of either
threshold, and the count with it."""
import numpy as np
import pytest

from sparlab_gb300 import problems as P
from sparlab_gb300.topopt import GpuSimpProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 2), (16, 16), (257, 1), (90, 91), (257, 256), (640, 411)])
def test_update_against_sequential_bisection(nx, ny):
    spec = P.ProblemSpec(dim=2, nx=nx, ny=ny, nz=0, lx=float(nx), ly=float(ny), lz=0.0)
    spec.fixed = P.clamp_left(spec)
    spec.loads = P.point_load(spec, [spec.node_index(nx, ny // 2)], (0.3, -1.0))[None, :]
    spec.weights = np.ones(1)
    spec.volume_fraction = 0.45
    gpu = GpuSimpProblem(spec)
    x = P.seeded_density(spec, 4, 0.3, 0.6)
    gpu.set_design(x)
    ev = gpu.evaluate()
    g = x * np.sqrt(np.maximum(0.0, -ev.dc_dx / ev.dv_dx))
    lo, hi = np.maximum(0.0, x - spec.move_limit), np.minimum(1.0, x + spec.move_limit)
    volume = lambda lam: float(ev.dv_dx @ np.clip(g / np.sqrt(lam), lo, hi))
    target = 0.45 * ev.volume / ev.volume_fraction
    a, b, count = 1e-12, 1e12, 0
    while count < 200:
        mid = np.sqrt(a * b)
        count += 1
        v = volume(mid)
        if abs(v - target) <= 1e-10 * target:
            break
        a, b = (mid, b) if v > target else (a, mid)
        if b / a - 1.0 < 1e-15:
            break
    step = gpu.oc_update(apply=False)
    assert step.bisections == count
    assert abs(step.lam / mid - 1) <= 1e-8
    assert abs(step.achieved_volume / (ev.dv_dx @ step.x) - 1) <= 1e-10
    assert step.max_change == np.abs(step.x - x).max()
    assert abs(ev.volume / (target / 0.45 * np.mean(ev.physical_density)) - 1) <= 1e-10
