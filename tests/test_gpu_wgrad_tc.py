"""The tensor-core weight gradient against FP64 sums, at grids around its tiles
(32 x 4 x 1 nodes), around the size where its accumulators run longer
(2^15 nodes), and for every width of segment; and the CUDA-core kernel for
channel counts it does not take.

Bound, of the largest gradient: a gradient sums at most 2^16 products of two
8-bit significands, exact in FP32, in accumulator runs of 64 truncated to
2^-24 each and partial sums rounded to nearest; signs are random here, so
2^-24 x (64 + sqrt(2^16 / 64)) of the root-mean-square sum, below 1e-5 of the
largest."""
import ctypes as C

import numpy as np
import pytest

from sparlab_gb300 import _lib

pytestmark = pytest.mark.gpu


def exact(xs, dy):
    import torch
    x = torch.nn.functional.pad(torch.cat(xs, 3).double(), (0, 0, 1, 1, 1, 1, 1, 1))
    nz, ny, nx, co = dy.shape
    d = dy.double().reshape(-1, co)
    taps = [d.t() @ x[k:k + nz, j:j + ny, i:i + nx].reshape(-1, x.shape[3])
            for k in range(3) for j in range(3) for i in range(3)]
    return torch.stack(taps), d.sum(0)


@pytest.mark.parametrize("cseg,cdy,cout,grid", [
    ((16,), 16, 16, (32, 4, 2)),       # whole tiles
    ((16,), 16, 3, (33, 5, 3)),        # one column and row more; fewer outputs than columns
    ((32,), 32, 32, (31, 3, 1)),       # less than a tile
    ((64,), 64, 64, (1, 1, 1)),        # one node
    ((64, 64), 64, 64, (20, 9, 4)),    # four segments
    ((32, 16), 16, 16, (40, 33, 25)),  # 33,000 nodes: long runs
    ((64, 32), 32, 32, (64, 32, 16)),  # 2^15 nodes: short runs
    ((24,), 40, 40, (9, 7, 5)),        # channel counts of the CUDA-core kernel
])
def test_weight_gradient(cseg, cdy, cout, grid):
    import torch
    nx, ny, nz = grid
    rng = np.random.default_rng(sum(cseg) + cout + nx)
    dev = torch.device("cuda", 0)

    def tensor(*shape):
        return torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).to(dev).to(torch.bfloat16)

    xs = [tensor(nz, ny, nx, c) for c in cseg]
    dy = tensor(nz, ny, nx, cdy)
    cin = sum(cseg)
    gw = torch.ones((27, cout, cin), device=dev)      # the gradient is added to what is there
    gb = torch.ones(cout, device=dev)
    ptrs = (C.c_void_p * 2)(*[t.data_ptr() for t in xs], *([0] * (2 - len(xs))))
    code = _lib.load().simp_conv3d_wgrad(C.c_int32(nx), C.c_int32(ny), C.c_int32(nz), C.c_int32(len(cseg)), ptrs,
                                         (C.c_int32 * 2)(*cseg, *([0] * (2 - len(cseg)))), C.c_void_p(dy.data_ptr()),
                                         C.c_int32(cdy), C.c_int32(cout), C.c_void_p(gw.data_ptr()),
                                         C.c_void_p(gb.data_ptr()))
    assert code == 0, _lib.load().simp_surrogate_last_error().decode()
    w, b = exact(xs, dy[..., :cout])
    assert (gw.double() - 1.0 - w).abs().max() <= 1e-5 * max(w.abs().max(), 1.0)
    assert (gb.double() - 1.0 - b).abs().max() <= 1e-5 * max(b.abs().max(), 1.0)
