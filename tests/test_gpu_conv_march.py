"""The marching convolution (weights resident, one loaded layer serving three
output layers) against FP64 sums: grids around its 32 x 4 node tiles and its
chunks of output layers, every pair of input segments it takes, both
directions, and a layer it leaves to the per-tap kernel.  FP32 outputs: at
most 27 x 64 products accumulated in FP32, below 1e-5 of the largest output."""
import ctypes as C

import numpy as np
import pytest

from sparlab_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cseg,n,grid,flip", [
    ((16,), 16, (32, 4, 16), 0),       # one full chunk of 16 layers
    ((16,), 16, (33, 5, 17), 1),       # a column, a row and a layer more, marching down
    ((16,), 48, (20, 9, 11), 1),       # 5 layers a chunk: the last has one
    ((16,), 32, (1, 1, 1), 0),         # one node
    ((32,), 32, (65, 3, 9), 1),
    ((32,), 64, (31, 8, 5), 0),        # 4 layers a chunk
    ((32, 16), 16, (40, 7, 18), 0),    # a concatenated input
    ((64,), 32, (33, 5, 3), 0),        # the per-tap kernel
])
def test_convolution(cseg, n, grid, flip):
    import torch
    nx, ny, nz = grid
    rng = np.random.default_rng(sum(cseg) + n + nx)
    dev = torch.device("cuda", 0)

    def tensor(*shape):
        return torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).to(dev).to(torch.bfloat16)

    xs = [tensor(nz, ny, nx, c) for c in cseg]
    w = tensor(27, n, sum(cseg))
    bias = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).to(dev)
    out = torch.full((nz, ny, nx, n), float("nan"), dtype=torch.float32, device=dev)
    pad = [0] * (2 - len(xs))
    pair = C.c_int32 * 2
    code = _lib.load().simp_conv3d_bf16(
        C.c_int32(nx), C.c_int32(ny), C.c_int32(nz), C.c_int32(len(xs)),
        (C.c_void_p * 2)(*[t.data_ptr() for t in xs], *pad), pair(*cseg, *pad), C.c_void_p(w.data_ptr()),
        C.c_int32(n), C.c_void_p(bias.data_ptr()), C.c_int32(0), C.c_int32(flip), C.c_int32(1),
        (C.c_void_p * 2)(out.data_ptr(), 0), pair(n, 0), pair(n, 0), pair(1, 0))
    assert code == 0, _lib.load().simp_surrogate_last_error().decode()
    torch.cuda.synchronize()
    x = torch.nn.functional.pad(torch.cat(xs, 3).double(), (0, 0, 1, 1, 1, 1, 1, 1))
    ref = bias.double().expand(nz, ny, nx, n).clone()
    for t in range(27):
        k, j, i = t // 9, t // 3 % 3, t % 3
        if flip:
            k, j, i = 2 - k, 2 - j, 2 - i
        ref += x[k:k + nz, j:j + ny, i:i + nx] @ w[t].double().t()
    assert (out.double() - ref).abs().max() <= 1e-5 * ref.abs().max()
