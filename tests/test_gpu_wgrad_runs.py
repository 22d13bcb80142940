"""The tensor-core weight gradient's accumulator runs, on sums of one sign, where
the tensor core's truncation (up to 2^-23 of the running sum an instruction,
always towards zero) adds up: runs of 2, 4 and 8 instructions of 16 nodes, of
which the longest loses up to (1 + .. + 8) / 8 x 2^-23 = 5.4e-7 of the sum.  The runs
are added rounded to nearest, in 50 walkers' partials: n / (128 x 50) additions
of 2^-24 each, random, below 1e-7 at 545,025 nodes.  Bound 1e-6; one unbroken
run of a walker's 681 instructions would lose 8e-6."""
import ctypes as C

import numpy as np
import pytest

from sparlab_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(20, 20, 20), (32, 31, 33), (129, 65, 65)])
def test_sums_of_one_sign(grid):
    import torch
    nx, ny, nz = grid
    rng = np.random.default_rng(nx)
    dev = torch.device("cuda", 0)
    x, dy = (torch.from_numpy(rng.uniform(0.5, 1.0, (nz, ny, nx, 16)).astype(np.float32)).to(dev).to(torch.bfloat16)
             for _ in range(2))
    gw, gb = torch.zeros((27, 16, 16), device=dev), torch.zeros(16, device=dev)
    code = _lib.load().simp_conv3d_wgrad(C.c_int32(nx), C.c_int32(ny), C.c_int32(nz), C.c_int32(1),
                                         (C.c_void_p * 2)(x.data_ptr(), 0), (C.c_int32 * 2)(16, 0),
                                         C.c_void_p(dy.data_ptr()), C.c_int32(16), C.c_int32(16),
                                         C.c_void_p(gw.data_ptr()), C.c_void_p(gb.data_ptr()))
    assert code == 0, _lib.load().simp_surrogate_last_error().decode()
    pad = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    d = dy.double().reshape(-1, 16)
    for t in range(27):
        k, j, i = t // 9, t // 3 % 3, t % 3
        ref = d.t() @ pad[k:k + nz, j:j + ny, i:i + nx].reshape(-1, 16)
        assert ((gw[t].double() - ref).abs() / ref).max() <= 1e-6
    assert ((gb.double() - d.sum(0)).abs() / d.sum(0)).max() <= 1e-6
