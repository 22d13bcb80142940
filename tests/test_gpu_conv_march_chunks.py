"""The marching convolution where a chunk of output layers is a single layer
behind whole ones (with c = ceil(nz / ceil(nz / m)) layers a chunk, m = 256 / n:
the march's start and end meet in it), in both directions; and its split BF16
outputs with ReLU.  Bounds: FP32 sums of at most 27 x 48 products, 1e-5 of the
largest output; a BF16 output is rounded once more, 2^-8 of itself."""
import ctypes as C

import numpy as np
import pytest

from sparlab_gb300 import _lib

pytestmark = pytest.mark.gpu


def convolve(cseg, n, grid, flip, relu, outputs):
    """(outputs of the kernel as FP64, FP64 sums) of random tensors."""
    import torch
    nx, ny, nz = grid
    rng = np.random.default_rng(sum(cseg) + n + nz + flip)
    dev = torch.device("cuda", 0)

    def tensor(*shape):
        return torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).to(dev).to(torch.bfloat16)

    xs = [tensor(nz, ny, nx, c) for c in cseg]
    w = tensor(27, n, sum(cseg))
    bias = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).to(dev)
    outs = [torch.full((nz, ny, nx, c), float("nan"), dtype=torch.float32 if f32 else torch.bfloat16, device=dev)
            for c, f32 in outputs]
    pair, ptrs = C.c_int32 * 2, C.c_void_p * 2
    pad, opad = [0] * (2 - len(xs)), [0] * (2 - len(outs))
    channels = [c for c, _ in outputs]
    code = _lib.load().simp_conv3d_bf16(
        C.c_int32(nx), C.c_int32(ny), C.c_int32(nz), C.c_int32(len(xs)), ptrs(*[t.data_ptr() for t in xs], *pad),
        pair(*cseg, *pad), C.c_void_p(w.data_ptr()), C.c_int32(n), C.c_void_p(bias.data_ptr()), C.c_int32(relu),
        C.c_int32(flip), C.c_int32(len(outs)), ptrs(*[t.data_ptr() for t in outs], *opad), pair(*channels, *opad),
        pair(*channels, *opad), pair(*[int(f) for _, f in outputs], *opad))
    assert code == 0, _lib.load().simp_surrogate_last_error().decode()
    torch.cuda.synchronize()
    x = torch.nn.functional.pad(torch.cat(xs, 3).double(), (0, 0, 1, 1, 1, 1, 1, 1))
    ref = bias.double().expand(nz, ny, nx, n).clone()
    for t in range(27):
        k, j, i = t // 9, t // 3 % 3, t % 3
        if flip:
            k, j, i = 2 - k, 2 - j, 2 - i
        ref += x[k:k + nz, j:j + ny, i:i + nx] @ w[t].double().t()
    return torch.cat([t.double() for t in outs], 3), ref.clamp(min=0.0) if relu else ref


@pytest.mark.parametrize("flip", [0, 1])
@pytest.mark.parametrize("cseg,n,nz", [
    ((32,), 64, 13),    # 4 + 4 + 4 + 1 layers
    ((16,), 48, 21),    # 5 x 4 + 1
    ((16,), 32, 57),    # 8 x 7 + 1
    ((16,), 16, 241),   # 16 x 15 + 1
    ((32, 16), 16, 241),
])
def test_last_chunk_of_one_layer(cseg, n, nz, flip):
    out, ref = convolve(cseg, n, (33, 5, nz), flip, 0, [(n, True)])
    assert (out - ref).abs().max() <= 1e-5 * ref.abs().max()


@pytest.mark.parametrize("flip", [0, 1])
def test_split_bf16_outputs(flip):
    out, ref = convolve((16,), 48, (40, 7, 11), flip, 1, [(32, False), (16, False)])
    assert ((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * ref.abs().max()).all()
