"""A convolution refuses pointers that its loads cannot take on the host, before
any device call: this runs without a GPU and launches nothing.  Both kernels'
channel counts (16, 32, 32 + 16: weights by 16-byte cp.async; 64: by TMA)."""
import ctypes as C

import pytest

from sparlab_gb300 import _lib

ADDRESS = 1 << 20  # never read


@pytest.mark.parametrize("flip", [0, 1])
@pytest.mark.parametrize("cseg", [(16,), (32,), (32, 16), (64,)])
@pytest.mark.parametrize("weights,inputs,what", [(ADDRESS + 2, ADDRESS, "weights"), (ADDRESS + 4, ADDRESS, "weights"),
                                                 (ADDRESS + 8, ADDRESS, "weights"), (None, ADDRESS, "weights"),
                                                 (ADDRESS, ADDRESS + 8, "activations")])
def test_misaligned_pointers_are_refused(cseg, flip, weights, inputs, what):
    pad = [0] * (2 - len(cseg))
    pair = C.c_int32 * 2
    code = _lib.load().simp_conv3d_bf16(
        C.c_int32(4), C.c_int32(4), C.c_int32(4), C.c_int32(len(cseg)), (C.c_void_p * 2)(*[inputs] * len(cseg), *pad),
        pair(*cseg, *pad), C.c_void_p(weights), C.c_int32(16), C.c_void_p(None), C.c_int32(0), C.c_int32(flip),
        C.c_int32(1), (C.c_void_p * 2)(ADDRESS, 0), pair(16, 0), pair(16, 0), pair(1, 0))
    assert code == _lib.SIMP_BAD_INPUT
    message = _lib.load().simp_surrogate_last_error().decode()
    assert what in message and "16-byte aligned" in message
