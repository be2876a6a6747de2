"""Scratch of the operator-level calls: an attention backward pass whose score gradients cannot be allocated recomputes the
scores and leaves no error behind it, and the memory kept between calls can be given back."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_attention_gpu import causal_spans
from tscale2_b200 import capi
from tscale2_b200.device import DeviceBuffer, check, sync

pytestmark = pytest.mark.gpu

T, H = 8192, 8
SCORE_GRADIENTS = 64 * 65 // 2 * 2 * 16384 * H  # one causal document


class Call:
    def __init__(self, T=T, H=H):
        self.T, self.H = T, H
        self.lib = capi.load_library()
        rng = np.random.default_rng(5)
        self.q, self.k, self.v, self.dout = (DeviceBuffer.from_numpy(rng.standard_normal((T, 128 * H)).astype(np.float16)) for _ in range(4))
        self.start, self.finish = causal_spans(T, T, T)
        self.o, self.lse = DeviceBuffer(T * 128 * H * 2), DeviceBuffer(T * H * 4)
        self.dscale = DeviceBuffer.from_numpy(rng.standard_normal((T, H)).astype(np.float32))
        self.grads = [DeviceBuffer(T * 128 * H * 4) for _ in range(3)]
        ip = [a.ctypes.data_as(C.c_void_p) for a in (self.start, self.finish)]
        check(self.lib.ts2_attention_forward(0, None, 2, self.q.ptr, self.k.ptr, self.v.ptr, *ip, T, H, 0.0, self.o.ptr, self.lse.ptr))
        self.spans = ip
        sync()

    def backward(self):
        check(self.lib.ts2_attention_backward(0, None, 2, self.q.ptr, self.k.ptr, self.v.ptr, self.dout.ptr, self.lse.ptr, self.dscale.ptr,
                                              *self.spans, self.T, self.H, 0.0, *[g.ptr for g in self.grads]))
        return [g.download((self.T, 128 * self.H), np.float32) for g in self.grads]


def free_bytes():
    return torch.cuda.mem_get_info()[0]


def test_without_room_for_the_score_gradients_the_call_succeeds_and_leaves_no_error():
    cudart = C.CDLL("libcudart.so.12")  # the one this library and the caller's framework share
    call = Call()
    want = call.backward()
    check(call.lib.ts2_dev_trim(0))
    text = call.lib.ts2_last_error(None)
    held, left = [], SCORE_GRADIENTS // 2
    try:
        while free_bytes() > left:
            held.append(DeviceBuffer(min(8 << 30, free_bytes() - left + (2 << 20))))
        assert free_bytes() < SCORE_GRADIENTS
        got = call.backward()
        assert cudart.cudaPeekAtLastError() == 0
        assert call.lib.ts2_last_error(None) == text
    finally:
        for b in held:
            b.free()
    # dK and dV come from the same kernel; dQ rounds the same score gradients to fp16 (2^-11 where the last bit differs)
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
    assert np.linalg.norm(got[0] - want[0]) < 5e-4 * np.linalg.norm(want[0])


def test_kept_scratch_is_given_back():
    call = Call()
    check(call.lib.ts2_dev_trim(0))
    before = free_bytes()
    call.backward()
    assert free_bytes() < before - SCORE_GRADIENTS // 2
    check(call.lib.ts2_dev_trim(0))
    assert free_bytes() > before - (64 << 20)


@pytest.mark.parametrize("heads,stored", [(6, True), (8, False)])  # 1.6 GB and 2.2 GB of score gradients
def test_a_call_takes_no_more_than_the_pool_keeps(heads, stored):
    """More would be mapped anew by every call, which takes longer than recomputing the scores."""
    call = Call(16384, heads)
    check(call.lib.ts2_dev_trim(0))
    before = free_bytes()
    call.backward()
    assert (free_bytes() < before - (1 << 30)) == stored
    check(call.lib.ts2_dev_trim(0))
