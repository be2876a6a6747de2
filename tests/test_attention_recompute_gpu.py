"""The attention backward pass without room for its score gradients (a batch beyond the engine's buffer): dQ comes from the
kernel that recomputes the scores, and the dK / dV kernel stores none.  Against the oracle at the sizes of
test_attention_gpu.py and its tolerances (fp16 rounding of the softmax weights and score gradients), with ragged ends and
ALiBi, and against the pass with room at the size where two CTAs' worth of tiles are in flight everywhere."""
import ctypes as C

import numpy as np
import pytest

from test_attention_gpu import causal_spans, csr, rel_l2
from tscale2_b200 import capi
from tscale2_b200.device import DeviceBuffer, check, sync

pytestmark = pytest.mark.gpu


def run(variant, q, k, v, dout, start, finish, H, slope, room):
    lib = capi.load_library()
    T = q.shape[0]
    ip = lambda a: a.ctypes.data_as(C.c_void_p)
    Q, K, V, DO = (DeviceBuffer.from_numpy(x) for x in (q, k, v, dout))
    O, LSE = DeviceBuffer(q.nbytes), DeviceBuffer(T * H * 4)
    check(lib.ts2_attention_forward(0, None, 2, Q.ptr, K.ptr, V.ptr, ip(start), ip(finish), T, H, slope, O.ptr, LSE.ptr))
    sync()
    o = O.download(q.shape, np.float16)
    DS = DeviceBuffer.from_numpy((dout.astype(np.float32) * o.astype(np.float32)).reshape(T, H, 128).sum(-1).astype(np.float32))
    out = [DeviceBuffer.from_numpy(np.full((T, H * 128), np.nan, np.float32)) for _ in range(3)]
    check(lib.ts2_op_attention_backward_limited(0, None, variant, Q.ptr, K.ptr, V.ptr, DO.ptr, LSE.ptr, DS.ptr, ip(start), ip(finish), T, H,
                                                slope, *[b.ptr for b in out], room))
    sync()
    return [b.download((T, H * 128), np.float16 if variant == 3 else np.float32).astype(np.float32) for b in out]


@pytest.mark.parametrize("variant", [2, 3])
@pytest.mark.parametrize("T,frag,width,H,slope", [(128, 128, 128, 1, 0.0), (300, 100, 48, 2, 0.5), (512, 256, 1000, 2, 0.0),
                                                  (70, 35, 20, 1, 0.25), (640, 640, 64, 1, 0.0), (257, 257, 257, 3, 0.125), (1, 1, 1, 1, 0.0)])
def test_recomputed_scores_match_the_oracle(oracle_port, variant, T, frag, width, H, slope):
    rng = np.random.default_rng(T + width + H)
    q, k, v, dout = (rng.standard_normal((T, 128 * H)).astype(np.float16) for _ in range(4))
    k = (k.astype(np.float32) * 1.7).astype(np.float16)
    start, finish = causal_spans(T, frag, width)
    ref = oracle_port.attention(q.astype(np.float32), k.astype(np.float32), v.astype(np.float32), H, slope, csr(start, finish),
                                dout.astype(np.float32))
    for name, got in zip(("dq", "dk", "dv"), run(variant, q, k, v, dout, start, finish, H, slope, 0)):
        assert np.isfinite(got).all() and rel_l2(got, ref[name]) < 3e-3 or not (got.any() or ref[name].any()), name


@pytest.mark.parametrize("variant", [2, 3])
def test_spans_that_are_not_monotone(oracle_port, variant):
    rng = np.random.default_rng(3)
    T, H = 200, 1
    q, k, v, dout = (rng.standard_normal((T, 128 * H)).astype(np.float16) for _ in range(4))
    start = rng.integers(0, T, T).astype(np.int32)
    finish = np.minimum(T - 1, start + rng.integers(-3, 60, T)).astype(np.int32)
    none = finish < start
    start[none], finish[none] = 0, -1
    ref = oracle_port.attention(q.astype(np.float32), k.astype(np.float32), v.astype(np.float32), H, 0.0, csr(start, finish),
                                dout.astype(np.float32))
    for name, got in zip(("dq", "dk", "dv"), run(variant, q, k, v, dout, start, finish, H, 0.0, 0)):
        assert rel_l2(got, ref[name]) < 3e-3, name


@pytest.mark.parametrize("slope", [0.0, 0.25])
def test_with_and_without_room_agree_at_scale(slope):
    T, H, frag = 16384, 12, 1024
    rng = np.random.default_rng(7)
    q, k, v, dout = (rng.standard_normal((T, H * 128)).astype(np.float16) for _ in range(4))
    start, finish = causal_spans(T, frag, frag)
    want = run(2, q, k, v, dout, start, finish, H, slope, 4 << 30)
    for variant in (2, 3):
        got = run(variant, q, k, v, dout, start, finish, H, slope, 0)
        for name, a, b in zip(("dq", "dk", "dv"), got, want):
            assert rel_l2(a, b) < 1e-3, name  # one fp16 rounding of the output in variant 3, and none or the last bit of dS in 2
