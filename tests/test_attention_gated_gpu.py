"""The attention forward with the output gate in its epilogue: o and lse are those of the plain form bit for bit, and
rg = s * sigmoid(2 gate) * o of that o, rounded to the operand format."""
import ctypes as C

import ml_dtypes
import numpy as np
import pytest

from tscale2_b200 import capi
from tscale2_b200.device import DeviceBuffer, check, sync

pytestmark = pytest.mark.gpu


# one node; a block less one, a block and one; several tiles with an odd tile count and blocks without keys
@pytest.mark.parametrize("prec", [capi.PREC_FP8, capi.PREC_F16, capi.PREC_INT8])
@pytest.mark.parametrize("T,H", [(1, 1), (127, 2), (129, 1), (700, 3)])
def test_gate_in_the_epilogue(prec, T, H):
    lib = capi.load_library()
    rng = np.random.default_rng(T + H)
    Q = 128 * H
    q, k, v = (rng.standard_normal((T, Q)).astype(np.float16) for _ in range(3))
    qkvg = (rng.standard_normal((T, 4 * Q)) * 2).astype(np.float16)
    t = np.arange(T)
    start, finish = np.maximum(0, t - 300).astype(np.int32), np.where(t // 128 % 3 == 1, -1, t - 1).astype(np.int32)
    start[finish < start] = 0
    ip = lambda a: a.ctypes.data_as(C.c_void_p)
    Qb, Kb, Vb, G = (DeviceBuffer.from_numpy(a) for a in (q, k, v, qkvg))
    O, O2, LSE, LSE2 = DeviceBuffer(T * Q * 2), DeviceBuffer(T * Q * 2), DeviceBuffer(T * H * 4), DeviceBuffer(T * H * 4)
    size = 2 if prec == capi.PREC_F16 else 1
    guard = 256
    RG = DeviceBuffer.from_numpy(np.full(T * Q * size + guard, 0x55, np.uint8))
    check(lib.ts2_attention_forward(0, None, 2, Qb.ptr, Kb.ptr, Vb.ptr, ip(start), ip(finish), T, H, 0.0, O.ptr, LSE.ptr))
    check(lib.ts2_op_attention_gated_forward(0, None, prec, Qb.ptr, Kb.ptr, Vb.ptr, ip(start), ip(finish), T, H, 0.0,
                                             G.ptr + 3 * Q * 2, 4 * Q,
                                             O2.ptr, LSE2.ptr, RG.ptr))
    sync()
    o = O2.download((T, Q), np.float16)
    assert np.array_equal(o.view(np.uint16), O.download((T, Q), np.float16).view(np.uint16))
    assert np.array_equal(LSE2.download((T, H), np.float32), LSE.download((T, H), np.float32))
    raw = RG.download(T * Q * size + guard, np.uint8)
    assert (raw[-guard:] == 0x55).all()
    s = {capi.PREC_FP8: 16.0, capi.PREC_F16: 1.0, capi.PREC_INT8: 24.0}[prec]
    want = s * o.astype(np.float64) / (1 + np.exp(-2 * qkvg[:, 3 * Q:].astype(np.float64)))
    if prec == capi.PREC_F16:  # one rounding to 11 bits; below the normal range half a step of 2^-24
        got = raw[:-guard].view(np.float16).reshape(T, Q).astype(np.float64)
        assert (np.abs(got - want) <= np.abs(want) * 2.0 ** -10 + 2.0 ** -24).all()
    elif prec == capi.PREC_INT8:  # nearest whole number
        got = raw[:-guard].view(np.int8).reshape(T, Q).astype(np.float64)
        assert (np.abs(got - np.clip(want, -128, 127)) <= 0.501).all()
    else:  # packed fp16 (three roundings and the tanh, 2^-9 in all), then 4 bits; half a step of 2^-9 below the normal range
        got = raw[:-guard].view(ml_dtypes.float8_e4m3fn).reshape(T, Q).astype(np.float64)
        assert (np.abs(got - want) <= np.abs(want) * (2.0 ** -4 + 2.0 ** -8) + 2.0 ** -10 + 16 * 2.0 ** -11 * np.abs(o)).all()
