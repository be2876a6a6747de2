"""The dX contraction of a branch with the backward of the activation (FFN) or of the gate (attention) in its epilogue, against the two kernels it replaces
(each of which is held to the oracle elsewhere).  Both sides round the product to fp16 and compute in packed fp16; only the
order of the 128-term projection sums differs (2^-22 relative), so a result differs where that moves an fp16 or e4m3 rounding:
a fraction of a percent of the elements, by a step."""
import ml_dtypes
import numpy as np
import pytest

from tscale2_b200 import capi
from tscale2_b200.device import DeviceBuffer, check, sync

pytestmark = pytest.mark.gpu


# rows: whole tiles, one short, one over a tile and over a CTA's half; columns: an even and an odd number of 128-wide tiles;
# K: one block, a ragged one, more blocks than the ring has stages
@pytest.mark.parametrize("T,D,F", [(5120, 128, 1024), (5119, 768, 1152), (5249, 208, 1152), (2561, 640, 3072)])
def test_fused_ffn_backward_equals_its_two_steps(T, D, F):
    lib = capi.load_library()
    rng = np.random.default_rng(T + F)
    e4m3 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(ml_dtypes.float8_e4m3fn).view(np.uint8)
    g, wt = e4m3(T, D), e4m3(F, D)
    wg = rng.standard_normal((T, 2 * F), dtype=np.float32).astype(np.float16)
    ws = (rng.random((T, F // 128), dtype=np.float32) + 0.5)
    G, WT, WG, WS = (DeviceBuffer.from_numpy(a) for a in (g, wt, wg, ws))
    DRG, WANT, GOT = DeviceBuffer(T * F * 2), DeviceBuffer(T * 2 * F), DeviceBuffer(T * 2 * F)
    alpha = 2.0 / D ** 0.5
    check(lib.ts2_gemm_dx(0, None, capi.PREC_FP8, capi.OUT_F16, T, F, D, G.ptr, WT.ptr, DRG.ptr, alpha, None, None))
    check(lib.ts2_op_ffn_act_backward(0, None, capi.PREC_FP8, DRG.ptr, WG.ptr, WS.ptr, T, F, WANT.ptr))
    check(lib.ts2_op_ffn_backward_fused(0, None, G.ptr, WT.ptr, alpha, WG.ptr, WS.ptr, T, D, F, GOT.ptr))
    sync()
    want, got = (b.download((T, 2 * F), np.uint8) for b in (WANT, GOT))
    assert np.array_equal(got[:, F:], want[:, F:])  # the gate's gradient has no sum in it
    assert np.mean(got[:, :F] != want[:, :F]) < 5e-3
    a, b = (x[:, :F].view(ml_dtypes.float8_e4m3fn).astype(np.float32) for x in (got, want))
    # a step of e4m3 is an eighth of the value at most (2^-9 below its normal range)
    assert (np.abs(a - b) <= np.maximum(np.abs(b) / 4, 2.0 ** -8)).all()


@pytest.mark.parametrize("T,D,Q", [(5120, 128, 1024), (5119, 768, 1152), (5249, 208, 1152), (3329, 640, 1536)])
def test_fused_attention_gate_backward_equals_its_two_steps(T, D, Q):
    lib = capi.load_library()
    rng = np.random.default_rng(T + Q)
    e4m3 = lambda *s: rng.standard_normal(s, dtype=np.float32).astype(ml_dtypes.float8_e4m3fn).view(np.uint8)
    G, WT = DeviceBuffer.from_numpy(e4m3(T, D)), DeviceBuffer.from_numpy(e4m3(Q, D))
    qkvg, o = (rng.standard_normal((T, n), dtype=np.float32).astype(np.float16) for n in (4 * Q, Q))
    QKVG, O = DeviceBuffer.from_numpy(qkvg), DeviceBuffer.from_numpy(o)
    DRG = DeviceBuffer(T * Q * 2)
    out = [(DeviceBuffer.from_numpy(np.zeros((T, 4 * Q), np.uint8)), DeviceBuffer(T * Q * 2), DeviceBuffer(T * Q // 128 * 4)) for _ in range(2)]
    alpha = 2.0 / D ** 0.5
    check(lib.ts2_gemm_dx(0, None, capi.PREC_FP8, capi.OUT_F16, T, Q, D, G.ptr, WT.ptr, DRG.ptr, alpha, None, None))
    check(lib.ts2_op_att_gate_backward(0, None, capi.PREC_FP8, DRG.ptr, QKVG.ptr, O.ptr, T, Q, *(b.ptr for b in out[0])))
    check(lib.ts2_op_att_gate_backward_fused(0, None, G.ptr, WT.ptr, alpha, QKVG.ptr, O.ptr, T, D, Q, *(b.ptr for b in out[1])))
    sync()
    (d4, dout, ds), (f4, fout, fs) = ((a.download((T, 4 * Q), np.uint8), b.download((T, Q), np.float16), c.download((T, Q // 128), np.float32))
                                      for a, b, c in out)
    assert np.array_equal(f4, d4) and np.array_equal(fout.view(np.uint16), dout.view(np.uint16))  # columns before the gate's stay zero
    # 128 fp32 terms in another order: 128 * 2^-24 of the sum of their magnitudes at most
    mag = np.abs(dout.astype(np.float32) * o.astype(np.float32)).reshape(T, Q // 128, 128).sum(-1)
    assert (np.abs(fs - ds) <= 128 * 2.0 ** -24 * mag).all()


def test_few_tiles_are_refused():
    lib = capi.load_library()
    B = DeviceBuffer(1 << 20)
    assert lib.ts2_op_ffn_backward_fused(0, None, B.ptr, B.ptr, 1.0, B.ptr, B.ptr, 128, 256, 256, B.ptr) == capi.TS2_ERR_UNSUPPORTED
