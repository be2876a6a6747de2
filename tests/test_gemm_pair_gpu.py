"""The contraction on pairs of CTAs (csrc/gemm_pair.cu): outputs of many 256 x 256 tiles, with edges that cut a pair's
second CTA, a lane quarter, a column half or a K block, every output form and operand format - against float64 products
of the same quantized operands on rows around the edges.  Tolerances: fp32 summation order (2e-5 relative L2), output
rounding of fp16 (2^-11: 6e-4) and bf16 (2^-8: 4e-3), as in test_gemm_gpu.py.  Which kernel a shape takes is the plan's
choice, so every case asks for it and fails when the plan no longer gives it to pairs (or, where it says so, to single CTAs)."""
import ctypes as C

import ml_dtypes
import numpy as np
import pytest

from tscale2_b200 import capi, host
from tscale2_b200.device import DeviceBuffer, check, sync
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu

DT = {capi.OUT_F32: np.float32, capi.OUT_F32_ADD: np.float32, capi.OUT_F16: np.float16, capi.OUT_BF16: ml_dtypes.bfloat16}
TOL = {capi.OUT_F32: 2e-5, capi.OUT_F32_ADD: 2e-5, capi.OUT_F16: 6e-4, capi.OUT_BF16: 4e-3}


def operand(rng, shape, prec):
    x = rng.standard_normal(shape).astype(np.float32)
    if prec == capi.PREC_INT8:
        return np.clip(np.rint(x * 20), -127, 127).astype(np.int8)
    return x.astype(np.float16 if prec == capi.PREC_F16 else ml_dtypes.float8_e4m3fn)


def plan_of(prec, out, token_major, M, N, K, gated=False):
    plan = (C.c_int32 * 3)()
    check(capi.load_library().ts2_op_gemm_plan(0, prec, out, int(token_major), int(gated), M, N, K, plan))
    return tuple(plan)


PAIR = (256, 256, 1)


@pytest.mark.parametrize("prec", [capi.PREC_FP8, capi.PREC_F16, capi.PREC_INT8])
@pytest.mark.parametrize("token_major", [False, True])
@pytest.mark.parametrize("M,N,K,out,plan", [
    (8192, 1024, 1024, capi.OUT_F32_ADD, PAIR),    # whole tiles, residual input
    (8208, 1152, 528, capi.OUT_F32_ADD, PAIR),     # the last pair has 16 rows: its second CTA none; columns end at half a tile
    (16400, 3040, 1056, capi.OUT_F16, PAIR),       # the same rows, 224 columns in the last tile, ragged K block
    (12272, 2080, 1600, capi.OUT_BF16, PAIR),      # rows end inside a lane quarter of the second CTA, 32 columns in the last tile
    (12304, 3264, 832, capi.OUT_F32, PAIR),        # columns end inside the second half of a tile
    (1008, 1568, 20464, capi.OUT_F32, (256, 256, 5)),  # few tiles and a long K: split, partial tiles in the workspace
    (1008, 1568, 20464, capi.OUT_F16, (256, 256, 5)),  # the reduction applies the epilogue
    # outputs of many tiles with a short K stay on single CTAs
    (16400, 1504, 384, capi.OUT_F16, None),
    (12256, 2080, 320, capi.OUT_BF16, None),
    (10128, 1664, 704, capi.OUT_F32, None),
    (768, 512, 16384, capi.OUT_F32, (128, 256, 12)),
])
def test_pairs_match_float64(prec, token_major, M, N, K, out, plan):
    got_plan = plan_of(prec, out, token_major, M, N, K)
    assert got_plan == plan if plan else got_plan[0] == 128, f"the plan takes {got_plan}"
    lib = capi.load_library()
    rng = np.random.default_rng(M + N + K + prec)
    a, b = operand(rng, (M, K), prec), operand(rng, (N, K), prec)
    rs, cs = rng.uniform(0.5, 1.5, M).astype(np.float32), rng.uniform(0.5, 1.5, N).astype(np.float32)
    c0 = rng.standard_normal((M, N)).astype(np.float32)
    alpha = 1.0 / 64
    RS, CS = DeviceBuffer.from_numpy(rs), DeviceBuffer.from_numpy(cs)
    C = DeviceBuffer.from_numpy(c0 if out == capi.OUT_F32_ADD else np.zeros((M, N), DT[out]))
    if token_major:
        A, B = DeviceBuffer.from_numpy(np.ascontiguousarray(a.T)), DeviceBuffer.from_numpy(np.ascontiguousarray(b.T))
        ws = lib.ts2_gemm_dw_workspace_bytes(K, N, M)
        WS = DeviceBuffer(max(ws, 16))
        check(lib.ts2_gemm_dw_scaled(0, None, prec, out, K, N, M, A.ptr, B.ptr, C.ptr, alpha, RS.ptr, CS.ptr, WS.ptr, ws))
    else:
        A, B = DeviceBuffer.from_numpy(a), DeviceBuffer.from_numpy(b)
        check(lib.ts2_gemm_tn(0, None, prec, out, M, N, K, A.ptr, K, B.ptr, K, C.ptr, N, alpha, RS.ptr, CS.ptr))
    sync()
    got = C.download((M, N), DT[out]).astype(np.float64)
    rows = np.unique(np.concatenate([np.arange(0, 40), np.arange(118, 140), np.arange(M - 170, M), rng.integers(0, M, 64)]))
    want = (a[rows].astype(np.float64) @ b.astype(np.float64).T) * alpha * rs[rows, None] * cs[None]
    if out == capi.OUT_F32_ADD:
        want += c0[rows]
    if out == capi.OUT_F16:
        want = np.clip(want, -65504, 65504)
    err = np.linalg.norm(got[rows] - want) / np.linalg.norm(want)
    assert err < TOL[out], err
    # and the far end of every row, where a clipped store would leave zeros
    tail = np.linalg.norm(got[rows, -32:] - want[:, -32:]) / np.linalg.norm(want[:, -32:])
    assert tail < 2 * TOL[out], tail


@pytest.mark.parametrize("prec", [capi.PREC_FP8, capi.PREC_F16, capi.PREC_INT8])
def test_gated_activation_on_pairs(prec):
    """The FFN's first contraction of a model: normalised wide values, gate and their product, in the epilogue of pairs; the
    last pair has 8 rows.  Operands as the step left them, so only the epilogue's own roundings are between both sides."""
    T, D, F = 8200, 256, 2048
    assert plan_of(prec, capi.OUT_F16, False, T, 2 * F, D, gated=True) == PAIR
    spec = host.ModelSpec(dim=D, head_count=2, ffn_tiles=F // 128, vocab=1024, attention_widths=[64], precision=prec).add_blocks(1)
    model = Model(spec, host.init_weights(spec, 4), T)
    model.set_batch(host.synthetic_batch(spec, 8, 1025, 5))
    model.compute_score()
    dtype = {capi.PREC_FP8: ml_dtypes.float8_e4m3fn, capi.PREC_F16: np.float16, capi.PREC_INT8: np.int8}[prec]
    s_act = {capi.PREC_FP8: 16.0, capi.PREC_F16: 1.0, capi.PREC_INT8: 24.0}[prec]
    rows = np.r_[0:40, 120:140, 250:270, T - 140:T]
    n = model.debug_read("n_fast", 1, (T, D), dtype)[rows].astype(np.float64)
    expand, gate = (model.get_fast_weights(i)[0].view(dtype).astype(np.float64) for i in (7, 8))
    alpha = D ** -0.5 / (s_act * 32)
    wide, g = n @ expand.T * alpha, n @ gate.T * alpha
    tiles = wide.reshape(len(rows), F // 128, 128)
    what = (tiles / np.sqrt((tiles ** 2).mean(-1, keepdims=True))).reshape(len(rows), F)
    cat = model.debug_read("cat16", 1, (T, 2 * F), np.float16)[rows].astype(np.float64)
    for got, want in ((cat[:, :F], what), (cat[:, F:], g)):
        assert np.linalg.norm(got - want) < 6e-4 * np.linalg.norm(want)
        assert (np.abs(got - want) <= 2e-3 * np.abs(want) + 1e-5).all()  # 2^-11 of fp16, twice for the accumulated sum
    rg = model.debug_read("rg", 1, (T, F), dtype)[rows].astype(np.float64)
    want = s_act * what / (1 + np.exp(-2 * g))
    if prec == capi.PREC_F16:
        assert np.linalg.norm(rg - want) < 1e-3 * np.linalg.norm(want)
    elif prec == capi.PREC_FP8:  # tanh.approx is 2^-11 off, a step is 2^-3 to 2^-4 of the value: few results change sides
        want = want.astype(np.float32).astype(dtype).astype(np.float64)
        assert np.mean(rg != want) < 2e-2 and (np.abs(rg - want) <= np.maximum(np.abs(want) / 8, 2.0 ** -9) * 1.01).all()
    else:
        want = np.clip(np.rint(want), -127, 127)
        assert np.mean(rg != want) < 5e-3 and (np.abs(rg - want) <= 1).all()
