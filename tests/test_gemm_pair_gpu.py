"""The contraction on pairs of CTAs (csrc/gemm_pair.cu): outputs of many 256 x 256 tiles, with edges that cut a pair's
second CTA, a lane quarter, a column half or a K block, every output form and operand format - against float64 products
of the same quantized operands on rows around the edges.  Tolerances: fp32 summation order (2e-5 relative L2), output
rounding of fp16 (2^-11: 6e-4) and bf16 (2^-8: 4e-3), as in test_gemm_gpu.py."""
import ml_dtypes
import numpy as np
import pytest

from tscale2_b200 import capi
from tscale2_b200.device import DeviceBuffer, check, sync

pytestmark = pytest.mark.gpu

DT = {capi.OUT_F32: np.float32, capi.OUT_F32_ADD: np.float32, capi.OUT_F16: np.float16, capi.OUT_BF16: ml_dtypes.bfloat16}
TOL = {capi.OUT_F32: 2e-5, capi.OUT_F32_ADD: 2e-5, capi.OUT_F16: 6e-4, capi.OUT_BF16: 4e-3}


def operand(rng, shape, prec):
    x = rng.standard_normal(shape).astype(np.float32)
    if prec == capi.PREC_INT8:
        return np.clip(np.rint(x * 20), -127, 127).astype(np.int8)
    return x.astype(np.float16 if prec == capi.PREC_F16 else ml_dtypes.float8_e4m3fn)


@pytest.mark.parametrize("prec", [capi.PREC_FP8, capi.PREC_F16, capi.PREC_INT8])
@pytest.mark.parametrize("token_major", [False, True])
@pytest.mark.parametrize("M,N,K,out", [
    (8192, 1024, 1024, capi.OUT_F32_ADD),      # whole tiles, residual input
    (16400, 1504, 384, capi.OUT_F16),          # the last pair has 16 rows: its second CTA none; 224 columns in the last tile
    (12256, 2080, 320, capi.OUT_BF16),         # rows end inside a lane quarter, 32 columns in the last tile, ragged K block
    (10128, 1664, 704, capi.OUT_F32),          # columns end in the second half of a tile
    (8208, 1152, 528, capi.OUT_F32_ADD),
    (768, 512, 16384, capi.OUT_F32),           # few tiles and a long K: split, partial tiles in the workspace
])
def test_pairs_match_float64(prec, token_major, M, N, K, out):
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
