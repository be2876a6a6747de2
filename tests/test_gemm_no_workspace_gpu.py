"""ts2_gemm_dw without scratch: an output whose tiles keep at least half the SMs busy is computed whole, also where the
fastest plan would split the tokens; one with few tiles and many tokens needs the workspace and says so."""
import ml_dtypes
import numpy as np
import pytest

from tscale2_b200 import capi
from tscale2_b200.device import DeviceBuffer, check, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,dtype", [(capi.PREC_FP8, ml_dtypes.float8_e4m3fn), (capi.PREC_F16, np.float16)])
@pytest.mark.parametrize("offered", [0, 1 << 16])  # bytes of workspace: none, too few
def test_many_tiles_need_no_workspace(prec, dtype, offered):
    lib = capi.load_library()
    T, n_in, n_out = 16384, 1280, 2048
    assert lib.ts2_gemm_dw_workspace_bytes(T, n_in, n_out) > max(offered, 0), "this shape is meant to be one the plan splits"
    rng = np.random.default_rng(1)
    dy, x = rng.standard_normal((T, n_out)).astype(dtype), rng.standard_normal((T, n_in)).astype(dtype)
    DY, X, DW, WS = DeviceBuffer.from_numpy(dy), DeviceBuffer.from_numpy(x), DeviceBuffer(n_out * n_in * 4), DeviceBuffer(max(offered, 16))
    check(lib.ts2_gemm_dw(0, None, prec, capi.OUT_F32, T, n_in, n_out, DY.ptr, X.ptr, DW.ptr, 0.5, WS.ptr if offered else None, offered))
    sync()
    got = DW.download((n_out, n_in), np.float32)
    rows = np.r_[0:64, 120:140, n_out - 64:n_out]
    want = 0.5 * dy[:, rows].astype(np.float64).T @ x.astype(np.float64)
    assert np.linalg.norm(got[rows] - want) < 2e-5 * np.linalg.norm(want)  # fp32 sums, as in test_gemm_gpu.py


def test_few_tiles_and_many_tokens_still_need_it():
    lib = capi.load_library()
    buf = DeviceBuffer(16384 * 256)
    out = DeviceBuffer(256 * 256 * 4)
    rc = lib.ts2_gemm_dw(0, None, capi.PREC_FP8, capi.OUT_F32, 16384, 256, 256, buf.ptr, buf.ptr, out.ptr, 1.0, None, 0)
    assert rc == capi.TS2_ERR_INVALID_ARG and b"workspace" in lib.ts2_last_error(None)
