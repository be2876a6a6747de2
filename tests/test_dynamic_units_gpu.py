"""TS2_GEMM_DYNAMIC_UNITS is read once per process, so it is set for a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes as C
import ml_dtypes, numpy as np
from tscale2_b200 import capi, host
from tscale2_b200.device import DeviceBuffer, check, sync
from tscale2_b200.model import Model
lib = capi.load_library()
M, N, K = 8192, 1024, 1024  # a shape that pairs of CTAs take otherwise
plan = (C.c_int32 * 3)()
check(lib.ts2_op_gemm_plan(0, capi.PREC_FP8, capi.OUT_F32_ADD, 0, 0, M, N, K, plan))
assert plan[0] == 128, list(plan)
T, D, F = 5120, 256, 1024
G, WT, WG, WS, DWG = (DeviceBuffer(n) for n in (T * D, F * D, 4 * T * F, 4 * T * F // 128, 2 * T * F))
assert lib.ts2_op_ffn_backward_fused(0, None, G.ptr, WT.ptr, 1.0, WG.ptr, WS.ptr, T, D, F, DWG.ptr) == capi.TS2_ERR_UNSUPPORTED
rng = np.random.default_rng(0)
a, b = (rng.standard_normal(s).astype(ml_dtypes.float8_e4m3fn) for s in ((M, K), (N, K)))
c0 = rng.standard_normal((M, N)).astype(np.float32)
A, B, C0 = (DeviceBuffer.from_numpy(x) for x in (a, b, c0))
for _ in range(3):
    check(lib.ts2_gemm_tn(0, None, capi.PREC_FP8, capi.OUT_F32_ADD, M, N, K, A.ptr, K, B.ptr, K, C0.ptr, N, 0.125, None, None))
sync()
rows = np.r_[0:40, M - 200:M]
want = c0[rows] + 3 * 0.125 * (a[rows].astype(np.float64) @ b.astype(np.float64).T)
assert np.linalg.norm(C0.download((M, N), np.float32)[rows] - want) < 2e-5 * np.linalg.norm(want)
spec = host.ModelSpec(dim=256, head_count=8, ffn_tiles=8, vocab=1024, attention_widths=[512]).add_blocks(1)
model = Model(spec, host.init_weights(spec, 1), 5120)
model.set_batch(host.synthetic_batch(spec, 10, 512, 2))
model.backprop(host.training_step(rate=0.0))
assert all(np.isfinite(g).all() and g.any() for g in model.get_gradients())
print("units drawn")
"""


def test_the_switch_reaches_every_contraction():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, TS2_GEMM_DYNAMIC_UNITS="1", PYTHONPATH=root)
    run = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "units drawn" in run.stdout, run.stderr[-3000:]
