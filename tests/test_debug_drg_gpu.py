"""The product before an activation's (or attention gate's) backward, "drg", stays on the chip where the contraction's
epilogue goes on with it: a plain step has nothing to read back, a traced step writes and records it and is otherwise the
same step."""
import ml_dtypes
import numpy as np
import pytest

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu


def test_a_traced_step_has_what_a_plain_one_keeps_on_the_chip():
    T, D, Q = 5120, 256, 1024  # 20 x 4 tiles of 256: one wave of CTA pairs
    spec = host.ModelSpec(dim=D, head_count=Q // 128, ffn_tiles=8, vocab=1024, attention_widths=[512],
                          precision=capi.PREC_FP8).add_blocks(2)
    model = Model(spec, host.init_weights(spec, 1), T)
    batch = host.synthetic_batch(spec, 10, 512, 2)

    def step():
        model.set_batch(batch)
        model.backprop(host.training_step(rate=0.0))
        return model.get_gradients()

    want = step()
    with pytest.raises(capi.Ts2Error) as e:
        model.debug_read("drg", 0, (T, Q), np.float16)
    assert e.value.code == capi.TS2_ERR_UNSUPPORTED
    model.set_debug_trace()
    captured = {}
    for name, size, dtype in (("drg[0]", Q, np.float16), ("g_fast[0]", D, ml_dtypes.float8_e4m3fn)):
        model.set_debug_capture(name, T * size * 2)
        got = step()
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
        captured[name] = model.debug_read("capture", 0, (T, size), dtype)
    assert {f"drg[{l}]" for l in range(4)} <= {r[0] for r in model.get_debug_trace()}
    # layer 0 comes last in the backward pass: the buffer still holds its product
    assert np.array_equal(model.debug_read("drg", 0, (T, Q), np.float16).view(np.uint16), captured["drg[0]"].view(np.uint16))
    combiner, _ = model.get_fast_weights(2 + 4)
    rows = np.r_[0:40, 1000:1040, T - 40:T]
    ref = captured["g_fast[0]"][rows].astype(np.float64) @ combiner.view(ml_dtypes.float8_e4m3fn).astype(np.float64) / (32 * D ** 0.5)
    err = np.linalg.norm(captured["drg[0]"][rows] - ref) / np.linalg.norm(ref)
    assert err < 6e-4  # fp16 output
    model.set_debug_trace(False)
    step()
    with pytest.raises(capi.Ts2Error):
        model.debug_read("drg", 0, (T, Q), np.float16)
