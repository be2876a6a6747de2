"""Operator-level attention calls take the caller's spans as they come: one that starts a little before the first key is the
span from key 0, in every kernel of the forward and backward pass, and the room for the score gradients counts it."""
import numpy as np
import pytest

from test_attention_gpu import causal_spans, run_device
from tscale2_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [2, 3])
@pytest.mark.parametrize("T,H,spans", [(64, 1, "window"), (700, 3, "window"), (700, 3, "first keys"), (1400, 2, "first keys")])
def test_a_span_that_starts_before_the_first_key(variant, T, H, spans):
    lib = capi.load_library()
    rng = np.random.default_rng(T)
    q, k, v, dout = (rng.standard_normal((T, 128 * H)).astype(np.float16) for _ in range(4))
    t = np.arange(T)
    if spans == "window":
        clamped, finish = causal_spans(T, T, 60)
        start = np.where(finish >= clamped, t - 60, clamped).astype(np.int32)
    else:  # every node looks at some of the first keys, the later half from before the first one
        start, finish = np.where(t < T // 2, t % 7, -1 - t % 7).astype(np.int32), (20 + t % 30).astype(np.int32)
        clamped = np.maximum(start, 0).astype(np.int32)
    assert (start < 0).any()
    want = run_device(lib, variant, q, k, v, dout, clamped, finish, H, 0.0)
    got = run_device(lib, variant, q, k, v, dout, start, finish, H, 0.0)
    for name, a, b in zip(["o", "lse", "dq", "dk", "dv"], got, want):
        assert np.array_equal(a, b), name
