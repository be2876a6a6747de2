"""Scoring takes the final layer in parts where the partial results of all nodes have no room: the same score from any division,
the last part ragged or small enough for another kernel."""
import numpy as np
import pytest

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [capi.PREC_FP8, capi.PREC_F16, capi.PREC_INT8])
@pytest.mark.parametrize("T,vocab", [(13003, 4128), (16640, 2080)])
def test_parts_add_up(prec, T, vocab):
    spec = host.ModelSpec(dim=256, head_count=1, ffn_tiles=2, vocab=vocab, attention_widths=[32], precision=prec).add_blocks(1)
    rng = np.random.default_rng(vocab)
    model = Model(spec, host.init_weights(spec, 2), T, bias=rng.standard_normal(vocab).astype(np.float32) * 2)
    model.set_batch(host.Batch(rng.integers(0, vocab, (1, T + 1)), spec.attention_widths))
    whole = model.compute_score()
    # sums of up to T / 32 values by atomic additions in any order, then one division: 2^-24 of the sum per addition; the logits
    # of the other kernel (a small last part) are rounded to fp16, 2^-11 of values of a few units averaged over T nodes
    for part in (8192, 5120, 4096):
        assert model.lib.ts2_selftest_score_part(model.h, part) == capi.TS2_OK
        assert abs(model.compute_score() - whole) < T / 32 * 2.0 ** -24 * abs(whole) + 2e-4
    assert model.lib.ts2_selftest_score_part(model.h, 100) == capi.TS2_ERR_INVALID_ARG
