"""MPF_DISABLE_TUNE_*: the matrices a flag names get no gradient and stay as they are; all others get the gradient they get
without the flag, bit for bit.  The gradient buffer is not zeroed as a whole, so the memory it may come to lie in is filled
with NaNs first, and the second accumulation starts on what an applied step left behind."""
import numpy as np
import pytest

from tscale2_b200 import capi, host
from tscale2_b200.device import DeviceBuffer, check
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu

EMBED, FINAL, LAYERS = capi.MPF_DISABLE_TUNE_EMBED, capi.MPF_DISABLE_TUNE_FINAL_LAYER, capi.MPF_DISABLE_TUNE_LAYERS


def spec_of(kind, prec, flags):
    spec = host.ModelSpec(dim=256, head_count=2, ffn_tiles=4, vocab=1024, attention_widths=[96], precision=prec, flags=flags,
                          expert_dim=128, moe_expert_count=4 if kind == "moe" else 0)
    return spec.add_blocks(2, moe=kind == "moe")


def poison(n):
    held = [DeviceBuffer(n) for _ in range(4)]
    for b in held:
        check(b.lib.ts2_dev_memset(0, b.ptr, 0xFF, n))
    check(held[0].lib.ts2_dev_sync(0))
    for b in held:
        b.free()


def gradients(spec, mats, batches):
    """Gradients of an applied step, of two accumulated ones after it, and the weights in the end."""
    poison(64 << 20)
    model = Model(spec, mats, max(b.node_count for b in batches))
    model.set_batch(batches[0])
    model.backprop(host.training_step(rate=0.0, iteration=0))
    out = [model.get_gradients()]
    for batch in batches[1:]:
        model.set_batch(batch)
        model.backprop(host.training_step(rate=0.0, iteration=1), apply=False)
    out.append(model.get_gradients())
    model.set_batch(batches[0])
    model.backprop(host.training_step(rate=0.01, iteration=2))
    out.append(model.get_weights())
    model.close()
    return out


# 5 x 900 nodes: more than a batch that is prepared (and sorted) in one launch takes
@pytest.mark.parametrize("seqs,seq", [(2, 100), (5, 900)])
@pytest.mark.parametrize("kind,prec", [("dense", capi.PREC_FP8), ("dense", capi.PREC_INT8), ("moe", capi.PREC_F16)])
@pytest.mark.parametrize("flags", [EMBED, FINAL, LAYERS, EMBED | FINAL | LAYERS])
def test_what_a_flag_names_keeps_still(kind, prec, flags, seqs, seq):
    spec = spec_of(kind, prec, 0)
    mats = host.init_weights(spec, 5)
    batches = [host.synthetic_batch(spec, seqs, seq, s) for s in range(3)]
    want = gradients(spec, mats, batches)
    got = gradients(spec_of(kind, prec, flags), mats, batches)
    for i, w0 in enumerate(mats):
        frozen = flags & (EMBED if i == 0 else FINAL if i == 1 else LAYERS)
        for step in range(2):
            if frozen:
                assert not got[step][i].any(), (i, step)
            else:
                assert np.array_equal(got[step][i], want[step][i]), (i, step)
        assert want[0][i].any() and not np.array_equal(want[2][i], w0), i
        assert not frozen or np.array_equal(got[2][i], w0), i
