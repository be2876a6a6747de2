"""ts2_get_params of a model that is updated in groups, while the step runs: the caller's arrays stay as they are when the call
fails for a reason that is known before its first copy."""
import numpy as np
import pytest
import torch

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu


def a_model():
    spec = host.ModelSpec(dim=512, head_count=2, ffn_tiles=8, vocab=32768, labels=32768, attention_widths=[256]).add_blocks(3)
    mats = host.init_weights(spec, 4)
    good = host.synthetic_batch(spec, 16, 256, 7)
    ti = good.target_id.copy()
    ti[9] = 10 ** 6
    bad = host.Batch.from_arrays(good.node_count, good.label_arr, good.label_ptr, good.target_node, ti, good.att)
    return spec, Model(spec, mats, good.node_count), good, bad


def arrays(spec, pinned):
    flat = torch.full((spec.param_count(),), 7.5, dtype=torch.float32, pin_memory=pinned).numpy()
    out, at = [], 0
    for y, x in spec.matrix_shapes():
        out.append(flat[at:at + y * x].reshape(y, x))
        at += y * x
    return flat, out


@pytest.mark.parametrize("what", [capi.PARAM_WEIGHTS, capi.PARAM_MOMENTUM, capi.PARAM_GRADIENT])
@pytest.mark.parametrize("pinned", [True, False])
def test_a_malformed_batch_leaves_the_arrays_alone(what, pinned):
    spec, model, good, bad = a_model()
    assert spec.param_count() >= 2 << 24, "meant to be a model that is updated in groups"
    flat, out = arrays(spec, pinned)
    views = host.matrix_views(out)
    for i in range(2):  # the second time with more of the same behind it, and an accumulated gradient in front
        if i:
            model.set_batch(good)
            model.backprop(host.training_step(rate=0.0), apply=False)
        model.set_batch(bad)
        model.backprop(host.training_step(rate=0.01, iteration=i))
        if i:
            model.backprop(host.training_step(rate=0.01, iteration=i))
        rc = model.lib.ts2_get_params(model.h, what, views, len(out))
        assert rc == capi.TS2_ERR_INVALID_ARG and b"1000000" in model.lib.ts2_last_error(model.h)
        assert (flat == 7.5).all()
    # reported once; the model goes on, and the next call fills them all
    model.set_batch(good)
    model.backprop(host.training_step(rate=0.01, iteration=2))
    model._check(model.lib.ts2_get_params(model.h, what, views, len(out)))
    got = [a.copy() for a in out]
    model.wait()
    model._check(model.lib.ts2_get_params(model.h, what, views, len(out)))
    for name, a, b in zip(spec.matrix_names(), got, out):
        assert np.array_equal(a, b) and not (a == 7.5).any(), name


def test_no_time_left_leaves_the_arrays_alone():
    spec, model, good, _ = a_model()
    flat, out = arrays(spec, True)
    views = host.matrix_views(out)
    model.set_batch(good)
    model.backprop(host.training_step(rate=0.01))
    model.wait()
    model._check(model.lib.ts2_set_wait_limit(model.h, 1e-4))
    for i in range(10):
        model.backprop(host.training_step(rate=0.01, iteration=1 + i))
    assert model.lib.ts2_get_params(model.h, capi.PARAM_WEIGHTS, views, len(out)) == capi.TS2_ERR_TIMEOUT
    assert (flat == 7.5).all()
    model._check(model.lib.ts2_set_wait_limit(model.h, 120.0))
    model._check(model.lib.ts2_get_params(model.h, capi.PARAM_WEIGHTS, views, len(out)))
    model.wait()
    for a, b in zip(out, model.get_weights()):
        assert np.array_equal(a, b)


def test_a_later_batch_that_is_known_to_be_malformed():
    spec, model, good, bad = a_model()
    flat, out = arrays(spec, True)
    views = host.matrix_views(out)
    model.set_batch(good)
    model.backprop(host.training_step(rate=0.01))
    model.set_batch(bad)
    torch.cuda.synchronize()  # it is checked by now
    assert model.lib.ts2_get_params(model.h, capi.PARAM_WEIGHTS, views, len(out)) == capi.TS2_ERR_INVALID_ARG
    assert (flat == 7.5).all()
    model._check(model.lib.ts2_get_params(model.h, capi.PARAM_WEIGHTS, views, len(out)))  # reported: the step's weights are there
    for a, b in zip(out, model.get_weights()):
        assert np.array_equal(a, b)
