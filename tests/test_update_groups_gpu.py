"""Matrices updated in groups beside the backward pass: the same bits as an update of everything behind it, with any number of
groups, dense and expert layers, accumulated gradients and frozen parts; and a step that fails while it is being queued has
changed nothing."""
import ctypes as C

import numpy as np
import pytest

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu

ONE_GO = 1 << 40


def a_spec(kind):
    if kind == "experts":
        return host.ModelSpec(dim=256, head_count=2, ffn_tiles=4, vocab=2048, attention_widths=[64], expert_dim=256, moe_expert_count=8,
                              moe_selected=2).add_blocks(3, moe=True)
    prec = {"e4m3": capi.PREC_FP8, "f16": capi.PREC_F16, "int8": capi.PREC_INT8}[kind]
    return host.ModelSpec(dim=256, head_count=2, ffn_tiles=4, vocab=2048, attention_widths=[64], precision=prec).add_blocks(4)


def groups(model, elems):
    n = C.c_int()
    model._check(model.lib.ts2_selftest_update_groups(model.h, elems, C.byref(n)))
    return n.value


def state(model):
    """Everything a step changes: weights, momentum, dispersion, what the contractions see of the weights."""
    out = model.get_weights() + model.get_momentum()
    for i in range(len(model.shapes)):
        rd, sw = model.get_row_disp(i)
        out += [rd, np.float32([sw])]
    moe = model.spec.moe_expert_count > 0
    for i in range(2 if moe else len(model.shapes)):  # expert matrices are laid out in another order
        q, sko = model.get_fast_weights(i)
        out += [q, np.float32([sko])]
    return out


def same(a, b):
    return len(a) == len(b) and all(np.array_equal(x, y) for x, y in zip(a, b))


def train(model, batches, steps, micro=1):
    k = 0
    for it in range(steps):
        for j in range(micro):
            model.set_batch(batches[k % len(batches)])
            model.backprop(host.training_step(rate=0.01, iteration=it), apply=j == micro - 1)
            k += 1


# elements per group: a group per layer and matrix outside the layers, two layers or so together, all layers in one
@pytest.mark.parametrize("kind", ["e4m3", "f16", "int8", "experts"])
@pytest.mark.parametrize("elems,micro", [(1000, 1), (700000, 1), (1500000, 3)])
def test_groups_are_one_update(kind, elems, micro):
    spec = a_spec(kind)
    assert elems * 2 <= spec.param_count()
    batches = [host.synthetic_batch(spec, 4, 64, 5 + i) for i in range(3)]
    mats = host.init_weights(spec, 3)
    results = []
    for e in (elems, ONE_GO):
        model = Model(spec, mats, batches[0].node_count)
        n = groups(model, e)
        assert n == 0 if e == ONE_GO else n >= 3
        if elems == 1000:
            assert n in (0, 2 + len(spec.layers))
        train(model, batches, 3, micro)
        results.append(state(model))
        model.set_batch(batches[0])
        results[-1].append(np.float32([model.compute_score()]))
        model.close()
    # the score is a sum of atomic additions
    assert abs(results[0][-1] - results[1][-1]) < 1e-5
    assert same(results[0][:-1], results[1][:-1])


@pytest.mark.parametrize("flags", [capi.MPF_DISABLE_TUNE_EMBED, capi.MPF_DISABLE_TUNE_FINAL_LAYER, capi.MPF_DISABLE_TUNE_LAYERS])
@pytest.mark.parametrize("kind", ["e4m3", "experts"])
def test_with_a_part_that_gets_no_gradient(kind, flags):
    spec = a_spec(kind)
    spec.flags = flags
    batches = [host.synthetic_batch(spec, 4, 64, 5)]
    mats = host.init_weights(spec, 3)
    results = []
    for e in (1000, ONE_GO):
        model = Model(spec, mats, batches[0].node_count)
        groups(model, e)
        train(model, batches, 2)
        results.append(state(model))
    assert same(*results)


@pytest.mark.parametrize("kind", ["e4m3", "experts"])
@pytest.mark.parametrize("elems", [1000, ONE_GO])
def test_a_step_that_fails_in_its_queueing_changes_nothing(kind, elems):
    spec = a_spec(kind)
    batches = [host.synthetic_batch(spec, 4, 64, 5 + i) for i in range(2)]
    mats = host.init_weights(spec, 3)
    model, other = (Model(spec, mats, batches[0].node_count) for _ in range(2))
    groups(model, elems), groups(other, elems)
    train(model, batches, 1), train(other, batches, 1)
    before = state(model)
    for layer in (len(spec.layers) - 2, 0):
        model._check(model.lib.ts2_selftest_fail_backward(model.h, layer))
        with pytest.raises(capi.Ts2Error) as e:
            model.backprop(host.training_step(rate=0.01, iteration=1))
        assert e.value.code == capi.TS2_ERR_UNSUPPORTED and "self-test" in str(e.value)
        assert same(state(model), before), f"failed at layer {layer}"
    # repeated, it is the step of a model that never failed
    for m in (model, other):
        m.backprop(host.training_step(rate=0.01, iteration=1))
    assert same(state(model), state(other))
