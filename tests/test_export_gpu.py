"""ts2_get_params merges the copies of matrices that follow one another in memory on both sides - but only inside one
page-locked range: matrices may lie side by side in host memory without belonging together."""
import ctypes as C
import mmap

import numpy as np
import pytest
import torch

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu


def model_and_weights():
    spec = host.ModelSpec(dim=256, head_count=2, ffn_tiles=4, vocab=2048, labels=2048, attention_widths=[64]).add_blocks(2)
    mats = host.init_weights(spec, 9)
    return spec, mats, Model(spec, mats, 128)


def views_of(spec, flat):
    out, at = [], 0
    for y, x in spec.matrix_shapes():
        out.append(flat[at:at + y * x].reshape(y, x))
        at += y * x
    return out


def export(model, views):
    model._check(model.lib.ts2_get_params(model.h, capi.PARAM_WEIGHTS, host.matrix_views(views), len(views)))


@pytest.mark.parametrize("pinned", [True, False])
def test_one_buffer_for_all(pinned):
    spec, mats, model = model_and_weights()
    flat = torch.zeros(spec.param_count(), pin_memory=pinned).numpy()
    views = views_of(spec, flat)
    export(model, views)
    for v, m in zip(views, mats):
        assert np.array_equal(v, m)


@pytest.mark.parametrize("which", ["each on its own", "every other one"])
def test_neighbours_that_are_locked_separately(which):
    """One mapping holds all matrices without gaps; each one (or every other one, the rest pageable) is page-locked by itself."""
    cudart = C.CDLL("libcudart.so.12")
    cudart.cudaHostRegister.argtypes, cudart.cudaHostUnregister.argtypes = [C.c_void_p, C.c_size_t, C.c_uint], [C.c_void_p]
    spec, mats, model = model_and_weights()
    page = mmap.PAGESIZE
    assert all(m.nbytes % page == 0 for m in mats)
    region = mmap.mmap(-1, sum(m.nbytes for m in mats))
    flat = np.frombuffer(region, np.float32)
    views = views_of(spec, flat)
    locked = []
    try:
        for v in views[::1 if which == "each on its own" else 2]:
            assert cudart.cudaHostRegister(v.ctypes.data, v.nbytes, 0) == 0
            locked.append(v.ctypes.data)
        export(model, views)
    finally:
        for p in locked:
            assert cudart.cudaHostUnregister(p) == 0
    for v, m in zip(views, mats):
        assert np.array_equal(v, m)


def test_a_wrong_shape_is_refused():
    spec, mats, model = model_and_weights()
    views = [np.zeros_like(m) for m in mats]
    views[3] = np.zeros((views[3].shape[0], views[3].shape[1] + 128), np.float32)
    rc = model.lib.ts2_get_params(model.h, capi.PARAM_WEIGHTS, host.matrix_views(views), len(views))
    assert rc == capi.TS2_ERR_INVALID_ARG


@pytest.mark.parametrize("micro", [1, 3])
def test_weights_and_error_are_read_while_the_step_goes_on(micro):
    """A model large enough to be updated in groups: what is read right behind ts2_backprop, beside the running backward pass,
    is what is there when the step is over; and the step equals that of a model which updates everything after it."""
    spec = host.ModelSpec(dim=512, head_count=2, ffn_tiles=8, vocab=32768, labels=32768, attention_widths=[256]).add_blocks(3)
    mats = host.init_weights(spec, 4)
    batches = [host.synthetic_batch(spec, 16, 256, 7 + i) for i in range(micro)]
    model = Model(spec, mats, batches[0].node_count)
    for it in range(2):
        for i, b in enumerate(batches):
            model.set_batch(b)
            model.backprop(host.training_step(rate=0.01, iteration=it), apply=i == micro - 1)
        err = model.avg_train_err()
        weights, momentum = model.get_weights(), model.get_momentum()
        model.wait()
        assert abs(model.avg_train_err() - err) < 1e-6
        for got in (weights, momentum):
            later = model.get_weights() if got is weights else model.get_momentum()
            for name, a, b in zip(spec.matrix_names(), got, later):
                assert np.array_equal(a, b), name
    assert all(not np.array_equal(a, b) for a, b in zip(weights, mats))
    # the update by its definition, from the gradient that was applied: one step of a fresh model, rate 0 for the weights' sake
    fresh = Model(spec, mats, batches[0].node_count)
    fresh.set_batch(batches[0])
    step = host.training_step(rate=0.01, iteration=0)
    fresh.backprop(step, apply=True)
    grads, after = fresh.get_gradients(), fresh.get_momentum()
    for i, (name, g, m) in enumerate(zip(spec.matrix_names(), grads, after)):
        disp = (g.astype(np.float64) ** 2).mean(1, keepdims=True) if i < 2 else (g.astype(np.float64) ** 2).mean()
        want = np.where(disp > 0, g / np.sqrt(np.where(disp > 0, disp, 1)), 0) * (1 - step.beta1)
        assert np.linalg.norm(m - want) <= 1e-5 * np.linalg.norm(want), name
