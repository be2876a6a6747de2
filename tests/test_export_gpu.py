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
