"""The buffer for the attention's score gradients is optional: a card without room for it still takes the model, a batch
that needs more than there is recomputes the scores, and the memory can be given back.

Both ways round the same fp32 values to fp16 (2^-11) before the dQ product and dQ itself to fp16 after it; where an order of
summation differs single roundings do, so gradients agree to well under 2^-11 = 5e-4 of their norm."""
import ctypes as C

import numpy as np
import pytest
import torch

from tscale2_b200 import capi, host
from tscale2_b200.device import DeviceBuffer
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu

HEADS, SEQ = 8, 1024


def spec_of(prec=capi.PREC_F16):
    return host.ModelSpec(dim=256, head_count=HEADS, ffn_tiles=4, vocab=1024, attention_widths=[8192], precision=prec).add_blocks(1)


def state(model):
    size, fits = C.c_int64(), C.c_int()
    model._check(model.lib.ts2_get_score_gradients(model.h, 0, C.byref(size), C.byref(fits)))
    return size.value, bool(fits.value)


def step(model, batch):
    model.set_batch(batch)
    fits = state(model)[1]
    model.backprop(host.training_step(rate=0.0))
    return fits, model.get_gradients()


def close(got, want):
    for i, (g, w) in enumerate(zip(got, want)):
        assert np.linalg.norm(g.astype(np.float64) - w) <= 5e-4 * np.linalg.norm(w.astype(np.float64)), i


def tile_bytes(seq, seqs):
    """Both 64-node tiles of every pair of 128-node blocks (key block, node block) of a causal document, all heads."""
    n = seq // 128
    return seqs * n * (n + 1) // 2 * 2 * 16384 * HEADS


@pytest.mark.parametrize("prec", [capi.PREC_F16, capi.PREC_FP8, capi.PREC_INT8])
def test_one_batch_fits_and_the_next_does_not(prec):
    spec = spec_of(prec)
    mats = host.init_weights(spec, 2)
    short, long = host.synthetic_batch(spec, 8, 1024, 3), host.synthetic_batch(spec, 1, 8192, 4)
    model = Model(spec, mats, 8192)
    assert state(model)[0] >= tile_bytes(8192, 1)
    want = [step(model, b) for b in (short, long)]
    assert want[0][0] and want[1][0]
    model._check(model.lib.ts2_set_score_gradient_limit(model.h, tile_bytes(1024, 8)))
    assert state(model) == (tile_bytes(1024, 8), False)
    for _ in range(2):
        fits, got = step(model, short)
        assert fits and all(np.array_equal(g, w) for g, w in zip(got, want[0][1]))
        fits, got = step(model, long)
        assert not fits
        if prec == capi.PREC_F16:
            close(got, want[1][1])
        else:  # a flipped rounding of dQ moves a one-byte operand by a whole step (up to 2^-3): few do
            for g, w in zip(got, want[1][1]):
                assert np.linalg.norm(g.astype(np.float64) - w) <= 2e-2 * np.linalg.norm(w.astype(np.float64))
    model._check(model.lib.ts2_set_score_gradient_limit(model.h, 0))
    assert state(model)[0] == 0 and not step(model, short)[0]
    model._check(model.lib.ts2_set_score_gradient_limit(model.h, 4 << 30))
    fits, got = step(model, long)
    assert fits and all(np.array_equal(g, w) for g, w in zip(got, want[1][1]))


def test_a_card_without_room_for_it_takes_the_model():
    """All device memory but what the model itself needs (and 256 MB) is taken; the buffer would be 1 GB."""
    spec = spec_of()
    mats = host.init_weights(spec, 2)
    batch = host.synthetic_batch(spec, 8192 // SEQ, SEQ, 3)
    torch.cuda.mem_get_info()  # the context exists
    Model(spec, mats, 8192).close()
    before = torch.cuda.mem_get_info()[0]
    model = Model(spec, mats, 8192)
    size = state(model)[0]
    assert size >= 1 << 30
    need = before - torch.cuda.mem_get_info()[0] - size
    _, want = step(model, batch)
    model.close()
    held = []
    try:
        while torch.cuda.mem_get_info()[0] > need + (256 << 20):
            held.append(DeviceBuffer(min(8 << 30, torch.cuda.mem_get_info()[0] - need - (256 << 20))))
        model = Model(spec, mats, 8192)
        size = state(model)[0]
        assert size < 256 << 20
        fits, got = step(model, batch)
        model.close()
    finally:
        for b in held:
            b.free()
    assert fits == (size >= tile_bytes(SEQ, 8192 // SEQ))
    close(got, want)
