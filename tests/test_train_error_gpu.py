"""ts2_avg_train_err reads the training error while the step goes on: what it reports belongs to its own step, whatever was
set since and however far the device has come."""
import time

import numpy as np
import pytest
import torch

from tscale2_b200 import capi, host
from tscale2_b200.capi import Ts2Error
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu


def with_bad_target(batch, entry):
    ti = batch.target_id.copy()
    ti[entry] = 10 ** 6
    return host.Batch.from_arrays(batch.node_count, batch.label_arr, batch.label_ptr, batch.target_node, ti, batch.att)


# one launch checks a batch of up to 4096 nodes, several a larger one
@pytest.mark.parametrize("seqs", [2, 40])
def test_the_next_batch_is_none_of_its_business(seqs):
    spec = host.ModelSpec(dim=256, head_count=2, ffn_tiles=4, vocab=1024, attention_widths=[128]).add_blocks(1)
    good = host.synthetic_batch(spec, seqs, 128, 1)
    model = Model(spec, host.init_weights(spec, 1), good.node_count)
    for _ in range(2):  # each of the two records
        model.set_batch(good)
        model.backprop(host.training_step(rate=0.0))
        err = model.avg_train_err()
        model.set_batch(with_bad_target(good, 5))
        torch.cuda.synchronize()  # the next batch is checked by now
        assert model.avg_train_err() == err  # the same word on the device
        with pytest.raises(Ts2Error) as e:  # reported once, by a call that waits for it
            model.wait()
        assert e.value.code == capi.TS2_ERR_INVALID_ARG and "1000000" in str(e.value), str(e.value)
        model.wait()


@pytest.mark.parametrize("seqs", [2, 40])
def test_its_own_batch_is(seqs):
    spec = host.ModelSpec(dim=256, head_count=2, ffn_tiles=4, vocab=1024, attention_widths=[128]).add_blocks(1)
    good = host.synthetic_batch(spec, seqs, 128, 1)
    model = Model(spec, host.init_weights(spec, 1), good.node_count)
    for i in range(2):
        model.set_batch(with_bad_target(good, 7 + i))
        model.backprop(host.training_step(rate=0.0))
        with pytest.raises(Ts2Error) as e:
            if i:
                model.set_batch(good)  # reports the step if it is over
            model.avg_train_err()
        assert e.value.code == capi.TS2_ERR_INVALID_ARG and f"node {7 + i}" in str(e.value), str(e.value)
        model.wait()
    model.backprop(host.training_step(rate=0.0))
    assert np.isfinite(model.avg_train_err())


def test_of_two_bad_batches_the_first_is_named():
    spec = host.ModelSpec(dim=256, head_count=2, ffn_tiles=4, vocab=1024, attention_widths=[128]).add_blocks(1)
    good = host.synthetic_batch(spec, 2, 128, 1)
    model = Model(spec, host.init_weights(spec, 1), good.node_count)
    for first, second in ((5, 9), (9, 5), (11, 3)):
        model.set_batch(with_bad_target(good, first))
        model.backprop(host.training_step(rate=0.0))
        with pytest.raises(Ts2Error) as e:
            model.set_batch(with_bad_target(good, second))  # reports the step if it is over
            model.wait()
        assert f"node {first} " in str(e.value), str(e.value)
        model.wait()


def test_a_call_that_gave_up_holds_no_later_one_back():
    """Twenty steps of some 5 ms are queued; reading the error gives up after 0.1 ms, and so does reading the gradient: it does not
    wait for what the first call would have read."""
    spec = host.ModelSpec(dim=512, head_count=4, ffn_tiles=16, vocab=8192, attention_widths=[1024]).add_blocks(4)
    batch = host.synthetic_batch(spec, 16, 1024, 3)
    model = Model(spec, host.init_weights(spec, 3), batch.node_count)
    outs = [np.empty(s, np.float32) for s in model.shapes]
    views = host.matrix_views(outs)
    model.set_batch(batch)
    model.backprop(host.training_step(rate=0.0))
    model.wait()
    model._check(model.lib.ts2_set_wait_limit(model.h, 1e-4))
    for _ in range(20):
        model.backprop(host.training_step(rate=0.0))
    with pytest.raises(Ts2Error) as e:
        model.avg_train_err()
    assert e.value.code == capi.TS2_ERR_TIMEOUT
    t0 = time.perf_counter()
    rc = model.lib.ts2_get_params(model.h, capi.PARAM_GRADIENT, views, len(outs))
    gave_up = time.perf_counter() - t0
    assert rc == capi.TS2_ERR_TIMEOUT
    t0 = time.perf_counter()
    torch.cuda.synchronize()
    left = time.perf_counter() - t0
    assert gave_up < 0.5 * left, (gave_up, left)
    model._check(model.lib.ts2_set_wait_limit(model.h, 120.0))
    assert np.isfinite(model.avg_train_err())
