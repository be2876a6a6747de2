"""ts2_set_batch waits for a staging slot when two batches are still queued; that wait has the limit of every other wait."""
import numpy as np
import pytest

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu


def test_the_wait_for_a_staging_slot_gives_up_and_can_be_repeated():
    """The steps take some 10 ms, the limit is 0.1 ms: the host runs ahead until no slot is free and the call returns the
    time-out; what was queued is unharmed, and the same batch can be set again."""
    spec = host.ModelSpec(dim=512, head_count=4, ffn_tiles=16, vocab=8192, attention_widths=[1024]).add_blocks(4)
    mats = host.init_weights(spec, 3)
    batches = [host.synthetic_batch(spec, 16, 1024, seed) for seed in range(8)]
    model = Model(spec, mats, batches[0].node_count)
    assert model.lib.ts2_set_wait_limit(model.h, 0.0) == capi.TS2_ERR_INVALID_ARG
    model._check(model.lib.ts2_set_wait_limit(model.h, 1e-4))
    done = 0
    with pytest.raises(capi.Ts2Error) as e:
        for i, batch in enumerate(batches):
            model.set_batch(batch)
            model.backprop(host.training_step(iteration=i))
            done += 1
    assert e.value.code == capi.TS2_ERR_TIMEOUT
    model._check(model.lib.ts2_set_wait_limit(model.h, 120.0))
    for i in range(done, len(batches)):
        model.set_batch(batches[i])
        model.backprop(host.training_step(iteration=i))
    got = model.get_weights()
    model.close()
    model = Model(spec, mats, batches[0].node_count)
    for i, batch in enumerate(batches):
        model.set_batch(batch)
        model.backprop(host.training_step(iteration=i))
        model.wait()
    for a, b in zip(got, model.get_weights()):
        assert np.array_equal(a, b)
