"""The head normalisation and rotation of Q, K and V and their backward take two (node, head) items per warp: an odd number of
items (odd heads x odd nodes) leaves half a warp without one.  Whole steps with fp16 operands against the oracle."""
import numpy as np
import pytest

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,seqs,length", [(1, 1, 1), (1, 1, 33), (3, 3, 17), (3, 1, 131), (2, 1, 5)])
def test_odd_numbers_of_items_against_the_oracle(oracle_port, heads, seqs, length):
    import oracle
    spec = host.ModelSpec(dim=128, head_count=heads, ffn_tiles=2, vocab=256, attention_widths=[64], precision=capi.PREC_F16).add_blocks(1)
    mats = host.init_weights(spec, 7)
    batch = host.synthetic_batch(spec, seqs, length, 8)
    ref = oracle_port.backprop(spec, mats, batch, oracle.QUANT_HALF)
    model = Model(spec, mats, batch.node_count)
    model.set_batch(batch)
    model.backprop(host.training_step(), apply=False)
    model.wait()
    for name, g, r in zip(spec.matrix_names(), model.get_gradients(), ref["grads"]):
        size = np.linalg.norm(r.astype(np.float64))
        # fp16 operands (2^-11 each) through one block: the bound of the other fp16 parity tests; a matrix without gradient stays zero
        assert np.linalg.norm(g.astype(np.float64) - r) <= 5e-3 * size + 1e-7, name
    model.close()
