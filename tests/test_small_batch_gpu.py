"""Batches small enough to be prepared in one launch (small_batch_kernel, up to 4096 nodes and labels) next to ones that
are just too big for it: span tables, reverse ranges, targets and the inverse label index, bit-exact with numpy."""
import numpy as np
import pytest

from test_batch_prep_gpu import NEG, check_reverse, expand, ragged_batch, small_spec
from tscale2_b200 import host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,labels_per_node", [(1, (1, 2)), (33, (1, 4)), (1025, (0, 3)), (4095, (1, 2)), (4096, (1, 2)), (4097, (1, 2)),
                                               (1400, (1, 5))])
def test_tables_at_the_edges_of_the_one_launch_form(T, labels_per_node):
    spec = small_spec(vocab=70016)
    batch = ragged_batch(spec, T, np.random.default_rng(T), labels_per_node=labels_per_node, used_labels=3000)
    model = Model(spec, host.init_weights(spec, 1), T)
    for _ in range(2):  # the second one queues up behind the first
        model.set_batch(batch)
    tab = model.batch_tables(0)
    start, finish = expand(batch.att[0], T)
    assert np.array_equal(tab["span_start"], start) and np.array_equal(tab["span_finish"], finish)
    check_reverse(start, finish, tab["rev_first"], tab["rev_last"], tight=True)
    target = np.full(T, -1, np.int32)
    target[batch.target_node] = batch.target_id
    assert np.array_equal(tab["target"], target)
    labels, nodes, negative = model.label_index()
    raw = batch.label_arr
    owner = np.repeat(np.arange(T), np.diff(batch.label_ptr.astype(np.int64)))
    order = np.argsort(raw & ~NEG, kind="stable")
    assert np.array_equal(labels, (raw & ~NEG)[order])
    assert np.array_equal(nodes, owner[order])
    assert np.array_equal(negative, (raw & NEG)[order] != 0)
