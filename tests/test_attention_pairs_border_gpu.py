"""Where the attention forward changes over to the kernel for long sequences: causal sequences of 3072 nodes, which that kernel
is faster for, are its own."""
import ctypes as C

import numpy as np
import pytest

from tscale2_b200 import capi
from tscale2_b200.device import DeviceBuffer, check, sync

pytestmark = pytest.mark.gpu


def forward(lib, variant, q, k, v, seq, H):
    T = len(q)
    t = np.arange(T)
    start, finish = (t // seq * seq).astype(np.int32), (t - 1).astype(np.int32)
    none = finish < start
    start[none], finish[none] = 0, -1
    ip = lambda a: a.ctypes.data_as(C.c_void_p)
    bufs = [DeviceBuffer.from_numpy(x) for x in (q, k, v)]
    o, lse = DeviceBuffer(q.nbytes), DeviceBuffer(T * H * 4)
    check(lib.ts2_attention_forward(0, None, variant, *(b.ptr for b in bufs), ip(start), ip(finish), T, H, 0.0, o.ptr, lse.ptr))
    sync()
    return o.download(q.shape, np.float16), lse.download((T, H), np.float32)


@pytest.mark.parametrize("seq,pairs", [(3072, True), (2816, False), (4096, True), (3200, False), (3073, False)])
def test_the_border(seq, pairs):
    """One sequence alone has too few work items and runs on the other kernel, whose sums come in another order: four of them give
    the same bits only if they run there too."""
    lib = capi.load_library()
    H, seqs = 16, 4
    assert -(-seq // 256) * H < 3 * 148 <= -(-seqs * seq // 256) * H
    rng = np.random.default_rng(seq)
    q, k, v = (rng.standard_normal((seqs * seq, 128 * H), dtype=np.float32).astype(np.float16) for _ in range(3))
    o, lse = forward(lib, 2, q, k, v, seq, H)
    alone, _ = forward(lib, 2, q[:seq], k[:seq], v[:seq], seq, H)
    assert np.array_equal(o[:seq], alone) == (not pairs)
    ref, ref_lse = forward(lib, 1, q, k, v, seq, H)
    ref = ref.astype(np.float64)
    # as in test_attention_pairs_gpu.py: softmax weights and results in fp16
    assert np.abs(lse - ref_lse).max() < 2e-3
    assert np.linalg.norm(o - ref) <= 1.5e-3 * np.linalg.norm(ref)
