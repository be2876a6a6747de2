"""The attention forward of long causal sequences (kernels_att_fwd_pair_tc.cu) against the row-wise kernel, which takes every
span by itself: sequences of an odd and an even number of 256-node pairs, nodes without a span, last blocks that are not full
or empty, keys scaled so that the running maximum moves often."""
import ctypes as C

import numpy as np
import pytest

from tscale2_b200 import capi
from tscale2_b200.device import DeviceBuffer, check, sync

pytestmark = pytest.mark.gpu


def forward(lib, variant, q, k, v, start, finish, H):
    T = len(start)
    ip = lambda a: a.ctypes.data_as(C.c_void_p)
    bufs = [DeviceBuffer.from_numpy(x) for x in (q, k, v)]
    o, lse = DeviceBuffer(q.nbytes), DeviceBuffer(T * H * 4)
    check(lib.ts2_attention_forward(0, None, variant, *(b.ptr for b in bufs), ip(start), ip(finish), T, H, 0.0, o.ptr, lse.ptr))
    sync()
    return o.download(q.shape, np.float16).astype(np.float64), lse.download((T, H), np.float32)


@pytest.mark.parametrize("seq,seqs,T,H,key_scale", [(4096, 2, 8192, 14, 1.0), (3328, 4, 13275, 9, 2.0), (4096, 4, 12289, 10, 1.0),
                                                    (3584, 3, 10752 - 128, 11, 0.1)])
def test_pairs_match_the_row_wise_kernel(seq, seqs, T, H, key_scale):
    lib = capi.load_library()
    rng = np.random.default_rng(T + H)
    q, k, v = (rng.standard_normal((T, 128 * H), dtype=np.float32) for _ in range(3))
    q, k, v = q.astype(np.float16), (k * key_scale).astype(np.float16), v.astype(np.float16)
    t = np.arange(T)
    start, finish = (t // seq * seq).astype(np.int32), (t - 1).astype(np.int32)
    none = finish < start
    none[700:900] = True  # a block of 128 nodes, and parts of two, without keys
    start[none], finish[none] = 0, -1
    assert (finish - start + 1).sum() >= 1536 * T and -(-T // 256) * H >= 3 * 148  # else the other kernel runs
    o, lse = forward(lib, 2, q, k, v, start, finish, H)
    ref, ref_lse = forward(lib, 1, q, k, v, start, finish, H)
    assert np.abs(lse - ref_lse).max() < 2e-3
    # softmax weights and result in fp16 (2^-11 each); the row-wise result in fp16 too
    assert np.linalg.norm(o - ref) <= 1.5e-3 * np.linalg.norm(ref)
    for rows in (slice(640, 960), slice(T - 130, T)):
        assert np.linalg.norm(o[rows] - ref[rows]) <= 1.5e-3 * np.linalg.norm(ref[rows])
    again, _ = forward(lib, 2, q, k, v, start, finish, H)
    assert np.array_equal(o, again)
