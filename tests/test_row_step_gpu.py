"""The row-wise steps that run behind a contraction in its own launch (few tiles: gemm_row.cu, many: the pairs of CTAs):
every result of a training step is recomputed in float64 from what the same step, traced, left in front of it.  Row counts
around the tiles' edges, widths of one and several 128-column tiles, all operand formats."""
import ml_dtypes
import numpy as np
import pytest

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

pytestmark = pytest.mark.gpu

DT = {capi.PREC_FP8: ml_dtypes.float8_e4m3fn, capi.PREC_F16: np.float16, capi.PREC_INT8: np.int8}
S_ACT = {capi.PREC_FP8: 16.0, capi.PREC_F16: 1.0, capi.PREC_INT8: 24.0}


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


def tiles(x):
    return np.asarray(x, np.float64).reshape(len(x), -1, 128)


def tilenorm(x):
    t = tiles(x)
    s = np.sqrt((t ** 2).mean(-1, keepdims=True))
    return (t / np.where(s == 0, 1, s)).reshape(len(x), -1)


def tilenorm_backward(x, d):
    x, d = tiles(x), tiles(d)
    s2 = (x ** 2).sum(-1, keepdims=True)
    return (np.sqrt(128 / s2) * (d - x * (x * d).sum(-1, keepdims=True) / s2)).reshape(len(x), -1)


def close_in_format(got, want, prec, share=2e-2):
    """want rounded to the operand format, a step of it aside where the value sits at a border between two"""
    got = got.astype(np.float64)
    if prec == capi.PREC_F16:
        assert rel(got, np.clip(want, -65504, 65504)) < 1e-3
    elif prec == capi.PREC_FP8:
        q = np.clip(want, -448, 448).astype(np.float32).astype(ml_dtypes.float8_e4m3fn).astype(np.float64)
        assert np.mean(got != q) < share and (np.abs(got - q) <= np.maximum(np.abs(q) / 8, 2.0 ** -9) * 1.01).all()
    else:
        q = np.clip(np.rint(want), -127, 127)
        assert np.mean(got != q) < share and (np.abs(got - q) <= 1).all()


class Traced:
    """One model and batch; `get` repeats the step and returns a buffer as the step had it at that point."""

    def __init__(self, prec, T, D, H, F, seq):
        self.prec, self.T, self.D, self.Q, self.F = prec, T, D, 128 * H, 128 * F
        spec = host.ModelSpec(dim=D, head_count=H, ffn_tiles=F, vocab=1024, attention_widths=[min(seq, 64)], precision=prec).add_blocks(1)
        self.model = Model(spec, host.init_weights(spec, 3), T)
        rng = np.random.default_rng(T)
        frags, rest = divmod(T, seq)
        assert rest == 0
        self.batch = host.Batch(rng.integers(0, spec.vocab, (frags, seq + 1)), spec.attention_widths)
        self.model.set_debug_taps()
        self.step()  # as it runs untraced: the taps below come from here
        self.states = [self.model.get_state_tap(l, False, T).reshape(T, D) for l in range(3)]
        self.grads = [self.model.get_state_tap(l, True, T).reshape(T, D) for l in range(3)]
        self.plain = self.model.get_gradients()
        self.n_fast = self.model.debug_read("n_fast", 1, (T, D), DT[prec])
        self.model.set_debug_trace()

    def step(self):
        self.model.set_batch(self.batch)
        self.model.backprop(host.training_step(rate=0.0), apply=True)
        self.model.wait()

    def get(self, name, width, dtype):
        self.model.set_debug_capture(name, self.T * width * np.dtype(dtype).itemsize)
        self.step()
        return self.model.debug_read("capture", 0, (self.T, width), dtype)


# (tokens, dim, heads, FFN tiles, sequence): one row; edges of a 128-row tile; odd widths; a K range shared by a cluster; then
# sizes whose contractions run on pairs of CTAs, the last pair not full
SIZES = [(1, 128, 1, 1, 1), (127, 256, 3, 2, 127), (129, 384, 2, 5, 43), (300, 256, 4, 8, 100), (512, 512, 4, 16, 128),
         (8200, 256, 3, 8, 1025), (24100, 768, 6, 12, 2410)]


@pytest.mark.parametrize("prec", [capi.PREC_FP8, capi.PREC_F16, capi.PREC_INT8])
@pytest.mark.parametrize("T,D,H,F,seq", SIZES)
def test_row_steps_of_a_training_step(prec, T, D, H, F, seq):
    m = Traced(prec, T, D, H, F, seq)
    Q, W = m.Q, m.F
    rows = np.unique(np.r_[0:min(T, 140), max(0, T - 300):T])
    # ---- forward: normalised states, Q | K | V | gate
    close_in_format(m.n_fast[rows], S_ACT[prec] * tilenorm(m.states[1][rows]), prec)
    nf = m.get("nF16", D, np.float16)[rows]
    assert rel(nf, tilenorm(m.states[2][rows])) < 5e-4
    cat = m.get("cat16[0]", 4 * Q, np.float16)[rows].astype(np.float64)
    angle = rows[:, None] * np.exp(-np.log(500000.0) * np.arange(64) / 64).astype(np.float32)[None]
    cos, sin = np.cos(angle), np.sin(angle)

    def rotate(x, back=1):
        p = x.reshape(len(rows), -1, 64, 2)
        c, s = cos[:, None], back * sin[:, None]
        return np.stack([p[..., 0] * c - p[..., 1] * s, p[..., 0] * s + p[..., 1] * c], -1).reshape(len(rows), -1)

    q, k, v = (m.get(f"{n}[0]", Q, np.float16)[rows].astype(np.float64) for n in "qkv")
    for got, want in ((q, rotate(tilenorm(cat[:, :Q]))), (k, rotate(cat[:, Q:2 * Q])), (v, tilenorm(cat[:, 2 * Q:3 * Q]))):
        assert rel(got, want) < 6e-4  # fp16; angles of many turns come from a table in fp32
    # ---- backward: final layer, activation, gate, normalisations
    g2 = tilenorm_backward(m.states[2][rows], m.get("dnF[0]", D, np.float32)[rows])
    assert rel(m.grads[2][rows], g2) < 1e-5
    for l in (1, 0):
        dn = m.get(f"dn[{l}]", D, np.float32)[rows]
        d = tilenorm_backward(m.states[l][rows], dn)
        got = m.grads[l][rows].astype(np.float64) - m.grads[l + 1][rows]
        scale = (got * d).sum() / max((d * d).sum(), 1e-300)  # the step's gradient scale, a device scalar
        # the differences of two fp32 gradients; dn in front of them is another launch's sum of the same products
        assert np.linalg.norm(got - scale * d) <= 1e-5 * np.linalg.norm(got) + 2e-7 * np.linalg.norm(m.grads[l + 1][rows])
    int8 = prec == capi.PREC_INT8
    cat_name, cat_dt, cat_prec = ("dcat16", np.float16, capi.PREC_F16) if int8 else ("dcat", DT[prec], prec)
    # FFN: layer 1
    drg = m.get("drg[1]", W, np.float16)[rows].astype(np.float64)
    wg = m.get("cat16[1]", 2 * W, np.float16)[rows].astype(np.float64)
    wscale = m.get("wscale[1]", W // 128, np.float32)[rows].astype(np.float64)
    dcat = m.get(f"{cat_name}[1]", 2 * W, cat_dt)[rows]
    s = 1 / (1 + np.exp(-2 * wg[:, W:]))
    dw = tiles(drg * s)
    wn = tiles(wg[:, :W])
    dwide = (wscale[..., None] * (dw - wn * (wn * dw).sum(-1, keepdims=True) / 128)).reshape(len(rows), W)
    dgate = drg * wg[:, :W] * 2 * s * (1 - s)
    # the e4m3 form computes in packed fp16: results near a border between two of its values change sides
    tol = {capi.PREC_F16: 1.5e-3, capi.PREC_FP8: 3.5e-2}[cat_prec]
    assert rel(dcat[:, :W], np.clip(dwide, -448, 448) if cat_prec == capi.PREC_FP8 else dwide) < tol
    assert rel(dcat[:, W:], np.clip(dgate, -448, 448) if cat_prec == capi.PREC_FP8 else dgate) < tol
    # attention gate: layer 0
    drg = m.get("drg[0]", Q, np.float16)[rows].astype(np.float64)
    o = m.get("att_o[0]", Q, np.float16)[rows].astype(np.float64)
    dcat = m.get(f"{cat_name}[0]", 4 * Q, cat_dt)[rows][:, 3 * Q:]
    s = 1 / (1 + np.exp(-2 * cat[:, 3 * Q:]))
    dgate = drg * o * 2 * s * (1 - s)
    assert rel(dcat, np.clip(dgate, -448, 448) if cat_prec == capi.PREC_FP8 else dgate) < tol
    if not int8:
        dout = m.get("dout[0]", Q, np.float16)[rows].astype(np.float64)
        assert rel(dout, drg * s) < (6e-4 if prec == capi.PREC_F16 else 2e-3)  # tanh.approx in packed fp16
        dscale = m.get("dscale[0]", H, np.float32)[rows]
        want = (dout * o).reshape(len(rows), H, 128).sum(-1)
        assert np.abs(dscale - want).max() < 2e-3 * max(np.abs(dout * o).reshape(len(rows), H, 128).sum(-1).max(), 1e-30)
    # a traced step is otherwise the same step
    for a, b in zip(m.plain, m.model.get_gradients()):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("prec", [capi.PREC_FP8, capi.PREC_F16, capi.PREC_INT8])
@pytest.mark.parametrize("T,vocab,bias", [(5003, 4128, True), (8192, 2080, False), (40, 1024, True)])
def test_score_without_logits_in_memory(prec, T, vocab, bias):
    """Scoring keeps the logits on the chip where its contraction runs on pairs; the training step rounds them to fp16 (2^-11 of
    values of a few units, averaged over T nodes).  Vocabularies that end inside a tile and inside a warp's 64 columns."""
    spec = host.ModelSpec(dim=256, head_count=1, ffn_tiles=2, vocab=vocab, attention_widths=[32], precision=prec).add_blocks(1)
    rng = np.random.default_rng(vocab)
    model = Model(spec, host.init_weights(spec, 2), T, bias=rng.standard_normal(vocab).astype(np.float32) * 2 if bias else None)
    batch = host.Batch(rng.integers(0, vocab, (1, T + 1)), spec.attention_widths)
    model.set_batch(batch)
    score = model.compute_score()
    model.backprop(host.training_step(rate=0.0))
    assert abs(score + model.avg_train_err()) < 2e-4
