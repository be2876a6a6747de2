"""The work that a user of this library has it do, as cases that can be timed.

Four kinds, each through the public entry points:

  train      an interval of training: every iteration hands the engine its batches (Model.set_batch), runs the step
             (Model.backprop; several micro-batches accumulate before one is applied) and reads the training error, and
             the interval ends with the weights exported to the host arrays the trainer keeps (ts2_get_params).
  score      evaluation: Model.set_batch + Model.compute_score over a few batches.
  gemm       the backward contractions of one linear layer, dX and dW, on device tensors (ts2_gemm_dx,
             ts2_gemm_dw_scaled).
  attention  the attention core of one layer on device tensors, forward and backward (ts2_attention_forward,
             ts2_attention_backward in the form the engine runs: fp16 gradients).

Weights are N(0, 0.02) (router matrices N(0, 1)), token frequencies fall off as 1 / rank like those of text, operands of
the operator-level cases are normal (e4m3, fp16) or uniform (int8)."""
import ctypes as C
import math

import numpy as np
import torch

from tscale2_b200 import capi, host
from tscale2_b200.model import Model

PREC = {"fp8": capi.PREC_FP8, "f16": capi.PREC_F16, "int8": capi.PREC_INT8}


def _train(**kw):
    c = dict(kind="train", prec="fp8", dim=256, heads=4, ffn_tiles=8, vocab=4096, blocks=2, seq=128, seqs=4, window=0, alibi=0.0,
             experts=0, selected=2, expert_dim=128, iterations=2, micro=1, loss_every_step=True)
    c.update(kw)
    return c


def _score(**kw):
    c = dict(kind="score", prec="fp8", dim=256, heads=4, ffn_tiles=8, vocab=4096, blocks=2, seq=128, seqs=4, window=0, alibi=0.0,
             experts=0, selected=2, expert_dim=128, batches=4)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest training set-up (2 blocks, dim 256, 4 x 128 tokens): smoke runs, tests, hyper-parameter sweeps; the
        # errors are read once per interval, so launches and gaps are what is left
        _train(name="train_small_f16", prec="f16", iterations=8, loss_every_step=False),
        # ragged little micro-batches with a short ALiBi window, four of them accumulated per applied step
        _train(name="train_ragged_fp8", seq=100, seqs=3, window=48, alibi=0.5, iterations=2, micro=4),
        # a small model of the int8 pipeline (the reference's default build), 8 x 2048 tokens per step
        _train(name="train_d512_int8", prec="int8", dim=512, heads=4, ffn_tiles=16, vocab=50304, blocks=8, seq=2048, seqs=8,
               iterations=3),
        # the dense 12-block model fed by little micro-batches (4 x 1000 tokens), four accumulated per applied step
        _train(name="train_d768_micro_fp8", dim=768, heads=12, ffn_tiles=24, vocab=50304, blocks=12, seq=1000, seqs=4,
               iterations=1, micro=4),
        # the headline: dense 12 blocks, dim 768, 64 x 1024 tokens per step, e4m3
        _train(name="train_d768_fp8", dim=768, heads=12, ffn_tiles=24, vocab=50304, blocks=12, seq=1024, seqs=64),
        # a wide model with long sequences (8 x 4096 tokens, dim 2048, FFN 8192), as many blocks as fit the card three times
        _train(name="train_d2048_long_fp8", dim=2048, heads=16, ffn_tiles=64, vocab=50304, blocks=4, seq=4096, seqs=8),
        # mixture of experts, 32 experts of width 1024, 2 selected, 32 x 1024 tokens
        _train(name="train_moe_d1024_fp8", dim=1024, heads=16, ffn_tiles=8, vocab=50304, blocks=3, seq=1024, seqs=32, experts=32,
               selected=2, expert_dim=1024),
        # evaluation of the dense model on held-out text, fp16 operands, fragments of 1000 tokens
        _score(name="score_d768_f16", prec="f16", dim=768, heads=12, ffn_tiles=24, vocab=50304, blocks=12, seq=1000, seqs=12),
        # scoring one short text: latency
        _score(name="score_short_fp8", seq=77, seqs=1, batches=4),
        # dX and dW of a 4096 x 4096 layer over 16384 tokens
        dict(name="gemm_4096_fp8", kind="gemm", prec="fp8", tokens=16384, n_in=4096, n_out=4096, out="bf16", scaled=True),
        # the same of an FFN contraction over an odd number of tokens, int8 operands, fp32 gradients
        dict(name="gemm_ragged_int8", kind="gemm", prec="int8", tokens=3001, n_in=768, n_out=3072, out="f32", scaled=True),
        # attention core over long causal sequences
        dict(name="attention_long", kind="attention", heads=16, seq=4096, seqs=4, window=4096, alibi=0.0),
    ]


# ---- sizes ----------------------------------------------------------------------------------------------------------

def _spec(c):
    s = host.ModelSpec(dim=c["dim"], head_count=c["heads"], ffn_tiles=c["ffn_tiles"], vocab=c["vocab"],
                       attention_widths=[c["window"] or c["seq"]], precision=PREC[c["prec"]], expert_dim=c["expert_dim"],
                       moe_expert_count=c["experts"], moe_selected=c["selected"])
    return s.add_blocks(c["blocks"], alibi_slope=c["alibi"], moe=c["experts"] > 0)


def _pairs(seq, seqs, window):
    """(node, key) pairs of causal spans [t - window, t - 1] inside fragments."""
    w = min(window or seq, seq)
    return seqs * (w * (w - 1) // 2 + (seq - w) * w)


def _linear_params(c):
    """Parameters every token is multiplied with, in the layers and the final layer."""
    d, q = c["dim"], 128 * c["heads"]
    if c["experts"]:
        ffn = 3 * d * c["expert_dim"] * c["selected"] + d * c["experts"]
    else:
        ffn = 3 * d * 128 * c["ffn_tiles"]
    return c["blocks"] * (5 * d * q + ffn) + c["vocab"] * d


def _activation_bytes(c):
    """About what the engine keeps per step: sizes a drawn case to the card."""
    q, f = 128 * c["heads"], 128 * c["ffn_tiles"]
    wide = c["expert_dim"] * c["selected"] if c["experts"] else f
    return c["seq"] * c["seqs"] * (c["blocks"] * (12 * c["dim"] + 22 * q + 8 * wide) + 40 * c["dim"] + 40 * max(q, wide))


def work(case):
    c = case
    if c["kind"] in ("train", "score"):
        tokens, p = c["seq"] * c["seqs"], _linear_params(c)
        att = c["blocks"] * 4.0 * _pairs(c["seq"], c["seqs"], c["window"]) * 128 * c["heads"]
        total = _spec(c).param_count()
        if c["kind"] == "score":
            es = 2 if c["prec"] == "f16" else 1
            return {"bytes": c["batches"] * (es * total + 24.0 * tokens), "flops": c["batches"] * (2.0 * p * tokens + att)}
        passes = c["iterations"] * c["micro"]
        # an applied step reads and writes weights and momentum (fp32); the export writes the weights once more
        return {"bytes": c["iterations"] * 16.0 * total + 4.0 * total + passes * 24.0 * tokens,
                "flops": passes * (6.0 * p * tokens + 3.5 * att)}
    if c["kind"] == "gemm":
        T, i, o = c["tokens"], c["n_in"], c["n_out"]
        es, os_ = (2 if c["prec"] == "f16" else 1), (2 if c["out"] == "bf16" else 4)
        return {"bytes": float(es * (T * o + i * o + T * o + T * i) + os_ * (T * i + i * o)), "flops": 4.0 * T * i * o}
    T, q = c["seq"] * c["seqs"], 128 * c["heads"]
    return {"bytes": 2.0 * T * q * (3 + 1 + 4 + 1 + 3), "flops": 14.0 * _pairs(c["seq"], c["seqs"], c["window"]) * q}


def tolerance(case):
    c = case
    if c["kind"] == "gemm":
        return {"rel": 4e-3, "max": 2e-2} if c["out"] == "bf16" else {"rel": 2e-5, "max": 5e-3}
    if c["kind"] == "attention":
        return {"rel": 3e-3, "max": 1e-1}  # fp16 softmax weights and score gradients before the second contraction
    # fp16 operands leave 1e-3 on a gradient, e4m3 and int8 operands up to 8e-2 on two correct pipelines' gradients (3 mantissa
    # bits, stochastic rounding); the weights carry them damped by the size of an update against a weight
    return {"rel": 2e-3, "max": 2e-1} if c["prec"] == "f16" else {"rel": 1e-2, "max": 4e-1}


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _tokens(rng, vocab, shape):
    return np.minimum(vocab - 1, np.power(float(vocab), rng.random(shape)).astype(np.int64) - 1)


def _batches(c, spec, seed, n):
    rng = np.random.default_rng(seed)
    return [host.Batch(_tokens(rng, spec.vocab, (c["seqs"], c["seq"] + 1)), spec.attention_widths) for _ in range(n)]


def _weights(spec, seed):
    """The trainer's host copy of the parameters: one pinned buffer, a view per matrix."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shapes = spec.matrix_shapes()
    n = sum(a * b for a, b in shapes)
    flat = torch.empty(n, dtype=torch.float32, pin_memory=True)
    dev = torch.randn(n, device="cuda", generator=gen)
    at, mats = 0, []
    for name, (y, x) in zip(spec.matrix_names(), shapes):
        dev[at:at + y * x] *= 1.0 if name.endswith("moe.select") else 0.02
        mats.append(flat[at:at + y * x].view(y, x).numpy())
        at += y * x
    flat.copy_(dev)
    return flat, mats


def _model_state(c, seed):
    spec = _spec(c)
    flat, mats = _weights(spec, seed)
    torch.cuda.empty_cache()  # the engine allocates for itself
    train = c["kind"] == "train"
    st = {"c": c, "model": Model(spec, mats, c["seq"] * c["seqs"]), "flat": flat, "mats": mats, "views": host.matrix_views(mats),
          "batches": _batches(c, spec, seed, c["iterations"] * c["micro"] if train else c["batches"])}
    if train:
        st["steps"] = [host.training_step(rate=0.001, iteration=10 + i) for i in range(c["iterations"])]
    return st


def _operand(prec, shape, gen):
    if prec == "int8":
        return torch.randint(-127, 128, shape, device="cuda", generator=gen, dtype=torch.int8)
    return torch.randn(shape, device="cuda", generator=gen).to(torch.float16 if prec == "f16" else torch.float8_e4m3fn)


def _gemm_state(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    T, i, o = c["tokens"], c["n_in"], c["n_out"]
    od = torch.bfloat16 if c["out"] == "bf16" else torch.float32
    ws = capi.load_library().ts2_gemm_dw_workspace_bytes(T, i, o)
    scale = lambda n: torch.rand(n, device="cuda", generator=gen) * 0.09 + 0.01
    return {"c": c, "dy": _operand(c["prec"], (T, o), gen), "wt": _operand(c["prec"], (i, o), gen), "x": _operand(c["prec"], (T, i), gen),
            "dx": torch.empty((T, i), device="cuda", dtype=od), "dw": torch.empty((o, i), device="cuda", dtype=od),
            "ws": torch.empty(max(ws, 16), device="cuda", dtype=torch.uint8), "ws_bytes": ws,
            "row": scale(T) if c["scaled"] else None, "col": scale(i) if c["scaled"] else None}


def _attention_state(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    T, H = c["seq"] * c["seqs"], c["heads"]
    half = lambda: torch.randn((T, 128 * H), device="cuda", generator=gen).to(torch.float16)
    t = np.arange(T)
    start = np.maximum(t // c["seq"] * c["seq"], t - c["window"]).astype(np.int32)
    finish = (t - 1).astype(np.int32)
    none = finish < start
    start[none], finish[none] = 0, -1
    st = {"c": c, "q": half(), "k": half(), "v": half(), "dout": half(), "start": start, "finish": finish}
    st.update({n: torch.empty((T, 128 * H), device="cuda", dtype=torch.float16) for n in ("o", "dq", "dk", "dv")})
    st["lse"] = torch.empty((T, H), device="cuda")
    # sum(dout * o) per head comes from the kernel before the attention core in a training step
    _attention_forward(st)
    torch.cuda.synchronize()
    st["dscale"] = (st["dout"].float() * st["o"].float()).view(T, H, 128).sum(-1).contiguous()
    return st


def prepare(case, seed):
    if case["kind"] in ("train", "score"):
        return _model_state(case, seed)
    return _gemm_state(case, seed) if case["kind"] == "gemm" else _attention_state(case, seed)


# ---- one pass -------------------------------------------------------------------------------------------------------

def _check(rc):
    if rc != capi.TS2_OK:
        raise capi.Ts2Error(rc, capi.load_library().ts2_last_error(None).decode())


def _ptr(t):
    return None if t is None else t.data_ptr()


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _run_train(st):
    c, model = st["c"], st["model"]
    losses, k = [], 0
    for step in st["steps"]:
        for j in range(c["micro"]):
            model.set_batch(st["batches"][k])
            model.backprop(step, apply=j == c["micro"] - 1)
            k += 1
        if c["loss_every_step"]:
            losses.append(model.avg_train_err())
    if not c["loss_every_step"]:
        losses = model.loss_history(k)
    _check(model.lib.ts2_get_params(model.h, capi.PARAM_WEIGHTS, st["views"], len(st["mats"])))
    return {"losses": np.asarray(losses, np.float32), "weights": st["flat"]}


def _run_score(st):
    scores = []
    for batch in st["batches"]:
        st["model"].set_batch(batch)
        scores.append(st["model"].compute_score())
    return np.asarray(scores, np.float32)


def _run_gemm(st):
    c, lib = st["c"], capi.load_library()
    out = capi.OUT_BF16 if c["out"] == "bf16" else capi.OUT_F32
    T, i, o, prec = c["tokens"], c["n_in"], c["n_out"], PREC[c["prec"]]
    _check(lib.ts2_gemm_dx(0, _stream(), prec, out, T, i, o, _ptr(st["dy"]), _ptr(st["wt"]), _ptr(st["dx"]), 1.0 / 64, _ptr(st["row"]), None))
    _check(lib.ts2_gemm_dw_scaled(0, _stream(), prec, out, T, i, o, _ptr(st["dy"]), _ptr(st["x"]), _ptr(st["dw"]), 1.0 / 64, None,
                                  _ptr(st["col"]), _ptr(st["ws"]), st["ws_bytes"]))
    return {"dx": st["dx"], "dw": st["dw"]}


def _host(a):
    return a.ctypes.data_as(C.c_void_p)


def _attention_forward(st):
    c = st["c"]
    _check(capi.load_library().ts2_attention_forward(
        0, _stream(), 2, _ptr(st["q"]), _ptr(st["k"]), _ptr(st["v"]), _host(st["start"]), _host(st["finish"]), c["seq"] * c["seqs"],
        c["heads"], c["alibi"], _ptr(st["o"]), _ptr(st["lse"])))


def _run_attention(st):
    c = st["c"]
    _attention_forward(st)
    _check(capi.load_library().ts2_attention_backward(
        0, _stream(), 3, _ptr(st["q"]), _ptr(st["k"]), _ptr(st["v"]), _ptr(st["dout"]), _ptr(st["lse"]), _ptr(st["dscale"]),
        _host(st["start"]), _host(st["finish"]), c["seq"] * c["seqs"], c["heads"], c["alibi"], _ptr(st["dq"]), _ptr(st["dk"]),
        _ptr(st["dv"])))
    return {n: st[n] for n in ("o", "lse", "dq", "dk", "dv")}


def run(state):
    return {"train": _run_train, "score": _run_score, "gemm": _run_gemm, "attention": _run_attention}[state["c"]["kind"]](state)


# ---- more cases of the same ranges ----------------------------------------------------------------------------------

def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _multiple(rng, lo, hi, of):
    return max(of, int(round(_log(rng, lo, hi) / of)) * of)


def _draw_model(rng, kind):
    dim = _multiple(rng, 128, 2048, 128)
    seq = int(_log(rng, 32, 4096))
    c = dict(prec=rng.choice(["fp8", "fp8", "f16", "int8"]), dim=dim, heads=max(1, int(_log(rng, dim / 256, dim / 64))),
             ffn_tiles=max(1, int(dim / 128 * rng.uniform(2, 4))), vocab=_multiple(rng, 1024, 50304, 32), blocks=int(_log(rng, 1, 12.99)),
             seq=seq, seqs=max(1, int(_log(rng, 128, 65536) / seq)), window=rng.choice([0, 0, max(8, seq // 3)]),
             alibi=rng.choice([0.0, 0.0, 0.5]))
    if c["prec"] != "int8" and rng.random() < 0.2:
        c.update(experts=rng.choice([4, 8, 16, 32]), selected=rng.choice([1, 2, 4]), expert_dim=_multiple(rng, 128, 1024, 128))
    if kind == "score":
        return _score(batches=rng.randint(1, 4), **c)
    return _train(iterations=rng.randint(1, 4), micro=rng.choice([1, 1, 2, 4]), loss_every_step=rng.random() < 0.5, **c)


def draw(rng):
    limit = max(work(c)["flops"] for c in listed() if c["kind"] == "train")
    while True:
        kind = rng.choice(["train", "train", "train", "score", "gemm", "attention"])
        if kind == "gemm":
            return dict(kind=kind, prec=rng.choice(["fp8", "f16", "int8"]), tokens=int(_log(rng, 100, 32768)), n_in=_multiple(rng, 128, 4096, 32),
                        n_out=_multiple(rng, 128, 8192, 32), out=rng.choice(["bf16", "f32"]), scaled=rng.random() < 0.5)
        if kind == "attention":
            seq = int(_log(rng, 64, 4096))
            return dict(kind=kind, heads=rng.randint(1, 16), seq=seq, seqs=max(1, int(_log(rng, 512, 16384) / seq)),
                        window=rng.choice([seq, max(16, seq // 4)]), alibi=rng.choice([0.0, 0.25]))
        c = _draw_model(rng, kind)
        if work(c)["flops"] <= 0.5 * limit and _activation_bytes(c) < 20e9 and _spec(c).param_count() < 3e8:
            return c
