"""Workloads of the package's public entry points, for timing and for comparing two builds.

`listed()` names the standing cases, `draw(rng)` gives further ones of the same ranges.  A case is a dict of plain values:

  kind           entry points it goes through
  prefill        mlstm_sequence: the mLSTM cell over whole sequences, rows of equal length or packed documents
  step           mlstm_step: one decode step, states in rows of their own or in a pool addressed by slots
  slstm_step     slstm_forward on a few tokens from a running state
  slstm_layer    causal_conv1d, headwise_proj, slstm_forward, headnorm_gate: an sLSTM layer's forward pass
  slstm_train    ops.SlstmFunction forward and backward: gradients of the cell input, recurrent matrix and bias
  model_prefill  LargeModel.forward on prompts (last position's logits and the final states)
  model_decode   LargeModel.forward on one token per stream with the states of the step before

Distributions follow the benchmark: q, k ~ N(0,1)/sqrt(d), v ~ N(0,1), input gates ~ N(0,1), forget gates ~ N(3,1), document
lengths log-normal (sigma 1), `docs` of them to a row, token ids uniform, weights random-initialised.
"""
import math

import torch

import xlstm_b200
from xlstm_b200 import ops
from xlstm_b200.large_model import LargeConfig, LargeModel, parameter_shapes, procedural_state_dict

DEV = "cuda"


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    big = dict(NH=8, DQ=256, DV=512)     # the heads of the 7B-shaped model
    return [
        # one user's short prompt: latency of a single call, a length that is no multiple of anything
        dict(name="prefill_short_prompt", kind="prefill", B=1, S=203, docs=0, state=False, **big),
        # one long document: a single sequence has to fill the machine
        dict(name="prefill_long_document", kind="prefill", B=1, S=8192, docs=0, state=False, **big),
        # the headline benchmark: four sequences of 8192 tokens
        dict(name="prefill_batch", kind="prefill", B=4, S=8192, docs=0, state=False, **big),
        # admission of a continuous batch: one row of 32768 tokens packed from documents of log-normal length
        dict(name="prefill_packed_row", kind="prefill", B=1, S=32768, docs=20, state=False, **big),
        # a few interactive streams
        dict(name="step_8_streams", kind="step", B=8, slots=0, **big),
        # a full serving batch in a slot pool, a few slots of it free
        dict(name="step_256_slots", kind="step", B=256, slots=256, **big),
        # token-by-token sLSTM inference: the smallest call of the package
        dict(name="slstm_one_token", kind="slstm_step", B=16, S=1, NH=4, DH=256),
        # one sLSTM layer of the block-stack configuration
        dict(name="slstm_layer", kind="slstm_layer", B=16, S=2048, NH=4, DH=256, docs=0),
        # training step of its cell
        dict(name="slstm_train", kind="slstm_train", B=16, S=2048, NH=4, DH=256, state=False),
        # decoding with the layers of the 7B-shaped model, sampling by the caller.  Two blocks: in a stack of random weights
        # bf16 rounding differences double every few blocks, deeper ones could not be compared.  The short vocabulary keeps
        # the head's share of the pass as small as it is behind 32 blocks.
        dict(name="model_decode_8_streams", kind="model_decode", B=8, D=4096, NH=8, blocks=2, vocab=2048, dtype="bf16"),
        # prefill of a prompt with the same layers
        dict(name="model_prefill", kind="model_prefill", B=1, S=2048, D=4096, NH=8, blocks=2, vocab=2048, dtype="bf16"),
        # the small fp32 model: 32-bit cells and many small operators
        dict(name="model_prefill_fp32", kind="model_prefill", B=3, S=256, D=512, NH=4, blocks=6, vocab=2048, dtype="f32"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["prefill", "prefill", "prefill", "step", "step", "slstm_step", "slstm_layer", "slstm_train", "model_decode",
                       "model_prefill", "model_prefill"])
    if kind == "prefill":
        NH, DQ, DV = rng.choice([(8, 256, 512), (8, 256, 512), (4, 128, 256), (4, 64, 128)])
        if rng.random() < 0.4:   # packed rows
            S = _log(rng, 512, 32768)
            B = 1 if S > 16384 else rng.randint(1, 2)
            return dict(kind=kind, B=B, S=S, docs=_log(rng, 1, max(2, S // 256)), state=False, NH=NH, DQ=DQ, DV=DV)
        B = _log(rng, 1, 8)
        S = _log(rng, 2, 32768 // B)
        return dict(kind=kind, B=B, S=min(S, 8192), docs=0, state=rng.random() < 0.3, NH=NH, DQ=DQ, DV=DV)
    if kind == "step":
        NH, DQ, DV = rng.choice([(8, 256, 512), (8, 256, 512), (4, 128, 256), (4, 64, 128)])
        B = _log(rng, 1, 256)
        return dict(kind=kind, B=B, slots=rng.choice([0, min(256, B + rng.randint(0, 16))]), NH=NH, DQ=DQ, DV=DV)
    if kind.startswith("slstm"):
        DH = rng.choice([64, 128, 256, 256])
        NH = rng.choice([2, 4])
        if kind == "slstm_step":
            return dict(kind=kind, B=_log(rng, 1, 64), S=rng.choice([1, 1, 2, 7]), NH=NH, DH=DH)
        B = _log(rng, 1, 32)
        S = _log(rng, 16, 2048)
        if kind == "slstm_layer":
            return dict(kind=kind, B=B, S=S, NH=NH, DH=DH, docs=rng.choice([0, 0, _log(rng, 1, max(2, S // 16))]))
        return dict(kind=kind, B=B, S=S, NH=NH, DH=DH, state=rng.random() < 0.3)
    if kind == "model_decode":
        D = rng.choice([2048, 4096, 4096])
        return dict(kind=kind, B=_log(rng, 1, 64), D=D, NH=D // 512, blocks=rng.choice([1, 2]), vocab=rng.choice([2048, 50304]), dtype="bf16")
    if rng.random() < 0.5:
        D = rng.choice([2048, 4096])
        return dict(kind=kind, B=1, S=_log(rng, 16, 2048), D=D, NH=D // 512, blocks=rng.choice([1, 2]), vocab=2048, dtype="bf16")
    return dict(kind=kind, B=_log(rng, 1, 4), S=_log(rng, 16, 512), D=512, NH=4, blocks=6, vocab=2048, dtype="f32")


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _documents(seed, B, S, docs):
    """Offsets of `docs` documents per row of S tokens: log-normal lengths, scaled so that they fill the row."""
    g = torch.Generator().manual_seed(seed)
    cu = [0]
    for b in range(B):
        ends = torch.cumsum(torch.exp(torch.randn(docs, generator=g, dtype=torch.float64)), 0)
        cu += [b * S + int(e) for e in torch.round(ends / ends[-1] * S)]
    return cu


def _model_config(c):
    return LargeConfig(embedding_dim=c["D"], num_heads=c["NH"], num_blocks=c["blocks"], vocab_size=c["vocab"])


def prepare(case, seed):
    c, kind = case, case["kind"]
    g = _generator(seed)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device=DEV)

    if kind in ("prefill", "step"):
        B, NH, DQ, DV = c["B"], c["NH"], c["DQ"], c["DV"]
        S = c.get("S", 1)
        # the layer hands the cell transposed views of its projections
        s = dict(kind=kind, q=(rnd(B, S, NH, DQ) / DQ ** 0.5).bfloat16().transpose(1, 2), k=(rnd(B, S, NH, DQ) / DQ ** 0.5).bfloat16().transpose(1, 2),
                 v=rnd(B, S, NH, DV).bfloat16().transpose(1, 2), i=rnd(B, S, NH).transpose(1, 2), f=(rnd(B, S, NH) + 3.0).transpose(1, 2))
        if kind == "step":
            N = c["slots"] or B
            for name in "qkv":
                s[name] = s[name][:, :, 0]
            s["c"], s["n"], s["m"] = rnd(N, NH, DQ, DV), rnd(N, NH, DQ), rnd(N, NH, 1).abs()
            s["slot"] = None
            if c["slots"]:
                # streams in no order, one in sixteen without a document
                slot = torch.randperm(N, generator=g, device=DEV)[:B].to(torch.int32)
                s["slot"] = torch.where(torch.rand(B, generator=g, device=DEV) < 1 / 16, torch.full_like(slot, -1), slot)
        else:
            s["cu"] = _documents(seed, B, S, c["docs"]) if c["docs"] else None
            s["init"] = (rnd(B, NH, DQ, DV), rnd(B, NH, DQ), rnd(B, NH, 1).abs()) if c["state"] else (None, None, None)
        return s
    if kind.startswith("slstm"):
        B, S, NH, DH = c["B"], c["S"], c["NH"], c["DH"]
        H = NH * DH
        R = ((torch.rand(NH, DH, 4, DH, generator=g, device=DEV) * 2 - 1) / H ** 0.5).bfloat16()
        s = dict(kind=kind, R=R, bias=rnd(NH, 4, DH) * 0.5)

        def running():
            st = rnd(4, B, H)
            st[2] = st[2].abs() + 0.5
            return st

        if kind == "slstm_layer":
            s["x"] = rnd(B, S, H).bfloat16()
            s["conv_w"], s["conv_b"] = (rnd(H, 1, 4) * 0.5).bfloat16(), (rnd(H) * 0.1).bfloat16()
            s["ws"] = [(rnd(NH, DH, DH) / DH ** 0.5).bfloat16() for _ in range(4)]
            s["norm_w"] = (1.0 + 0.1 * rnd(H)).bfloat16()
            s["cu"] = _documents(seed, B, S, c["docs"]) if c["docs"] else None
            return s
        s["wx"] = rnd(B, S, 4 * H).bfloat16()
        s["state"] = running() if kind == "slstm_step" or c["state"] else None
        if kind == "slstm_train":
            s["gh"] = rnd(B, NH, S, DH).bfloat16()
            for name in ("wx", "R", "bias"):
                s[name].requires_grad_()
        return s
    cfg = _model_config(c)
    dtype = torch.bfloat16 if c["dtype"] == "bf16" else torch.float32
    weights = procedural_state_dict(cfg, seed=seed, dtype=dtype, device=DEV, gen_device=DEV)
    s = dict(kind=kind, model=LargeModel(cfg, weights, torch.device(DEV, torch.cuda.current_device()), dtype))
    s["tokens"] = torch.randint(0, cfg.vocab_size, (c["B"], c.get("S", 1)), generator=g, device=DEV)
    if kind == "model_decode":
        dq, dv = cfg.qk_dim // c["NH"], cfg.v_dim // c["NH"]
        s["state"] = {i: (rnd(c["B"], c["NH"], dq, dv), rnd(c["B"], c["NH"], dq), rnd(c["B"], c["NH"], 1).abs()) for i in range(c["blocks"])}
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "prefill":
        h, (c, n, m) = xlstm_b200.mlstm_sequence(s["q"], s["k"], s["v"], s["i"], s["f"], *s["init"], cu_seqlens=s["cu"])
        return h, c, n, m
    if kind == "step":
        h, (s["c"], s["n"], s["m"]) = xlstm_b200.mlstm_step(s["q"], s["k"], s["v"], s["i"], s["f"], s["c"], s["n"], s["m"], slot=s["slot"])
        return h, s["c"], s["n"], s["m"]
    if kind == "slstm_step":
        h, s["state"] = xlstm_b200.slstm_forward(s["wx"], s["R"], s["bias"], s["state"])
        return h, s["state"]
    if kind == "slstm_layer":
        xc = xlstm_b200.causal_conv1d(s["x"], s["conv_w"], s["conv_b"], cu_seqlens=s["cu"])
        wx = xlstm_b200.headwise_proj([s["x"], xc], s["ws"], [1, 1, 0, 0])
        h, last = xlstm_b200.slstm_forward(wx, s["R"], s["bias"], cu_seqlens=s["cu"])
        return xlstm_b200.headnorm_gate(h, None, s["norm_w"]), last
    if kind == "slstm_train":
        h, last = ops.SlstmFunction.apply(s["wx"], s["R"], s["bias"], s["state"])
        dwx, dR, db = torch.autograd.grad(h, (s["wx"], s["R"], s["bias"]), s["gh"])
        return h.detach(), last.detach(), dwx, dR, db
    with torch.no_grad():
        if kind == "model_prefill":
            logits, st = s["model"].forward(s["tokens"], last_only=True)
        else:
            logits, st = s["model"].forward(s["tokens"], s["state"])
            s["state"] = st
    return [logits] + [t for i in sorted(st) for t in st[i]]


# ------------------------------------------------------------------------------------------------ work and tolerance
def _cell_work(B, S, NH, DQ, DV, docs, state):
    """q, k, v, gates in, h out, the final state of every document; every token updates and reads a DQ x DV state."""
    st = NH * (DQ * DV + DQ + 1) * 4 * docs
    return B * S * NH * (2 * (2 * DQ + 2 * DV) + 8) + st * (2 if state else 1), B * S * NH * 4 * DQ * DV


def work(case):
    c, kind = case, case["kind"]
    if kind == "prefill":
        by, fl = _cell_work(c["B"], c["S"], c["NH"], c["DQ"], c["DV"], c["B"] * max(1, c["docs"]), c["state"])
        return {"bytes": by, "flops": fl}
    if kind == "step":
        B, NH, DQ, DV = c["B"], c["NH"], c["DQ"], c["DV"]
        live = B * NH * (15 / 16 if c["slots"] else 1)
        return {"bytes": live * (2 * (DQ * DV + DQ + 1) * 4 + 2 * (2 * DQ + 2 * DV) + 8), "flops": live * 4 * DQ * DV}
    if kind.startswith("slstm"):
        B, S, NH, DH = c["B"], c["S"], c["NH"], c["DH"]
        H, T = NH * DH, B * S
        rec = T * NH * 2 * DH * 4 * DH
        fixed = NH * DH * 4 * DH * 2 + 2 * 4 * B * H * 4
        if kind == "slstm_layer":    # x in, the layer's output out; the four projections and the recurrence
            return {"bytes": 2 * T * H * 2 + fixed + 4 * NH * DH * DH * 2, "flops": 2 * rec}
        if kind == "slstm_train":    # wx, dh in, h, dwx out; forward, backward and the gradient of R
            return {"bytes": T * (4 + 1 + 1 + 4) * H * 2 + 3 * fixed, "flops": 3 * rec}
        return {"bytes": T * 5 * H * 2 + fixed, "flops": rec}
    cfg, esz = _model_config(c), 2 if c["dtype"] == "bf16" else 4
    B, S = c["B"], c.get("S", 1)
    shapes = parameter_shapes(cfg)
    dense = sum(math.prod(s) for n, s in shapes.items() if len(s) == 2 and n.startswith("backbone"))
    head = cfg.vocab_size * cfg.embedding_dim
    dq, dv = cfg.qk_dim // c["NH"], cfg.v_dim // c["NH"]
    state = c["blocks"] * B * c["NH"] * (dq * dv + dq + 1) * 4
    by = (dense + head) * esz + B * S * cfg.embedding_dim * esz + B * cfg.vocab_size * esz + state * (2 if kind == "model_decode" else 1)
    fl = 2 * B * (S * dense + head) + c["blocks"] * B * S * c["NH"] * 4 * dq * dv
    return {"bytes": by, "flops": fl}


def tolerance(case):
    kind = case["kind"]
    if kind.startswith("model"):
        # fp32: the cells' exponentials and long sums through six blocks; bf16: two blocks of seven rounded operators each
        return {"rel": 5e-5} if case["dtype"] == "f32" else {"rel": 2e-2, "max": 0.4}
    return {"rel": 1e-2}    # bf16 operands and outputs
