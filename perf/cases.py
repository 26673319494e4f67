"""Performance cases of the KDA framework: the calls its users make, over the sizes they make them at.

Seven kinds of work, each through the package's public entry points:

  step      ``recurrent_kda_step``: one decoded token for every running sequence, state updated in place or not
  burst     ``fused_recurrent_kda``: a few tokens per sequence (a verified draft, a short continuation)
  prefill   ``chunk_kda`` under ``no_grad``: a prompt in, outputs and the final state for decoding out
  train     ``chunk_kda`` forward and backward on a dense batch, both recompute policies
  packed    the same on documents packed with ``cu_seqlens``, with an initial state per document
  serve     the whole ``KimiDeltaAttention`` sublayer, forward only, under autocast
  layer     the whole sublayer, forward and backward, under autocast

Values follow ``openkimi_b200.synthetic``: q, k, v, do ~ N(0,1); gate input ~ N(0,1) with A_log ~ U(ln 1, ln 16), or, with
``spans``, N(3,1) with A_log ~ U(ln 8, ln 64) and beta logits ~ N(2,1), so that the decay inside a chunk reaches the span
guard; initial states ~ N(0, 0.02); sublayer weights ~ N(0, 0.02).
"""

from __future__ import annotations

import math

import torch

from openkimi_b200 import KimiDeltaAttention, chunk_kda, fused_recurrent_kda, recurrent_kda_step
from openkimi_b200.synthetic import random_cu_seqlens

DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
FUSED = dict(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True, state_v_first=True)


def listed():
    return [
        # one user's chat: a token at a time, the latency of a single call
        dict(name="step_one", kind="step", seqs=1, heads=6, dim=128, dtype="bf16", inplace=True),
        # a serving batch: every state is read and written once per token
        dict(name="step_batch", kind="step", seqs=256, heads=6, dim=128, dtype="bf16", inplace=True),
        # a draft of eight tokens checked for four sequences
        dict(name="burst_draft", kind="burst", seqs=4, time=8, heads=6, dim=128, dtype="bf16"),
        # a chat prompt of an odd length
        dict(name="prefill_short", kind="prefill", batch=1, time=509, heads=6, dim=128, dtype="bf16", state=False),
        # one long document continued from a state: a single chain of chunks per head
        dict(name="prefill_long", kind="prefill", batch=1, time=16381, heads=6, dim=128, dtype="bf16", state=True),
        # the primary profile of the benchmark, intermediates kept
        dict(name="train_primary", kind="train", batch=16, time=2048, heads=6, dim=128, dtype="bf16", keep=True, spans=False),
        # decay so strong that tiles of the diagonal fail the span guard; intermediates rebuilt in the backward (the default)
        dict(name="train_spans", kind="train", batch=4, time=4096, heads=6, dim=128, dtype="bf16", keep=False, spans=True),
        # the smallest micro-batch: one sequence, odd length
        dict(name="train_micro", kind="train", batch=1, time=2047, heads=6, dim=128, dtype="bf16", keep=True, spans=False),
        # sixteen documents of uneven length packed to 65536 tokens
        dict(name="packed_long", kind="packed", time=65536, docs=16, heads=6, dim=128, dtype="bf16", keep=True),
        # the FP32 mode that other runs are validated against
        dict(name="train_fp32", kind="train", batch=2, time=512, heads=4, dim=64, dtype="fp32", keep=True, spans=False),
        # the sublayer of a serving step over a few prompts
        dict(name="serve_layer", kind="serve", batch=4, time=1000, heads=6, dim=128, dtype="bf16"),
        # the sublayer of the primary model over its training batch
        dict(name="layer_train", kind="layer", batch=64, time=2048, heads=6, dim=128, dtype="bf16", keep=True),
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm; most of what comes out is odd or ragged
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("step", "burst", "prefill", "train", "packed", "fp32", "serve", "layer"))
    heads = rng.choice((2, 3, 4, 6, 8, 12))
    if kind == "step":
        return dict(kind="step", seqs=size(2, 512), heads=heads, dim=rng.choice((64, 128, 128)),
                    dtype=rng.choice(("bf16", "bf16", "fp32")), inplace=rng.random() < 0.75)
    if kind == "burst":
        return dict(kind="burst", seqs=size(1, 64), time=rng.randint(2, 16), heads=heads, dim=128, dtype="bf16")
    if kind == "prefill":
        time = size(16, 32768)
        return dict(kind="prefill", batch=max(1, min(size(1, 16), 65536 // time)), time=time, heads=heads, dim=128, dtype="bf16",
                    state=rng.random() < 0.5)
    if kind == "packed":
        time = size(1024, 65536)
        return dict(kind="packed", time=time, docs=size(2, max(2, min(32, time // 64))), heads=min(heads, 6), dim=128,
                    dtype="bf16", keep=rng.random() < 0.5)
    if kind == "fp32":
        return dict(kind="train", batch=rng.randint(1, 4), time=size(64, 1024), heads=min(heads, 6), dim=rng.choice((64, 64, 128)),
                    dtype="fp32", keep=rng.random() < 0.5, spans=rng.random() < 0.25)
    if kind == "train":
        time = size(64, 8192)
        return dict(kind="train", batch=max(1, min(size(1, 32), 32768 // time)), time=time, heads=heads, dim=128, dtype="bf16",
                    keep=rng.random() < 0.5, spans=rng.random() < 0.25)
    time = size(64, 4096)
    most = 16384 if kind == "serve" else 65536
    return dict(kind=kind, batch=max(1, min(size(1, 64), most // time)), time=time, heads=rng.choice((4, 6, 8)), dim=128,
                dtype="bf16", **({} if kind == "serve" else {"keep": rng.random() < 0.5}))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(gen, shape, dtype=torch.float32, mean=0.0, std=1.0):
    return (torch.randn(shape, generator=gen, device="cuda") * std + mean).to(dtype)


def _inputs(case, gen, lead, spans=False):
    """Tensors of one call whose leading dimensions are ``lead``: [B, T] or, for a decoding step, [N]."""
    H, d, dt = case["heads"], case["dim"], DTYPES[case["dtype"]]
    lo, hi = (8.0, 64.0) if spans else (1.0, 16.0)
    s = {n: _normal(gen, (*lead, H, d), dt) for n in ("q", "k", "v")}
    s["g"] = _normal(gen, (*lead, H, d), dt, mean=3.0 if spans else 0.0)
    s["beta"] = _normal(gen, (*lead, H), dt, mean=2.0 if spans else 0.0)
    s["A_log"] = torch.rand(H, generator=gen, device="cuda") * math.log(hi / lo) + math.log(lo)
    s["dt_bias"] = torch.zeros(H * d, device="cuda")
    return s


def _layer(case, gen):
    """The sublayer with random weights N(0, 0.02); norm weight 1, dt_bias 0, A_log ~ U(ln 1, ln 16)."""
    H, d = case["heads"], case["dim"]
    with torch.device("cuda"):
        m = KimiDeltaAttention(H * d, H, d, conv_kernel=4, disable_recompute=case.get("keep", True))
    with torch.no_grad():
        for name, prm in m.named_parameters():
            if prm.dim() >= 2 and name != "dt_bias":
                prm.normal_(0.0, 0.02, generator=gen)
        m.A_log.uniform_(0.0, math.log(16.0), generator=gen)
    return m


def prepare(case, seed):
    gen, kind = _generator(seed), case["kind"]
    H, d, dt = case["heads"], case["dim"], DTYPES[case["dtype"]]
    if kind == "step":
        return dict(case=case, x=_inputs(case, gen, (case["seqs"],)), state=_normal(gen, (case["seqs"], H, d, d), std=0.02))
    if kind == "burst":
        return dict(case=case, x=_inputs(case, gen, (case["seqs"], case["time"])),
                    state=_normal(gen, (case["seqs"], H, d, d), std=0.02))
    if kind == "prefill":
        return dict(case=case, x=_inputs(case, gen, (case["batch"], case["time"])),
                    state=_normal(gen, (case["batch"], H, d, d), std=0.02) if case["state"] else None)
    if kind in ("train", "packed"):
        batch = case.get("batch", 1)
        x = _inputs(case, gen, (batch, case["time"]), case.get("spans", False))
        s = dict(case=case, x=x, do=_normal(gen, (batch, case["time"], H, d), dt), cu=None, cu_cpu=None, state=None)
        if kind == "packed":
            s["cu_cpu"] = random_cu_seqlens(case["time"], case["docs"], seed=seed)
            s["cu"] = s["cu_cpu"].cuda()
            s["state"] = _normal(gen, (case["docs"], H, d, d), std=0.02)
        s["leaves"] = [t for t in (*x.values(), s["state"]) if t is not None]
        for t in s["leaves"]:
            t.requires_grad_(True)
        return s
    s = dict(case=case, layer=_layer(case, gen), x=_normal(gen, (case["batch"], case["time"], H * d), dt))
    if kind == "layer":
        s["x"].requires_grad_(True)
        s["dout"] = _normal(gen, s["x"].shape, dt)
        s["leaves"] = [s["x"], *s["layer"].parameters()]
    return s


def run(s):
    case, x = s["case"], s["x"]
    kind, scale = case["kind"], case["dim"] ** -0.5
    if kind == "step":
        return recurrent_kda_step(**x, state=s["state"], scale=scale, inplace=case["inplace"], **FUSED)
    if kind == "burst":
        return fused_recurrent_kda(**x, scale=scale, initial_state=s["state"], output_final_state=True, **FUSED)
    if kind == "prefill":
        with torch.no_grad():
            return chunk_kda(**x, scale=scale, initial_state=s["state"], output_final_state=True, **FUSED)
    if kind == "serve":
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return s["layer"](x)
    for t in s["leaves"]:
        t.grad = None
    if kind == "layer":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = s["layer"](x)
        out.backward(s["dout"])
        return [out, *(t.grad for t in s["leaves"])]
    o, ht = chunk_kda(**x, scale=scale, initial_state=s["state"], output_final_state=True, cu_seqlens=s["cu"],
                      cu_seqlens_cpu=s["cu_cpu"], disable_recompute=case["keep"], **FUSED)
    o.backward(s["do"])
    return [o, ht, *(t.grad for t in s["leaves"])]


def work(case):
    """Inputs read once, outputs written once; operations of the recurrence itself (prediction, update and output of a
    [d, d] state, 2 d^2 each, the backward twice that) and of the sublayer's projections."""
    kind, H, d = case["kind"], case["heads"], case["dim"]
    es = 2 if case["dtype"] == "bf16" else 4
    seqs = case.get("seqs") or case.get("docs") or case["batch"]
    tokens = case["time"] if kind == "packed" else case.get("batch", seqs) * case.get("time", 1)
    back = kind in ("train", "packed", "layer")
    flops = tokens * H * 6 * d * d * (3 if back else 1)
    row = H * d * es                                   # one token of q, k, g, v or o
    params = (H + H * d) * 4
    if kind in ("serve", "layer"):
        width, proj = H * d, H * d
        weights = 4 * width * proj + width * (2 * d + H) + 2 * d * proj
        flops += 2 * tokens * weights * (3 if back else 1)
        small = params + (3 * proj * 4 + d) * 4        # gate, filters, norm weight
        acts = tokens * width * es
        return dict(bytes=(2 * acts + weights * 4 + small) + ((2 * acts + weights * 4 + small) if back else 0), flops=flops)
    state = seqs * H * d * d * 4
    has_state = kind in ("step", "burst", "packed") or case.get("state", False)
    total = tokens * (5 * row + H * es) + params + state * (2 if has_state else 1)
    if back:                                           # do in; dq, dk, dv, dg, dbeta, the parameters' and the state's out
        total += tokens * (5 * row + H * es) + params + (state if has_state else 0)
    return dict(bytes=total, flops=flops)


def tolerance(case):
    """BF16 operands and outputs with FP32 accumulation, or FP32 throughout (decays reach 2^-100 and more inside a chunk, and
    the gate gradient is a difference of sums of such terms)."""
    return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 1e-4}
