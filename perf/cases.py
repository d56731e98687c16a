"""What the framework's speed is measured on: calls of its public entry points over the range of sizes they serve.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` one more of the same ranges; `prepare`
makes what a caller has in hand, `run` is one pass.  Kinds:

  forward   gdn_chunk on tensors in GPU memory: one or a few new tokens on a stored state (decode), prompts, long
            sequences, batches; with or without what a layer adds around it (q/k normalisation, gate activations,
            gated output normalisation)
  packed    gdn_chunk_varlen on sequences of different lengths laid end to end
  host      gdn_chunk_host with inputs and results in page-locked host memory

The operator is forward only.  Head dimension 128 everywhere (fixed in the kernels).
"""

import math
import random

import torch
import torch.nn.functional as F

from gdn_qsa_sm80 import gdn_chunk, gdn_chunk_host, gdn_chunk_varlen

D = 128

FORWARD = {"kind": "forward", "B": 1, "S": 1, "Hq": 16, "Hv": 32, "gates": "fp32", "state": True, "decay": 0.5, "layer": False}


def _forward(name, **sizes):
    return dict(FORWARD, name=name, **sizes)


def listed():
    return [
        # one stream generating text: the smallest call, latency and launches only
        _forward("decode one sequence", gates="bf16"),
        # a serving batch generating text, called the way a layer calls it: raw projections in, gated rows out
        _forward("decode 64 sequences, layer", B=64, gates="bf16", layer=True),
        # a few drafted tokens verified at once on stored states
        _forward("verify 4 tokens of 8", B=8, S=4),
        # a short chat prompt of ragged length, called the way a layer calls it
        _forward("prompt of 333, layer", S=333, gates="bf16", state=False, layer=True),
        # two prompts through a layer with as many q/k heads as value heads
        _forward("two prompts, equal heads", B=2, S=1500, Hq=8, Hv=8, gates="bf16", state=False),
        # a batch of prompts with everything a layer adds, length one short of a multiple
        _forward("four prompts, layer", B=4, S=1999, gates="bf16", layer=True),
        # the default model shape (synthetic.WORKLOADS["default"])
        _forward("default", S=8192),
        # many short sequences (synthetic.WORKLOADS["short_batch"])
        _forward("short batch", B=16, S=2048, state=False),
        # the largest: a throughput batch (synthetic.WORKLOADS["throughput"])
        _forward("throughput", B=64, S=4096),
        # one long document with slow decay (synthetic.WORKLOADS["long_context"])
        _forward("long context", S=131072, decay=0.1, state=False),
        # prompts of different lengths packed end to end, as a serving scheduler hands them over
        {"name": "packed prompts", "kind": "packed", "n": 24, "T": 12011, "Hq": 16, "Hv": 32, "gates": "bf16", "decay": 0.5,
         "state": True, "layer": False},
        # the default model shape with inputs and results in host memory, one call at a time into kept buffers
        {"name": "default from host memory", "kind": "host", "B": 1, "S": 8192, "Hq": 16, "Hv": 32, "gates": "fp32",
         "decay": 0.5, "state": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    Hq, Hv = rng.choice([(16, 32), (16, 32), (8, 16), (4, 8), (2, 4), (8, 8), (16, 16), (3, 3), (4, 16), (2, 16)])
    common = {"Hq": Hq, "Hv": Hv, "gates": rng.choice(["bf16", "fp32"]), "state": rng.random() < 0.6,
              "decay": round(math.exp(rng.uniform(math.log(0.05), math.log(2.0))), 3)}
    what = rng.choices(["decode", "prompt", "long", "packed", "host"], weights=[3, 4, 3, 2, 1])[0]
    if what == "decode":      # one to eight new tokens on stored states
        c = dict(common, kind="forward", B=_log_int(rng, 1, 256), S=rng.choice([1, 1, 1, 2, 3, 4, 6, 8]), layer=rng.random() < 0.5)
        c["state"] = True
        return c
    if what == "prompt":      # batches of sequences of up to 4096 tokens, at most 262144 tokens of 32 heads together
        S = _log_int(rng, 9, 4096)
        most = min(64, 262144 * 32 // (S * Hv))
        return dict(common, kind="forward", B=_log_int(rng, 1, max(1, most)), S=S, layer=rng.random() < 0.5)
    if what == "long":        # a few long sequences
        S = _log_int(rng, 4096, 65536)
        return dict(common, kind="forward", B=rng.randint(1, max(1, min(4, 131072 // S))), S=S, layer=rng.random() < 0.3)
    if what == "packed":      # sequences of 1 to a few thousand tokens, end to end
        n = _log_int(rng, 2, 64)
        return dict(common, kind="packed", n=n, T=n * _log_int(rng, 16, 2048), layer=rng.random() < 0.5)
    S = _log_int(rng, 512, 8192)
    return dict(common, kind="host", B=rng.randint(1, max(1, min(4, 8192 // S))), S=S)


def lengths(n, T):
    """n sequence lengths that add up to T, spread by about a factor of four; the same ones for every seed."""
    rng = random.Random(n * 1000003 + T)
    w = [math.exp(rng.uniform(-0.7, 0.7)) for _ in range(n)]
    cut = [0] + [round(T * sum(w[:i + 1]) / sum(w)) for i in range(n)]
    for i in range(1, n + 1):          # none empty
        cut[i] = max(cut[i], cut[i - 1] + 1)
    cut[n] = T
    for i in range(n - 1, 0, -1):
        cut[i] = min(cut[i], cut[i + 1] - 1)
    return cut


def prepare(case, seed):
    """Inputs with the distributions of gdn_qsa_sm80_b200/synthetic.py, generated on the GPU from the seed."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    packed = case["kind"] == "packed"
    B, S = (1, case["T"]) if packed else (case["B"], case["S"])
    Hq, Hv = case["Hq"], case["Hv"]
    layer = bool(case.get("layer", False))

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device=dev)

    def qk():   # a layer hands its projections over as they are; otherwise head vectors of unit norm
        x = randn(B, S, Hq, D)
        return (x if layer else F.normalize(x, dim=-1)).bfloat16()

    q, k, v = qk(), qk(), randn(B, S, Hv, D).bfloat16()
    g, beta = randn(B, S, Hv), randn(B, S, Hv)
    if layer:   # raw projections; the decay's scale sits in the projection: softplus(x + log(scale)) ~ scale softplus(x)
        g = g + math.log(case["decay"])
    else:
        g, beta = -F.softplus(g) * case["decay"], torch.sigmoid(beta)
    if case["gates"] == "bf16":
        g, beta = g.bfloat16(), beta.bfloat16()
    n_states = case["n"] if packed else B
    h0 = 0.1 * randn(n_states, Hv, D, D) if case["state"] else None
    s = {"kind": case["kind"], "x": (q, k, v, g, beta), "h0": h0, "options": {}}
    if layer:
        s["options"] = {"use_qk_l2norm_in_kernel": True, "gate_activations": True}
    if packed:
        s["cu"] = lengths(case["n"], case["T"])
    elif layer:
        s["options"]["output_gate"] = (randn(B, S, Hv, D).bfloat16(), (1 + 0.1 * randn(D)).bfloat16())
    if case["kind"] == "host":
        s["x"] = tuple(t.cpu().pin_memory() for t in s["x"])
        s["h0"] = None if h0 is None else h0.cpu().pin_memory()
        s["out"] = torch.empty(B, S, Hv, D, dtype=torch.bfloat16, pin_memory=True)
        s["hT"] = torch.empty(B, Hv, D, D, pin_memory=True)
    return s


def run(s):
    if s["kind"] == "host":
        return gdn_chunk_host(*s["x"], initial_state=s["h0"], out=s["out"], final_state_out=s["hT"])
    if s["kind"] == "packed":
        return gdn_chunk_varlen(*s["x"], s["cu"], initial_state=s["h0"], **s["options"])
    return gdn_chunk(*s["x"], initial_state=s["h0"], **s["options"])


def work(case):
    """Bytes: q, k, v, gates and states read once, outputs and states written once.  Flops: the operator's dense
    products by 64-token chunks (products of q and k once per q/k head), or, up to 8 tokens, the recurrence itself."""
    Hq, Hv = case["Hq"], case["Hv"]
    packed = case["kind"] == "packed"
    tokens = case["T"] if packed else case["B"] * case["S"]
    n_states = case["n"] if packed else case["B"]
    gate = 2 if case["gates"] == "bf16" else 4
    b = tokens * (Hq * 2 * D * 2 + Hv * 2 * D * 2 + Hv * 2 * gate) + n_states * Hv * D * D * 4 * (2 if case["state"] else 1)
    if case.get("layer", False) and not packed:
        b += tokens * Hv * D * 2 + 2 * D
    if not packed and case["S"] <= 8:
        f = tokens * Hv * 7 * D * D
    else:
        f = tokens * (Hq * 4 * 64 * D + Hv * (6 * 64 * D + 6 * D * D))
    return {"bytes": b, "flops": f}


def tolerance(case):
    """bf16 operands of the chunked products (the operator's parity bar: 1e-2); up to 8 tokens the arithmetic is fp32
    and only the bf16 rounding of the rows, once or (normalised rows) twice, separates two implementations."""
    if case["kind"] == "forward" and case["S"] <= 8:
        return {"rel": 4e-3, "max": 2e-2}
    return {"rel": 1e-2}
