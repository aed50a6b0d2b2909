"""The work whose time counts: passes through the package's public entry points as a serving program makes them.

Kinds of pass (``case["kind"]``):

* ``forward``  one ``gdn_forward`` on prepared tensors: prompts from a few tokens to 131072, one request or a batch,
  both gate types, with and without a carried-in state.
* ``varlen``   one ``gdn_forward_varlen``: requests of unequal length packed along the token axis, offsets on the
  host or on the device.
* ``prefill``  a layer's prefill from its raw projections: ``gdn_forward_projections`` -> ``rmsnorm_gated`` ->
  ``out_proj_gemm``.
* ``decode``   a layer's single-token step: ``gdn_prepare_inputs`` -> ``gdn_decode_step`` (state updated in place) ->
  ``rmsnorm_gated`` -> ``out_proj_gemm``.
* ``verify``   a speculative-decoding step: ``gdn_verify_step`` on a window of draft tokens, then
  ``gdn_commit_step`` of the accepted prefixes (state updated in place).

Head counts, sizes and value distributions are those of ``actlizela_b200/workloads.py``, the tests and ``bench.py``
(out_proj: 2560 output features); lengths off the 64-token chunk are as common in use as multiples of it.
"""
import random

import torch
import torch.nn.functional as F

from actlizela_b200 import (gdn_commit_step, gdn_decode_step, gdn_forward, gdn_forward_projections, gdn_forward_varlen,
                            gdn_prepare_inputs, gdn_verify_step, out_proj_gemm, rmsnorm_gated)

DIM = 128
FEATURES = 2560                 # output features of out_proj
LARGEST = 131072 * 32           # token-heads of the largest forward


def _forward(name, batch, tokens, hk, hv, gate="logsigmoid", gate_fp32=True, initial=False):
    return dict(name=name, kind="forward", batch=batch, tokens=tokens, hk=hk, hv=hv, gate=gate, gate_fp32=gate_fp32,
                initial=initial)


def listed():
    return [
        # a short prompt, length off the chunk: launches and latency are what it costs
        _forward("forward_t100", 1, 100, 16, 32),
        # an ordinary prompt and the headline prompt
        _forward("forward_t2048", 1, 2048, 16, 32),
        _forward("forward_t8192", 1, 8192, 16, 32),
        # a continued prompt (state carried in) with three value heads to a key head
        _forward("forward_t8192_hv48", 1, 8192, 16, 48, initial=True),
        # a full batch, BF16 gates, states carried in
        _forward("forward_b8_t4096", 8, 4096, 16, 32, gate_fp32=False, initial=True),
        # a batch of ragged prompts whose gates hardly decay, four value heads to a key head
        _forward("forward_b4_t3000_slow", 4, 3000, 8, 32, gate="slow", initial=True),
        # a long document
        _forward("forward_t131072", 1, 131072, 16, 32, initial=True),
        # a scheduler's packed prefill batch: unequal requests, offsets in device memory
        dict(name="varlen_24x300", kind="varlen", sequences=24, tokens=7200, layout=1, hk=16, hv=32, gate="logsigmoid",
             gate_fp32=True, initial=False, offsets="device"),
        # a whole layer's prefill from raw projections to the output projection, two ragged prompts
        dict(name="layer_prefill_b2_t1500", kind="prefill", batch=2, tokens=1500, hk=16, hv=32, initial=True),
        # a whole layer's decode step: few requests (latency) and many (state bandwidth)
        dict(name="layer_decode_b4", kind="decode", batch=4, hk=16, hv=32),
        dict(name="layer_decode_b128", kind="decode", batch=128, hk=16, hv=32),
        # speculative decoding: four draft tokens for each of 16 requests, then the accepted prefixes
        dict(name="verify_b16_w4", kind="verify", batch=16, width=4, hk=16, hv=32, gate_fp32=True),
    ]


def _log_uniform(rng, low, high):
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def draw(rng):
    """One more case: any of the kinds, sizes spread over the logarithm of the range, odd ones among them."""
    kind = rng.choice(("forward", "forward", "forward", "forward", "varlen", "prefill", "decode", "verify"))
    hk, hv = rng.choice(((16, 32), (16, 32), (16, 48), (8, 32), (16, 16), (4, 8), (2, 6), (32, 64)))
    if kind == "forward":
        batch = rng.choice((1, 1, 1, 2, 3, 4, 8))
        tokens = _log_uniform(rng, 17, min(131072, LARGEST // (batch * hv)))
        if rng.random() < 0.4:
            tokens = max(64, tokens // 64 * 64)
        return dict(kind=kind, batch=batch, tokens=tokens, hk=hk, hv=hv,
                    gate=rng.choice(("logsigmoid", "logsigmoid", "logsigmoid", "slow")),
                    gate_fp32=rng.random() < 0.6, initial=rng.random() < 0.5)
    if kind == "varlen":
        sequences = _log_uniform(rng, 2, 64)
        return dict(kind=kind, sequences=sequences, tokens=sequences * _log_uniform(rng, 40, 1200),
                    layout=rng.randrange(1 << 20), hk=hk, hv=hv, gate=rng.choice(("logsigmoid", "logsigmoid", "slow")),
                    gate_fp32=rng.random() < 0.6, initial=rng.random() < 0.5, offsets=rng.choice(("device", "host")))
    if kind == "prefill":
        batch = rng.choice((1, 1, 2, 4))
        return dict(kind=kind, batch=batch, tokens=_log_uniform(rng, 50, 16000 // batch), hk=hk, hv=hv,
                    initial=rng.random() < 0.5)
    if kind == "decode":
        return dict(kind=kind, batch=_log_uniform(rng, 1, 256), hk=hk, hv=hv)
    return dict(kind=kind, batch=_log_uniform(rng, 1, 96), width=rng.randint(2, 8), hk=hk, hv=hv,
                gate_fp32=rng.random() < 0.6)


def _bounds(case):
    """Offsets of the packed requests: lengths spread around their mean, every request at least one token."""
    rng = random.Random(case["layout"])
    n, tokens = case["sequences"], case["tokens"]
    weights = [rng.uniform(0.1, 2.0) for _ in range(n)]
    total, run, bounds = sum(weights), 0.0, [0]
    for w in weights[:-1]:
        run += w
        bounds.append(max(bounds[-1] + 1, int(run / total * (tokens - n))))
    return bounds + [tokens]


def _inputs(gen, batch, tokens, hk, hv, gate, gate_fp32):
    """q, k normalised per head vector, v ~ N(0,1), natural-log decay, beta in (0,1)."""
    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    q = F.normalize(normal(batch, tokens, hk, DIM), dim=-1).to(torch.bfloat16)
    k = F.normalize(normal(batch, tokens, hk, DIM), dim=-1).to(torch.bfloat16)
    v = normal(batch, tokens, hv, DIM).to(torch.bfloat16)
    if gate == "slow":
        g = -0.01 * torch.rand(batch, tokens, hv, generator=gen, device="cuda")
        beta = torch.sigmoid(normal(batch, tokens, hv) + 1.0)
    else:
        g = F.logsigmoid(normal(batch, tokens, hv) + 2.0)
        beta = torch.sigmoid(normal(batch, tokens, hv))
    return q, k, v, g.to(torch.float32 if gate_fp32 else torch.bfloat16), beta.to(torch.bfloat16)


def _state(gen, rows, hv):
    return 0.05 * torch.randn(rows, hv, DIM, DIM, generator=gen, device="cuda")


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, hk, hv = case["kind"], case["hk"], case["hv"]
    s = dict(case)

    def normal(*shape, dtype=torch.bfloat16):
        return torch.randn(*shape, generator=gen, device="cuda").to(dtype)

    if kind in ("forward", "varlen"):
        batch = 1 if kind == "varlen" else case["batch"]
        s["x"] = _inputs(gen, batch, case["tokens"], hk, hv, case["gate"], case["gate_fp32"])
        s["initial_state"] = _state(gen, case["sequences"] if kind == "varlen" else batch, hv) if case["initial"] else None
        if kind == "varlen":
            bounds = _bounds(case)
            s["cu_seqlens"] = torch.tensor(bounds, dtype=torch.int32, device="cuda") if case["offsets"] == "device" else bounds
    elif kind == "verify":
        batch, width = case["batch"], case["width"]
        s["x"] = _inputs(gen, batch, width, hk, hv, "logsigmoid", case["gate_fp32"])
        s["state"] = _state(gen, batch, hv)
        s["counts"] = torch.randint(0, width + 1, (batch,), generator=gen, device="cuda", dtype=torch.int32)
    else:
        # raw projections of a layer and its weights
        rows = (case["batch"], case["tokens"]) if kind == "prefill" else (case["batch"],)
        s["mixed"] = normal(*rows, (2 * hk + hv) * DIM)
        s["a"], s["b"] = normal(*rows, hv), normal(*rows, hv)
        s["a_log"], s["dt_bias"] = 0.5 * normal(hv, dtype=torch.float32), normal(hv, dtype=torch.float32)
        s["z"] = normal(*rows, hv, DIM)
        s["norm_weight"] = (1.0 + 0.1 * normal(DIM, dtype=torch.float32)).to(torch.bfloat16)
        s["out_weight"] = (normal(FEATURES, hv * DIM, dtype=torch.float32) * (hv * DIM) ** -0.5).to(torch.bfloat16)
        s["state"] = _state(gen, case["batch"], hv) if kind == "decode" or case["initial"] else None
    return s


def run(s):
    kind = s["kind"]
    if kind == "forward":
        return gdn_forward(*s["x"], s["initial_state"])
    if kind == "varlen":
        return gdn_forward_varlen(*s["x"], s["cu_seqlens"], s["initial_state"])
    if kind == "verify":
        q, k, v, g, beta = s["x"]
        out, delta = gdn_verify_step(q, k, v, g, beta, s["state"])
        state = gdn_commit_step(k, g, delta, s["counts"], s["state"])
        return out, delta, state
    if kind == "prefill":
        out, state = gdn_forward_projections(s["mixed"], s["a"], s["b"], s["a_log"], s["dt_bias"], s["hk"], s["hv"], s["state"])
        gated = rmsnorm_gated(out, s["z"], s["norm_weight"])
        return out, state, out_proj_gemm(gated.view(-1, s["hv"] * DIM), s["out_weight"])
    q, k, v, g, beta = gdn_prepare_inputs(s["mixed"], s["a"], s["b"], s["a_log"], s["dt_bias"], s["hk"], s["hv"])
    out = gdn_decode_step(q, k, v, g, beta, s["state"])
    gated = rmsnorm_gated(out, s["z"], s["norm_weight"])
    return out, s["state"], out_proj_gemm(gated.view(-1, s["hv"] * DIM), s["out_weight"])


def work(case):
    """Inputs once and outputs once; of the layer passes every entry point's own (their results are separate tensors)."""
    kind, hk, hv = case["kind"], case["hk"], case["hv"]
    n = case["tokens"] if kind == "varlen" else case["batch"] * case.get("width", case.get("tokens", 1))
    state = (case["sequences"] if kind == "varlen" else case["batch"]) * hv * DIM * DIM * 4
    qk, heads = n * hk * DIM * 2, n * hv * DIM * 2            # one BF16 tensor with key heads / value heads
    if kind in ("forward", "varlen"):
        moved = 2 * qk + 2 * heads + n * hv * ((4 if case["gate_fp32"] else 2) + 2) + state * (2 if case["initial"] else 1)
        return {"bytes": moved, "flops": 180224 * n * hv}       # eight dense contractions of the chunk form per token-head
    if kind == "verify":
        # state read by both steps and written by the second, deltas (FP32) written and read
        moved = 3 * qk + 2 * heads + 2 * (2 * heads) + n * hv * (2 * (4 if case["gate_fp32"] else 2) + 2) + 3 * state
        return {"bytes": moved, "flops": (7 + 2) * n * hv * DIM * DIM}
    gate = 3 * heads + n * FEATURES * 2 + heads + FEATURES * hv * DIM * 2       # rmsnorm_gated, then out_proj_gemm
    gemm = 2 * n * FEATURES * hv * DIM
    if kind == "prefill":
        moved = 2 * qk + heads + 2 * n * hv * 2 + heads + state * (2 if case["initial"] else 1)
        return {"bytes": moved + gate, "flops": 180224 * n * hv + gemm}
    moved = 2 * (2 * qk + heads) + n * hv * (4 + 6) + (2 * qk + 2 * heads + n * hv * 6) + 2 * state
    return {"bytes": moved + gate, "flops": 7 * n * hv * DIM * DIM + gemm}


def tolerance(case):
    """BF16 results: about 2e-3 from their own rounding and as much again from the BF16 operands behind them; the steps
    of one token at a time round nothing but their results."""
    if case["kind"] == "verify":
        return {"rel": 5e-3, "max": 0.02}
    return {"rel": 1e-2, "max": 0.1}
