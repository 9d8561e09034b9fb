"""What a user of this package has it do, as cases that can be timed: decode steps of a server, prompts that are read in,
training steps.  Every case goes through the public entry points (`fused_recurrent_kda_fwd`, `chunk_kda` and its autograd).

A case is a dict:
  kind         "decode" (states updated in place), "prefill" (forward only) or "train" (forward and backward)
  seqs, tokens sequences and tokens per sequence; with `packed` the sequences are of uneven length, from `shortest` to
               `tokens`, concatenated in one row with cu_seqlens (`lengths` picks which)
  heads, value_heads, dim   q/k heads, value heads, K = V
  dtype        of q, k, v
  layer        the call that the attention layer makes: raw gate (with A_log and dt_bias), beta logits and unnormalised q, k, all
               activated inside the operator; otherwise log-decays, betas and normalised q, k are handed over
  bounded      the layer's gate is bounded from below (lower_bound = -5, safe_gate)
  slots        decode: states live in a pool that is larger than the batch, and a slot table says where
  states       initial states are given and final states are wanted
"""
from __future__ import annotations

import math
import random

import torch

from kda_b200 import chunk_kda, fused_recurrent_kda_fwd
from kda_b200.inputs import flops_per_token_head

_DEFAULTS = dict(seqs=1, tokens=1, packed=False, shortest=1, lengths=0, heads=32, value_heads=32, dim=128, dtype="bf16", layer=False,
                 bounded=False, slots=False, states=True)


def _case(**kw) -> dict:
    return {**_DEFAULTS, **kw}


def listed() -> list[dict]:
    return [
        # one conversation: every generated token is one such call per layer, so its latency is what the user waits for
        _case(name="decode_1", kind="decode", layer=True),
        # a server with some dozens of running requests, states in a pool
        _case(name="decode_48_slots", kind="decode", seqs=48, layer=True, slots=True),
        # draft tokens being checked: four tokens a request, each token's state kept in a slot of its own
        _case(name="decode_24_draft_4", kind="decode", seqs=24, tokens=4, layer=True, slots=True),
        # the stated decode workload: 1,024 sequences, states from end to end
        _case(name="decode_1024", kind="decode", seqs=1024),
        # a short prompt: time to the first token
        _case(name="prefill_1x333", kind="prefill", tokens=333, layer=True),
        # a server's batch of prompts of all lengths, with grouped value heads
        _case(name="prefill_packed_12", kind="prefill", seqs=12, tokens=2500, shortest=40, packed=True, lengths=1, heads=8, layer=True),
        # the stated prefill workload
        _case(name="prefill_4x4096", kind="prefill", seqs=4, tokens=4096),
        # one long document, bounded gates
        _case(name="prefill_1x32768_bounded", kind="prefill", tokens=32768, layer=True, bounded=True),
        # a small model with heads of 64 and rows that are no multiple of anything
        _case(name="train_2x1000_d64", kind="train", seqs=2, tokens=1000, heads=8, value_heads=8, dim=64, states=False),
        # the stated training workload
        _case(name="train_8x8192", kind="train", seqs=8, tokens=8192),
        # pretraining on packed documents, the way the layer calls the operator
        _case(name="train_packed_8", kind="train", seqs=8, tokens=16384, shortest=128, packed=True, lengths=3, layer=True, states=False),
        # float32 training: parity runs and gradient checks
        _case(name="train_fp32_8x2048", kind="train", seqs=8, tokens=2048, dtype="fp32"),
    ]


_MOST = 8 * 8192 * 32        # (token, value head) pairs of the largest training case
_MOST_FP32 = 8 * 2048 * 32


def _log_int(rng: random.Random, low: int, high: int) -> int:
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["decode", "prefill", "train"])
    if kind == "decode":
        draft = rng.random() < 0.25
        heads = rng.choice([16, 32])
        return _case(kind=kind, seqs=_log_int(rng, 1, 128 if draft else 1024), tokens=rng.randint(2, 6) if draft else 1, heads=heads,
                     value_heads=heads, layer=rng.random() < 0.75, slots=draft or rng.random() < 0.5)
    fp32 = kind == "train" and rng.random() < 0.25
    heads = rng.choice([8, 16, 32])
    grouped = kind == "prefill" and heads < 32 and rng.random() < 0.5
    value_heads = 32 if grouped else heads
    most = (_MOST_FP32 if fp32 else _MOST) // value_heads
    packed = not fp32 and rng.random() < 0.4
    layer = not fp32 and rng.random() < 0.6
    c = dict(kind=kind, heads=heads, value_heads=value_heads, dtype="fp32" if fp32 else "bf16", layer=layer,
             bounded=layer and rng.random() < 0.3, dim=64 if rng.random() < 0.2 else 128, states=kind == "prefill" or rng.random() < 0.5)
    if packed:
        c.update(packed=True, seqs=_log_int(rng, 2, 32), lengths=rng.randrange(1 << 20), shortest=16 if kind == "prefill" else 128)
        c["tokens"] = max(2 * c["shortest"], min(_log_int(rng, 300, 16384), most // c["seqs"]))
    else:
        c["seqs"] = _log_int(rng, 1, 8)
        low, high = (16, 32768) if kind == "prefill" else (128, 2048 if fp32 else 8192)
        c["tokens"] = max(low, min(_log_int(rng, low, high), most // c["seqs"]))
    return _case(**c)


def _lengths(case: dict) -> list[int]:
    if not case["packed"]:
        return [case["tokens"]] * case["seqs"]
    rng = random.Random(case["lengths"])
    return [rng.randint(case["shortest"], case["tokens"]) for _ in range(case["seqs"])]


def prepare(case: dict, seed: int) -> dict:
    """Values as in `kda_b200/inputs.py`: q, k of unit norm (raw normal values for the layer's call), v normal, beta a sigmoid,
    g = -exp(a) softplus(x) with a = log U(1, 16) per head, states of standard deviation 0.02."""
    H, HV, D = case["heads"], case["value_heads"], case["dim"]
    dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")      # noqa: E731
    lengths = _lengths(case)
    N, total = len(lengths), sum(lengths)
    B, T = (1, total) if case["packed"] else (N, case["tokens"])
    unit = lambda x: x if case["layer"] else x / x.norm(dim=-1, keepdim=True)    # noqa: E731
    x = dict(q=unit(rn(B, T, H, D)).to(dt), k=unit(rn(B, T, H, D)).to(dt), v=rn(B, T, HV, D).to(dt))
    a_log = torch.log(1.0 + 15.0 * torch.rand(HV, generator=gen, device="cuda"))
    options = {}
    if case["layer"]:
        x["g"], x["beta"] = rn(B, T, HV, D).to(dt), rn(B, T, HV).to(dt)
        x["A_log"], x["dt_bias"] = a_log, rn(HV * D)
        options.update(use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True)
        if case["bounded"]:
            options.update(lower_bound=-5.0)
            if case["kind"] != "decode":
                options.update(safe_gate=True)
    else:
        x["g"] = -torch.exp(a_log).view(1, 1, HV, 1) * torch.nn.functional.softplus(rn(B, T, HV, D))
        x["beta"] = torch.sigmoid(rn(B, T, HV))
    if case["kind"] == "decode":
        pool = N * T + N if case["slots"] else N           # a slot for every token, and room for more requests
        x["initial_state"] = rn(pool, HV, D, D) * 0.02
        if case["slots"]:
            slots = torch.randperm(pool, generator=gen, device="cuda")[:N * T].to(torch.int32)
            x["ssm_state_indices"] = slots if T == 1 else slots.view(N, T)
            if T > 1:
                x["num_accepted_tokens"] = torch.randint(1, T + 1, (N,), generator=gen, device="cuda").to(torch.int32)
        return dict(kind="decode", args=x, options=options)
    if case["packed"]:
        ends = [0]
        for n in lengths:
            ends.append(ends[-1] + n)
        options["cu_seqlens"] = torch.tensor(ends, dtype=torch.int32, device="cuda")
    if case["states"]:
        x["initial_state"] = rn(N, HV, D, D) * 0.02
        options["output_final_state"] = True
    state = dict(kind=case["kind"], args=x, options=options)
    if case["kind"] == "train":
        for t in x.values():
            t.requires_grad_(True)
        state["up"] = [rn(B, T, HV, D).to(dt)] + ([rn(N, HV, D, D) * 0.01] if case["states"] else [])
    return state


def run(state: dict):
    args, options = state["args"], state["options"]
    if state["kind"] == "decode":
        o, pool = fused_recurrent_kda_fwd(**args, **options)
        return dict(o=o, states=pool)
    if state["kind"] == "prefill":
        with torch.inference_mode():
            o, ht = chunk_kda(**args, **options)
        return dict(o=o, states=ht)
    o, ht = chunk_kda(**args, **options)
    up = state["up"]
    grads = torch.autograd.grad([o, ht][:len(up)], list(args.values()), up)
    return dict(o=o, states=ht, **{"d_" + n: g for n, g in zip(args, grads)})


def work(case: dict) -> dict:
    HV, D = case["value_heads"], case["dim"]
    lengths = _lengths(case)
    N, tokens = len(lengths), sum(lengths)
    qkv_el = 2 if case["dtype"] == "bf16" else 4
    gate_el = qkv_el if case["layer"] else 4
    qk, vo = 2 * tokens * case["heads"] * D * qkv_el, tokens * HV * D * qkv_el
    gb = tokens * HV * (D + 1) * gate_el
    state = N * HV * D * D * 4
    flops = tokens * HV * flops_per_token_head(D, D, backward=case["kind"] == "train")
    if case["kind"] == "decode":
        # one state read per sequence, one written per token where each has its slot
        return dict(bytes=qk + 2 * vo + gb + state * (1 + (case["tokens"] if case["slots"] else 1)), flops=7 * tokens * HV * D * D)
    once = qk + 2 * vo + gb + (2 * state if case["states"] else 0)      # inputs and o (and, going back, the gradients and do)
    return dict(bytes=once * (2 if case["kind"] == "train" else 1), flops=flops)


def tolerance(case: dict):
    if case["dtype"] == "fp32":
        return {"rel": 3e-5}         # sums of fp32 products over thousands of dependent steps, decays of accumulated exponents
    if case["kind"] == "decode":
        return {"rel": 4e-3}         # o rounded once to bf16; the states are fp32
    if case["kind"] == "train" and case["layer"]:
        return {"rel": 2e-2}         # gradients of A_log and dt_bias: sums over all tokens of gate gradients that carry bf16 noise
    return {"rel": 1e-2}             # bf16 operands of the chunk products
