"""The work that a user of this library has it do, as measurable cases.

Every case is one step (or one layer-by-layer pass) through the public interface `mugen_b200.mla.MlaContext`, repeated at
the same sequence lengths: a pass begins a step, runs its layers, ends it and rolls the sequences back to where they
stood, as the caller of a speculative step does (`rollback` is host bookkeeping).  `kind` names how the caller drives the
library:

  decode   step_begin, step_layers over the whole attention stack, step_end: one new token per sequence
  calls    the same step through the per-layer calls step_append and step_attend, as an engine calls them that runs its
           feed-forward part between the layers
  verify   a decode step of a few new tokens per sequence (the verify pass of speculative decoding)
  chunk    a step in which some sequences take a long prompt chunk, possibly next to plain decode rows of other sequences
  block    step_block for every layer: hidden states in, hidden states out (projections around the attention included);
           one new token per sequence, or a prompt
  range    one long sequence in the form used when its cache is cut by KV range: step_layer_partial and merge_partials
  host     step_layer_host for every layer: page-locked host buffers in and out

Shapes are the two that the benchmark and the tests use: 16 heads, hidden 2048, full q projection, 27 layers, fp16, and
128 heads, hidden 7168, q_lora_rank 1536, bf16 (fewer layers than a model has where one layer is large: every layer costs
the same), with 8 to 64 heads between them for heads that are split over GPUs.  Lengths reach from an empty cache to
131072 tokens.  Latent rows and queries have the distributions of `mugen_b200.synth`.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from mugen_b200 import synth
from mugen_b200.mla import MlaContext

ROW, QDIM, VDIM, RANK = 576, 192, 128, 512
ROPE = dict(rope_theta=10000.0, rope_scaling_factor=40.0, rope_original_ctx=4096, rms_norm_eps=1e-6)
CHUNK_MIN = 64      # new tokens from which a sequence counts as a prompt chunk below


def _case(kind, heads, dtype, layers, batch, ctx, *, ctx_min=0, new=1, chunks=0, chunk=0, chunk_start=0, rope=False,
          hidden=0, q_lora=0, **more):
    """batch sequences whose cached lengths are log-uniform in ctx_min..ctx (ctx_min = 0: all of them ctx), `new` tokens
    each, and `chunks` further sequences that take `chunk` tokens each on top of chunk_start cached ones."""
    return dict(kind=kind, heads=heads, dtype=dtype, layers=layers, batch=batch, ctx=ctx, ctx_min=ctx_min, new=new,
                chunks=chunks, chunk=chunk, chunk_start=chunk_start, rope=rope, hidden=hidden, q_lora=q_lora, **more)


def listed():
    return [
        # one chat user on a small model, short context: launches and latency are everything
        _case("decode", 16, "f16", 27, 1, 2047, name="decode_16h_one_user"),
        # the same model serving a batch: the benchmark's 27-layer workload
        _case("decode", 16, "f16", 27, 32, 8191, name="decode_16h_batch32"),
        # the large model serving a full batch: the benchmark's headline step, four of its layers
        _case("decode", 128, "bf16", 4, 64, 16383, name="decode_128h_batch64"),
        # a serving batch as it comes: contexts of every length at once
        _case("decode", 128, "bf16", 3, 128, 32767, ctx_min=256, name="decode_128h_ragged128"),
        # one GPU's share of that batch when it is spread over eight, driven layer by layer, q rotated by the library
        _case("calls", 128, "bf16", 8, 8, 16383, rope=True, name="calls_128h_batch8"),
        # speculative decoding on the small model: five positions per sequence to verify
        _case("verify", 16, "f16", 27, 16, 4096, ctx_min=1000, new=5, rope=True, name="verify_16h_batch16"),
        # whole attention blocks of the small model for a few users
        _case("block", 16, "f16", 27, 4, 3000, ctx_min=300, rope=True, hidden=2048, name="block_16h_batch4"),
        # whole attention blocks of the large model for a batch
        _case("block", 128, "bf16", 3, 32, 4095, ctx_min=512, rope=True, hidden=7168, q_lora=1536, name="block_128h_batch32"),
        # a prompt of ordinary, odd length entering the small model
        _case("block", 16, "f16", 27, 0, 0, chunks=1, chunk=777, rope=True, hidden=2048, name="prompt_16h_777"),
        # long prompts in chunks next to the decode rows of a running batch on the large model
        _case("chunk", 128, "bf16", 1, 32, 16000, ctx_min=256, chunks=2, chunk=4096, chunk_start=8192, name="chunk_128h_4096"),
        # one very long context
        _case("range", 128, "bf16", 4, 1, 131071, name="range_128h_131072"),
        # an engine that keeps its activations on the host; the heads of the large model split over two GPUs
        _case("host", 64, "bf16", 8, 16, 4095, ctx_min=700, name="host_64h_batch16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """Another case of the same ranges."""
    while True:
        kind = rng.choice(["decode", "decode", "calls", "verify", "block", "prompt", "chunk", "range", "host"])
        heads = rng.choice([16, 16, 128, 128, 64, 32, rng.randint(5, 100)])
        dtype = rng.choice(["f16", "bf16"])
        layers = rng.randint(8, 27) if heads <= 32 else rng.randint(2, 8)
        batch, ctx, rope = _log_int(rng, 1, 128), _log_int(rng, 64, 32768), rng.random() < 0.5
        ctx_min = rng.choice([0, max(1, ctx // rng.randint(2, 64))])
        hidden, q_lora = rng.choice([(2048, 0), (2048, 0), (4096, 512), (7168, 1536)])
        if kind in ("decode", "calls", "host"):
            c = _case(kind, heads, dtype, layers, batch, ctx, ctx_min=ctx_min, rope=rope)
        elif kind == "verify":
            c = _case(kind, heads, dtype, layers, max(1, batch // 2), ctx, ctx_min=ctx_min, new=rng.randint(2, 8), rope=rope)
        elif kind == "block":
            c = _case("block", heads, dtype, layers, batch, ctx, ctx_min=ctx_min, rope=True, hidden=hidden, q_lora=q_lora)
        elif kind == "prompt":
            c = _case("block", heads, dtype, layers, 0, 0, chunks=rng.choice([1, 1, 2]), chunk=_log_int(rng, 64, 4096),
                      chunk_start=rng.choice([0, 0, _log_int(rng, 64, 8192)]), rope=True, hidden=hidden, q_lora=q_lora)
        elif kind == "chunk":
            c = _case(kind, heads, dtype, max(1, layers // 4), batch, min(ctx, 16384), ctx_min=min(ctx_min, 16384),
                      chunks=rng.randint(1, 4), chunk=_log_int(rng, 64, 4096), chunk_start=rng.choice([0, _log_int(rng, 64, 8192)]),
                      rope=rope)
        else:
            c = _case(kind, heads, dtype, layers, 1, _log_int(rng, 8192, 131072))
        w = work(c)
        # within what the largest listed cases do and hold; weights are made on the host, which bounds their size
        weights = c["layers"] * (c["heads"] * 131072 + (_block_values(c) if c["kind"] == "block" else 0))
        if w["bytes"] <= 5e9 and w["flops"] <= 5e12 and _cache_bytes(c) <= 5e9 and weights <= 6e8:
            return c


def _lengths(case):
    """(cached tokens, new tokens) of every sequence: the batch first, then the chunks."""
    rng = random.Random(case["batch"] * 1000003 + case["ctx"])
    lo, hi = case["ctx_min"], case["ctx"]
    cached = [_log_int(rng, lo, hi) if lo else hi for _ in range(case["batch"])]
    return (cached + [case["chunk_start"]] * case["chunks"], [case["new"]] * case["batch"] + [case["chunk"]] * case["chunks"])


def _cache_bytes(case):
    cached, new = _lengths(case)
    return case["layers"] * sum(a + b + 64 for a, b in zip(cached, new)) * ROW * 2


def _block_values(case):
    """Values in the projection weights of one layer."""
    h, e, r = case["heads"], case["hidden"], case["q_lora"]
    return 576 * e + e * h * VDIM + ((r * e + h * QDIM * r) if r else h * QDIM * e)


def prepare(case, seed):
    H, L = case["heads"], case["layers"]
    dt, tdt = (synth.DT_F16, torch.float16) if case["dtype"] == "f16" else (synth.DT_BF16, torch.bfloat16)
    cached, new = _lengths(case)
    rows = sum(new)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def randn(shape, scale=1.0):
        return (torch.randn(shape, device="cuda", generator=gen) * scale).to(tdt)

    def host_bits(t):
        return t.view(torch.int16).cpu().numpy().view(np.uint16)

    top = max(a + b for a, b in zip(cached, new))
    ctx = MlaContext(n_layers=L, n_heads=H, dtype=dt, n_pages=sum((a + b + 63) // 64 + 1 for a, b in zip(cached, new)) + 8,
                     max_seqs=len(cached), max_seq_len=top + 64, max_rows=rows, **ROPE)
    ctx.shuffle_free_pages(seed)
    w_type = synth.W_F16 if dt == synth.DT_F16 else synth.W_BF16
    w_uk, w_uv = (host_bits(randn((H * 128, RANK), 0.02)) for _ in range(2))
    norm = host_bits(1.0 + randn((RANK,), 0.1))
    for layer in range(L):
        ctx.set_layer_weights(layer, w_uk, w_uv, w_type, norm)
    if case["kind"] == "block":
        e, r = case["hidden"], case["q_lora"]
        w = dict(attn_norm=1.0 + randn((e,), 0.1), kv_a_mqa=randn((576, e), e ** -0.5), wo=randn((e, H * VDIM), (H * VDIM) ** -0.5))
        if r:
            w.update(q_a=randn((r, e), e ** -0.5), q_a_norm=1.0 + randn((r,), 0.1), q_b=randn((H * QDIM, r), r ** -0.5))
        else:
            w.update(q=randn((H * QDIM, e), e ** -0.5))
        w = {k: host_bits(v) for k, v in w.items()}
        for layer in range(L):
            ctx.set_block_weights(layer, **w)
    ctx.set_q_rope(case["rope"])
    seqs = [ctx.seq_create() for _ in cached]
    for layer in range(L):                      # every sequence holds its own window of the layer's rows
        pool = randn((max(cached) + 7 * len(cached) + 1, ROW)).view(torch.int16)
        for i, (s, n) in enumerate(zip(seqs, cached)):
            if n:
                ctx.write_rows(layer, s, 0, pool[7 * i:7 * i + n])
    for s, n in zip(seqs, cached):
        ctx.advance_seq_len(s, n)
    state = dict(kind=case["kind"], layers=L, ctx=ctx, seqs=seqs, cached=cached, new=None if max(new) == 1 else new)
    if case["kind"] == "block":
        state["input"] = randn((rows, case["hidden"]))
        state["hidden"] = torch.empty_like(state["input"])
    else:
        state["q"] = randn((L, rows, H, QDIM), 0.9)
        state["kv"] = randn((L, rows, ROW))
        state["out"] = torch.zeros((L, rows, H, VDIM), device="cuda", dtype=tdt)
    if case["kind"] == "range":
        state["partial"] = torch.zeros((1, rows, H, RANK + 2), device="cuda")
    if case["kind"] == "host":
        for k in ("q", "kv", "out"):
            state[k] = state[k].cpu().pin_memory()
    assert ctx.status() == 0
    return state


def run(state):
    ctx, seqs, layers, kind = state["ctx"], state["seqs"], state["layers"], state["kind"]
    ctx.step_begin(seqs, state["new"])
    if kind == "block":
        result = state["hidden"]
        result.copy_(state["input"])            # the embedded tokens of the step
        for layer in range(layers):
            ctx.step_block(layer, result)
    else:
        q, kv, result = state["q"], state["kv"], state["out"]
        if kind == "calls":
            for layer in range(layers):
                ctx.step_append(layer, kv[layer])
                ctx.step_attend(layer, q[layer], result[layer])
        elif kind == "range":
            partial = state["partial"]
            for layer in range(layers):
                ctx.step_layer_partial(layer, kv[layer], q[layer], partial[0])
                ctx.merge_partials(layer, 1, partial.shape[1], partial, result[layer])
        elif kind == "host":
            for layer in range(layers):
                ctx.step_layer_host(layer, kv[layer], q[layer], result[layer])
        else:
            ctx.step_layers(0, layers, kv, q, result)
    ctx.step_end()
    ctx.rollback(seqs, state["cached"])
    return result


def work(case):
    """What a pass cannot do without: the latent rows that its queries see once per layer, the new rows, the weights, what
    goes in and what comes out; absorbed attention for single rows, expanded keys and values for prompt chunks where that
    takes fewer operations."""
    H, L = case["heads"], case["layers"]
    cached, new = _lengths(case)
    rows, bts, flops = sum(new), 0.0, 0.0
    for a, n in zip(cached, new):
        pairs = n * a + n * (n + 1) / 2
        absorbed = pairs * H * 2.0 * (576 + 512) + n * H * 2.0 * 2 * 128 * 512
        expanded = pairs * H * 2.0 * (192 + 128) + (a + n) * H * 2.0 * 512 * 256
        flops += min(absorbed, expanded) if n >= CHUNK_MIN else absorbed
        bts += (a + n) * ROW * 2.0
    bts += 2.0 * H * 128 * RANK * 2                                     # W_UK, W_UV
    if case["kind"] == "block":
        flops += 2.0 * rows * _block_values(case)
        bts += 2.0 * _block_values(case)
        io = 2.0 * rows * case["hidden"] * 2                            # hidden states cross once for the whole stack
    else:
        bts += rows * (ROW + H * (QDIM + VDIM)) * 2.0
        io = 0.0
    return {"bytes": bts * L + io, "flops": flops * L}


def tolerance(case):
    """Probabilities, absorbed queries and outputs are rounded to the storage type (11 or 8 significant bits) and sums may
    be cut in other places."""
    return {"rel": 4e-3} if case["dtype"] == "f16" else {"rel": 1.2e-2}
