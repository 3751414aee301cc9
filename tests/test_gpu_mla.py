"""Parity of the CUDA path (through the C ABI) with the CPU checker.

Bars: the append is bit-exact; attention outputs stay within max-abs 2e-2 and relative-L2 5e-3
of the CPU result on the same seeded inputs (the tolerance the task states for fp16/bf16
caches).  Every test runs once per attention kernel family the library offers.
"""
import base64
import os
import time

import numpy as np
import pytest

from mugen_b200 import capi, synth

pytestmark = pytest.mark.gpu

MAX_ABS, REL_L2 = 2e-2, 5e-3
YARN = dict(rope_theta=10000.0, rope_scaling_factor=40.0, rope_original_ctx=4096, rms_norm_eps=1e-6)

KERNELS = [capi.KERNEL_MMA, capi.KERNEL_TCGEN05, capi.KERNEL_TCGEN05_PAIR128, capi.KERNEL_TCGEN05_T16]
if os.environ.get("MLA_TEST_KERNELS"):
    KERNELS = [int(k) for k in os.environ["MLA_TEST_KERNELS"].split(",")]


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return torch


def _dev(torch, bits: np.ndarray):
    return torch.from_numpy(np.ascontiguousarray(bits).view(np.int16)).cuda()


def _host(t) -> np.ndarray:
    return t.cpu().numpy().view(np.uint16)


def make_ctx(case: synth.LayerCase, kernel, n_layers=1, extra_pages=8, max_rows=0, shuffle=None, **kw):
    from mugen_b200.mla import MlaContext
    pages = sum((s + 63) // 64 + 1 for s in case.seq_lens) + extra_pages
    args = dict(n_layers=n_layers, n_heads=case.n_heads, dtype=case.dt, n_pages=pages,
                max_seqs=max(len(case.seq_lens), 1) + 2, max_seq_len=max(case.seq_lens + [64]) + 256,
                max_rows=max_rows, kernel=kernel, **YARN)
    args.update(kw)
    ctx = MlaContext(**args)
    if shuffle is not None:
        ctx.shuffle_free_pages(shuffle)
    for layer in range(n_layers):
        ctx.set_layer_weights(layer, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    return ctx


def fill(torch, ctx, case, layer=0, upto=None):
    seqs = []
    for b, cache in enumerate(case.caches):
        s = ctx.seq_create()
        n = case.seq_lens[b] if upto is None else upto[b]
        if n:
            ctx.write_rows(layer, s, 0, _dev(torch, cache[:n]))
        ctx.advance_seq_len(s, n)
        seqs.append(s)
    return seqs


def check_close(got_bits, want_bits, dt, what=""):
    mx, rl = synth.error_norms(got_bits, want_bits, dt, dt)
    assert mx <= MAX_ABS and rl <= REL_L2, f"{what}: max-abs {mx:.3e}, rel-L2 {rl:.3e}"
    return mx, rl


def oracle_out(oracle, case, b, seq_len=None, q=None):
    n = case.seq_lens[b] if seq_len is None else seq_len
    return oracle.attention(case.q[b] if q is None else q, case.caches[b], n, case.w_uk, case.w_uv,
                            case.w_type, case.n_heads, case.dt)


# ---------------------------------------------------------------------------------------------
# append: bit-exact
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dt", [synth.DT_F16, synth.DT_BF16])
@pytest.mark.parametrize("factor,ctx_len", [(40.0, 4096), (0.0, 0)])
def test_append_bit_exact(torch, oracle, dt, factor, ctx_len):
    positions = [0, 1, 31, 32, 63, 64, 65, 127, 128, 1000, 4095, 4096, 8191, 20000, 40000]
    case = synth.make_layer_case(11, 4, [1] * len(positions), dt)
    kw = dict(YARN, rope_scaling_factor=factor, rope_original_ctx=ctx_len)
    from mugen_b200.mla import MlaContext
    ctx = MlaContext(n_layers=2, n_heads=4, dtype=dt, n_pages=640, max_seqs=4,
                     max_seq_len=40064, max_rows=len(positions), kernel=capi.KERNEL_MMA, **kw)
    for layer in range(2):
        ctx.set_layer_weights(layer, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    s = ctx.seq_create()
    ctx.append_rows(1, [s] * len(positions), positions, _dev(torch, case.kv_a))
    want = oracle.append_rows(case.kv_a, positions, case.norm_w, kw["rms_norm_eps"], factor, ctx_len,
                              kw["rope_theta"], dt)
    for i, p in enumerate(positions):
        got = ctx.read_rows(1, s, p, 1)[0]
        assert np.array_equal(got, want[i]), f"position {p}"
    # the other layer's slots were not touched
    assert not ctx.read_rows(0, s, 0, 64).any()
    assert ctx.status() == 0
    ctx.close()


def test_append_reproduces_the_rows_of_the_reference_forward(torch, golden):
    """Golden rows written by the reference's own inline append (RMSNorm + NeoX/YaRN RoPE + scatter inside
    forward(), transformer.cpp:3930-3987, run on a tiny deepseek2 GGUF file): the append kernel, fed the kv_a the
    reference's code read, must store the very bits the reference stored."""
    import base64
    from mugen_b200.mla import MlaContext
    unb = lambda t: np.frombuffer(base64.b64decode(t), np.uint16).copy()
    groups = {}
    for c in golden["append"]:
        groups.setdefault((c["model"], c["layer"]), []).append(c)
    assert len(groups) >= 4
    dummy_w = np.zeros((128, 512), np.uint16)
    for (model, layer), entries in groups.items():
        c0 = entries[0]
        assert c0["source"].startswith("reference forward()") and c0["dt"] == synth.DT_F16
        top = max(c["position"] for c in entries)
        ctx = MlaContext(n_layers=1, n_heads=1, dtype=synth.DT_F16, n_pages=len(entries) + 1, max_seqs=1,
                         max_seq_len=64, max_position=top + 1, max_rows=len(entries), kernel=capi.KERNEL_MMA, rope_theta=c0["theta"],
                         rope_scaling_factor=c0["factor"], rope_original_ctx=c0["orig_ctx"], rms_norm_eps=c0["eps"])
        ctx.set_layer_weights(0, dummy_w, dummy_w, synth.W_F16, unb(c0["norm_w"]))
        # one sequence per entry would need a page table per position; instead place each row at its position
        # modulo the page size (the rotation uses the true position through a base offset)
        for c in entries:
            s = ctx.seq_create()
            ctx.seq_set_base(s, c["position"] - c["position"] % 64)
            ctx.append_rows(0, [s], [c["position"]], _dev(torch, unb(c["kv_a"])[None]))
            got = ctx.read_rows(0, s, c["position"] % 64, 1)[0]
            assert np.array_equal(got, unb(c["row"])), (model, layer, c["position"])
            ctx.seq_free(s)
        assert ctx.status() == 0
        ctx.close()


def test_append_many_rows_bit_exact(torch, oracle):
    """A 300-row chunk appended in one call (the batched twin, transformer.cpp:1263-1323)."""
    n = 300
    case = synth.make_layer_case(12, 2, [1] * n, synth.DT_F16)
    from mugen_b200.mla import MlaContext
    ctx = MlaContext(n_layers=1, n_heads=2, dtype=synth.DT_F16, n_pages=8, max_seqs=2, max_seq_len=512,
                     max_rows=n, kernel=capi.KERNEL_MMA, **YARN)
    ctx.set_layer_weights(0, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    s = ctx.seq_create()
    pos = list(range(7, 7 + n))
    ctx.append_rows(0, [s] * n, pos, _dev(torch, case.kv_a))
    want = oracle.append_rows(case.kv_a, pos, case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0,
                              synth.DT_F16)
    assert np.array_equal(ctx.read_rows(0, s, 7, n), want)
    ctx.close()


# ---------------------------------------------------------------------------------------------
# attention vs the CPU checker
# ---------------------------------------------------------------------------------------------
ATTN_CASES = [
    # heads, seq_lens, dtype, w_type, q_scale
    (16, [1], synth.DT_F16, synth.W_F16, 1.0),
    (16, [63, 64, 65], synth.DT_F16, synth.W_F16, 1.0),
    (16, [2048], synth.DT_F16, synth.W_F16, 1.0),            # configs[0] shape
    (16, [700, 33, 1500, 256], synth.DT_BF16, synth.W_BF16, 1.0),
    (128, [513, 100], synth.DT_BF16, synth.W_BF16, 1.0),      # V3 head count
    (128, [300], synth.DT_F16, synth.W_F16, 6.0),             # peaky softmax: rescaling exercised
    (64, [1000, 31], synth.DT_BF16, synth.W_BF16, 8.0),
    (5, [129, 1], synth.DT_F16, synth.W_F16, 1.0),            # head count not a tile multiple
    (16, [384], synth.DT_F16, synth.W_Q8_0, 1.0),
    (16, [384], synth.DT_F16, synth.W_Q4_0, 1.0),
]


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("n_heads,seq_lens,dt,w_type,q_scale", ATTN_CASES)
def test_attend_matches_cpu(torch, oracle, kernel, n_heads, seq_lens, dt, w_type, q_scale):
    case = synth.make_layer_case(500 + n_heads + sum(seq_lens), n_heads, seq_lens, dt, w_type, q_scale)
    ctx = make_ctx(case, kernel, shuffle=3)
    seqs = fill(torch, ctx, case)
    out = torch.zeros((len(seq_lens), n_heads, 128), dtype=torch.int16, device="cuda")
    ctx.attend_rows(0, seqs, seq_lens, _dev(torch, case.q), out)
    got = _host(out)
    assert ctx.status() == 0
    for b in range(len(seq_lens)):
        check_close(got[b], oracle_out(oracle, case, b), dt, f"seq {b} len {seq_lens[b]}")
    ctx.close()


@pytest.mark.parametrize("kernel", KERNELS)
def test_golden_reference_outputs(torch, golden, kernel):
    """Against fixtures produced by the reference's own cpu_mla_attention."""
    for c in golden["attention"]:
        case = synth.make_layer_case(c["seed"], c["n_heads"], [c["seq_len"]], synth.DT_F16, c["w_type"],
                                     c["q_scale"], c["exact_in_both"])
        assert case.digest() == c["inputs_sha256"]
        ctx = make_ctx(case, kernel)
        seqs = fill(torch, ctx, case)
        out = torch.zeros((1, c["n_heads"], 128), dtype=torch.int16, device="cuda")
        ctx.attend_rows(0, seqs, [c["seq_len"]], _dev(torch, case.q), out)
        want = np.frombuffer(base64.b64decode(c["out_f16"]), np.uint16).reshape(c["n_heads"], 128)
        check_close(_host(out)[0], want, synth.DT_F16, f"golden seed {c['seed']}")
        ctx.close()


@pytest.mark.parametrize("kernel", KERNELS)
def test_bf16_cache_against_f16_reference_values(torch, oracle, kernel):
    """bf16 context on numbers exact in both formats, checked against the f16 CPU result."""
    c16 = synth.make_layer_case(77, 32, [900], synth.DT_F16, synth.W_F16, 1.0, True)
    want = oracle_out(oracle, c16, 0)
    tobf = lambda b: synth.to_bits(synth.from_bits(b, synth.DT_F16), synth.DT_BF16)
    cbf = synth.LayerCase(32, synth.DT_BF16, synth.W_BF16, [900], tobf(c16.q), [tobf(c16.caches[0])],
                          tobf(c16.w_uk), tobf(c16.w_uv), c16.w_uk_f32, c16.w_uv_f32, tobf(c16.norm_w),
                          tobf(c16.kv_a))
    ctx = make_ctx(cbf, kernel)
    seqs = fill(torch, ctx, cbf)
    out = torch.zeros((1, 32, 128), dtype=torch.int16, device="cuda")
    ctx.attend_rows(0, seqs, [900], _dev(torch, cbf.q), out)
    mx, rl = synth.error_norms(_host(out)[0], want, synth.DT_BF16, synth.DT_F16)
    assert mx <= MAX_ABS and rl <= REL_L2, (mx, rl)
    ctx.close()


@pytest.mark.parametrize("kernel", KERNELS)
def test_attend_shorter_than_cache_and_empty(torch, oracle, kernel):
    """attend_len is the caller's (cpu_mla_attention's seq_len argument), not the cache length;
    a zero-length row yields zeros."""
    case = synth.make_layer_case(91, 16, [500, 200], synth.DT_F16)
    ctx = make_ctx(case, kernel)
    seqs = fill(torch, ctx, case)
    lens = [131, 0]
    out = torch.full((2, 16, 128), 7, dtype=torch.int16, device="cuda")
    ctx.attend_rows(0, seqs, lens, _dev(torch, case.q), out)
    got = _host(out)
    check_close(got[0], oracle_out(oracle, case, 0, 131), synth.DT_F16)
    assert not got[1].any()
    ctx.close()


# ---------------------------------------------------------------------------------------------
# the decode-step scheduler
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("dt", [synth.DT_F16, synth.DT_BF16])
def test_decode_steps_multi_layer(torch, oracle, kernel, dt):
    """3 decode steps over 2 layers and 3 ragged sequences: append-then-attend ordering,
    counters moving once per step, truncate rollback and re-append (speculative-decode contract)."""
    H, L = 16, 2
    lens0 = [130, 64, 5]
    cases = [synth.make_layer_case(300 + l, H, [n + 8 for n in lens0], dt) for l in range(L)]
    from mugen_b200.mla import MlaContext
    ctx = MlaContext(n_layers=L, n_heads=H, dtype=dt, n_pages=16, max_seqs=4, max_seq_len=512,
                     kernel=kernel, **YARN)
    ctx.shuffle_free_pages(9)
    host = [[None] * 3 for _ in range(L)]   # the CPU-side mirror of each (layer, seq) cache
    seqs = [ctx.seq_create() for _ in lens0]
    for l in range(L):
        ctx.set_layer_weights(l, cases[l].w_uk, cases[l].w_uv, cases[l].w_type, cases[l].norm_w)
        for b, s in enumerate(seqs):
            host[l][b] = cases[l].caches[b].copy()
            ctx.write_rows(l, s, 0, _dev(torch, host[l][b][:lens0[b]]))
    for b, s in enumerate(seqs):
        ctx.advance_seq_len(s, lens0[b])
    rng = np.random.default_rng(5)

    def one_step(expect_len):
        ctx.step_begin(seqs)
        for l in range(L):
            kv_a = synth.to_bits(rng.standard_normal((3, 576), np.float32), dt)
            q = synth.to_bits(rng.standard_normal((3, H, 192), np.float32) * np.float32(0.9), dt)
            out = torch.zeros((3, H, 128), dtype=torch.int16, device="cuda")
            ctx.step_append(l, _dev(torch, kv_a))
            ctx.step_attend(l, _dev(torch, q), out)
            got = _host(out)
            pos = [expect_len[b] for b in range(3)]
            rows = oracle.append_rows(kv_a, pos, cases[l].norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
            for b in range(3):
                host[l][b][pos[b]] = rows[b]
                assert np.array_equal(ctx.read_rows(l, seqs[b], pos[b], 1)[0], rows[b])
                want = oracle.attention(q[b], host[l][b], pos[b] + 1, cases[l].w_uk, cases[l].w_uv,
                                        cases[l].w_type, H, dt)
                check_close(got[b], want, dt, f"layer {l} seq {b}")
            # counters do not move inside the step
            assert [ctx.seq_len(s) for s in seqs] == expect_len
        ctx.step_end()
        return [n + 1 for n in expect_len]

    cur = list(lens0)
    cur = one_step(cur)
    cur = one_step(cur)
    assert [ctx.seq_len(s) for s in seqs] == [n + 2 for n in lens0]
    # roll back one token on sequence 0 (rejected draft), then continue: the row is rewritten
    ctx.truncate(seqs[0], cur[0] - 1)
    cur[0] -= 1
    cur = one_step(cur)
    assert ctx.status() == 0
    ctx.close()


@pytest.mark.parametrize("kernel", KERNELS)
def test_step_layers_equals_per_layer_calls(torch, kernel):
    """The multi-layer call runs the append inside the absorb launch (same arithmetic, other blocks):
    outputs and appended rows are bit-identical to the per-layer calls with their separate append kernel."""
    H, L, dt, lens = 64, 3, synth.DT_BF16, [200, 65]
    case = synth.make_layer_case(333, H, [n + 1 for n in lens], dt)
    rng = np.random.default_rng(4)
    kv = _dev(torch, synth.to_bits(rng.standard_normal((L, 2, 576), np.float32), dt))
    q = _dev(torch, synth.to_bits(rng.standard_normal((L, 2, H, 192), np.float32) * np.float32(0.9), dt))
    outs, rows = [], []
    for mode in (0, 1):
        ctx = make_ctx(case, kernel, n_layers=L)
        seqs = []
        for b, n in enumerate(lens):
            s_ = ctx.seq_create()
            for l in range(L):
                ctx.write_rows(l, s_, 0, _dev(torch, case.caches[b][:n]))
            ctx.advance_seq_len(s_, n)
            seqs.append(s_)
        out = torch.zeros((L, 2, H, 128), dtype=torch.int16, device="cuda")
        ctx.step_begin(seqs)
        if mode == 0:
            for l in range(L):
                ctx.step_append(l, kv[l])
                ctx.step_attend(l, q[l], out[l])
        else:
            ctx.step_layers(0, L, kv, q, out)
        ctx.step_end()
        outs.append(_host(out).copy())
        rows.append(np.stack([ctx.read_rows(l, seqs[b], lens[b], 1) for l in range(L) for b in range(2)]))
        assert ctx.status() == 0
        ctx.close()
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(rows[0], rows[1])


@pytest.mark.parametrize("dt", [synth.DT_F16, synth.DT_BF16])
def test_q_rope_inside_the_absorb_kernel(torch, oracle, dt):
    """Step E of the reference's decode driver (transformer.cpp:3882-3921) folded into the absorb
    kernel: queries passed before their RoPE give bit-identical outputs to queries the checker
    rotated at the same positions, for decode rows, a prefill chunk (one position per row) and the
    explicit-length call; and they agree with the CPU attention over the rotated queries."""
    H, lens, chunk = 64, [130, 64], 5
    case = synth.make_layer_case(777, H, [n + chunk for n in lens], dt)
    rng = np.random.default_rng(12)
    n_new = [1, chunk]
    R = sum(n_new)
    kv = synth.to_bits(rng.standard_normal((R, 576), np.float32), dt)
    q_raw = synth.to_bits(rng.standard_normal((R, H, 192), np.float32) * np.float32(0.9), dt)
    pos = [lens[0]] + [lens[1] + t for t in range(chunk)]
    q_rot = q_raw.copy()
    for r in range(R):
        q_rot[r] = oracle.q_rope(q_raw[r], pos[r], 40.0, 4096, 10000.0, dt)
    assert not np.array_equal(q_rot, q_raw)
    outs = []
    for in_kernel in (False, True):
        ctx = make_ctx(case, capi.KERNEL_AUTO, max_rows=R)
        seqs = fill(torch, ctx, case, upto=lens)
        ctx.set_q_rope(in_kernel)
        out = torch.zeros((R, H, 128), dtype=torch.int16, device="cuda")
        ctx.step_begin(seqs, n_new)
        ctx.step_layers(0, 1, _dev(torch, kv)[None], _dev(torch, q_raw if in_kernel else q_rot)[None], out[None])
        ctx.step_end()
        got = [_host(out).copy()]
        # explicit-length call: the query stands at the last attended position
        out2 = torch.zeros((2, H, 128), dtype=torch.int16, device="cuda")
        sel = [0, R - 1]
        ctx.attend_rows(0, seqs, [lens[0] + 1, lens[1] + chunk],
                        _dev(torch, (q_raw if in_kernel else q_rot)[sel]), out2)
        got.append(_host(out2).copy())
        assert ctx.status() == 0
        if in_kernel:                      # refused where a row has no position of its own
            with pytest.raises(Exception):
                ctx.step_begin(seqs, [0, 1])
        outs.append(got)
        if not in_kernel:
            rows = oracle.append_rows(kv, pos, case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
            cache1 = np.concatenate([case.caches[1][:lens[1]], rows[1:]])
            want = oracle.attention(q_rot[R - 1], cache1, lens[1] + chunk, case.w_uk, case.w_uv, case.w_type, H, dt)
            check_close(got[0][R - 1], want, dt, "last chunk row")
        ctx.close()
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
    for k, r in enumerate([0, R - 1]):    # other split points, so equal only within the tolerance
        check_close(outs[0][1][k], outs[0][0][r], dt, "explicit-length call")


@pytest.mark.parametrize("kernel", KERNELS)
def test_prefill_chunk_is_causal(torch, oracle, kernel):
    """A 70-token chunk appended at start_position 50 next to a plain decode row: token t attends
    [0, start+t+1) (transformer.cpp:1325-1337)."""
    H, dt = 16, synth.DT_F16
    case = synth.make_layer_case(61, H, [50 + 70, 33 + 1], dt)
    from mugen_b200.mla import MlaContext
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=dt, n_pages=8, max_seqs=2, max_seq_len=256, max_rows=80,
                     kernel=kernel, **YARN)
    ctx.set_layer_weights(0, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    s0, s1 = ctx.seq_create(), ctx.seq_create()
    ctx.write_rows(0, s0, 0, _dev(torch, case.caches[0][:50])); ctx.advance_seq_len(s0, 50)
    ctx.write_rows(0, s1, 0, _dev(torch, case.caches[1][:33])); ctx.advance_seq_len(s1, 33)
    rng = np.random.default_rng(8)
    kv_a = synth.to_bits(rng.standard_normal((71, 576), np.float32), dt)
    q = synth.to_bits(rng.standard_normal((71, H, 192), np.float32) * np.float32(0.9), dt)
    out = torch.zeros((71, H, 128), dtype=torch.int16, device="cuda")
    ctx.step_begin([s0, s1], [70, 1])
    assert ctx.step_info()[0] == 71
    ctx.step_append(0, _dev(torch, kv_a))
    ctx.step_attend(0, _dev(torch, q), out)
    ctx.step_end()
    got = _host(out)
    pos = list(range(50, 120)) + [33]
    rows = oracle.append_rows(kv_a, pos, case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
    c0 = np.concatenate([case.caches[0][:50], rows[:70]])
    c1 = np.concatenate([case.caches[1][:33], rows[70:]])
    for t in (0, 1, 13, 14, 69):
        want = oracle.attention(q[t], c0, 50 + t + 1, case.w_uk, case.w_uv, case.w_type, H, dt)
        check_close(got[t], want, dt, f"chunk token {t}")
    check_close(got[70], oracle.attention(q[70], c1, 34, case.w_uk, case.w_uv, case.w_type, H, dt), dt)
    assert ctx.seq_len(s0) == 120 and ctx.seq_len(s1) == 34
    ctx.close()


@pytest.mark.parametrize("H,dt,spec,q_rope", [
    (16, synth.DT_F16, [(50, 70), (33, 1)], False),                  # one chunk next to a decode row
    (5, synth.DT_BF16, [(0, 64), (0, 129)], False),                  # chunks from empty sequences, odd head count
    (128, synth.DT_BF16, [(100, 1), (200, 300), (64, 2), (77, 128)], False),   # chunks, a decode row and a 2-token verify row
    (32, synth.DT_F16, [(130, 200), (40, 1)], True),                 # queries arrive before their RoPE
])
def test_prefill_chunks_take_the_expanded_path(torch, oracle, H, dt, spec, q_rope):
    """Sequences that take >= 64 new tokens in a step are routed, by mla_step_layers, through the prefill kernels
    (latent rows expanded into per-head keys / values, causal flash attention), the other rows of the same step through
    the decode kernels.  Chunk token t must see exactly [0, start + t + 1) (transformer.cpp:1325-1337): sampled tokens
    of every chunk, and every other row, against the CPU attention; appended rows bit-equal to the checker's."""
    from mugen_b200.mla import MlaContext
    starts, n_new = [a for a, _ in spec], [b for _, b in spec]
    R = sum(n_new)
    case = synth.make_layer_case(4000 + H, H, [a + b for a, b in spec], dt)
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=dt, n_pages=sum((a + b) // 64 + 2 for a, b in spec), max_seqs=len(spec),
                     max_seq_len=max(a + b for a, b in spec) + 64, max_rows=R, kernel=capi.KERNEL_AUTO, **YARN)
    ctx.shuffle_free_pages(3)
    ctx.set_layer_weights(0, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    seqs = fill(torch, ctx, case, upto=starts)
    rng = np.random.default_rng(77)
    kv = synth.to_bits(rng.standard_normal((R, 576), np.float32), dt)
    q_raw = synth.to_bits(rng.standard_normal((R, H, 192), np.float32) * np.float32(0.9), dt)
    pos, row0 = [], []
    for a, b in spec:
        row0.append(len(pos))
        pos += [a + t for t in range(b)]
    q_rot = q_raw
    if q_rope:
        q_rot = q_raw.copy()
        for r in range(R):
            q_rot[r] = oracle.q_rope(q_raw[r], pos[r], 40.0, 4096, 10000.0, dt)
        ctx.set_q_rope(True)
    out = torch.zeros((R, H, 128), dtype=torch.int16, device="cuda")
    ctx.step_begin(seqs, n_new)
    ctx.step_layers(0, 1, _dev(torch, kv)[None], _dev(torch, q_raw)[None], out[None])
    ctx.step_end()
    assert ctx.status() == 0
    got = _host(out)
    rows = oracle.append_rows(kv, pos, case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
    for i, (a, b) in enumerate(spec):
        assert ctx.seq_len(seqs[i]) == a + b
        assert np.array_equal(ctx.read_rows(0, seqs[i], a, b), rows[row0[i]:row0[i] + b]), f"appended rows of sequence {i}"
        cache = np.concatenate([case.caches[i][:a], rows[row0[i]:row0[i] + b]])
        ts = sorted(set(t for t in (0, 1, 62, 63, 64, 65, 127, 128, b // 2, b - 2, b - 1) if 0 <= t < b))
        for t in ts:
            want = oracle.attention(q_rot[row0[i] + t], cache, a + t + 1, case.w_uk, case.w_uv, case.w_type, H, dt)
            check_close(got[row0[i] + t], want, dt, f"sequence {i} (start {a}, {b} new), token {t}")
    ctx.close()


@pytest.mark.parametrize("decode_rows,launches", [(0, 3), (2, 5)])
def test_launches_of_a_step_with_a_chunk_are_counted(torch, decode_rows, launches):
    """The append or, with decode rows, absorb, attention and merge; then the expansion and the chunk's attention."""
    n = 1 + decode_rows
    case = synth.make_layer_case(4400, 4, [100] * n, synth.DT_F16)
    ctx = make_ctx(case, capi.KERNEL_AUTO, max_rows=130)
    seqs = fill(torch, ctx, case)
    new = [100] + [1] * decode_rows
    kv, q, out = (torch.zeros((1, sum(new)) + d, dtype=torch.int16, device="cuda") for d in ((576,), (4, 192), (4, 128)))
    before = ctx.launch_count()
    ctx.step_begin(seqs, new)
    ctx.step_layers(0, 1, kv, q, out)
    ctx.step_end()
    assert ctx.launch_count() - before == launches and ctx.status() == 0
    ctx.close()


@pytest.mark.parametrize("start,n_new", [(0, 64), (1, 127), (0, 129), (120, 137), (300, 212), (0, 1025)])
def test_prefill_maxima_that_move_at_every_step(torch, start, n_new):
    """1 to 9 steps of 128 keys whose rows grow along the sequence, so that the maxima move (and the output is rescaled) in
    steps of both softmax groups, with the sums spread over them; sharp queries, so that most exponents lie far below zero.
    Against float64 from the rows the cache holds.  Expanded keys are rounded to fp16 (2^-12 of each value): scores of
    standard deviation ~8 carry an error of ~1e-3, within the usual 5e-3 / 2e-2."""
    H, dt = 8, synth.DT_F16
    total = start + n_new
    case = synth.make_layer_case(5100 + n_new, H, [total], dt)
    from mugen_b200.mla import MlaContext
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=dt, n_pages=total // 64 + 3, max_seqs=1, max_seq_len=total + 64, max_rows=n_new, **YARN)
    ctx.shuffle_free_pages(2)
    ctx.set_layer_weights(0, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    s = ctx.seq_create()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n_new)
    grow = torch.linspace(0.5, 2.0, total, device="cuda")[:, None]
    rows = (torch.randn((total, 576), device="cuda", generator=gen) * grow).half()
    if start:
        ctx.write_rows(0, s, 0, rows[:start].view(torch.int16))
        ctx.advance_seq_len(s, start)
    kv = rows[start:].contiguous()
    kv[:, 512:] *= 4                                       # the append normalises the latent part: the rope part keeps growing
    q = (torch.randn((n_new, H, 192), device="cuda", generator=gen) * 3).half()
    out = torch.zeros((n_new, H, 128), dtype=torch.float16, device="cuda")
    ctx.step_begin([s], [n_new])
    ctx.step_layers(0, 1, kv[None], q[None], out[None])
    ctx.step_end()
    assert ctx.status() == 0
    held = torch.from_numpy(ctx.read_rows(0, s, 0, total).view(np.int16)).cuda().view(torch.float16).double()
    uk, uv = (torch.from_numpy(w.view(np.int16)).cuda().view(torch.float16).double().view(H, 128, 512) for w in (case.w_uk, case.w_uv))
    qd = q.double()
    sc = torch.einsum("nhi,hid,td->hnt", qd[..., :128], uk, held[:, :512]) + torch.einsum("nhi,ti->hnt", qd[..., 128:], held[:, 512:])
    pos = torch.arange(total, device="cuda")
    sc = (sc / 192 ** 0.5).masked_fill(pos[None, None] > pos[None, start:, None], -torch.inf)
    want = torch.einsum("hnt,td,hid->nhi", torch.softmax(sc, -1), held[:, :512], uv)
    err = (out.double() - want).abs()
    assert err.max() <= 2e-2 * max(1.0, want.abs().max().item()) and err.norm() <= 5e-3 * want.norm(), (err.max(), err.norm() / want.norm())
    ctx.close()


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("kernel", KERNELS)
def test_kv_range_shards_merge(torch, oracle, kernel, fused):
    """One sequence cut into 3 KV ranges held by 3 contexts (stand-ins for 3 GPUs): each emits
    (m, l, acc) partials; the merged + projected result equals the unsharded CPU result.  `fused`: the append rides in
    the launch that absorbs q (mla_step_layer_partial; the shards without a new row pass no kv_a)."""
    H, dt, S = 32, synth.DT_BF16, 64 * 9 + 17
    case = synth.make_layer_case(71, H, [S], dt)
    cuts = [0, 64 * 3, 64 * 6, S]
    from mugen_b200.mla import MlaContext
    parts = torch.zeros((3, 1, H, 514), dtype=torch.float32, device="cuda")
    ctxs = []
    rng = np.random.default_rng(3)
    kv_a = synth.to_bits(rng.standard_normal((1, 576), np.float32), dt)
    new_row = oracle.append_rows(kv_a, [S], case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
    full = np.concatenate([case.caches[0], new_row])
    q = _dev(torch, case.q)
    for g in range(3):
        ctx = MlaContext(n_layers=1, n_heads=H, dtype=dt, n_pages=8, max_seqs=1, max_seq_len=512,
                         max_position=4096, kernel=kernel, **YARN)
        ctx.set_layer_weights(0, case.w_uk, case.w_uv, case.w_type, case.norm_w)
        s = ctx.seq_create()
        ctx.seq_set_base(s, cuts[g])
        n = cuts[g + 1] - cuts[g]
        ctx.write_rows(0, s, 0, _dev(torch, case.caches[0][cuts[g]:cuts[g + 1]]))
        ctx.advance_seq_len(s, n)
        # the shard owning the tail takes the appended token; the others only answer the query
        ctx.step_begin([s], [1 if g == 2 else 0])
        if fused:
            ctx.step_layer_partial(0, _dev(torch, kv_a) if g == 2 else None, q, parts[g])
        else:
            ctx.step_append(0, _dev(torch, kv_a))
            ctx.step_attend_partial(0, q, parts[g])
        ctx.step_end()
        if g == 2:
            assert np.array_equal(ctx.read_rows(0, s, n, 1)[0], new_row[0])
            assert ctx.seq_len(s) == n + 1
        else:
            assert ctx.seq_len(s) == n
        ctxs.append(ctx)
    out = torch.zeros((1, H, 128), dtype=torch.int16, device="cuda")
    ctxs[0].merge_partials(0, 3, 1, parts, out)
    want = oracle.attention(case.q[0], full, S + 1, case.w_uk, case.w_uv, case.w_type, H, dt)
    check_close(_host(out)[0], want, dt, "merged shards")
    # the exported state itself: m is a log2-domain maximum, l and acc follow it
    p = parts.cpu().numpy()
    for g in range(3):
        end = cuts[g + 1] + (1 if g == 2 else 0)
        ref = oracle.partial(case.q[0], full, cuts[g], end, case.w_uk, case.w_type, H, dt)
        o_gpu = p[g, 0, :, 2:] / p[g, 0, :, 1:2]
        o_ref = ref[:, 2:] / ref[:, 1:2]
        assert np.abs(o_gpu - o_ref).max() < 2e-2
        np.testing.assert_allclose(p[g, 0, :, 0], ref[:, 0] * np.log2(np.e), rtol=2e-2, atol=5e-2)
    for ctx in ctxs:
        assert ctx.status() == 0
        ctx.close()


@pytest.mark.parametrize("kernel", KERNELS)
def test_host_buffer_entry_point(torch, oracle, kernel):
    H, dt = 16, synth.DT_F16
    case = synth.make_layer_case(81, H, [200, 77], dt)
    ctx = make_ctx(case, kernel)
    seqs = fill(torch, ctx, case, upto=[199, 76])
    out = np.zeros((2, H, 128), np.uint16)
    ctx.step_begin(seqs)
    ctx.step_layer_host(0, case.kv_a, case.q, out)
    ctx.step_end()
    rows = oracle.append_rows(case.kv_a, [199, 76], case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
    for b, n in enumerate([200, 77]):
        cache = np.concatenate([case.caches[b][:n - 1], rows[b:b + 1]])
        want = oracle.attention(case.q[b], cache, n, case.w_uk, case.w_uv, case.w_type, H, dt)
        check_close(out[b], want, dt)
    ctx.close()


def test_host_buffer_entry_point_page_locked_overlaps_and_matches_device_path(torch):
    """Page-locked caller buffers: copies run on the context's own copy streams (inputs of the next
    layer and outputs of the previous one move while a layer computes).  Two steps over three
    layers must give, bit for bit, what the device-buffer call gives, and the outputs must be in
    the host buffers when step_end returns."""
    H, L, dt, lens = 128, 3, synth.DT_BF16, [300, 65]
    case = synth.make_layer_case(91, H, [n + 2 for n in lens], dt)
    rng = np.random.default_rng(6)
    kv = [synth.to_bits(rng.standard_normal((L, 2, 576), np.float32), dt) for _ in range(2)]
    q = [synth.to_bits(rng.standard_normal((L, 2, H, 192), np.float32) * np.float32(0.9), dt) for _ in range(2)]
    results = []
    for mode in ("device", "host"):
        ctx = make_ctx(case, capi.KERNEL_AUTO, n_layers=L)
        seqs = []
        for b, n in enumerate(lens):
            s_ = ctx.seq_create()
            for l in range(L):
                ctx.write_rows(l, s_, 0, _dev(torch, case.caches[b][:n]))
            ctx.advance_seq_len(s_, n)
            seqs.append(s_)
        outs = []
        for step in range(2):
            if mode == "device":
                out = torch.zeros((L, 2, H, 128), dtype=torch.int16, device="cuda")
                ctx.step_begin(seqs)
                ctx.step_layers(0, L, _dev(torch, kv[step]), _dev(torch, q[step]), out)
                ctx.step_end()
                outs.append(_host(out).copy())
            else:
                hkv = torch.from_numpy(kv[step].view(np.int16)).pin_memory()
                hq = torch.from_numpy(q[step].view(np.int16)).pin_memory()
                hout = torch.zeros((L, 2, H, 128), dtype=torch.int16).pin_memory()
                ctx.step_begin(seqs)
                for l in range(L):
                    ctx.step_layer_host(l, hkv[l], hq[l], hout[l])
                ctx.step_end()                      # no stream synchronisation: step_end waits for the copies
                outs.append(hout.numpy().view(np.uint16).copy())
        assert ctx.status() == 0
        results.append(outs)
        ctx.close()
    for step in range(2):
        assert results[1][step].any()
        assert np.array_equal(results[0][step], results[1][step])


# ---------------------------------------------------------------------------------------------
# bookkeeping and error behaviour on the device-backed context
# ---------------------------------------------------------------------------------------------
def test_cache_bookkeeping_and_errors(torch):
    from mugen_b200.mla import MlaContext
    case = synth.make_layer_case(1, 2, [1], synth.DT_F16)
    ctx = MlaContext(n_layers=1, n_heads=2, dtype=synth.DT_F16, n_pages=4, max_seqs=2, max_seq_len=200,
                     kernel=capi.KERNEL_MMA, **YARN)
    ctx.set_layer_weights(0, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    a, b = ctx.seq_create(), ctx.seq_create()
    with pytest.raises(capi.MlaError) as e:
        ctx.seq_create()
    assert e.value.code == 4
    rows = torch.zeros((130, 576), dtype=torch.int16, device="cuda")
    ctx.write_rows(0, a, 0, rows)
    assert ctx.free_pages() == 1
    ctx.advance_seq_len(a, 130)
    with pytest.raises(capi.MlaError):          # advancing past appended rows
        ctx.advance_seq_len(a, 100)
    with pytest.raises(capi.MlaError) as e:     # pool exhausted (needs 2 pages, 1 free)
        ctx.write_rows(0, b, 0, rows[:100])
    assert e.value.code == 3
    with pytest.raises(capi.MlaError) as e:     # beyond max_seq_len
        ctx.append_rows(0, [a], [200], rows[:1])
    assert e.value.code == 4
    with pytest.raises(capi.MlaError):          # truncate never grows
        ctx.truncate(a, 131)
    ctx.truncate(a, 64)
    assert ctx.seq_len(a) == 64 and ctx.free_pages() == 3
    ctx.truncate(a, 1)
    assert ctx.free_pages() == 3                # partial last page is kept
    ctx.clear(a)
    assert ctx.seq_len(a) == 0 and ctx.free_pages() == 4
    with pytest.raises(capi.MlaError) as e:     # out-of-order scheduler calls
        ctx.step_end()
    assert e.value.code == 5
    ctx.step_begin([a, b])
    with pytest.raises(capi.MlaError):
        ctx.step_begin([a])
    ctx.step_end()
    assert ctx.seq_len(a) == 1 and ctx.seq_len(b) == 1
    assert ctx.status() == 0
    ctx.close()


def test_a_wait_that_runs_out_raises_the_status_bit_and_leaves_the_context_usable(torch, oracle):
    """Failure detection on the device, without faulting it: the self-test block waits on a barrier nothing
    completes, with a limit of a million cycles; the wait must give up (never hang, never trap), raise
    ST_WAIT_TIMEOUT (4) in the status word, free its tensor memory and return.  The host reads the bit through
    mla_status, which clears it, and the same context then computes a correct attention."""
    case = synth.make_layer_case(4242, 128, [200], synth.DT_BF16)
    ctx = make_ctx(case, capi.KERNEL_AUTO)
    seqs = fill(torch, ctx, case)
    assert ctx.status() == 0
    waited = ctx.selftest_wait_timeout(1_000_000)
    assert 1_000_000 <= waited < 400_000_000, waited          # gave up after the limit, within a fraction of a second
    with pytest.raises(capi.MlaError) as ei:
        ctx.status()
    assert ei.value.code == 6 and "= 4" in str(ei.value)          # MLA_ERR_DEVICE, ST_WAIT_TIMEOUT
    assert ctx.status() == 0                                   # reading cleared it
    out = torch.zeros((1, 128, 128), dtype=torch.int16, device="cuda")
    ctx.attend_rows(0, seqs, [200], _dev(torch, case.q), out)
    check_close(_host(out)[0], oracle_out(oracle, case, 0), case.dt, "after the timed-out wait")
    assert ctx.status() == 0
    with pytest.raises(capi.MlaError):                         # limits beyond about a second are refused
        ctx.selftest_wait_timeout(3_000_000_000)
    ctx.close()


def test_a_share_that_never_comes_is_not_added(torch):
    """The blocks of a cluster put a projection's sums together.  Where one of them gives up, the others must not take what their
    shared memory holds for its share: the self-test's second launch reports any block that does (and raises here)."""
    ctx = make_ctx(synth.make_layer_case(11, 2, [3], synth.DT_F16), capi.KERNEL_AUTO)
    before = ctx.launch_count()
    ctx.selftest_wait_timeout(200_000)
    assert ctx.launch_count() - before == 2
    with pytest.raises(capi.MlaError) as ei:
        ctx.status()
    assert "= 4" in str(ei.value) and ctx.status() == 0
    ctx.close()


def test_block_tables_are_permuted_pages(torch):
    from mugen_b200.mla import MlaContext
    ctx = MlaContext(n_layers=1, n_heads=2, dtype=synth.DT_F16, n_pages=64, max_seqs=2, max_seq_len=4096,
                     kernel=capi.KERNEL_MMA, **YARN)
    ctx.shuffle_free_pages(42)
    s = ctx.seq_create()
    ctx.write_rows(0, s, 0, torch.zeros((64 * 40, 576), dtype=torch.int16, device="cuda"))
    pages = ctx.seq_pages(s)
    assert len(pages) == 40 and len(set(pages.tolist())) == 40
    assert not np.array_equal(pages, np.sort(pages))
    ctx.close()


@pytest.mark.parametrize("H,dt,L,lens", [
    (16, synth.DT_F16, 5, [200]),                                   # one row per layer: all layers in one group
    (40, synth.DT_BF16, 3, [1, 64, 65, 700, 0]),                    # tile edges and an empty sequence
    (128, synth.DT_BF16, 7, [(37 * i) % 190 for i in range(100)]),  # 700 rows: a group of 4 layers and one of 3
])
def test_step_layers_in_groups_of_layers(torch, H, dt, L, lens):
    """step_layers plans groups of layers as one launch series; its cuts may differ from the per-layer calls', so outputs
    agree within the attention tolerance and appended rows bit for bit."""
    from mugen_b200.mla import MlaContext
    B = len(lens)
    case = synth.make_layer_case(900 + H, H, [n + 1 for n in lens], dt)
    rng = np.random.default_rng(5)
    kv = _dev(torch, synth.to_bits(rng.standard_normal((L, B, 576), np.float32), dt))
    q = _dev(torch, synth.to_bits(rng.standard_normal((L, B, H, 192), np.float32) * np.float32(0.9), dt))
    outs, rows = [], []
    for grouped in (False, True):
        ctx = MlaContext(n_layers=L, n_heads=H, dtype=dt, n_pages=sum(n // 64 + 1 for n in lens), max_seqs=B, max_seq_len=1024, **YARN)
        ctx.shuffle_free_pages(9)
        for l in range(L):          # every layer its own weights: scaled by an exact power of two
            scale = 2.0 ** -(l % 3)
            ctx.set_layer_weights(l, synth.to_bits(case.w_uk_f32 * scale, dt), synth.to_bits(case.w_uv_f32, dt), case.w_type, case.norm_w)
        seqs = []
        for b, n in enumerate(lens):
            s_ = ctx.seq_create()
            for l in range(L):
                if n:
                    ctx.write_rows(l, s_, 0, _dev(torch, np.roll(case.caches[b][:n], l, axis=0)))
            ctx.advance_seq_len(s_, n)
            seqs.append(s_)
        out = torch.zeros((L, B, H, 128), dtype=torch.int16, device="cuda")
        ctx.step_begin(seqs)
        if grouped:
            ctx.step_layers(0, L, kv, q, out)
        else:
            for l in range(L):
                ctx.step_append(l, kv[l])
                ctx.step_attend(l, q[l], out[l])
        ctx.step_end()
        outs.append(_host(out).copy())
        rows.append(np.stack([ctx.read_rows(l, seqs[b], lens[b], 1) for l in range(L) for b in range(B)]))
        assert ctx.status() == 0
        ctx.close()
    assert np.array_equal(rows[0], rows[1])
    for l in range(L):
        check_close(outs[1][l], outs[0][l], dt, f"layer {l}")


@pytest.mark.parametrize("H,dt,spec", [
    (16, synth.DT_F16, [(62, 5), (0, 5), (1000, 5)]),               # 80 head rows per stream; a page that only the later rows reach
    (16, synth.DT_BF16, [(127, 2), (63, 2), (500, 1)]),             # 32 head rows, and a single row beside them
    (16, synth.DT_F16, [(190, 4)]),                                 # 64: a full tile
    (8, synth.DT_BF16, [(63, 2), (64, 1)]),                         # 16 columns of the transposed kernel
    (5, synth.DT_F16, [(60, 7), (200, 3)]),                         # 35 head rows off every tile
    (32, synth.DT_BF16, [(125, 7)]),                                # 7 rows in groups of 4 and 3
    (16, synth.DT_F16, [(10, 1)] * 40 + [(300, 40)]),               # many single rows beside a long run
    (100, synth.DT_BF16, [(130, 2), (64, 1)]),                      # no grouping; heads between 64 and 128
    (16, synth.DT_BF16, [(62, 5), (500, 1), (1000, 2)]),            # 80 head rows, 48 per block of the pair, beside groups of 16 and 32
    (16, synth.DT_F16, [(300, 6), (0, 1)]),                         # 96 beside 16: the second block's queries reach past the last row
    (16, synth.DT_F16, [(40, 2), (700, 3), (129, 1)]),              # 48 columns of the transposed kernel, groups of 32, 48 and 16
])
def test_rows_of_one_sequence_share_a_stream(torch, oracle, H, dt, spec):
    """Several new tokens of a sequence in one step are attended over one stream of its pages; every row against the CPU
    attention at its own length."""
    from mugen_b200.mla import MlaContext
    case = synth.make_layer_case(700 + H + len(spec), H, [a + b for a, b in spec], dt)
    R = sum(b for _, b in spec)
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=dt, n_pages=sum((a + b) // 64 + 1 for a, b in spec), max_seqs=len(spec),
                     max_seq_len=max(a + b for a, b in spec), max_rows=R, **YARN)
    ctx.shuffle_free_pages(13)
    ctx.set_layer_weights(0, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    seqs = fill(torch, ctx, case, upto=[a for a, _ in spec])
    rng = np.random.default_rng(31)
    kv = synth.to_bits(rng.standard_normal((R, 576), np.float32), dt)
    q = synth.to_bits(rng.standard_normal((R, H, 192), np.float32) * np.float32(0.9), dt)
    out = torch.zeros((R, H, 128), dtype=torch.int16, device="cuda")
    ctx.step_begin(seqs, [b for _, b in spec])
    ctx.step_layers(0, 1, _dev(torch, kv)[None], _dev(torch, q)[None], out[None])
    ctx.step_end()
    assert ctx.status() == 0
    got, r = _host(out), 0
    for i, (a, b) in enumerate(spec):
        rows = oracle.append_rows(kv[r:r + b], list(range(a, a + b)), case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
        cache = np.concatenate([case.caches[i][:a], rows])
        for t in range(b):
            want = oracle.attention(q[r + t], cache, a + t + 1, case.w_uk, case.w_uv, case.w_type, H, dt)
            check_close(got[r + t], want, dt, f"sequence {i} (start {a}), token {t}")
        r += b
    ctx.close()


@pytest.mark.parametrize("H,dt", [(16, synth.DT_BF16), (17, synth.DT_F16), (32, synth.DT_BF16), (33, synth.DT_F16), (48, synth.DT_BF16),
                                  (49, synth.DT_F16), (64, synth.DT_BF16), (65, synth.DT_F16), (96, synth.DT_BF16), (97, synth.DT_BF16)])
def test_attention_at_the_edges_of_its_widths(torch, oracle, H, dt):
    """Both sides of every width of the transposed kernel and of the SM-pair kernel: rows of one token, a full page, one token more, and long ones whose scores rise
    from page to page, so that references move on later pages; 320 rows, so that a block walks several segments and its rings of
    pages wrap many times.  Bounds as everywhere here."""
    lens = [1, 64, 65, 1100]
    case = synth.make_layer_case(9100 + H, H, lens, dt, q_scale=3.0)
    for i, n in enumerate(lens):
        ramp = np.linspace(0.2, 2.0, n, dtype=np.float32)[:, None]
        case.caches[i] = synth.to_bits(synth.from_bits(case.caches[i], dt) * ramp, dt)
    times = 80
    ctx = make_ctx(case, capi.KERNEL_AUTO, shuffle=5, max_rows=len(lens) * times)
    seqs = fill(torch, ctx, case)
    want = [oracle_out(oracle, case, b) for b in range(len(lens))]
    out = torch.zeros((len(lens) * times, H, 128), dtype=torch.int16, device="cuda")
    ctx.attend_rows(0, seqs * times, lens * times, _dev(torch, np.tile(case.q, (times, 1, 1))), out)
    got = _host(out)
    assert ctx.status() == 0 and ctx.kernel_name() == ("tcgen05-t16" if H <= 16 else "tcgen05" if H <= 64 else "tcgen05-pair128")
    for r in range(len(lens) * times):
        check_close(got[r], want[r % len(lens)], dt, f"row {r}")
    again = torch.zeros_like(out)
    ctx.attend_rows(0, seqs * times, lens * times, _dev(torch, np.tile(case.q, (times, 1, 1))), again)
    assert np.array_equal(_host(again), got)
    ctx.close()


@pytest.mark.parametrize("H", [5, 16, 32, 48, 64])
def test_scores_far_beyond_the_precision_of_their_exponents(torch, H):
    """Finite scores of 2^36 and more, where one step of a float is thousands: the largest score's distance to the reference is 0 all
    the same, and the softmax picks its token.  All rows of a sequence lie along one direction u, one of them is u, one -u,
    the others at most half as long: the output is W_UV u, with the sign of the head's score."""
    from mugen_b200.mla import MlaContext
    lens = [1, 64, 65, 130, 1100]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(H)
    rn = lambda *shape, s=1.0: (torch.randn(shape, device="cuda", generator=gen) * s).bfloat16()
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=synth.DT_BF16, n_pages=64, max_seqs=len(lens), max_seq_len=2048, max_rows=len(lens), **YARN)
    w_uk, w_uv = rn(H * 128, 512, s=0.02), rn(H * 128, 512, s=0.02)
    ctx.set_layer_weights(0, bits(w_uk), bits(w_uv), synth.W_BF16, np.full(512, 0x3F80, np.uint16))
    u, q = rn(576), rn(len(lens), H, 192, s=1e13)
    seqs = []
    for n in lens:
        a = (torch.rand(n, device="cuda", generator=gen) - 0.5).double()
        a[-1], a[n // 3] = (-1.0, 1.0) if n > 1 else (1.0, 1.0)
        s = ctx.seq_create()
        ctx.write_rows(0, s, 0, (a[:, None] * u.double()).bfloat16().view(torch.int16))
        ctx.advance_seq_len(s, n)
        seqs.append(s)
    out = torch.zeros((len(lens), H, 128), dtype=torch.int16, device="cuda")
    ctx.attend_rows(0, seqs, lens, q.view(torch.int16), out)
    got = out.view(torch.bfloat16).double()
    assert ctx.status() == 0
    score = torch.einsum("rhi,hid,d->rh", q[..., :128].double(), w_uk.double().view(H, 128, 512), u[:512].double()) + q[..., 128:].double() @ u[512:].double()
    sure = score.abs() > 0.02 * score.square().mean().sqrt()               # the absorbed queries' rounding cannot turn the sign
    assert sure.double().mean() > 0.9 and score.abs()[sure].min() > 2.0 ** 36 / (1.4427 / 192 ** 0.5)
    sign = torch.where(torch.tensor(lens, device="cuda")[:, None] > 1, score.sign(), torch.ones_like(score))
    want = sign[..., None] * (w_uv.double().view(H, 128, 512) @ u[:512].double())
    err = (got - want).norm(dim=-1) / want.norm(dim=-1)
    assert err[sure].max().item() <= 2.0 ** -8                             # the outputs' rounding to 8 bits
    ctx.close()


@pytest.mark.parametrize("H,dt", [(128, synth.DT_F16), (96, synth.DT_BF16)])
def test_references_move_on_the_last_tile_of_every_segment(torch, oracle, H, dt):
    """Segments of two and three tiles of the SM-pair kernel, several per pair, whose scores rise by more than 2^8 from tile to tile: the request to
    move a reference comes on a segment's last tile, and again on the second one of the next segment, with one flag for both and no
    round between the blocks on the first tile in between."""
    lens, times = [256, 384, 130, 257], 80
    case = synth.make_layer_case(9300 + H, H, lens, dt, q_scale=3.0)
    for i, n in enumerate(lens):
        steps = np.asarray([0.05, 1.0, 2.2], np.float32)[np.arange(n) // 128][:, None]
        case.caches[i] = synth.to_bits(synth.from_bits(case.caches[i], dt) * steps, dt)
    w_uk = synth.from_bits(case.w_uk, dt).reshape(H, 128, 512)
    for i, n in enumerate(lens):
        q, c = synth.from_bits(case.q[i], dt), synth.from_bits(case.caches[i], dt)
        s = (np.einsum("hi,hid,td->ht", q[:, :128], w_uk, c[:, :512], optimize=True) + q[:, 128:] @ c[:, 512:].T) / np.sqrt(192) * np.log2(np.e)
        tops = np.stack([s[:, t:t + 128].max(1) for t in range(0, n, 128)])
        assert i > 1 or (np.diff(tops, axis=0).max(1) > 9).all()             # some head moves on every tile but the first
    ctx = make_ctx(case, capi.KERNEL_AUTO, shuffle=5, max_rows=len(lens) * times)
    seqs = fill(torch, ctx, case)
    want = [oracle_out(oracle, case, b) for b in range(len(lens))]
    q = _dev(torch, np.tile(case.q, (times, 1, 1)))
    first = None
    for _ in range(4):
        out = torch.zeros((len(lens) * times, H, 128), dtype=torch.int16, device="cuda")
        ctx.attend_rows(0, seqs * times, lens * times, q, out)
        got = _host(out)
        assert ctx.status() == 0 and ctx.kernel_name() == "tcgen05-pair128"
        assert first is None or np.array_equal(got, first)
        first = got
    for r in range(len(lens) * times):
        check_close(first[r], want[r % len(lens)], dt, f"row {r}")
    ctx.close()


@pytest.mark.parametrize("H,dt,lens", [
    (5, synth.DT_F16, [6000]),                             # one row in 94 parts: sixteen warps share its dims
    (32, synth.DT_BF16, [2100]),
    (70, synth.DT_F16, [65]),                              # few parts
    (16, synth.DT_BF16, [4100, 40]),                       # two rows: eight warps each
])
def test_merge_of_few_rows_in_many_parts(torch, oracle, H, dt, lens):
    """The merge's warps per row for the smallest steps (mla_merge_tc5.cu), every head against the CPU."""
    case = synth.make_layer_case(6100 + H, H, [n + 1 for n in lens], dt)
    ctx = make_ctx(case, capi.KERNEL_AUTO, shuffle=5, max_rows=len(lens), max_seqs=len(lens))
    seqs = fill(torch, ctx, case, upto=lens)
    out = torch.zeros((len(lens), H, 128), dtype=torch.int16, device="cuda")
    ctx.step_begin(seqs)
    ctx.step_layers(0, 1, _dev(torch, case.kv_a)[None], _dev(torch, case.q)[None], out[None])
    ctx.step_end()
    assert ctx.status() == 0
    got = _host(out)
    rows = oracle.append_rows(case.kv_a, lens, case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
    for b, n in enumerate(lens):
        cache = np.concatenate([case.caches[b][:n], rows[b:b + 1]])
        check_close(got[b], oracle.attention(case.q[b], cache, n + 1, case.w_uk, case.w_uv, case.w_type, H, dt), dt, f"row {b}")
    ctx.close()


@pytest.mark.parametrize("H,dt,rows,L", [
    (16, synth.DT_F16, 16, 5),       # alone a layer's heads are cut into nine parts of one or two rows, five layers take whole heads
    (5, synth.DT_F16, 29, 7),        # parts of one row; four of seven and eight
    (40, synth.DT_BF16, 11, 4),      # three of three and four; one
    (24, synth.DT_BF16, 70, 3),      # six of eleven and twelve; two of 35
])
def test_a_rows_projection_is_the_same_whoever_shares_its_launch(torch, oracle, H, dt, rows, L):
    """Contexts of one page are never cut, so a layer's outputs are the same bits alone and in a launch of several layers, whichever
    kernel the merge takes for the rows that a block has; and they are the CPU's."""
    lens = [(11 * i) % 60 for i in range(rows)]
    case = synth.make_layer_case(7300 + H, H, [n + 1 for n in lens], dt)
    kv, q = _dev(torch, case.kv_a), _dev(torch, case.q)
    outs = []
    for grouped in (False, True):
        ctx = make_ctx(case, capi.KERNEL_AUTO, n_layers=L, shuffle=3, max_rows=rows, max_seqs=rows)
        seqs = []
        for b, n in enumerate(lens):
            seqs.append(ctx.seq_create())
            for l in range(L):
                if n:
                    ctx.write_rows(l, seqs[b], 0, _dev(torch, case.caches[b][:n]))
            ctx.advance_seq_len(seqs[b], n)
        out = torch.zeros((L, rows, H, 128), dtype=torch.int16, device="cuda")
        ctx.step_begin(seqs)
        if grouped:
            before = ctx.launch_count()
            ctx.step_layers(0, L, torch.stack([kv] * L), torch.stack([q] * L), out)
            assert ctx.launch_count() - before == 3          # all layers in one absorb, one attention, one merge
        else:
            for l in range(L):
                ctx.step_append(l, kv)
                ctx.step_attend(l, q, out[l])
        ctx.step_end()
        outs.append(_host(out).copy())
        assert ctx.status() == 0
        ctx.close()
    assert np.array_equal(outs[0], outs[1])
    appended = oracle.append_rows(case.kv_a, lens, case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
    for b, n in enumerate(lens):
        want = oracle.attention(case.q[b], np.concatenate([case.caches[b][:n], appended[b:b + 1]]), n + 1, case.w_uk, case.w_uv, case.w_type, H, dt)
        check_close(outs[0][0][b], want, dt, f"row {b}")


@pytest.mark.parametrize("rows,L", [(8, 6), (24, 6), (48, 6), (70, 3)])
def test_absorb_streams_the_weights_of_many_units_per_block(torch, rows, L):
    """128 heads x L layers in one launch: every block of the absorb walks several (layer, head) units through its ring, with
    query tiles of 16, 32 and 64 rows.  Every layer has weights of its own; all rows and heads against float64."""
    from mugen_b200.mla import MlaContext
    H, dt = 128, synth.DT_BF16
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows)
    rn = lambda *shape, scale=1.0: (torch.randn(shape, device="cuda", generator=gen) * scale).bfloat16()
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    lens = [5 + 7 * i % 61 for i in range(rows)]
    ctx = MlaContext(n_layers=L, n_heads=H, dtype=dt, n_pages=2 * rows, max_seqs=rows, max_seq_len=128, **YARN)
    ctx.shuffle_free_pages(3)
    w_uk, w_uv = rn(L, H, 128, 512, scale=0.02), rn(L, H, 128, 512, scale=0.02)
    for l in range(L):
        ctx.set_layer_weights(l, bits(w_uk[l]), bits(w_uv[l]), synth.W_BF16, bits(1 + rn(512, scale=0.1)))
    seqs = [ctx.seq_create() for _ in lens]
    for l in range(L):
        for s, n in zip(seqs, lens):
            ctx.write_rows(l, s, 0, rn(n, 576).view(torch.int16))
    for s, n in zip(seqs, lens):
        ctx.advance_seq_len(s, n)
    kv, q = rn(L, rows, 576), rn(L, rows, H, 192, scale=0.9)
    out = torch.zeros((L, rows, H, 128), device="cuda", dtype=torch.bfloat16)
    for rep in range(20):                     # the copies of a launch land in another order every time
        out.zero_()
        ctx.step_begin(seqs)
        ctx.step_layers(0, L, kv, q, out)
        ctx.step_end()
        if rep < 19:
            ctx.rollback(seqs, lens)
        assert ctx.status() == 0
        first = out.clone() if rep == 0 else first
        assert torch.equal(out, first)
    for l in range(L):
        for r, (s, n) in enumerate(zip(seqs, lens)):
            c = torch.from_numpy(ctx.read_rows(l, s, 0, n + 1).view(np.int16)).cuda().view(torch.bfloat16).double()
            qa = torch.einsum("hi,hid->hd", q[l, r, :, :128].double(), w_uk[l].double())
            p = torch.softmax((qa @ c[:, :512].T + q[l, r, :, 128:].double() @ c[:, 512:].T) / 192 ** 0.5, -1)
            want = torch.einsum("hd,hjd->hj", p @ c[:, :512], w_uv[l].double())
            e = ((out[l, r].double() - want).norm(dim=-1) / want.norm(dim=-1)).max().item()      # per head
            # absorbed queries, probabilities and outputs are rounded to 8 bits once each (2^-9 at most); REL_L2 holds over all heads
            assert e <= 4 * REL_L2, f"layer {l}, row {r}: rel-L2 of the worst head {e:.2e}"
    ctx.close()


def test_merge_of_partials_beyond_4g_floats(torch):
    """mla_merge_partials over a caller's buffer of more than 2^32 floats (17 GB): what the parts behind that line hold must reach
    the outputs.  All states are empty (l = 0) but a few in the last two parts, so every other output is exactly 0."""
    from mugen_b200.mla import MlaContext
    H, rows, parts = 128, 2107, 33
    assert (parts - 2) * rows * H * 514 > 1 << 32
    if torch.cuda.mem_get_info()[0] < 20 << 30:
        pytest.skip("needs 20 GB of device memory")
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=synth.DT_F16, n_pages=2, max_seqs=1, max_seq_len=64, **YARN)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    w_uv = (torch.randn(H, 128, 512, device="cuda", generator=gen) * 0.05).half()
    bits = w_uv.view(torch.int16).cpu().numpy().view(np.uint16)
    ctx.set_layer_weights(0, bits, bits, synth.W_F16, np.full(512, 0x3C00, np.uint16))
    p = torch.zeros((parts, rows, H, 514), device="cuda")
    want = torch.zeros((rows, H, 128), device="cuda", dtype=torch.float64)
    for part, row, head in [(31, 0, 0), (31, 1000, 64), (31, rows - 1, H - 1), (32, 17, 5), (32, rows - 1, 0)]:
        acc = torch.randn(512, device="cuda", generator=gen)
        p[part, row, head, 1] = 1.0
        p[part, row, head, 2:] = acc
        want[row, head] = w_uv[head].double() @ acc.double()
    out = torch.full((rows, H, 128), 7.0, device="cuda", dtype=torch.float16)
    ctx.merge_partials(0, parts, rows, p, out)
    assert ctx.status() == 0
    # the state goes to the product in two halves of 11 bits each: what is left is the rounding of the output
    assert (out.double() - want).abs().max().item() <= 2.0 ** -11 * want.abs().max().item() * 1.1
    ctx.close()


@pytest.mark.parametrize("rows", [2, 8, 12])
def test_merge_of_one_part_is_the_merge_of_parts(torch, rows):
    """A row with one part takes a path of its own where a block has many rows (12 rows of 128 heads): it must give the bits of the
    general one, here the same part beside one that is empty, also for states that finite scores do not leave.  An empty part
    (m = -inf) adds nothing, whatever lies behind it."""
    from mugen_b200.mla import MlaContext
    H = 128
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=synth.DT_F16, n_pages=2, max_seqs=1, max_seq_len=64, **YARN)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    w_uv = (torch.randn(H, 128, 512, device="cuda", generator=gen) * 0.05).half()
    bits = w_uv.view(torch.int16).cpu().numpy().view(np.uint16)
    ctx.set_layer_weights(0, bits, bits, synth.W_F16, np.full(512, 0x3C00, np.uint16))
    inf, nan = float("inf"), float("nan")
    p = torch.randn((1, rows, H, 514), device="cuda", generator=gen)
    p[..., 1] = p[..., 1].abs() + 0.5
    empty = [(0, 0), (1, 3), (rows - 1, 127)]
    for (r, h), acc in zip(empty, (nan, inf, -inf)):
        p[0, r, h, 0], p[0, r, h, 1], p[0, r, h, 2:] = -inf, 0.0, acc
    for h, (m, l) in zip((10, 11, 12, 13), ((inf, 1.0), (nan, 1.0), (0.5, 0.0), (0.5, nan))):
        p[0, 1, h, 0], p[0, 1, h, 1] = m, l
    beside = torch.zeros_like(p)
    beside[..., 0] = -inf
    one, two = (torch.full((rows, H, 128), 7.0, device="cuda", dtype=torch.float16) for _ in range(2))
    ctx.merge_partials(0, 1, rows, p, one)
    ctx.merge_partials(0, 2, rows, torch.cat([p, beside]), two)
    assert ctx.status() == 0
    for r, h in empty:
        assert not one[r, h].any(), f"empty part of row {r}, head {h}"
    assert torch.equal(one.isnan(), two.isnan())
    assert torch.equal(one.nan_to_num(), two.nan_to_num())
    ctx.close()


def test_bounded_waits_do_not_run_while_an_earlier_kernel_does(torch, oracle):
    """A kernel ahead of the absorb and the merge that lets them start early and then runs for longer than the limit of their
    barrier waits (about two seconds): the limits must start when it ends, and the results must stand."""
    spin = torch.cuda._compile_kernel('extern "C" __global__ void spin(int mcycles) {'
                                      ' asm volatile("griddepcontrol.launch_dependents;");'
                                      ' const long long t0 = clock64(); while (clock64() - t0 < mcycles * 1000000LL) __nanosleep(1000); }', "spin")
    H, dt, lens = 128, synth.DT_BF16, [100, 300]
    case = synth.make_layer_case(77, H, [n + 1 for n in lens], dt)
    ctx = make_ctx(case, capi.KERNEL_AUTO, max_rows=len(lens))
    seqs = fill(torch, ctx, case, upto=lens)
    q, kv = _dev(torch, case.q), _dev(torch, case.kv_a)
    out, again = (torch.zeros((len(lens), H, 128), dtype=torch.int16, device="cuda") for _ in range(2))
    partial = torch.zeros((len(lens), H, 514), device="cuda")
    long = 4_800                                         # 2.4 s at the highest clock; the limit is 4e9 cycles
    ctx.step_begin(seqs)
    ctx.step_append(0, kv)
    ctx.step_attend_partial(0, q, partial)               # also: the step's plan is on the device
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    spin((1, 1, 1), (1, 1, 1), (long,))
    ctx.step_attend(0, q, out)
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 > 2.1
    spin((1, 1, 1), (1, 1, 1), (long,))
    ctx.merge_partials(0, 1, len(lens), partial, again)
    torch.cuda.synchronize()
    ctx.step_end()
    assert ctx.status() == 0
    rows = oracle.append_rows(case.kv_a, lens, case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
    for b, n in enumerate(lens):
        want = oracle.attention(case.q[b], np.concatenate([case.caches[b][:n], rows[b:b + 1]]), n + 1, case.w_uk, case.w_uv, case.w_type, H, dt)
        check_close(_host(out)[b], want, dt, f"row {b}")
        check_close(_host(again)[b], want, dt, f"row {b}, merged partial")
    ctx.close()


def _step_ctx(torch, H=16, dt=synth.DT_F16, L=3, lens=(100, 700, 64, 5)):
    """L layers over sequences of `lens` cached tokens, with one new token each: context, sequences, kv_a and q of all layers."""
    from mugen_b200.mla import MlaContext
    case = synth.make_layer_case(4400 + H, H, [n + 1 for n in lens], dt)
    ctx = MlaContext(n_layers=L, n_heads=H, dtype=dt, n_pages=sum(n // 64 + 3 for n in lens) + 8, max_seqs=len(lens) + 1, max_seq_len=2048,
                     max_rows=256, **YARN)
    for l in range(L):
        ctx.set_layer_weights(l, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    seqs = []
    for b, n in enumerate(lens):
        s = ctx.seq_create()
        for l in range(L):
            ctx.write_rows(l, s, 0, _dev(torch, np.roll(case.caches[b][:n], l, axis=0)))
        ctx.advance_seq_len(s, n)
        seqs.append(s)
    rng = np.random.default_rng(8)
    kv = _dev(torch, synth.to_bits(rng.standard_normal((L, len(lens), 576), np.float32), dt))
    q = _dev(torch, synth.to_bits(rng.standard_normal((L, len(lens), H, 192), np.float32) * np.float32(0.9), dt))
    return ctx, seqs, list(lens), kv, q


def test_step_info_and_balance_describe_the_open_step(torch):
    """From step_begin on, whichever calls follow: rows, segments and balance of ONE layer of the step that is open."""
    ctx, seqs, lens, kv, q = _step_ctx(torch)
    L, B = kv.shape[:2]
    out = torch.zeros((L, B, 16, 128), dtype=torch.int16, device="cuda")
    pages = [(n + 1 + 63) // 64 for n in lens]
    seen = []
    for part in (seqs, seqs[:1], seqs):
        n, k = len(part), sum(pages[:len(part)])
        ctx.step_begin(part)
        first = (ctx.step_info(), ctx.step_balance())
        assert first[0][0] == n and n <= first[0][1] <= k and first[1][0] <= k and 1 <= first[1][1] <= first[1][2] <= k
        ctx.step_layers(0, L, kv[:, :n].contiguous(), q[:, :n].contiguous(), out[:, :n].contiguous())       # one group of three layers
        assert (ctx.step_info(), ctx.step_balance()) == first
        ctx.step_append(0, kv[0, :n].contiguous())
        ctx.step_attend(0, q[0, :n].contiguous(), out[0, :n].contiguous())
        assert (ctx.step_info(), ctx.step_balance()) == first
        ctx.step_end()
        ctx.rollback(seqs, lens)
        seen.append(first)
    assert seen[0] == seen[2] != seen[1]
    ctx.step_begin(seqs[:1], [130])               # a prompt chunk alone: no row is left to the decode kernels
    assert ctx.step_info()[0] == 130 and ctx.step_balance() == (1, 0, 0)
    ctx.step_end()
    assert ctx.status() == 0
    ctx.close()


def test_calls_of_a_step_on_streams_of_their_own(torch):
    """The step's metadata is on the device when step_begin's stream says so: appends of two layers (which share no workspace) on
    two streams, both ordered behind that stream and not behind each other.  The first is held back by a busy stream."""
    ctx, seqs, lens, kv, q = _step_ctx(torch)
    L = kv.shape[0]
    ctx.step_begin(seqs)
    for l in range(L):
        ctx.step_append(l, kv[l])
    ctx.step_end()
    want = [[ctx.read_rows(l, s, n, 1).copy() for s, n in zip(seqs, lens)] for l in range(L)]
    ctx.rollback(seqs, lens)
    other = ctx.seq_create()                       # a step of other rows in between: what a stale upload would hold
    ctx.step_begin([other])
    ctx.step_append(0, kv[0, :1].contiguous())
    ctx.step_end()
    for s, n in zip(seqs, lens):
        for l in range(L):
            ctx.write_rows(l, s, n, torch.zeros((1, 576), dtype=torch.int16, device="cuda"))
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    ctx.step_begin(seqs)
    a.wait_stream(torch.cuda.current_stream())
    b.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(a):
        torch.cuda._sleep(100_000_000)             # about 50 ms
        ctx.step_append(0, kv[0])
    with torch.cuda.stream(b):
        ctx.step_append(1, kv[1])
    b.synchronize()
    assert not a.query()                           # layer 1 did not wait for layer 0's stream
    a.synchronize()
    ctx.step_append(2, kv[2])
    ctx.step_end()
    assert ctx.status() == 0
    for l in range(L):
        for i, (s, n) in enumerate(zip(seqs, lens)):
            assert np.array_equal(ctx.read_rows(l, s, n, 1), want[l][i]), (l, i)
    ctx.close()


@pytest.mark.parametrize("how", ["another stream", "another handle"])
def test_the_first_call_behind_an_upload_waits_for_it_whatever_went_elsewhere(torch, how):
    """step_begin behind a busy stream, then a group of layers on a stream ordered behind it, whose own upload has its first launch
    there, then an append on the first stream with nothing between it and the step's upload.  And the default stream by its other handle
    (cudaStreamLegacy).  The rows of a step in between are what a call that is too early would write to."""
    ctx, seqs, lens, kv, q = _step_ctx(torch)
    L, B, H = q.shape[:3]
    last = L - 1
    ctx.step_begin(seqs)
    ctx.step_append(last, kv[last])
    ctx.step_end()
    want = [ctx.read_rows(last, s, n, 1).copy() for s, n in zip(seqs, lens)]
    ctx.rollback(seqs, lens)
    other = ctx.seq_create()
    ctx.step_begin([other])
    ctx.step_append(last, kv[last, :1].contiguous())
    ctx.step_end()
    stale = ctx.read_rows(last, other, 0, 1).copy()
    for s, n in zip(seqs, lens):
        ctx.write_rows(last, s, n, torch.zeros((1, 576), dtype=torch.int16, device="cuda"))
    ctx.write_rows(last, other, 0, torch.zeros((1, 576), dtype=torch.int16, device="cuda"))
    out = torch.zeros((last, B, H, 128), dtype=torch.int16, device="cuda")
    torch.cuda.synchronize()
    a, b = torch.cuda.default_stream() if how == "another handle" else torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(20_000_000)              # about 10 ms
        ctx.step_begin(seqs)
    if how == "another stream":
        b.wait_stream(a)
        with torch.cuda.stream(b):
            ctx.step_layers(0, last, kv[:last], q[:last], out)
        with torch.cuda.stream(a):
            ctx.step_append(last, kv[last])
    else:
        assert a.cuda_stream == 0
        assert ctx.lib.mla_step_append(ctx.h, last, kv[last].data_ptr(), 1) == capi.OK
    torch.cuda.synchronize()
    ctx.step_end()
    assert ctx.status() == 0
    for s, n, w in zip(seqs, lens, want):
        assert np.array_equal(ctx.read_rows(last, s, n, 1)[0], w[0])
    assert not ctx.read_rows(last, other, 0, 1).any() and stale.any()
    ctx.close()


@pytest.mark.parametrize("H,dt", [(16, synth.DT_F16), (128, synth.DT_BF16)])
def test_groups_of_layers_start_early_behind_their_own_upload(torch, H, dt):
    """Steps over other sequences in turn, enqueued behind a busy stream without a wait in between: the first kernel of a group starts
    before its upload has stored anything, and neither it nor a kernel behind it may use what the step before had left there."""
    ctx, seqs, lens, kv, q = _step_ctx(torch, H=H, dt=dt, lens=(100, 700, 64, 1, 333, 129))
    L, B = kv.shape[:2]
    picks = [[0, 1, 2], [5, 4], [3], [1, 5, 0, 2], [2, 0]]

    def step(p, out):
        rows = torch.tensor(p, device="cuda")
        k, x = kv[:, rows].contiguous(), q[:, rows].contiguous()
        ctx.step_begin([seqs[i] for i in p])
        ctx.step_layers(0, L, k, x, out)
        ctx.step_end()
        ctx.rollback([seqs[i] for i in p], [lens[i] for i in p])
        return k, x

    outs = [[torch.zeros((L, len(p), H, 128), dtype=torch.int16, device="cuda") for p in picks] for _ in range(3)]
    for p, o in zip(picks, outs[0]):
        step(p, o)
        torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)              # about 10 ms
    keep = [step(p, o) for r in outs[1:] for p, o in zip(picks, r)]
    torch.cuda.synchronize()
    assert ctx.status() == 0 and len(keep) == 2 * len(picks)
    for r in outs[1:]:
        for want, got in zip(outs[0], r):
            assert np.array_equal(_host(got), _host(want))
    ctx.close()


@pytest.mark.parametrize("how", ["layers", "calls"])
def test_the_calls_of_an_open_step_can_be_captured(torch, how):
    """step_begin uploads; the calls behind it are launches alone, also inside a stream capture.  The graph is replayed over other
    inputs and after later steps have used the upload ring, and must give what the direct calls give."""
    ctx, seqs, lens, kv, q = _step_ctx(torch, H=128, dt=synth.DT_BF16, lens=(100, 700, 64))
    L, B = kv.shape[:2]
    out, want = (torch.zeros((L, B, 128, 128), dtype=torch.int16, device="cuda") for _ in range(2))

    def calls(o):
        if how == "layers":
            ctx.step_layers(0, L, kv, q, o)
        for l in range(L if how == "calls" else 0):
            ctx.step_append(l, kv[l])
            ctx.step_attend(l, q[l], o[l])

    for _ in range(20):                            # the ring goes round; kernels are loaded
        ctx.step_begin(seqs)
        calls(want)
        ctx.step_end()
        ctx.rollback(seqs, lens)
    torch.cuda.synchronize()
    ctx.step_begin(seqs)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        calls(out)
    q.copy_(torch.flip(q, (1,)))
    g.replay()
    calls(want)
    torch.cuda.synchronize()
    for l in range(L):
        check_close(_host(out[l]), _host(want[l]), synth.DT_BF16, f"layer {l}")
    ctx.step_end()
    ctx.rollback(seqs, lens)
    for _ in range(10):
        ctx.step_begin(seqs)
        calls(want)
        ctx.step_end()
        ctx.rollback(seqs, lens)
    assert ctx.status() == 0
    del g
    ctx.close()


@pytest.mark.parametrize("how", ["layers", "calls", "block"])
def test_calls_captured_on_the_stream_of_step_begin_keep_their_overlap(torch, how):
    """Captured with nothing between them and the step's upload, the launches of a step follow each other by programmatic edges, all of
    them.  Replayed at once behind the upload of a step, with another step's metadata in its place before and the stream
    busy, the graph writes this step's rows and outputs."""
    import ctypes as C
    ctx, seqs, lens, kv, q = _step_ctx(torch)
    L, B, H = q.shape[:3]
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    E = 256
    rn = lambda *shape: (torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(len(shape))) * 0.05).half()
    for l in range(L if how == "block" else 0):
        ctx.set_block_weights(l, attn_norm=bits(1 + rn(E)), kv_a_mqa=bits(rn(576, E)), wo=bits(rn(E, H * 128)), q=bits(rn(H * 192, E)))
    ctx.set_q_rope(how == "block")
    hidden, start = rn(B, E), rn(B, E)
    out = torch.zeros((L, B, H, 128), dtype=torch.int16, device="cuda")

    def calls():
        if how == "layers":
            ctx.step_layers(0, L, kv, q, out)
        for l in range(L if how == "calls" else 0):
            ctx.step_append(l, kv[l])
            ctx.step_attend(l, q[l], out[l])
        for l in range(L if how == "block" else 0):
            ctx.step_block(l, hidden)

    def end():
        """Closes the step: its rows and outputs, which are zeros again behind it."""
        got = [ctx.read_rows(l, s, n, 1).copy() for l in range(L) for s, n in zip(seqs, lens)], (hidden if how == "block" else out).clone()
        ctx.step_end()
        ctx.rollback(seqs, lens)
        for l in range(L):
            for s, n in zip(seqs, lens):
                ctx.write_rows(l, s, n, torch.zeros((1, 576), dtype=torch.int16, device="cuda"))
        hidden.copy_(start)
        out.zero_()
        return got

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        hidden.copy_(start)
        for _ in range(2):                         # workspaces are there, kernels are loaded
            ctx.step_begin(seqs)
            calls()
            end()
        ctx.step_begin(seqs)
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g, stream=stream):
            before = ctx.launch_count()
            calls()
            n = ctx.launch_count() - before
        # an edge's data are 8 bytes: ports of either end, kind of dependency (1: programmatic), nothing
        edges, data = C.c_size_t(n - 1), (C.c_uint8 * 8 * (n - 1))()
        ends = [(C.c_void_p * (n - 1))() for _ in range(2)]
        assert C.CDLL("libcuda.so.1").cuGraphGetEdges_v2(C.c_void_p(g.raw_cuda_graph()), *ends, data, C.byref(edges)) == 0
        assert edges.value == n - 1 and all(ends[1]) and [d[2] for d in data] == [1] * (n - 1)
        g.instantiate()
        stream.synchronize()
        g.replay()
        want = end()
        for _ in range(3):
            other = ctx.seq_create()
            ctx.step_begin([other])
            ctx.step_append(0, kv[0, :1].contiguous())
            ctx.step_end()
            ctx.seq_free(other)
            torch.cuda._sleep(2_000_000)           # about a millisecond
            ctx.step_begin(seqs)
            g.replay()
            got = end()
            assert torch.equal(got[1], want[1]) and got[1].any() and all(np.array_equal(x, y) and x.any() for x, y in zip(got[0], want[0]))
        assert ctx.status() == 0
    del g
    ctx.close()


def test_a_step_that_is_captured_whole(torch):
    """step_begin inside the capture as well (which waits for its turn in the upload ring: a relaxed capture lets it): its upload is
    part of the graph, and the launches behind it find it complete."""
    ctx, seqs, lens, kv, q = _step_ctx(torch)
    L, B, H = q.shape[:3]
    out, want = (torch.zeros((L, B, H, 128), dtype=torch.int16, device="cuda") for _ in range(2))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx.step_begin(seqs)
        for l in range(L):
            ctx.step_append(l, kv[l])
            ctx.step_attend(l, q[l], want[l])
        rows = [ctx.read_rows(l, s, n, 1).copy() for l in range(L) for s, n in zip(seqs, lens)]
        ctx.step_end()
        ctx.rollback(seqs, lens)
        for l in range(L):
            for s, n in zip(seqs, lens):
                ctx.write_rows(l, s, n, torch.zeros((1, 576), dtype=torch.int16, device="cuda"))
        stream.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream, capture_error_mode="relaxed"):
            ctx.step_begin(seqs)
            for l in range(L):
                ctx.step_append(l, kv[l])
                ctx.step_attend(l, q[l], out[l])
        torch.cuda._sleep(2_000_000)
        g.replay()
        got = [ctx.read_rows(l, s, n, 1).copy() for l in range(L) for s, n in zip(seqs, lens)]
        ctx.step_end()
        assert ctx.status() == 0
    assert torch.equal(out, want) and all(np.array_equal(x, y) and x.any() for x, y in zip(got, rows))
    del g
    ctx.close()


def test_a_context_on_a_device_with_little_room_left(torch, oracle):
    """The workspace for groups of layers is a matter of speed: where it does not fit any more the context is created without it,
    and its steps give the same."""
    from mugen_b200.mla import MlaContext
    H, dt, L, lens = 16, synth.DT_F16, 27, [200, 65]
    case = synth.make_layer_case(31, H, [n + 1 for n in lens], dt)
    make = lambda: MlaContext(n_layers=L, n_heads=H, dtype=dt, n_pages=16, max_seqs=2, max_seq_len=256, max_rows=10, **YARN)
    make().close()                                         # what the process itself allocates is there
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    ctx = make()
    need = free0 - torch.cuda.mem_get_info()[0]
    ctx.close()
    # records: 148 workers x 128 head rows more than one layer's rows need, and 27 x 10 rows instead of 10; half of it is missing
    extra = 148 * 128 * 514 * 4
    filler = torch.empty(torch.cuda.mem_get_info()[0] - need + extra // 2, dtype=torch.uint8, device="cuda")
    try:
        ctx = make()
    finally:
        del filler
        torch.cuda.empty_cache()
    for l in range(L):
        ctx.set_layer_weights(l, case.w_uk, case.w_uv, case.w_type, case.norm_w)
    seqs = []
    for b, n in enumerate(lens):
        s = ctx.seq_create()
        for l in range(L):
            ctx.write_rows(l, s, 0, _dev(torch, case.caches[b][:n]))
        ctx.advance_seq_len(s, n)
        seqs.append(s)
    rng = np.random.default_rng(2)
    kv = synth.to_bits(rng.standard_normal((L, 10, 576), np.float32), dt)          # five new tokens each
    q = synth.to_bits(rng.standard_normal((L, 10, H, 192), np.float32) * np.float32(0.9), dt)
    out = torch.zeros((L, 10, H, 128), dtype=torch.int16, device="cuda")
    before = ctx.launch_count()
    ctx.step_begin(seqs, [5, 5])
    ctx.step_layers(0, L, _dev(torch, kv), _dev(torch, q), out)
    ctx.step_end()
    assert ctx.status() == 0 and ctx.launch_count() - before == 3 * L          # layer by layer
    for l in (0, L - 1):
        for b, n in enumerate(lens):
            rows = oracle.append_rows(kv[l, 5 * b:5 * b + 5], list(range(n, n + 5)), case.norm_w, YARN["rms_norm_eps"], 40.0, 4096, 10000.0, dt)
            cache = np.concatenate([case.caches[b][:n], rows])
            for t in range(5):
                want = oracle.attention(q[l, 5 * b + t], cache, n + t + 1, case.w_uk, case.w_uv, case.w_type, H, dt)
                check_close(_host(out[l, 5 * b + t]), want, dt, f"layer {l}, sequence {b}, token {t}")
    ctx.close()


@pytest.mark.parametrize("room, groups", [(12 << 30, 1), (1 << 29, 3)])
def test_what_else_is_on_the_device_does_not_change_the_groups(torch, room, groups):
    """A context made with `room` bytes of the device left behind it, beside one with all of it: 27 layers of 101 rows are one group
    whether 12 or 180 GB are free, and give the same bits.  Only where less than a gigabyte is left the groups are smaller."""
    make = lambda: _step_ctx(torch, L=27, lens=[(29 * i) % 150 for i in range(101)])
    outs = []
    for full in (False, True):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        if full:
            filler = torch.empty(torch.cuda.mem_get_info()[0] - need - room, dtype=torch.uint8, device="cuda")
        else:
            free = torch.cuda.mem_get_info()[0]
        ctx, seqs, lens, kv, q = make()
        if full:
            del filler
            torch.cuda.empty_cache()
        else:
            torch.cuda.synchronize()
            need = free - torch.cuda.mem_get_info()[0]
        out = torch.zeros((27, 101, 16, 128), dtype=torch.int16, device="cuda")
        before = ctx.launch_count()
        ctx.step_begin(seqs)
        ctx.step_layers(0, 27, kv, q, out)
        ctx.step_end()
        assert ctx.status() == 0 and ctx.launch_count() - before == 3 * (groups if full else 1)
        outs.append(_host(out))
        ctx.close()
    if groups == 1:
        assert np.array_equal(outs[0], outs[1])
    for l in (0, 13, 26):
        check_close(outs[1][l], outs[0][l], synth.DT_F16, f"layer {l}")


@pytest.mark.parametrize("n_seq, pages", [(1, 1), (85, 1), (86, 1), (300, 1), (40, 120)])
def test_step_metadata_of_any_size_reaches_the_kernels(torch, n_seq, pages):
    """The metadata goes up in pieces of 16 bytes, 1,024 to a block: a step of many rows, or of many pages, writes the same cache rows
    as the same tokens one sequence to a step, whose metadata is a piece or two, and again when the steps follow each other at once."""
    from mugen_b200.mla import MlaContext
    rng = np.random.default_rng(n_seq)
    norm = synth.to_bits(rng.standard_normal(512, np.float32), synth.DT_F16)
    w = synth.to_bits(rng.standard_normal((16 * 128, 512), np.float32), synth.DT_F16)
    kv = _dev(torch, synth.to_bits(rng.standard_normal((3, n_seq, 576), np.float32), synth.DT_F16))
    rows = []
    for together in (True, False):
        ctx = MlaContext(n_layers=1, n_heads=16, dtype=synth.DT_F16, n_pages=n_seq * (pages + 1), max_seqs=n_seq, max_seq_len=64 * pages + 8, **YARN)
        ctx.set_layer_weights(0, w, w, synth.W_F16, norm)
        seqs = [ctx.seq_create() for _ in range(n_seq)]
        start = torch.zeros((64 * pages - 1, 576), dtype=torch.int16, device="cuda")
        for s in seqs:
            ctx.write_rows(0, s, 0, start)
            ctx.advance_seq_len(s, 64 * pages - 1)
        for t in range(3):
            for some in [slice(None)] if together else [slice(i, i + 1) for i in range(n_seq)]:
                ctx.step_begin(seqs[some])
                ctx.step_append(0, kv[t, some].contiguous())
                ctx.step_end()
        assert ctx.status() == 0
        rows.append(np.stack([ctx.read_rows(0, s, 64 * pages - 1, 3) for s in seqs]))
        ctx.close()
    assert np.array_equal(rows[0], rows[1]) and rows[0].any(axis=(1, 2)).all()


@pytest.mark.parametrize("H,dt,L,rows,groups", [
    (5, synth.DT_F16, 27, 60, 1),          # 1,620 rows
    (16, synth.DT_BF16, 27, 101, 1),       # 2,727
    (5, synth.DT_BF16, 9, 455, 1),         # 4,095 of the 4,096 that a group may have
    (5, synth.DT_BF16, 9, 456, 2),         # 4,104: five layers and four
    (64, synth.DT_BF16, 5, 273, 1),        # 1,365 rows of 73,728 bytes: as many as 96 MB of queries hold
    (64, synth.DT_F16, 5, 274, 2),         # 1,370: three layers and two
    (128, synth.DT_BF16, 3, 227, 1),       # 681 of 682
    (128, synth.DT_BF16, 3, 228, 2),       # 684: two layers and one
])
def test_groups_of_layers_of_thousands_of_rows(torch, monkeypatch, H, dt, L, rows, groups):
    from mugen_b200.mla import MlaContext
    launches, step_layers = [], MlaContext.step_layers

    def counted(ctx, *args):
        before = ctx.launch_count()
        step_layers(ctx, *args)
        launches.append(ctx.launch_count() - before)

    monkeypatch.setattr(MlaContext, "step_layers", counted)
    test_step_layers_in_groups_of_layers(torch, H, dt, L, [(29 * i) % 150 for i in range(rows)])
    assert launches == [3 * groups]                # absorb, attention, merge
