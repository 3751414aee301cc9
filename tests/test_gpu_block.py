"""The projections around the attention op (mla_set_block_weights, mla_block_project_in / _out, mla_step_block):
steps A-D, F, J, K of the reference's MLA decode driver (src/core/model/transformer.cpp:3849-3929, 4002-4015).

Two oracles.  (1) The recorded trace of the reference's own forward() on a tiny deepseek2 model (tests/golden, "block"
entries; the model is re-created here from its seed): what went into and came out of every layer's attention block at
every position.  (2) A plain numpy restatement of the reference's kernels for the DeepSeek-V3 projection shapes:
matvec = float accumulation rounded once to the storage type, rms_norm = x * rsqrt(mean(x^2) + eps) * w rounded once,
residual = sum rounded once (src/metal/kernel_sources.h:55-98, 264-312, 357-366).  The tensor core adds the products
in another order than the reference's lanes, so results are compared within a tolerance, stated below."""
import base64
import os
import sys

import numpy as np
import pytest

from mugen_b200 import capi, synth

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import tiny_gguf  # noqa: E402

pytestmark = pytest.mark.gpu
# a projection output is one rounding of a float sum: two correct implementations differ by at most one unit in the last
# place of a few elements.  max-abs is relative to the tensor's largest magnitude.
REL_L2, MAX_REL = 2e-3, 1.6e-2


@pytest.fixture(scope="module")
def torch():
    import torch
    assert torch.cuda.is_available()
    return torch


def _dev(torch, bits):
    return torch.from_numpy(np.ascontiguousarray(bits).view(np.int16)).cuda()


def _bits(t):
    return t.cpu().numpy().view(np.uint16)


def _close(got, want, dt, what):
    g, w = synth.from_bits(got, dt).astype(np.float64).ravel(), synth.from_bits(want, dt).astype(np.float64).ravel()
    rl = np.sqrt(((g - w) ** 2).sum()) / max(np.sqrt((w ** 2).sum()), 1e-30)
    mx = np.abs(g - w).max() / max(np.abs(w).max(), 1e-30)
    assert rl <= REL_L2 and mx <= MAX_REL, f"{what}: rel-L2 {rl:.2e}, max/peak {mx:.2e}"


def _unb(t):
    return np.frombuffer(base64.b64decode(t), np.uint16).copy()


def test_block_trace_of_the_reference_forward(torch, golden):
    from mugen_b200.mla import MlaContext
    blk = golden["block"]
    m = tiny_gguf.TinyModel(**blk["model"])
    tiny_gguf.build(m)
    f16 = lambda name: np.frombuffer(m.tensors[name][2], np.float16 if m.tensors[name][0] == 1 else np.float32).astype(np.float16).view(np.uint16).reshape(m.tensors[name][1][::-1])
    H, E, L, dt = m.n_heads, m.embed, m.n_layers, synth.DT_F16
    ctx = MlaContext(n_layers=L, n_heads=H, dtype=dt, n_pages=4, max_seqs=L, max_seq_len=64, rope_theta=m.rope_theta,
                     rope_scaling_factor=m.rope_factor, rope_original_ctx=m.rope_orig_ctx, rms_norm_eps=m.eps)
    for l in range(L):
        b = f"blk.{l}."
        ctx.set_layer_weights(l, f16(b + "attn_k_b.weight"), f16(b + "attn_v_b.weight"), synth.W_F16, f16(b + "attn_kv_a_norm.weight"))
        ctx.set_block_weights(l, attn_norm=f16(b + "attn_norm.weight"), q_a=f16(b + "attn_q_a.weight"),
                              q_a_norm=f16(b + "attn_q_a_norm.weight"), q_b=f16(b + "attn_q_b.weight"),
                              kv_a_mqa=f16(b + "attn_kv_a_mqa.weight"), wo=f16(b + "attn_output.weight"))
    ctx.set_q_rope(True)
    # one sequence per layer: the layers of the reference share a position counter but not a cache, and here every
    # layer is replayed from its own recorded input (the FFN between the blocks is not part of this library)
    seqs = [ctx.seq_create() for _ in range(L)]
    for pos, step in enumerate(blk["steps"]):
        taps = {k: _unb(v) for k, v in step.items()}
        for l in range(L):
            hidden_in = taps["hidden_in"].reshape(L, E)[l]
            # the pieces
            q = torch.zeros((1, H, 192), dtype=torch.int16, device="cuda")
            kv = torch.zeros((1, 576), dtype=torch.int16, device="cuda")
            ctx.block_project_in(l, _dev(torch, hidden_in[None]), q, kv)
            _close(_bits(q)[0], taps["q_pre"].reshape(L, H, 192)[l], dt, f"q, layer {l}, position {pos}")
            _close(_bits(kv)[0], taps["kv_a_pre"].reshape(L, 576)[l], dt, f"kv_a, layer {l}, position {pos}")
            h2 = _dev(torch, hidden_in[None].copy())
            ctx.block_project_out(l, _dev(torch, taps["attn_out"].reshape(L, 1, H, 128)[l]), h2)
            _close(_bits(h2)[0], taps["hidden_mid"].reshape(L, E)[l], dt, f"Wo + residual, layer {l}, position {pos}")
            # the whole block through the step interface: hidden in -> hidden out, cache growing by one row per position
            h = _dev(torch, hidden_in[None].copy())
            ctx.step_begin([seqs[l]])
            ctx.step_block(l, h)
            ctx.step_end()
            _close(_bits(h)[0], taps["hidden_mid"].reshape(L, E)[l], dt, f"whole block, layer {l}, position {pos}")
    assert ctx.status() == 0 and [ctx.seq_len(s) for s in seqs] == [len(blk["steps"])] * L
    ctx.close()


def _np_project(x_bits, w_bits, dt):
    y = synth.from_bits(x_bits, dt).astype(np.float32) @ synth.from_bits(w_bits, dt).astype(np.float32).T
    return synth.to_bits(y, dt)


def _np_rmsnorm(x_bits, w_bits, eps, dt):
    x = synth.from_bits(x_bits, dt).astype(np.float32)
    inv = 1.0 / np.sqrt((x * x).mean(axis=-1, keepdims=True) + np.float32(eps))
    return synth.to_bits(x * inv * synth.from_bits(w_bits, dt).astype(np.float32), dt)


@pytest.mark.parametrize("dt,rows,H,E,R", [(synth.DT_BF16, 64, 128, 7168, 1536),      # DeepSeek-V3 attention block, batch 64
                                           (synth.DT_F16, 32, 16, 2048, 0),           # V2-Lite: full q projection
                                           (synth.DT_BF16, 5, 8, 264, 72)])           # ragged sizes: tiles cut by M, N and K
def test_projection_shapes_against_numpy_restatement(torch, dt, rows, H, E, R):
    from mugen_b200.mla import MlaContext
    rng = np.random.default_rng(E + R)
    rnd = lambda shape, s: synth.to_bits((rng.standard_normal(shape) * s).astype(np.float32), dt)
    w = dict(attn_norm=synth.to_bits((1 + 0.1 * rng.standard_normal(E)).astype(np.float32), dt), kv_a_mqa=rnd((576, E), E ** -0.5),
             wo=rnd((E, H * 128), (H * 128) ** -0.5))
    if R:
        w.update(q_a=rnd((R, E), E ** -0.5), q_a_norm=synth.to_bits((1 + 0.1 * rng.standard_normal(R)).astype(np.float32), dt),
                 q_b=rnd((H * 192, R), R ** -0.5))
    else:
        w.update(q=rnd((H * 192, E), E ** -0.5))
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=dt, n_pages=2, max_seqs=1, max_seq_len=64, rms_norm_eps=1e-6)
    ctx.set_block_weights(0, **w)
    hidden = rnd((rows, E), 1.0)
    q = torch.zeros((rows, H, 192), dtype=torch.int16, device="cuda")
    kv = torch.zeros((rows, 576), dtype=torch.int16, device="cuda")
    ctx.block_project_in(0, _dev(torch, hidden), q, kv)
    h2 = _np_rmsnorm(hidden, w["attn_norm"], 1e-6, dt)
    if R:
        want_q = _np_project(_np_rmsnorm(_np_project(h2, w["q_a"], dt), w["q_a_norm"], 1e-6, dt), w["q_b"], dt)
    else:
        want_q = _np_project(h2, w["q"], dt)
    _close(_bits(q).reshape(rows, -1), want_q, dt, "q")
    _close(_bits(kv), _np_project(h2, w["kv_a_mqa"], dt), dt, "kv_a")
    attn = rnd((rows, H, 128), 0.05)
    hid = _dev(torch, hidden.copy())
    ctx.block_project_out(0, _dev(torch, attn), hid)
    wo_out = synth.from_bits(_np_project(attn.reshape(rows, -1), w["wo"], dt), dt)
    want_h = synth.to_bits(synth.from_bits(hidden, dt).astype(np.float32) + wo_out, dt)
    _close(_bits(hid), want_h, dt, "Wo + residual")
    assert ctx.status() == 0
    ctx.close()


@pytest.mark.parametrize("rows,H,E,R,shift", [
    (1, 5, 72, 0, 0),               # a k-block of 8 values behind a whole one; outputs off every tile
    (16, 16, 2048, 0, 0), (17, 16, 2048, 0, 4),       # the widths of gemm_rows_kernel and one row more; outputs off 16 bytes
    (33, 5, 1000, 200, 0), (65, 16, 520, 64, 0), (128, 3, 2048, 0, 1),
    (129, 16, 2048, 0, 0),          # SM pairs: a second tile of one row ...
    (256, 5, 72, 0, 4), (257, 128, 1000, 136, 0), (700, 16, 2048, 0, 0),
])
def test_projections_at_the_edges_of_their_tiles(torch, rows, H, E, R, shift):
    """Both projection kernels against float64 of the same rounded operands: norms and q_a are rounded to fp16 as the reference
    rounds them, so what remains is one rounding per output (2^-11 at most, 2.9e-4 in the mean square), a few last places
    of the normalised rows that fall the other way, and in the residual a second rounding: rel-L2 1e-3."""
    from mugen_b200.mla import MlaContext
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows * 7 + E)
    rn = lambda *shape, scale=1.0: (torch.randn(shape, device="cuda", generator=gen) * scale).half()
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    eps, QD, VD = 1e-6, H * 192, H * 128
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=synth.DT_F16, n_pages=2, max_seqs=1, max_seq_len=64, rope_theta=1e4,
                     rope_scaling_factor=1.0, rope_original_ctx=4096, rms_norm_eps=eps)
    w = dict(attn_norm=1 + rn(E, scale=0.1), kv_a_mqa=rn(576, E, scale=E ** -0.5), wo=rn(E, VD, scale=VD ** -0.5))
    w.update(dict(q_a=rn(R, E, scale=E ** -0.5), q_a_norm=1 + rn(R, scale=0.1), q_b=rn(QD, R, scale=R ** -0.5)) if R
             else dict(q=rn(QD, E, scale=E ** -0.5)))
    ctx.set_block_weights(0, **{k: bits(v) for k, v in w.items()})

    def at(n_cols):                 # an output that starts `shift` values behind a 16-byte boundary
        return torch.zeros(rows * n_cols + 8, dtype=torch.float16, device="cuda")[shift:shift + rows * n_cols].view(rows, n_cols)

    def norm(x, g):
        return (x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + eps) * g.double()).half()

    def close(got, want, what):
        e = (got.double() - want).norm() / want.norm()
        assert e <= 1e-3, f"{what}: rel-L2 {e:.2e}"

    hidden, q, kv = rn(rows, E), at(QD), at(576)
    ctx.block_project_in(0, hidden, q, kv)
    x = norm(hidden, w["attn_norm"])
    a = x
    if R:
        a = norm((x.double() @ w["q_a"].double().T).half(), w["q_a_norm"])
    close(q, a.double() @ (w["q_b"] if R else w["q"]).double().T, "q")
    close(kv, x.double() @ w["kv_a_mqa"].double().T, "kv_a")
    att, out = rn(rows, VD), at(E)
    out.copy_(hidden)
    ctx.block_project_out(0, att, out)
    close(out, hidden.double() + (att.double() @ w["wo"].double().T).half().double(), "hidden")
    assert ctx.status() == 0
    ctx.close()


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("rows,H,E,R,shift", [
    (1, 5, 72, 0, 0), (16, 16, 2048, 0, 0), (17, 16, 520, 64, 4), (33, 5, 1000, 200, 0), (65, 3, 520, 0, 1), (128, 3, 2048, 0, 8),
    (129, 16, 2048, 0, 0), (256, 5, 72, 0, 4), (257, 64, 1000, 136, 0), (700, 16, 2048, 0, 8),
    # the order of the tiles, Wo: two by two with one over; one by one; 9 tiles of rows side by side, the last one of 252 rows
    (1100, 72, 520, 0, 0), (600, 80, 520, 0, 0), (2300, 3, 1032, 0, 0),
    # outputs off a 16-byte boundary in both widths of tile, in whole runs and cut ones
    (1100, 72, 520, 0, 4), (777, 16, 2048, 0, 1),
    # cut tiles ahead of a round of whole ones: the input projections, with TMA and without; the output projection
    (1300, 16, 5120, 0, 0), (1500, 16, 5120, 0, 4), (2000, 48, 3072, 0, 0),
])
def test_every_output_of_the_projections_and_nothing_beside_them(torch, rows, H, E, R, shift, dt):
    """Element by element against float64, and the values in front of and behind each output untouched.  An output is one rounding
    of a float sum (u = 2^-11 or 2^-8 of it) over operands that were rounded to the storage type: a normalised value or a q_a
    that falls the other way (u of ITS magnitude, independent) moves an output by about u * |x| * |w|, here with |w| = 1 / sqrt(K)
    and |x| near 1 by u in the mean square; six of those beside one rounding (two in the residual) hold every element."""
    from mugen_b200.mla import MlaContext
    tdt, code, u = (torch.float16, synth.DT_F16, 2.0 ** -11) if dt == "f16" else (torch.bfloat16, synth.DT_BF16, 2.0 ** -8)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows * 11 + E)
    rn = lambda *shape, scale=1.0: (torch.randn(shape, device="cuda", generator=gen) * scale).to(tdt)
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    eps, QD, VD, pad, mark = 1e-6, H * 192, H * 128, 256, 0x7BAD
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=code, n_pages=2, max_seqs=1, max_seq_len=64, rope_theta=1e4,
                     rope_scaling_factor=1.0, rope_original_ctx=4096, rms_norm_eps=eps)
    w = dict(attn_norm=1 + rn(E, scale=0.1), kv_a_mqa=rn(576, E, scale=E ** -0.5), wo=rn(E, VD, scale=VD ** -0.5))
    w.update(dict(q_a=rn(R, E, scale=E ** -0.5), q_a_norm=1 + rn(R, scale=0.1), q_b=rn(QD, R, scale=R ** -0.5)) if R
             else dict(q=rn(QD, E, scale=E ** -0.5)))
    ctx.set_block_weights(0, **{k: bits(v) for k, v in w.items()})
    whole = {}

    def at(what, n_cols):
        whole[what] = torch.full((pad + shift + rows * n_cols + pad,), mark, dtype=torch.int16, device="cuda")
        return whole[what].view(tdt)[pad + shift:pad + shift + rows * n_cols].view(rows, n_cols)

    def norm(x, g):
        return (x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + eps) * g.double()).to(tdt)

    def close(got, want, what, roundings=1):
        bad = (got.double() - want).abs() > u * (roundings * want.abs() + 6)
        assert not bad.any(), f"{what}: {int(bad.sum())} elements, the first at {bad.nonzero()[0].tolist()}"
        buf = whole[what]
        assert (buf[:pad + shift] == mark).all() and (buf[pad + shift + got.numel():] == mark).all(), f"{what}: written beside the output"

    hidden, q, kv = rn(rows, E), at("q", QD), at("kv_a", 576)
    ctx.block_project_in(0, hidden, q, kv)
    x = norm(hidden, w["attn_norm"])
    a = norm((x.double() @ w["q_a"].double().T).to(tdt), w["q_a_norm"]) if R else x
    close(q, a.double() @ (w["q_b"] if R else w["q"]).double().T, "q")
    close(kv, x.double() @ w["kv_a_mqa"].double().T, "kv_a")
    att, out = rn(rows, VD), at("hidden", E)
    out.copy_(hidden)
    ctx.block_project_out(0, att, out)
    close(out, hidden.double() + (att.double() @ w["wo"].double().T).to(tdt).double(), "hidden", 2)
    assert ctx.status() == 0
    ctx.close()


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("rows,H,E,R", [
    (1, 1, 64, 0), (2, 2, 1024, 0), (3, 2, 1032, 8), (4, 5, 2048, 0), (5, 16, 4096, 512), (8, 5, 72, 64), (9, 16, 2048, 0), (16, 4, 7168, 1536),
    (17, 2, 1024, 0), (24, 5, 520, 200), (31, 2, 4096, 136), (32, 16, 2048, 0),
    (8, 64, 4096, 512), (4, 64, 1024, 0),          # single blocks of 8 and of 16 k-blocks
    (16, 4, 7168, 1024),                           # 14 k-blocks per block of a cluster of 8
])
def test_projections_of_few_rows_in_every_cluster_size(torch, rows, H, E, R, dt):
    """Clusters of 1, 2, 4 and 8 blocks per tile, shared and whole rows per warp, k-blocks that end early.  The operands of one row
    go to no other: the rows of a call equal, bit for bit, the same rows of a call with other rows beside them, where both calls
    have rows of the same number per warp; and every output is within the bounds of the test above.  That the input projections
    ran in this kernel shows in the launches: the norm is not one of them."""
    from mugen_b200.mla import MlaContext
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows * 13 + E)
    tdt, code, u = (torch.float16, synth.DT_F16, 2.0 ** -11) if dt == "f16" else (torch.bfloat16, synth.DT_BF16, 2.0 ** -8)
    rn = lambda *shape, scale=1.0: (torch.randn(shape, device="cuda", generator=gen) * scale).to(tdt)
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    eps, QD, VD = 1e-6, H * 192, H * 128
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=code, n_pages=2, max_seqs=1, max_seq_len=64, rope_theta=1e4,
                     rope_scaling_factor=1.0, rope_original_ctx=4096, rms_norm_eps=eps)
    w = dict(attn_norm=1 + rn(E, scale=0.1), kv_a_mqa=rn(576, E, scale=E ** -0.5), wo=rn(E, VD, scale=VD ** -0.5))
    w.update(dict(q_a=rn(R, E, scale=E ** -0.5), q_a_norm=1 + rn(R, scale=0.1), q_b=rn(QD, R, scale=R ** -0.5)) if R
             else dict(q=rn(QD, E, scale=E ** -0.5)))
    ctx.set_block_weights(0, **{k: bits(v) for k, v in w.items()})
    norm = lambda x, g: (x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + eps) * g.double()).to(tdt)

    def run(hidden, att):
        q, kv, out = torch.zeros((len(hidden), QD), device="cuda").to(tdt), torch.zeros((len(hidden), 576), device="cuda").to(tdt), hidden.clone()
        ctx.block_project_in(0, hidden, q, kv)
        ctx.block_project_out(0, att, out)
        return q, kv, out

    hidden, att = rn(rows, E), rn(rows, VD)
    before = ctx.launch_count()
    q, kv, out = run(hidden, att)
    if (E, R) != (7168, 1536):               # 17 tiles of 112 k-blocks: a device holds 17 clusters of 8, or the call goes elsewhere
        assert ctx.launch_count() - before == (3 if R else 2)
    x = norm(hidden, w["attn_norm"])
    a = norm((x.double() @ w["q_a"].double().T).to(tdt), w["q_a_norm"]) if R else x
    for got, want, n in ((q, a.double() @ (w["q_b"] if R else w["q"]).double().T, 1), (kv, x.double() @ w["kv_a_mqa"].double().T, 1),
                         (out, hidden.double() + (att.double() @ w["wo"].double().T).to(tdt).double(), 2)):
        assert not ((got.double() - want).abs() > u * (n * want.abs() + 6)).any()
    other_hidden, other_att = rn(rows, E, scale=30.0), rn(rows, VD, scale=30.0)
    other_hidden[rows // 2], other_att[rows // 2] = hidden[rows // 2], att[rows // 2]
    for got, want in zip(run(other_hidden, other_att), (q, kv, out)):
        assert torch.equal(got[rows // 2], want[rows // 2])
    # an output over the rows themselves: they are read before it is written
    if not R and QD <= E:
        buf = hidden.clone()
        ctx.block_project_in(0, buf, buf.view(-1)[:rows * QD], kv)
        assert not ((buf.view(-1)[:rows * QD].view(rows, QD).double() - a.double() @ w["q"].double().T).abs() > u * ((a.double() @ w["q"].double().T).abs() + 6)).any()
    assert ctx.status() == 0
    ctx.close()


@pytest.mark.parametrize("rows,H,E,R,dt", [
    (4, 64, 1024, 0, "bf16"),            # Wo: 16 k-blocks per block in clusters of 8
    (16, 32, 4096, 512, "f16"),          # Wo: 16 in clusters of 4
    (9, 16, 7168, 1536, "bf16"),         # Wo: 16 in clusters of 2; q_a and kv_a: 14 where 17 clusters of 8 are resident
    (16, 16, 7168, 1536, "f16"),
])
def test_projections_of_few_rows_whose_weight_ring_comes_round(torch, rows, H, E, R, dt):
    """10 to 16 k-blocks per block: every stage of the weight ring is used again (which issuer may then wait for it is tested on the
    CPU, tests/host).  Six layers, launched as close as launches can follow each other, must leave the bits that the same calls leave
    with the device idle before each; and one call's outputs are those of float64."""
    from mugen_b200.mla import MlaContext
    tdt, code, u = (torch.float16, synth.DT_F16, 2.0 ** -11) if dt == "f16" else (torch.bfloat16, synth.DT_BF16, 2.0 ** -8)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows * 17 + E)
    rn = lambda *shape, scale=1.0: (torch.randn(shape, device="cuda", generator=gen) * scale).to(tdt)
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    L, QD, VD, eps = 6, H * 192, H * 128, 1e-6
    ctx = MlaContext(n_layers=L, n_heads=H, dtype=code, n_pages=2, max_seqs=1, max_seq_len=64, rope_theta=1e4,
                     rope_scaling_factor=1.0, rope_original_ctx=4096, rms_norm_eps=eps)
    g, ga = 1 + rn(E, scale=0.1), 1 + rn(max(R, 8), scale=0.1)
    kv_w = [rn(576, E, scale=E ** -0.5) for _ in range(L)]
    wo = [rn(E, VD, scale=VD ** -0.5) for _ in range(L)]
    q_w = rn(QD, R or E, scale=(R or E) ** -0.5)
    for l in range(L):
        more = dict(q_a=bits(rn(R, E, scale=E ** -0.5)), q_a_norm=bits(ga), q_b=bits(q_w)) if R else dict(q=bits(q_w))
        ctx.set_block_weights(l, attn_norm=bits(g), kv_a_mqa=bits(kv_w[l]), wo=bits(wo[l]), **more)
    hidden, att = rn(rows, E), rn(rows, VD)
    q, kv, out = torch.zeros((L, rows, QD), device="cuda", dtype=tdt), torch.zeros((L, rows, 576), device="cuda", dtype=tdt), hidden.clone()

    def calls(between):
        for l in range(L):
            ctx.block_project_in(l, hidden, q[l], kv[l])
            between()
        for l in range(L):
            ctx.block_project_out(l, att, out)
            between()

    calls(torch.cuda.synchronize)
    want = [t.clone() for t in (q, kv, out)]
    x = (hidden.double() * torch.rsqrt((hidden.double() ** 2).mean(-1, keepdim=True) + eps) * g.double()).to(tdt)
    for l in range(L):                       # the bounds of the element-by-element test above
        ref = x.double() @ kv_w[l].double().T
        assert not ((kv[l].double() - ref).abs() > u * (ref.abs() + 6)).any()
    one = hidden.clone()
    ctx.block_project_out(0, att, one)
    ref = hidden.double() + (att.double() @ wo[0].double().T).to(tdt).double()
    assert not ((one.double() - ref).abs() > u * (2 * ref.abs() + 6)).any()
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        calls(lambda: None)
    for _ in range(50):
        q.zero_(), kv.zero_(), out.copy_(hidden)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        for got, w in zip((q, kv, out), want):
            assert torch.equal(got, w)
    assert ctx.status() == 0
    del graph
    ctx.close()


@pytest.mark.parametrize("rows,H,E,R,launches", [
    (1, 16, 2048, 0, 1), (32, 16, 2048, 0, 1), (33, 16, 2048, 0, 2),
    (32, 16, 4096, 512, 2),              # q_b in clusters of 4
    (8, 64, 4096, 512, 2),               # q_b: 96 tiles, single blocks, up to 8 rows
    (9, 64, 4096, 512, 3), (32, 64, 4096, 512, 3),
    (32, 128, 7168, 1536, 4),            # more k-blocks than a block holds, more tiles than SMs
])
def test_which_input_projections_take_the_kernel_for_few_rows(torch, rows, H, E, R, launches):
    """That kernel normalises the rows itself; the general one has the norm as a launch ahead of it."""
    from mugen_b200.mla import MlaContext
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=synth.DT_F16, n_pages=2, max_seqs=1, max_seq_len=64)
    one = lambda *shape: np.full(shape, 0x3C00 if len(shape) == 1 else 0x2000, np.uint16)
    w = dict(attn_norm=one(E), kv_a_mqa=one(576, E), wo=one(E, H * 128))
    w.update(dict(q_a=one(R, E), q_a_norm=one(R), q_b=one(H * 192, R)) if R else dict(q=one(H * 192, E)))
    ctx.set_block_weights(0, **w)
    q, kv = (torch.zeros((rows, n), device="cuda", dtype=torch.float16) for n in (H * 192, 576))
    before = ctx.launch_count()
    ctx.block_project_in(0, torch.ones((rows, E), device="cuda", dtype=torch.float16), q, kv)
    assert ctx.launch_count() - before == launches
    # all values equal: a row of ones is its own norm, and an output the sum of its weights (0x2000 = 2^-7), of twice the roundings
    a = E * 2.0 ** -7
    want = R * 2.0 ** -7 if R else a                       # q_a's rows are equal values again: the norm makes ones of them
    assert (kv.double() - a).abs().max() <= a * 2.0 ** -10 and (q.double() - want).abs().max() <= want * 2.0 ** -9
    assert ctx.status() == 0
    ctx.close()


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("rows,E", [(40, 2048), (777, 2048), (40, 2056), (1300, 4096), (40, 8192), (40, 8200), (33, 72)])
def test_the_norm_ahead_of_a_projection_in_every_block_shape(torch, rows, E, dt):
    """Blocks of 256 threads with one piece or four, of 512 with four and more: the kv_a rows are unit vectors, so that its outputs are
    the normalised values themselves.  They are one rounding of a value whose float error (a sum of E squares, two products, a
    reciprocal root of two units in the last place) is below 2^-17 of it."""
    from mugen_b200.mla import MlaContext
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows + E)
    tdt, code, u = (torch.float16, synth.DT_F16, 2.0 ** -11) if dt == "f16" else (torch.bfloat16, synth.DT_BF16, 2.0 ** -8)
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    ctx = MlaContext(n_layers=1, n_heads=1, dtype=code, n_pages=2, max_seqs=1, max_seq_len=64, rope_theta=1e4, rope_scaling_factor=1.0,
                     rope_original_ctx=4096, rms_norm_eps=1e-6)
    at = torch.linspace(0, E - 1, 576).long() if E >= 576 else torch.arange(576) % E
    unit = torch.zeros((576, E), dtype=tdt)
    unit[torch.arange(576), at] = 1.0
    zeros = torch.zeros((192, E), dtype=tdt)
    g = (1.0 + 0.1 * torch.randn((E,), device="cuda", generator=gen)).to(tdt)
    ctx.set_block_weights(0, attn_norm=bits(g), kv_a_mqa=bits(unit), wo=bits(torch.zeros((E, 128), dtype=tdt)), q=bits(zeros))
    hidden = (torch.randn((rows, E), device="cuda", generator=gen) * torch.logspace(-2, 2, rows, device="cuda")[:, None]).to(tdt)
    q, kv = torch.zeros((rows, 192), device="cuda").to(tdt), torch.zeros((rows, 576), device="cuda").to(tdt)
    before = ctx.launch_count()
    ctx.block_project_in(0, hidden, q, kv)
    assert ctx.launch_count() - before == 2 and ctx.status() == 0
    x = hidden.double()
    want = (x * torch.rsqrt((x ** 2).mean(-1, keepdim=True) + 1e-6) * g.double())[:, at.cuda()]
    tiny = 2.0 ** -25 if dt == "f16" else 0.0                  # half a unit of the subnormal numbers
    assert not ((kv.double() - want).abs() > (u + 2.0 ** -17) * want.abs() + tiny).any()
    ctx.close()


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("rows", [1, 16, 17, 32, 33, 128])
@pytest.mark.parametrize("E", [64, 136, 200, 320, 704])
def test_projections_whose_tiles_have_fewer_k_blocks_than_issuers(torch, E, rows, dt):
    """The general kernel of up to 128 rows (155 tiles are more than the device has SMs, which the one for few rows does not take) with
    up to 32 rows deals a block's k-blocks out to three issuers with accumulators of their own: whole tiles of 1 to 11 k-blocks, and in
    the output projection tiles of 200 k-blocks cut into runs of a few, so that an issuer has none, one or several of a tile."""
    from mugen_b200.mla import MlaContext
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows * 17 + E)
    tdt, code, u = (torch.float16, synth.DT_F16, 2.0 ** -11) if dt == "f16" else (torch.bfloat16, synth.DT_BF16, 2.0 ** -8)
    H, QD, VD = 100, 19200, 12800
    rn = lambda *shape, scale=1.0: (torch.randn(shape, device="cuda", generator=gen) * scale).to(tdt)
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16)
    ctx = MlaContext(n_layers=1, n_heads=H, dtype=code, n_pages=2, max_seqs=1, max_seq_len=64, rope_theta=1e4, rope_scaling_factor=1.0,
                     rope_original_ctx=4096, rms_norm_eps=1e-6)
    w = dict(attn_norm=1 + rn(E, scale=0.1), kv_a_mqa=rn(576, E, scale=E ** -0.5), wo=rn(E, VD, scale=VD ** -0.5), q=rn(QD, E, scale=E ** -0.5))
    ctx.set_block_weights(0, **{k: bits(v) for k, v in w.items()})
    hidden, att = rn(rows, E), rn(rows, VD)
    q, kv, out = torch.zeros((rows, QD), device="cuda").to(tdt), torch.zeros((rows, 576), device="cuda").to(tdt), hidden.clone()
    before = ctx.launch_count()
    ctx.block_project_in(0, hidden, q, kv)
    ctx.block_project_out(0, att, out)
    assert ctx.status() == 0 and ctx.launch_count() - before == 3
    x = (hidden.double() * torch.rsqrt((hidden.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w["attn_norm"].double()).to(tdt).double()
    # one rounding of the output (two with the residual), and as the bound beside it six units of the storage type on sums of order one:
    # where the normalised rows round the other way than here
    for got, want, n in ((q, x @ w["q"].double().T, 1), (kv, x @ w["kv_a_mqa"].double().T, 1),
                         (out, hidden.double() + (att.double() @ w["wo"].double().T).to(tdt).double(), 2)):
        assert not ((got.double() - want).abs() > u * (n * want.abs() + 6)).any()
    q2, out2 = torch.zeros_like(q), hidden.clone()
    ctx.block_project_in(0, hidden, q2, kv)
    ctx.block_project_out(0, att, out2)
    assert torch.equal(q, q2) and torch.equal(out, out2)
    ctx.close()


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("rows,H,E,R", [
    (1, 2, 4096, 0), (1, 2, 4104, 0), (4, 2, 7168, 0), (8, 5, 6144, 136),         # up to 8 rows: whole rows up to 4,096 values, exchanged sums behind that
    (9, 2, 1016, 0), (9, 2, 1024, 0), (16, 5, 2048, 0), (16, 2, 2056, 256),       # up to 16: whole up to 2,048
    (17, 2, 1016, 0), (25, 2, 1032, 0), (32, 5, 2048, 1024), (31, 2, 2056, 0),    # up to 32
    (10, 3, 1032, 72), (16, 5, 4096, 264), (18, 2, 2048, 1016), (32, 5, 2056, 264),      # short rows of q_a: as the projection before
])
def test_projections_of_few_rows_in_every_form_of_the_norm(torch, rows, H, E, R, dt):
    test_projections_of_few_rows_in_every_cluster_size(torch, rows, H, E, R, dt)
