"""Block-level parity on the GPU: B200Block / B200FrameAttention against outputs recorded from the reference's
FlashInferBlock (paged fp32 path), SDPABlock and Attention on CPU (tests/golden/*.npz).

Weights are fp32 and the Linear layers run in fp32; q/k/v are rounded to bf16 by the CUDA prologue, attention runs
on bf16 tensor cores.  Tolerance on block outputs: 2e-2 max-abs and cosine >= 0.9999 (float64)."""
import os

import numpy as np
import pytest
import torch

import seeded
import lingbot_map_b200 as P

pytestmark = pytest.mark.gpu
G = os.path.join(os.path.dirname(__file__), "golden")
DEV = "cuda:0"


class Rope2dStub:
    """Carries the base frequency the way RotaryPositionEmbedding2D does (rope.py:81-86)."""
    base_frequency = 100.0


def close(got, want, tag, max_abs=2e-2, cos=0.9999):
    g = got.double().cpu().numpy().ravel()
    w = np.asarray(want, np.float64).ravel()
    c = float(g @ w / (np.linalg.norm(g) * np.linalg.norm(w)))
    d = float(np.abs(g - w).max())
    assert np.isfinite(g).all() and d <= max_abs and c >= cos, f"{tag}: max_abs={d:.3e} cosine={c:.7f}"


def rope3d_pos(f_start, n_frames, pph, ppw, ns):
    """Complex frequency tensor [1,1,N,32] as WanRotaryPosEmbed.forward returns it (rope.py:336-425)."""
    from oracle import gct_oracle as O
    ang = np.concatenate([O.rope3d_angles(f, pph, ppw, ns) for f in range(f_start, f_start + n_frames)], axis=0)
    z = torch.polar(torch.ones(ang.shape, dtype=torch.float64), torch.from_numpy(ang))
    return z[None, None].to(DEV)


@pytest.mark.parametrize("kf", [2, 1])
def test_block_stream_matches_reference(kf):
    z = np.load(os.path.join(G, "block_stream_fp32.npz"))
    dim, H, pph, ppw, ns, scale, window = 128, 2, 3, 4, 6, 2, 3
    Ptok = ns + pph * ppw
    blk = P.B200Block(dim=dim, num_heads=H, init_values=0.01, qk_norm=True, rope=Rope2dStub(),
                      kv_cache_sliding_window=window, kv_cache_scale_frames=scale).eval().to(DEV)
    seeded.fill_module_(blk, 21)
    mgr = P.B200KVCacheManager(num_blocks=1, max_num_frames=scale + window + 16, tokens_per_frame=Ptok, num_heads=H,
                               head_dim=64, dtype=torch.float32, device=DEV, scale_frames=scale,
                               sliding_window=window, max_total_frames=40)
    tag = f"paged_kf{kf}"
    kw = dict(num_patches=Ptok - ns, num_special=ns, enable_3d_rope=True, kv_cache=mgr, global_idx=0,
              num_frame_for_scale=scale, num_register_tokens=4)
    tfp = 0
    with torch.no_grad():
        x = torch.from_numpy(seeded.randn(500, 1, scale * Ptok, dim)).to(DEV)
        y = blk(x, pos=rope3d_pos(0, scale, pph, ppw, ns), num_frames=scale, num_frame_per_block=scale, **kw)
        close(y, z[f"{tag}_phase1"], "phase 1")
        tfp += scale
        for i in range(scale, scale + 8):
            is_kf = kf <= 1 or (i - scale) % kf == 0
            mgr._skip_append = not is_kf
            x = torch.from_numpy(seeded.randn(500 + i, 1, Ptok, dim)).to(DEV)
            y = blk(x, pos=rope3d_pos(tfp, 1, pph, ppw, ns), num_frames=1, num_frame_per_block=1, **kw)
            close(y, z[f"{tag}_frame{i}"], f"frame {i} ({'KF' if is_kf else 'non-KF'})")
            if is_kf:
                tfp += 1
    mgr._skip_append = False
    # page table and eviction decisions bit-exact with the reference run
    assert mgr.build_visible_page_table(0) == list(z[f"{tag}_visible_end"])
    assert mgr.compute_last_page_len(0) == int(z[f"{tag}_last_len_end"][0])
    assert mgr.device_status() == 0


def test_block_attn_pre_contract():
    """attn_pre returns (q, k, v) [tokens, H, 64] like block.py:217-227 and equals what the fused append writes."""
    dim, H, pph, ppw, ns = 128, 2, 3, 4, 6
    Ptok = ns + pph * ppw
    blk = P.B200Block(dim=dim, num_heads=H, init_values=0.01, qk_norm=True, rope=Rope2dStub()).eval().to(DEV)
    seeded.fill_module_(blk, 5)
    mgr = P.B200KVCacheManager(1, 21, Ptok, H, 64, device=DEV, scale_frames=2, sliding_window=3, max_total_frames=40)
    x = torch.from_numpy(seeded.randn(1, 1, Ptok, dim)).to(DEV)
    pos = rope3d_pos(3, 1, pph, ppw, ns)
    with torch.no_grad():
        q, k, v = blk.attn_pre(x, pos=pos, enable_3d_rope=True)
        blk(x, pos=pos, num_frames=1, enable_3d_rope=True, kv_cache=mgr, global_idx=0)
    assert q.shape == (Ptok, H, 64) and q.dtype == torch.bfloat16
    kk, vv = mgr._gather_kv(0)
    # cache order: patch page first, then the special page (flashinfer_cache.py:446-450)
    assert torch.equal(kk, torch.cat([k[ns:], k[:ns]])) and torch.equal(vv, torch.cat([v[ns:], v[:ns]]))


def test_frame_attention_matches_reference():
    z = np.load(os.path.join(G, "prepare_qkv_fp32.npz"))
    dim, H, pph, ppw, ns = 128, 2, 3, 4, 6
    N = ns + pph * ppw
    fa = P.B200FrameAttention(dim, num_heads=H, qk_norm=True, rope=Rope2dStub()).eval().to(DEV)
    seeded.fill_module_(fa, 11)
    x = torch.from_numpy(seeded.randn(123, 2, N, dim)).to(DEV)
    pos = torch.from_numpy(z["rope2d_pos"]).to(DEV)[None].expand(2, -1, -1)
    with torch.no_grad():
        y = fa(x, pos=pos)
    close(y, z["frame_attn_out"], "frame attention")


def test_bf16_autocast_path():
    """demo.py casts the aggregator to bf16 and runs under autocast (demo.py:458-460,545): bf16 weights and
    activations, bf16 LayerNorm parameters.  Golden: the reference's own FlashInferBlock with `.to(bfloat16)` under
    bf16 autocast on CPU (tests/golden/block_stream_bf16.npz, make_goldens.py block_stream_bf16_values).

    Tolerance.  Both sides return bf16, whose spacing at the outputs' magnitude (up to 5.8 here) is 2^-5 = 3.1e-2
    for |y| in [4, 8) and 2^-6 for [2, 4); the two runs round every intermediate (LayerNorm output, qkv, attention
    output, proj, two MLP layers, two residual sums) to bf16 at slightly different values, so final results that
    differ by one or two output rounding steps are expected: max-abs bound = 2 steps at the largest magnitude
    = 6.3e-2.  The cosine over the whole output is insensitive to single steps and keeps 0.9999."""
    z = np.load(os.path.join(G, "block_stream_bf16.npz"))
    dim, H, pph, ppw, ns, scale, window = 128, 2, 3, 4, 6, 2, 3
    Ptok = ns + pph * ppw
    blk = P.B200Block(dim=dim, num_heads=H, init_values=0.01, qk_norm=True, rope=Rope2dStub(),
                      kv_cache_sliding_window=window, kv_cache_scale_frames=scale).eval().to(DEV)
    seeded.fill_module_(blk, 21)
    blk = blk.to(torch.bfloat16)
    mgr = P.B200KVCacheManager(1, scale + window + 16, Ptok, H, 64, device=DEV, scale_frames=scale,
                               sliding_window=window, max_total_frames=40)
    kw = dict(num_patches=Ptok - ns, num_special=ns, enable_3d_rope=True, kv_cache=mgr, global_idx=0,
              num_frame_for_scale=scale, num_register_tokens=4)
    tol = dict(max_abs=6.3e-2, cos=0.9999)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        x = torch.from_numpy(seeded.randn(900, 1, scale * Ptok, dim)).to(DEV).to(torch.bfloat16)
        y = blk(x, pos=rope3d_pos(0, scale, pph, ppw, ns), num_frames=scale, num_frame_per_block=scale, **kw)
        assert y.dtype == torch.bfloat16
        close(y, z["phase1"], "bf16 phase 1", **tol)
        for i in range(5):
            x = torch.from_numpy(seeded.randn(901 + i, 1, Ptok, dim)).to(DEV).to(torch.bfloat16)
            y = blk(x, pos=rope3d_pos(scale + i, 1, pph, ppw, ns), num_frames=1, num_frame_per_block=1, **kw)
            assert y.dtype == torch.bfloat16
            close(y, z[f"frame{i}"], f"bf16 frame {i}", **tol)
    assert mgr.build_visible_page_table(0) == list(z["visible_end"])
    assert mgr.device_status() == 0


def test_block_with_compiled_style_attn_pre_equals_fused_path():
    """With blk.attn_pre rebound on the instance (what compile_model does) the streaming forward goes through
    attn_pre + append_frame instead of the fused append; both write the same pages and give the same output."""
    dim, H, pph, ppw, ns = 128, 2, 3, 4, 6
    Ptok = ns + pph * ppw
    mk_blk = lambda: P.B200Block(dim=dim, num_heads=H, init_values=0.01, qk_norm=True, rope=Rope2dStub(),
                                 kv_cache_sliding_window=3, kv_cache_scale_frames=2).eval().to(DEV)
    a, b = mk_blk(), mk_blk()
    seeded.fill_module_(a, 9)
    seeded.fill_module_(b, 9)
    b.attn_pre = b.attn_pre                       # instance attribute, as after `b.attn_pre = torch.compile(b.attn_pre)`
    mk = lambda: P.B200KVCacheManager(1, 21, Ptok, H, 64, device=DEV, scale_frames=2, sliding_window=3, max_total_frames=40)
    ma, mb = mk(), mk()
    for i in range(7):
        skip = i in (3, 5)
        ma._skip_append = mb._skip_append = skip
        x = torch.from_numpy(seeded.randn(40 + i, 1, Ptok, dim)).to(DEV)
        pos = rope3d_pos(i, 1, pph, ppw, ns)
        with torch.no_grad():
            ya = a(x, pos=pos, num_frames=1, enable_3d_rope=True, kv_cache=ma, global_idx=0)
            yb = b(x, pos=pos, num_frames=1, enable_3d_rope=True, kv_cache=mb, global_idx=0)
        assert torch.equal(ya, yb)
        assert ma.build_visible_page_table(0) == mb.build_visible_page_table(0)
    assert torch.equal(ma._gather_kv(0)[0], mb._gather_kv(0)[0])


def test_plain_attention_without_norm_and_rope():
    """The DINOv2 patch-embed attention (vision_transformer.py:144-171 builds Block(attn_class=Attention) with
    qk_norm off and no RoPE; 1 class + 4 register + 999 patch tokens): B200FrameAttention against fp32 SDPA."""
    dim, H, N = 128, 2, 1004
    fa = P.B200FrameAttention(dim, num_heads=H, qk_norm=False, rope=None).eval().to(DEV)
    seeded.fill_module_(fa, 31)
    x = torch.from_numpy(seeded.randn(77, 2, N, dim)).to(DEV)
    with torch.no_grad():
        y = fa(x)
        qkv = fa.qkv(x).reshape(2, N, 3, H, 64).permute(2, 0, 3, 1, 4)
        ref = torch.nn.functional.scaled_dot_product_attention(qkv[0], qkv[1], qkv[2])
        ref = fa.proj(ref.transpose(1, 2).reshape(2, N, dim))
    close(y, ref.double().cpu().numpy(), "plain attention")


@pytest.mark.parametrize("dim,H,weights,x_dtype,rope", [(128, 2, "bf16", "bf16", "3d"), (192, 3, "f32", "f32", "3d"), (576, 9, "bf16", "f32", "none"),
                                                        (1024, 16, "f32", "bf16", "2d"), (128, 2, "bf16", "bf16", "no autocast"),
                                                        (320, 5, "bf16", "f32", "3d"), (1088, 17, "f32", "bf16", "none"), (2048, 32, "bf16", "f32", "3d")])
@pytest.mark.parametrize("scaled", [True, False])
def test_layers_as_one_call_equal_the_module_code(monkeypatch, dim, H, weights, x_dtype, rope, scaled):
    """B200Block and B200FrameAttention as single native calls against the same modules run operation by operation: scale
    pass, keyframes with eviction, a non-keyframe, batch mode without a cache, a rebound ffn_residual; columns for one to
    eight warps per row, row counts that leave warps idle, and every combination of parameter and activation precision.

    Both sides round the same intermediates to bf16, the native call fewer of them (scale and sum in one step), and return
    bf16 or fp32; results may differ by two bf16 rounding steps at the largest magnitude of the output, 2 * 2^-7 * max.  That shows a
    missing or misplaced term; how close the sums are is measured against float64 further down."""
    from lingbot_map_b200 import block as block_mod
    pph, ppw, ns, scale, window = 3, 5, 6, 2, 2
    T = ns + pph * ppw
    dt = {"bf16": torch.bfloat16, "f32": torch.float32}
    blk = P.B200Block(dim=dim, num_heads=H, init_values=0.5 if scaled else None, qk_norm=scaled, rope=None if rope == "none" else Rope2dStub(),
                      kv_cache_sliding_window=window, kv_cache_scale_frames=scale).eval().to(DEV)
    fa = P.B200FrameAttention(dim, num_heads=H, qk_norm=scaled, rope=None if rope == "none" else Rope2dStub()).eval().to(DEV)
    seeded.fill_module_(blk, 3)
    seeded.fill_module_(fa, 4)
    blk, fa = blk.to(dt[weights]), fa.to(dt[weights])
    three_d = rope not in ("2d", "none")
    y, x = torch.meshgrid(torch.arange(1, pph + 1), torch.arange(1, ppw + 1), indexing="ij")
    pos2d = torch.cat([torch.zeros(ns, 2, dtype=torch.int64), torch.stack([y, x], -1).reshape(-1, 2)])[None].to(DEV)
    calls = []
    real = block_mod._native.block_layer

    class Counting:
        def __getattr__(self, name):
            return getattr(_lib_native, name)

        def block_layer(self, *a):
            calls.append("block")
            r = real(*a)
            assert r is not NotImplemented
            return r

        def frame_layer(self, *a):
            calls.append("frame")
            r = _lib_native.frame_layer(*a)
            assert r is not NotImplemented
            return r

    _lib_native = block_mod._native
    monkeypatch.setattr(block_mod, "_native", Counting())

    def run(fused):
        monkeypatch.setattr(block_mod, "_may_fuse", lambda: fused)
        mgr = P.B200KVCacheManager(1, scale + window + 16, T, H, 64, device=DEV, scale_frames=scale, sliding_window=window, max_total_frames=40)
        kw = dict(num_patches=T - ns, num_special=ns, enable_3d_rope=three_d, global_idx=0, num_frame_for_scale=scale)
        pos = lambda f, n: rope3d_pos(f, n, pph, ppw, ns) if three_d else pos2d.repeat(1, n, 1)
        data = lambda i, *s: torch.from_numpy(seeded.randn(i, *s, dim)).to(DEV).to(dt[x_dtype])
        out = [fa(data(1, 3, T), pos=pos2d.expand(3, -1, -1)), blk(data(2, 2, T), pos=pos(0, 1), **kw),
               blk(data(3, 1, scale * T), pos=pos(0, scale), num_frames=scale, kv_cache=mgr, **kw)]
        for i in range(5):
            mgr._skip_append = i == 2
            out.append(blk(data(4 + i, 1, T), pos=pos(scale + i, 1), num_frames=1, kv_cache=mgr, **kw))
        blk.ffn_residual = lambda v: 2 * v
        out.append(blk(data(9, 1, T), pos=pos(9, 1), num_frames=1, kv_cache=mgr, **kw))
        del blk.__dict__["ffn_residual"]
        assert mgr.device_status() == 0
        return out, mgr.build_visible_page_table(0), mgr._gather_kv(0)

    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16, enabled=rope != "no autocast"):
        got, table, kv = run(True)
        want, wtable, wkv = run(False)
    assert calls == ["frame"] + ["block"] * 8
    assert table == wtable
    for i, (a, b) in enumerate(zip(got + list(kv), want + list(wkv))):
        assert a.dtype == b.dtype and a.shape == b.shape, i
        d, top = float((a.float() - b.float()).abs().max()), float(b.float().abs().max())
        assert d <= 2 * 2 ** -7 * top, (i, d, top)


@pytest.mark.parametrize("frames,scale,window", [(2, 2, 1), (8, 8, 4), (9, 16, 4), (17, 17, 2), (11, 2, 1), (20, 3, 2)])
def test_scale_pass_appends_its_frames_as_one_by_one(monkeypatch, frames, scale, window):
    """The native scale pass appends up to eight frames per launch, and ends a launch where an evicted page comes back: page tables and
    pages as the modules make them, which append and evict frame by frame (K and V differ by the rounding steps of the test above).  The
    hidden layer has 33 columns, so that the activation ends in the middle of eight values."""
    from lingbot_map_b200 import block as block_mod
    pph, ppw, ns, dim, H = 3, 5, 6, 128, 2
    T = ns + pph * ppw
    blk = P.B200Block(dim=dim, num_heads=H, mlp_ratio=33 / 128, init_values=0.5, qk_norm=True, rope=Rope2dStub(), kv_cache_sliding_window=window,
                      kv_cache_scale_frames=scale).eval().to(DEV)
    seeded.fill_module_(blk, 3)
    blk = blk.to(torch.bfloat16)
    x = torch.from_numpy(seeded.randn(3, 1, frames * T, dim)).to(DEV).to(torch.bfloat16)

    def run(fused):
        monkeypatch.setattr(block_mod, "_may_fuse", lambda: fused)
        mgr = P.B200KVCacheManager(1, scale + window + 16, T, H, 64, device=DEV, scale_frames=scale, sliding_window=window, max_total_frames=40)
        y = blk(x, pos=rope3d_pos(0, frames, pph, ppw, ns), num_frames=frames, kv_cache=mgr, num_patches=T - ns, num_special=ns,
                enable_3d_rope=True, global_idx=0, num_frame_for_scale=scale)
        assert mgr.device_status() == 0
        return [y, *mgr._gather_kv(0)], mgr.build_visible_page_table(0), mgr.key_norm_max.clone()

    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        got, table, norms = run(True)
        want, wtable, wnorms = run(False)
    assert table == wtable
    assert torch.allclose(norms, wnorms, rtol=2 ** -7)
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert float((a.float() - b.float()).abs().max()) <= 2 * 2 ** -7 * float(b.float().abs().max())


def _layer_pair(dim=128, H=2):
    blk = P.B200Block(dim=dim, num_heads=H, init_values=0.5, qk_norm=True, rope=Rope2dStub()).eval().to(DEV)
    fa = P.B200FrameAttention(dim, num_heads=H, qk_norm=True, rope=Rope2dStub()).eval().to(DEV)
    seeded.fill_module_(blk, 3)
    seeded.fill_module_(fa, 4)
    return blk.to(torch.bfloat16), fa.to(torch.bfloat16)


def _off_alignment(t):
    """The same values one element off a 16-byte boundary, as a slice of a flat parameter buffer lies."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:].copy_(t.reshape(-1))
    return flat[1:].view(t.shape)


@pytest.mark.parametrize("what", ["norm", "gamma", "qk norm", "input", "conjugated positions"])
def test_layers_take_what_the_modules_take(what):
    """Parameters and inputs off the 16-byte alignment of the vector loads, and positions whose conjugation is still to be
    done: as one native call or through the modules, with the result of the aligned, resolved tensors.  Where the modules run instead
    of the native layer a value may be rounded to bf16 once more on the way: two rounding steps, 2 * 2^-7 * max."""
    blk, fa = _layer_pair()
    pph, ppw, ns = 3, 5, 6
    x = torch.from_numpy(seeded.randn(11, 1, ns + pph * ppw, 128)).to(DEV).bfloat16()
    pos = rope3d_pos(3, 1, pph, ppw, ns)
    kw = dict(num_patches=pph * ppw, num_special=ns, enable_3d_rope=True)

    def run(x, pos):
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return [blk(x, pos=pos, **kw), fa(x, pos=pos, enable_3d_rope=True)]

    want = run(x, pos)
    if what == "norm":
        blk.norm1.weight.data, blk.norm2.bias.data = _off_alignment(blk.norm1.weight.data), _off_alignment(blk.norm2.bias.data)
    elif what == "gamma":
        blk.ls1.gamma.data, blk.ls2.gamma.data = _off_alignment(blk.ls1.gamma.data), _off_alignment(blk.ls2.gamma.data)
    elif what == "qk norm":
        for m in (blk.attn, fa):
            m.q_norm.weight.data, m.k_norm.bias.data = _off_alignment(m.q_norm.weight.data), _off_alignment(m.k_norm.bias.data)
    elif what == "input":
        x = _off_alignment(x)
    else:
        pos = torch.conj(torch.conj_physical(pos))
        assert pos.is_conj()
    for got, ref in zip(run(x, pos), want):
        assert float((got.float() - ref.float()).abs().max()) <= 2 * 2 ** -7 * float(ref.float().abs().max())


def _strided(t, form):
    """The values of t [B, N, C] in memory of another layout."""
    B, N, C = t.shape
    if form == "columns":                       # a slice of wider rows
        return torch.cat([t, t.flip(-1)], dim=-1)[..., :C]
    if form == "every other token":
        return torch.stack([t, t.flip(-1)], dim=2).reshape(B, 2 * N, C)[:, ::2]
    if form == "transposed":                    # what flatten(2).transpose(1, 2) of a feature map gives
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    if form == "transposed, off alignment":
        return _off_alignment(t.transpose(1, 2).contiguous()).transpose(1, 2)
    if form == "batches apart":
        return torch.cat([t, t.flip(-1)], dim=1)[:, :N]
    return t[:, :1].expand(B, N, C)             # one row for every token


@pytest.mark.parametrize("form", ["columns", "every other token", "transposed", "transposed, off alignment", "batches apart", "expanded"])
@pytest.mark.parametrize("how", ["batch of 1", "batch of 2", "scale pass", "streamed", "non-keyframe"])
@pytest.mark.parametrize("x_dtype", ["bf16", "f32"])
def test_block_takes_inputs_of_any_strides(form, how, x_dtype):
    """Output and cache pages of a strided input equal those of its contiguous copy, bit for bit: both run the same kernels on
    the same rows."""
    blk, fa = _layer_pair()
    pph, ppw, ns, scale = 3, 5, 6, 2
    T, frames = ns + pph * ppw, scale if how == "scale pass" else 1
    x = torch.from_numpy(seeded.randn(13, 2 if how == "batch of 2" else 1, frames * T, 128)).to(DEV).to({"bf16": torch.bfloat16, "f32": torch.float32}[x_dtype])
    x = _strided(x, form)
    kw = dict(num_patches=T - ns, num_special=ns, enable_3d_rope=True, num_frames=frames, global_idx=0, pos=rope3d_pos(0, frames, pph, ppw, ns))

    def run(x):
        mgr = None
        if not how.startswith("batch"):
            mgr = P.B200KVCacheManager(1, scale + 2 + 16, T, 2, 64, device=DEV, scale_frames=scale, sliding_window=2, max_total_frames=40)
            mgr._skip_append = how == "non-keyframe"
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            y = blk(x, kv_cache=mgr, **kw)
            return [y, fa(x, pos=kw["pos"], enable_3d_rope=True)] + ([] if mgr is None else [mgr.kv_caches[0].clone()])

    got, want = run(x), run(x.clone(memory_format=torch.contiguous_format))
    assert torch.equal(got[0], want[0]) and all(torch.equal(a, b) for a, b in zip(got[2:], want[2:]))
    # the frame layer's first matrix product reads x with its strides: its sums may run in another order (one bf16 rounding
    # step of an intermediate, as everywhere in this file two steps of the largest output)
    assert float((got[1].float() - want[1].float()).abs().max()) <= 2 * 2 ** -7 * float(want[1].float().abs().max())


@pytest.mark.parametrize("where", ["norm1.weight", "norm1.bias", "attn.qkv.weight", "attn.qkv.bias", "attn.q_norm.weight", "attn.k_norm.bias", "attn.proj.weight",
                                   "ls1.gamma", "norm2.weight", "norm2.bias", "mlp.fc1.weight", "mlp.fc2.bias", "ls2.gamma", "positions"])
@pytest.mark.parametrize("three_d", [True, False])
def test_layers_refuse_what_lies_on_another_device(monkeypatch, where, three_d):
    """A parameter or positions on another device than the input: nothing is launched with its address, the native call hands
    over to the modules (NotImplemented) and these raise.  The host stands for any other device: the rule compares devices."""
    from lingbot_map_b200 import block as block_mod
    blk, fa = _layer_pair()
    pph, ppw, ns = 3, 5, 6
    T = ns + pph * ppw
    x = torch.from_numpy(seeded.randn(11, 1, T, 128)).to(DEV).bfloat16()
    pos = rope3d_pos(3, 1, pph, ppw, ns) if three_d else torch.ones(1, T, 2, dtype=torch.int64, device=DEV)
    answers, real = [], block_mod._native

    class Watching:
        def __getattr__(self, name):
            def call(*a):
                r = getattr(real, name)(*a)
                answers.append((name, r is NotImplemented))
                return r
            return call

    monkeypatch.setattr(block_mod, "_native", Watching())
    if where == "positions":
        pos = pos.cpu()
    else:
        path, name = where.rsplit(".", 1)
        p = getattr(blk.get_submodule(path), name)
        p.data = p.data.cpu()
        if where.startswith("attn."):
            p = getattr(fa.get_submodule(path[5:]), name)
            p.data = p.data.cpu()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        with pytest.raises((RuntimeError, ValueError)):
            blk(x, pos=pos, enable_3d_rope=three_d)
        assert answers == [("block_layer", True)]
        if where.startswith("attn.") or where == "positions":
            with pytest.raises((RuntimeError, ValueError)):
                fa(x, pos=pos, enable_3d_rope=three_d)
            assert answers[1:] == [("frame_layer", True)]
    torch.cuda.synchronize()


@pytest.mark.parametrize("kind", ["function", "dispatch"])
def test_a_mode_sees_the_operations_of_the_modules(kind):
    """The four Linear layers and two norms of a block, and the two Linear layers of a frame layer, under a mode that records them."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    seen = []

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", ""))
            return func(*args, **(kwargs or {}))

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append({"addmm": "linear", "native_layer_norm": "layer_norm"}.get(func.overloadpacket.__name__, ""))
            return func(*args, **(kwargs or {}))

    blk, fa = _layer_pair()
    x = torch.from_numpy(seeded.randn(11, 1, 21, 128)).to(DEV).bfloat16()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16), (Function if kind == "function" else Dispatch)():
        blk(x, pos=rope3d_pos(3, 1, 3, 5, 6), enable_3d_rope=True)
        assert (seen.count("linear"), seen.count("layer_norm")) == (4, 2)
        fa(x, pos=rope3d_pos(3, 1, 3, 5, 6), enable_3d_rope=True)
        assert seen.count("linear") == 6


@pytest.mark.parametrize("where", ["F.linear", "F.layer_norm", "F.gelu", "ops.prep_qkv", "ops.dense_attention", "block.LayerScale.forward", "block.Mlp.forward",
                                   "P.B200Block.ffn_residual", "P.B200Attention.stream_frame", "P.B200Attention.forward", "P.B200Attention._evict",
                                   "P.B200FrameAttention._dense", "P.B200KVCacheManager.append_frame", "P.B200KVCacheManager.append_frame_fused",
                                   "P.B200KVCacheManager.evict_frames", "P.B200KVCacheManager.compute_attention", "P.B200KVCacheManager.plan",
                                   "P.B200KVCacheManager.rollback_last_frame"])
def test_a_replaced_function_or_method_is_called(monkeypatch, where):
    """What a profiler or a test puts in the place of a function or class method sees the calls of a frame layer, a batch-mode block, a scale
    pass, a keyframe and a non-keyframe; outputs as without it (two bf16 rounding steps of the largest, as everywhere here)."""
    import torch.nn.functional as F
    from lingbot_map_b200 import block, ops
    blk, fa = _layer_pair()
    pph, ppw, ns, scale = 3, 5, 6, 2
    T = ns + pph * ppw
    data = lambda i, n: torch.from_numpy(seeded.randn(i, 1, n * T, 128)).to(DEV).bfloat16()

    def run():
        mgr = P.B200KVCacheManager(1, scale + 2 + 16, T, 2, 64, device=DEV, scale_frames=scale, sliding_window=2, max_total_frames=40)
        kw = dict(num_patches=T - ns, num_special=ns, enable_3d_rope=True, global_idx=0)
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            out = [fa(data(1, 1), pos=rope3d_pos(0, 1, pph, ppw, ns), enable_3d_rope=True), blk(data(2, 1), pos=rope3d_pos(0, 1, pph, ppw, ns), **kw),
                   blk(data(3, scale), pos=rope3d_pos(0, scale, pph, ppw, ns), num_frames=scale, kv_cache=mgr, **kw)]
            for i in range(2):
                mgr._skip_append = i == 1
                out.append(blk(data(4 + i, 1), pos=rope3d_pos(scale + i, 1, pph, ppw, ns), num_frames=1, kv_cache=mgr, **kw))
        return out

    want = run()
    owner, name = where.rsplit(".", 1)
    owner = eval(owner)
    calls, real = [], getattr(owner, name)

    def counted(*a, **k):
        calls.append(name)
        return real(*a, **k)

    monkeypatch.setattr(owner, name, counted)
    got = run()
    assert calls
    for a, b in zip(got, want):
        assert float((a.float() - b.float()).abs().max()) <= 2 * 2 ** -7 * float(b.float().abs().max())


@pytest.mark.parametrize("what", ["complex32", "complex64", "no batch entry"])
def test_layers_take_positions_as_the_modules_do(what):
    """Half-precision complex positions are converted (the modules' result, two bf16 rounding steps of the largest output); 2-D positions
    without a batch entry are an error before anything is launched."""
    blk, fa = _layer_pair()
    T = 21
    x = torch.from_numpy(seeded.randn(11, 1, T, 128)).to(DEV).bfloat16()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        if what == "no batch entry":
            none = torch.zeros(0, T, 2, dtype=torch.int64, device=DEV)
            for layer in (blk, fa):
                with pytest.raises(IndexError):
                    layer(x, pos=none)
            return
        pos = rope3d_pos(3, 1, 3, 5, 6).to(getattr(torch, what))
        for layer in (blk, fa):
            got, want = layer(x, pos=pos, enable_3d_rope=True), layer(x, pos=pos.to(torch.complex128), enable_3d_rope=True)
            assert float((got.float() - want.float()).abs().max()) <= 2 * 2 ** -7 * float(want.float().abs().max())


@pytest.mark.parametrize("width", [64, 128, 200])
def test_frame_layer_with_an_output_projection_of_another_width(monkeypatch, width):
    """proj may have been replaced by a Linear layer of another output width; as one native call and as modules (two bf16 rounding
    steps of the largest output)."""
    from lingbot_map_b200 import block
    _, fa = _layer_pair()
    fa.proj = torch.nn.Linear(128, width).to(DEV).bfloat16()
    x, pos = torch.from_numpy(seeded.randn(11, 2, 21, 128)).to(DEV).bfloat16(), rope3d_pos(3, 1, 3, 5, 6)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        got = fa(x, pos=pos, enable_3d_rope=True)
        monkeypatch.setattr(block, "_may_fuse", lambda: False)
        want = fa(x, pos=pos, enable_3d_rope=True)
    assert got.shape == want.shape == (2, 21, width) and got.dtype == want.dtype
    assert float((got.float() - want.float()).abs().max()) <= 2 * 2 ** -7 * float(want.float().abs().max())


class _In64Bits:
    """The two layers in float64 from the module's parameters: LayerNorm, Linear, rotations and softmax attention as they are
    defined, without a rounding in between."""

    @staticmethod
    def linear(x, m):
        return x @ m.weight.double().t() + m.bias.double()

    @staticmethod
    def norm(x, m):
        return torch.nn.functional.layer_norm(x, (x.shape[-1],), m.weight.double(), m.bias.double(), m.eps)

    @staticmethod
    def rotate(x, ang, three_d):                # x [N, H, 64], ang [N, 32]
        c, s = ang.cos()[:, None], ang.sin()[:, None]
        if three_d:
            a, b = x[..., 0::2], x[..., 1::2]
            return torch.stack([a * c - b * s, a * s + b * c], -1).reshape(x.shape)
        y = x.reshape(*x.shape[:2], 2, 2, 16)
        a, b = y[:, :, :, 0], y[:, :, :, 1]
        c, s = c.reshape(-1, 1, 2, 16), s.reshape(-1, 1, 2, 16)
        return torch.stack([a * c - b * s, a * s + b * c], 3).reshape(x.shape)

    @classmethod
    def attention(cls, m, x, ang, three_d, cached=None):        # x [N, C]
        q, k, v = cls.linear(x, m.qkv).reshape(x.shape[0], 3, m.num_heads, 64).unbind(1)
        q, k = cls.rotate(cls.norm(q, m.q_norm), ang, three_d), cls.rotate(cls.norm(k, m.k_norm), ang, three_d)
        if cached is not None:
            k, v = torch.cat([cached[0].double(), k]), torch.cat([cached[1].double(), v])
        p = torch.softmax(torch.einsum("qhd,khd->hqk", q, k) / 8, -1)
        return cls.linear(torch.einsum("hqk,khd->qhd", p, v).reshape(x.shape), m.proj)

    @classmethod
    def frame(cls, m, x, ang, three_d):
        return torch.stack([cls.attention(m, t.double(), ang, three_d) for t in x])

    @classmethod
    def block(cls, m, x, ang, three_d, cached=None):
        out = []
        for t in x.double():
            t = t + cls.attention(m.attn, cls.norm(t, m.norm1), ang, three_d, cached) * m.ls1.gamma.double()
            out.append(t + cls.linear(torch.nn.functional.gelu(cls.linear(cls.norm(t, m.norm2), m.mlp.fc1)), m.mlp.fc2) * m.ls2.gamma.double())
        return torch.stack(out)


@pytest.mark.parametrize("dim,H,weights,x_dtype,three_d", [(128, 2, "bf16", "bf16", True), (192, 3, "f32", "f32", True), (1024, 16, "bf16", "bf16", False),
                                                           (1024, 16, "bf16", "f32", True), (320, 5, "f32", "bf16", False)])
def test_native_layers_are_no_further_from_64_bits_than_the_modules(monkeypatch, dim, H, weights, x_dtype, three_d):
    """Error of both ways against float64, 2-norm over 2-norm.  The native call rounds the same operands to bf16 and fewer sums, so
    its error is not larger than the modules' but for the spread of two sets of some thousand roundings of the same size (2 %; an error of
    its own of a fifth of the roundings would show).  Neither exceeds 2^-7, which is fifty roundings of 2^-9 / sqrt(3) in quadrature: a
    path has about ten, and those before the softmax weigh several times."""
    from lingbot_map_b200 import block as block_mod
    pph, ppw, ns, scale = 9, 13, 6, 2
    T, dt = ns + pph * ppw, {"bf16": torch.bfloat16, "f32": torch.float32}
    blk = P.B200Block(dim=dim, num_heads=H, init_values=0.5, qk_norm=True, rope=Rope2dStub(), kv_cache_sliding_window=4, kv_cache_scale_frames=scale)
    fa = P.B200FrameAttention(dim, num_heads=H, qk_norm=True, rope=Rope2dStub())
    blk, fa = blk.eval().to(DEV), fa.eval().to(DEV)
    seeded.fill_module_(blk, 3)
    seeded.fill_module_(fa, 4)
    blk, fa = blk.to(dt[weights]), fa.to(dt[weights])
    y, x = torch.meshgrid(torch.arange(1, pph + 1), torch.arange(1, ppw + 1), indexing="ij")
    pos2d = torch.cat([torch.zeros(ns, 2, dtype=torch.int64), torch.stack([y, x], -1).reshape(-1, 2)])[None].to(DEV)
    pos = lambda f, n: rope3d_pos(f, n, pph, ppw, ns) if three_d else pos2d.repeat(1, n, 1)
    inv = 100.0 ** -(torch.arange(16, device=DEV, dtype=torch.float64) / 16)
    ang = lambda f, n: (pos(f, n).reshape(-1, 32).angle() if three_d else (pos(f, n)[0].double()[:, :, None] * inv).reshape(-1, 32))
    data = [torch.from_numpy(seeded.randn(i, *s, dim)).to(DEV).to(dt[x_dtype]) for i, s in enumerate([(2, T), (2, T), (1, scale * T), (1, T)])]

    def run(fused):
        monkeypatch.setattr(block_mod, "_may_fuse", lambda: fused)
        mgr = P.B200KVCacheManager(1, scale + 4 + 16, T, H, 64, device=DEV, scale_frames=scale, sliding_window=4, max_total_frames=40)
        kw = dict(num_patches=T - ns, num_special=ns, enable_3d_rope=three_d, global_idx=0)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = [fa(data[0], pos=pos(0, 1), enable_3d_rope=three_d),
                   blk(data[1], pos=pos(0, 1), **kw), blk(data[2], pos=pos(0, scale), num_frames=scale, kv_cache=mgr, **kw)]
            cached = mgr._gather_kv(0)
            out.append(blk(data[3], pos=pos(scale, 1), num_frames=1, kv_cache=mgr, **kw))
        want = [_In64Bits.frame(fa, data[0], ang(0, 1), three_d), _In64Bits.block(blk, data[1], ang(0, 1), three_d),
                _In64Bits.block(blk, data[2], ang(0, scale), three_d), _In64Bits.block(blk, data[3], ang(scale, 1), three_d, cached)]
        return [float((a.double() - w).norm() / w.norm()) for a, w in zip(out, want)]

    with torch.no_grad():
        native, modules = run(True), run(False)
    for i, (a, b) in enumerate(zip(native, modules)):
        assert a <= 1.02 * b and a <= 2 ** -7, (i, a, b)
