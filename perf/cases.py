"""The performance cases of this framework: what a user's program has it do, at the sizes it meets.

A model behind this backend streams video frames of 518 x (294 ... 392) pixels (patch 14: 21 x 37 ... 28 x 37 patches,
1005 tokens at 518 x 378) through 24 pairs of frame and global attention with 16 heads of 64, starts a sequence with a
scale pass over its first frames, keeps one token per frame in 16 camera-head caches, and culls and voxelises the point
clouds it makes.  Every case runs through the public entry points of the package.

Kinds
  stream    one streamed frame through the operator-level hot path of `layers` layer pairs: q/k norm + 2-D RoPE prologue and
            dense attention of the frame, then fused append with 3-D RoPE, eviction and attention over the paged cache.
            The frame is a non-keyframe (appended, attended over, rolled back: most frames at a keyframe interval above
            one), so that the cache is the same before every pass.
  block     the same step through the modules (B200FrameAttention + B200Block with its Linear layers and MLP).
  sequence  the start of a sequence through the modules: reset, scale pass over `scale` frames, then keyframes.
  frames    B200FrameAttention on a batch of frames (frame blocks of the scale pass; patch-embed layers without q/k norm
            and RoPE).
  dense     the dense attention operator alone, on views of one qkv buffer (scale pass of a global layer; odd sizes).
  camera    one frame of the camera head: `caches` one-token attentions over `cached` past frames, fp32.
  cull      frustum culling of a point cloud.      voxel     Morton voxelisation of one frame's points.
"""
import math

import torch

import lingbot_map_b200 as P
from lingbot_map_b200 import _lib, render_ops

DEV = "cuda"
SPECIAL = 6                    # camera + register + scale tokens of a frame
HEAD_DIM = 64


def listed():
    return [
        # the headline workload: all 24 layers at the steady state of a 10,000-frame sequence (131,928 visible tokens)
        dict(name="stream_10k", kind="stream", layers=24, pph=27, ppw=37, heads=16, cached=10000, scale=8, window=64, src="bf16"),
        # the same at the trained context of 320 frames (window full, 73,848 visible tokens)
        dict(name="stream_320", kind="stream", layers=24, pph=27, ppw=37, heads=16, cached=320, scale=8, window=64, src="bf16"),
        # the first frames after the scale pass: short cache, launches and latency count
        dict(name="stream_start", kind="stream", layers=24, pph=27, ppw=37, heads=16, cached=9, scale=8, window=64, src="bf16"),
        # a small frame (126 x 182 pixels), small cache, fp32 activations (a model without autocast)
        dict(name="stream_small_f32", kind="stream", layers=4, pph=9, ppw=13, heads=16, cached=40, scale=2, window=8, src="f32"),
        # one global layer with one anchor frame, a 16-frame window and 1,000 frames of memory
        dict(name="memory_1k", kind="stream", layers=1, pph=27, ppw=37, heads=16, cached=1017, scale=1, window=16, src="bf16"),
        # layer pairs as modules, bf16 weights under autocast, at the trained context
        dict(name="block_320", kind="block", layers=2, pph=27, ppw=37, heads=16, cached=320, scale=8, window=64, weights="bf16"),
        # a sequence's first sixteen frames at 518 x 294 as modules: scale pass over 8, then 8 keyframes with a short window
        dict(name="sequence_16", kind="sequence", layers=2, pph=21, ppw=37, heads=16, frames=8, scale=8, window=4, weights="bf16"),
        # frame attention of the scale pass: eight frames as a batch
        dict(name="frames_8", kind="frames", batch=8, pph=27, ppw=37, heads=16, rope=True, weights="bf16"),
        # camera head at 10,000 cached frames and at the start of a sequence (the smallest calls)
        dict(name="camera_10k", kind="camera", caches=16, cached=10000, new=1, heads=16, head_dim=128),
        dict(name="camera_start", kind="camera", caches=16, cached=12, new=1, heads=16, head_dim=128),
        # the accumulated cloud of about forty frames, and one frame's points
        dict(name="cull_8m", kind="cull", points=8000000, camera_on="cuda"),
        dict(name="voxel_frame", kind="voxel", width=518, height=378, voxel=0.02),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _one(rng):
    kind = rng.choice(["stream", "stream", "stream", "block", "block", "sequence", "frames", "dense", "camera", "camera", "cull", "voxel"])
    # square and wide frames, patches of 14 pixels, the long side 518 or the small test model's 182
    pph, ppw = rng.choice([(rng.randint(18, 37), 37), (rng.randint(18, 37), 37), (37, rng.randint(18, 36)), (rng.randint(7, 13), 13)])
    scale, window = rng.choice([(8, 64), (8, 64), (1, 16), (2, 8), (rng.randint(1, 8), rng.randint(2, 64))])
    if kind == "stream":
        return dict(kind=kind, layers=rng.choice([1, 2, 4, 12, 24]), pph=pph, ppw=ppw, heads=rng.choice([16, 16, 16, 2, 3]),
                    cached=_log(rng, 1, 10000), scale=scale, window=window, src=rng.choice(["bf16", "bf16", "bf16", "f32"]))
    if kind == "block":
        return dict(kind=kind, layers=rng.randint(1, 3), pph=pph, ppw=ppw, heads=rng.choice([16, 16, 16, 2]), cached=_log(rng, 1, 2000),
                    scale=scale, window=window, weights=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "sequence":
        return dict(kind=kind, layers=rng.randint(1, 2), pph=pph, ppw=ppw, heads=rng.choice([16, 16, 2]), frames=rng.randint(1, 12),
                    scale=rng.randint(2, 8), window=rng.choice([4, 8, 64]), weights=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "frames":
        return dict(kind=kind, batch=rng.randint(1, 8), pph=pph, ppw=ppw, heads=rng.choice([16, 16, 2]), rope=rng.random() < 0.6,
                    weights=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "dense":
        n_kv = _log(rng, 40, 8400)
        return dict(kind=kind, batch=rng.choice([1, 1, 2, 3]), n_q=n_kv if rng.random() < 0.7 else _log(rng, 1, n_kv), n_kv=n_kv,
                    heads=rng.choice([16, 16, 2, 3]))
    if kind == "camera":
        new = 1 if rng.random() < 0.75 else rng.randint(2, 8)
        return dict(kind=kind, caches=16, cached=_log(rng, 1, 10000) if new == 1 else rng.choice([0, _log(rng, 1, 300)]), new=new,
                    heads=rng.choice([16, 16, 16, 2]), head_dim=rng.choice([128, 128, 128, 64]))
    if kind == "cull":
        return dict(kind=kind, points=_log(rng, 1000, 16000000), camera_on=rng.choice(["cuda", "cuda", "cpu"]))
    return dict(kind=kind, width=14 * ppw, height=14 * pph, voxel=rng.choice([0.005, 0.01, 0.02, 0.05, 0.1]))


def draw(rng):
    most = work(listed()[0])
    while True:
        c = _one(rng)
        w = work(c)
        if w["bytes"] <= most["bytes"] and w["flops"] <= most["flops"] and _pool_bytes(c) <= 20e9:
            return c


# ---------------------------------------------------------------------------------------------- sizes
def _tokens(c):
    return c["pph"] * c["ppw"] + SPECIAL


def _visible(c, cached, current):
    """Visible K/V tokens with `cached` frames kept and the current frame (1: it stays beside the full window)."""
    full = min(cached, c["scale"] + c["window"]) + current
    return (_tokens(c) - SPECIAL) * full + SPECIAL * (cached + current)


def _pool_bytes(c):
    if c["kind"] not in ("stream", "block"):
        return 0
    pages = c["scale"] + c["window"] + 16 + SPECIAL * (c["cached"] + 110) // (_tokens(c) - SPECIAL) + 17
    return c["layers"] * pages * (_tokens(c) - SPECIAL) * c["heads"] * HEAD_DIM * 4


def work(c):
    """Bytes and operations of one pass: every input read once, every output written once."""
    kind = c["kind"]
    if kind == "cull":
        return {"bytes": 13 * c["points"], "flops": 28 * c["points"]}
    if kind == "voxel":
        n = c["width"] * c["height"]           # an occupied voxel writes 32 bytes; at most one per point, about one in three
        return {"bytes": 24 * n + 32 * n // 3, "flops": 20 * n}
    if kind == "camera":
        rows, width = c["cached"] + c["new"], c["heads"] * c["head_dim"]
        return {"bytes": c["caches"] * (2 * rows + 2 * c["new"]) * width * 4, "flops": c["caches"] * 4 * c["new"] * rows * width}
    C = c["heads"] * HEAD_DIM
    if kind == "dense":
        return {"bytes": c["batch"] * (2 * c["n_q"] + 2 * c["n_kv"]) * C * 2, "flops": 4 * c["batch"] * c["n_q"] * c["n_kv"] * C}
    T = _tokens(c)
    w = 4 if c.get("weights") == "f32" else 2
    if kind == "frames":
        n = c["batch"] * T
        return {"bytes": n * C * (4 + 2) + 4 * C * C * w, "flops": 4 * n * T * C + 8 * n * C * C}
    if kind == "stream":
        esz, kv = (4 if c["src"] == "f32" else 2), _visible(c, c["cached"], 1)
        return {"bytes": c["layers"] * (2 * 3 * T * C * esz + 2 * T * C * 2 + kv * C * 4 + T * C * 4),
                "flops": c["layers"] * 4 * T * C * (T + kv)}
    if kind == "block":
        kv = _visible(c, c["cached"], 1)
        return {"bytes": c["layers"] * (kv * C * 4 + T * C * 4 + 16 * C * C * w) + 2 * T * C * w,
                "flops": c["layers"] * (4 * T * C * (T + kv) + 32 * T * C * C)}
    S, b, f = c["scale"], 0, 0                 # sequence
    for i in range(c["frames"] + 1):
        n = S * T if i == 0 else T
        kv = S * T if i == 0 else _visible(c, S + i, 0)
        b += kv * C * 4 + n * C * 4 + 16 * C * C * w + 2 * n * C * w
        f += 4 * n * C * (T + kv) + 32 * n * C * C
    return {"bytes": c["layers"] * b, "flops": c["layers"] * f}


def tolerance(c):
    if c["kind"] in ("cull", "voxel"):
        return "exact"
    if c["kind"] == "camera":
        return {"rel": 1e-5}                   # fp32 throughout
    return {"rel": 1e-2}                       # bf16 operands and outputs, fp32 accumulation


# ---------------------------------------------------------------------------------------------- inputs
class _Rope2d:
    """What the frame blocks' 2-D rotary embedding tells the attention module."""
    base_frequency = 100.0


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _filled_cache(c, g):
    """A cache manager at the state after `cached` keyframes, its pages filled with N(0, 1) keys and values."""
    m = P.B200KVCacheManager(c["layers"], c["scale"] + c["window"] + 16, _tokens(c), c["heads"], HEAD_DIM, device=torch.device(DEV, 0),
                             scale_frames=c["scale"], sliding_window=c["window"], max_total_frames=c["cached"] + 110)
    for b, pool in enumerate(m.kv_caches):
        pool.normal_(generator=g)
        for _ in range(c["cached"]):
            m.append_frame_bookkeeping(b)
            m.evict_frames(b, c["scale"], c["window"])
    m.rescan_key_norms()
    return m


def _filled_module(mod, g, weights):
    mod = mod.eval().to(DEV)
    with torch.no_grad():
        for name, p in mod.named_parameters():
            p.normal_(generator=g)
            if p.dim() == 2:
                p.mul_(p.shape[1] ** -0.5)
            elif name.endswith("gamma"):
                p.mul_(0.1).add_(0.5)
            else:
                p.mul_(0.1).add_(1.0 if "norm" in name and name.endswith("weight") else 0.0)
    return mod.to(torch.bfloat16) if weights == "bf16" else mod


def _pos2d(c, batch):
    y, x = torch.meshgrid(torch.arange(1, c["pph"] + 1), torch.arange(1, c["ppw"] + 1), indexing="ij")
    p = torch.cat([torch.zeros(SPECIAL, 2, dtype=torch.int64), torch.stack([y, x], dim=-1).reshape(-1, 2)])
    return p[None].expand(batch, -1, -1).contiguous().to(DEV)


def _pos3d(c, first, frames):
    """Complex rotations [1, 1, tokens, 32] of `frames` frames from frame `first` on: 10 time, 11 row and 11 column
    frequencies per token."""
    T, ppw = _tokens(c), c["ppw"]
    i = torch.arange(T, dtype=torch.float64)
    patch = i >= SPECIAL
    row = torch.where(patch, SPECIAL + torch.div(i - SPECIAL, ppw, rounding_mode="floor"), i)
    col = torch.where(patch, SPECIAL + torch.remainder(i - SPECIAL, ppw), i)
    freq = lambda n, dim: 10000.0 ** -(2.0 * torch.arange(n, dtype=torch.float64) / dim)
    ang = torch.cat([torch.cat([(torch.full_like(i, float(f)))[:, None] * freq(10, 20), row[:, None] * freq(11, 22), col[:, None] * freq(11, 22)], dim=1)
                     for f in range(first, first + frames)])
    return torch.polar(torch.ones_like(ang), ang)[None, None].to(DEV)


def _modules(c, g):
    C = c["heads"] * HEAD_DIM
    frame = [_filled_module(P.B200FrameAttention(C, num_heads=c["heads"], qk_norm=True, rope=_Rope2d()), g, c["weights"]) for _ in range(c["layers"])]
    glob = [_filled_module(P.B200Block(dim=C, num_heads=c["heads"], init_values=0.01, qk_norm=True, rope=_Rope2d(),
                                       kv_cache_sliding_window=c["window"], kv_cache_scale_frames=c["scale"]), g, c["weights"])
            for _ in range(c["layers"])]
    return frame, glob


def prepare(case, seed):
    c, g = case, _gen(seed)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    s = {"case": c}
    if c["kind"] in ("stream", "block", "sequence", "frames"):
        T, C = _tokens(c), c["heads"] * HEAD_DIM
        act = torch.float32 if c.get("weights", c.get("src")) == "f32" else torch.bfloat16
    if c["kind"] == "stream":
        s["mgr"] = _filled_cache(c, g)
        for k in ("qkv_frame", "qkv_global"):
            s[k] = [rn(T, 3 * C).to(act) for _ in range(c["layers"])]
        s["norm"] = [[1 + 0.1 * rn(64), 0.1 * rn(64), 1 + 0.1 * rn(64), 0.1 * rn(64)] for _ in range(2 * c["layers"])]
        s["cs2d"] = P.ops.rope2d_table(c["pph"], c["ppw"], SPECIAL, DEV)
        s["cs3d"] = torch.empty(T, 32, 2, dtype=torch.float32, device=DEV)
    elif c["kind"] == "block":
        s["mgr"] = _filled_cache(c, g)
        s["mgr"]._skip_append = True           # a non-keyframe
        s["frame"], s["glob"] = _modules(c, g)
        s["pos2d"], s["pos3d"], s["x"] = _pos2d(c, 1), _pos3d(c, c["cached"], 1), rn(1, T, C).to(act)
    elif c["kind"] == "sequence":
        S = c["scale"]
        s["mgr"] = P.B200KVCacheManager(c["layers"], S + c["window"] + 16, T, c["heads"], HEAD_DIM, device=torch.device(DEV, 0), scale_frames=S,
                                        sliding_window=c["window"], max_total_frames=320)
        s["frame"], s["glob"] = _modules(c, g)
        s["pos2d"] = [_pos2d(c, S), _pos2d(c, 1)]
        s["pos3d"] = [_pos3d(c, 0, S)] + [_pos3d(c, S + i, 1) for i in range(c["frames"])]
        s["x"] = [rn(S, T, C).to(act)] + [rn(1, T, C).to(act) for _ in range(c["frames"])]
    elif c["kind"] == "frames":
        s["attn"] = _filled_module(P.B200FrameAttention(C, num_heads=c["heads"], qk_norm=c["rope"], rope=_Rope2d() if c["rope"] else None), g, c["weights"])
        s["pos"] = _pos2d(c, c["batch"]) if c["rope"] else None
        s["x"] = rn(c["batch"], T, C)          # fp32: what a LayerNorm under autocast hands over
    elif c["kind"] == "dense":
        B, H = c["batch"], c["heads"]
        kv = rn(B, c["n_kv"], 3, H, HEAD_DIM).to(torch.bfloat16)
        s["q"], s["k"], s["v"] = (kv[:, :, 0] if c["n_q"] == c["n_kv"] else rn(B, c["n_q"], H, HEAD_DIM).to(torch.bfloat16)), kv[:, :, 1], kv[:, :, 2]
    elif c["kind"] == "camera":
        H, D, n = c["heads"], c["head_dim"], c["new"]
        s["caches"] = [P.DecodeCache(H, D, torch.device(DEV, 0), capacity=max(1024, c["cached"] + n)) for _ in range(c["caches"])]
        for d in s["caches"]:
            d.k[:c["cached"]].normal_(generator=g)
            d.v[:c["cached"]].normal_(generator=g)
            d.count = c["cached"]
        s["qkv"] = [(rn(n, H, D), rn(n, H, D), rn(n, H, D)) for _ in range(c["caches"])]
    elif c["kind"] == "cull":
        s["pts"] = rn(c["points"], 3) * 3
        q, _ = torch.linalg.qr(rn(3, 3).cpu())
        s["R"], s["t"] = q.to(c["camera_on"]), (0.5 * rn(3)).to(c["camera_on"])
    else:                                      # voxel: the points of a smooth, noisy depth image, rotated into the world
        h, w, fixed = c["height"], c["width"], _gen(1)
        v, u = torch.meshgrid(torch.arange(h, device=DEV) / h - 0.5, torch.arange(w, device=DEV) / w - 0.5, indexing="ij")
        depth = 2.5 + torch.sin(4 * u + 1) * torch.cos(5 * v + 2) + 0.5 * torch.sin(17 * (0.7 * u - 0.4 * v))
        depth = depth * (1 + 0.01 * torch.randn(h, w, device=DEV, generator=fixed))
        turn = torch.tensor([[0.36, 0.48, -0.8], [-0.8, 0.6, 0.0], [0.48, 0.64, 0.6]], device=DEV)
        cell = torch.floor(torch.stack([u * depth, v * depth, depth], dim=-1).reshape(-1, 3) @ turn / c["voxel"])
        # where the cloud lies, where in its voxel a point lies and the colours come from the seed; how many voxels it occupies does not
        shift = torch.randint(-40, 40, (3,), device=DEV, generator=g)
        s["xyz"] = ((cell + shift + 0.1 + 0.8 * torch.rand(h * w, 3, device=DEV, generator=g)) * c["voxel"]).contiguous()
        s["rgb"] = torch.rand(h * w, 3, device=DEV, generator=g)
    return s


# ---------------------------------------------------------------------------------------------- one pass
def _stream(s):
    c, m, out = s["case"], s["mgr"], []
    P.ops.rope3d_table(c["cached"] % 1024, c["pph"], c["ppw"], SPECIAL, DEV, out=s["cs3d"])
    m._defer_eviction = True
    for b in range(c["layers"]):
        q, k, v = P.ops.prep_qkv(s["qkv_frame"][b], c["heads"], _tokens(c), *s["norm"][2 * b], s["cs2d"], _lib.ROPE_2D)
        out.append(P.ops.dense_attention(q[None], k[None], v[None]))
        qg = m.append_frame_fused(b, s["qkv_global"][b], *s["norm"][2 * b + 1], s["cs3d"], _lib.ROPE_3D)
        m.evict_frames(b, c["scale"], c["window"])
        out.append(m.compute_attention(b, qg))
        m.rollback_last_frame(b)
    m._defer_eviction = False
    return out


def _layers(s, x, pos2d, pos3d, frames):
    """`frames` frames [frames, T, C] through the layer pairs: frame attention, then the global block on all tokens."""
    c = s["case"]
    T, C = _tokens(c), c["heads"] * HEAD_DIM
    kw = dict(num_patches=T - SPECIAL, num_special=SPECIAL, num_frames=frames, num_frame_per_block=frames, num_frame_for_scale=c["scale"],
              enable_3d_rope=True, kv_cache=s["mgr"])
    for b in range(c["layers"]):
        x = x + s["frame"][b](x, pos=pos2d)
        x = s["glob"][b](x.view(1, frames * T, C), pos=pos3d, global_idx=b, **kw).view(frames, T, C)
    return x


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "stream":
        return _stream(s)
    if kind == "block":
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return _layers(s, s["x"], s["pos2d"], s["pos3d"], 1)
    if kind == "sequence":
        s["mgr"].reset()
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            out = [_layers(s, s["x"][0], s["pos2d"][0], s["pos3d"][0], c["scale"])]
            for i in range(c["frames"]):
                out.append(_layers(s, s["x"][1 + i], s["pos2d"][1], s["pos3d"][1 + i], 1))
        return out + list(s["mgr"].kv_caches)
    if kind == "frames":
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return s["attn"](s["x"], pos=s["pos"])
    if kind == "dense":
        return P.ops.dense_attention(s["q"], s["k"], s["v"])
    if kind == "camera":
        return [d.attend(q, k, v, False) for d, (q, k, v) in zip(s["caches"], s["qkv"])]
    if kind == "cull":
        return render_ops.frustum_cull(s["pts"], s["R"], s["t"], 300.0, 310.0, 259.0, 189.0, 518, 378, 0.1, 6.0)
    return render_ops.voxelize_frame(s["xyz"], s["rgb"], c["voxel"])
