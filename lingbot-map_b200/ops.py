"""Stand-alone operators of the B200 backend (thin wrappers over the C ABI): dense attention for the
frame blocks and the phase-1 scale pass, the fused q/k-norm + RoPE + bf16 prologue, RoPE tables and the
log-sum-exp merge of partial attention results.  All of them need a CUDA device.

Dense attention and the prologue are also registered as torch.library custom operators
(`gct_b200::dense_attention`, `gct_b200::prep_qkv`) with shape-only fake implementations: the reference
wraps whole frame blocks and `attn_pre` in torch.compile (demo.py:177-186, gct_profile.py:47-57), and a
custom operator is traced as one opaque node instead of breaking the graph at the ctypes call."""
from typing import Optional

import torch
from torch import Tensor

from . import _lib
from .cache import _stream_ptr

_native = _lib.binding()


def _require_cuda(t: Tensor, name: str):
    if not t.is_cuda:
        raise RuntimeError(f"{name} must be a CUDA tensor: the B200 backend has no CPU path")


def dense_attention(q: Tensor, k: Tensor, v: Tensor, out: Optional[Tensor] = None) -> Tensor:
    """softmax(q k^T / 8) v, non-causal (the SDPA call of lingbot_map/layers/attention.py:76,490).

    q [B, Nq, H, 64], k/v [B, Nkv, H, 64] bf16 with arbitrary strides (head_dim contiguous, strides
    multiples of 8 elements) -> [B, Nq, H, 64] bf16 contiguous."""
    if out is None and torch.compiler.is_compiling():
        return torch.ops.gct_b200.dense_attention(q, k, v)      # one opaque node in the traced graph
    return _native.dense_attention(q, k, v, out)                # eager: straight to the C ABI


def prep_qkv(qkv: Tensor, heads: int, tokens_per_frame: int, q_norm_w, q_norm_b, k_norm_w, k_norm_b,
             rope_cs: Optional[Tensor], rope_mode: int):
    """qkv Linear output [tokens, 3*H*64] -> (q, k, v) bf16 [tokens, H, 64]: LayerNorm(64) on q and k,
    RoPE from the per-token cos/sin table (indexed by token % tokens_per_frame), v cast only
    (lingbot_map/layers/attention.py:67-73)."""
    if torch.compiler.is_compiling():
        return torch.ops.gct_b200.prep_qkv(qkv, heads, tokens_per_frame, q_norm_w, q_norm_b, k_norm_w, k_norm_b, rope_cs,
                                           rope_mode)
    return _native.prep_qkv(qkv, heads, tokens_per_frame, q_norm_w, q_norm_b, k_norm_w, k_norm_b, rope_cs, rope_mode)


@torch.library.custom_op("gct_b200::dense_attention", mutates_args=())
def _dense_attention_op(q: Tensor, k: Tensor, v: Tensor) -> Tensor:
    return _native.dense_attention(q, k, v, None)


@_dense_attention_op.register_fake
def _dense_attention_fake(q: Tensor, k: Tensor, v: Tensor) -> Tensor:
    return q.new_empty((q.shape[0], q.shape[1], q.shape[2], 64), dtype=torch.bfloat16)


@torch.library.custom_op("gct_b200::prep_qkv", mutates_args=())
def _prep_qkv_op(qkv: Tensor, heads: int, tokens_per_frame: int, q_norm_w: Optional[Tensor], q_norm_b: Optional[Tensor],
                 k_norm_w: Optional[Tensor], k_norm_b: Optional[Tensor], rope_cs: Optional[Tensor],
                 rope_mode: int) -> tuple[Tensor, Tensor, Tensor]:
    return _native.prep_qkv(qkv, heads, tokens_per_frame, q_norm_w, q_norm_b, k_norm_w, k_norm_b, rope_cs, rope_mode)


@_prep_qkv_op.register_fake
def _prep_qkv_fake(qkv, heads, tokens_per_frame, q_norm_w, q_norm_b, k_norm_w, k_norm_b, rope_cs, rope_mode):
    mk = lambda: qkv.new_empty((qkv.shape[0], heads, 64), dtype=torch.bfloat16)
    return mk(), mk(), mk()


def rope3d_table(frame_index: int, pph: int, ppw: int, num_special: int, device, out: Optional[Tensor] = None) -> Tensor:
    """cos/sin [tokens, 32, 2] fp32 of the 3-D RoPE for one frame (lingbot_map/layers/rope.py:293-433)."""
    n = num_special + pph * ppw
    if out is None:
        out = torch.empty(n, 32, 2, dtype=torch.float32, device=device)
    _native.rope3d_table(frame_index, pph, ppw, num_special, out)
    return out


def rope2d_table(pph: int, ppw: int, num_special: int, device, base: float = 100.0) -> Tensor:
    """cos/sin [tokens, 32, 2] fp32 of the frame blocks' 2-D RoPE (lingbot_map/layers/rope.py:88-122)."""
    out = torch.empty(num_special + pph * ppw, 32, 2, dtype=torch.float32, device=device)
    _require_cuda(out, "out")
    with torch.cuda.device(out.device):
        _lib.check(_lib.load().gct_rope2d_table(pph, ppw, num_special, base, out.data_ptr(), _stream_ptr(out.device)))
    return out


def lse_merge(parts: Tensor, lse: Tensor, return_lse: bool = False):
    """parts [G, Nq, H, 64] fp32 (normalised partial outputs), lse [G, Nq, H] fp32 -> [Nq, H, 64] bf16."""
    _require_cuda(parts, "parts")
    G, Nq, H, D = parts.shape
    parts, lse = parts.contiguous(), lse.contiguous()
    out = torch.empty(Nq, H, D, dtype=torch.bfloat16, device=parts.device)
    lo = torch.empty(Nq, H, dtype=torch.float32, device=parts.device) if return_lse else None
    with torch.cuda.device(parts.device):
        _lib.check(_lib.load().gct_lse_merge(parts.data_ptr(), lse.data_ptr(), G, Nq, H, out.data_ptr(),
                                             None if lo is None else lo.data_ptr(), _stream_ptr(parts.device)))
    return (out, lo) if return_lse else out


def device_status(device) -> int:
    """Status word of the manager-less operators on `device` (0 = ok; 1 = a bounded wait timed out,
    2 = an index check failed).  Synchronises the device."""
    index = torch.device(device).index
    return _native.operator_status(torch.cuda.current_device() if index is None else index)
