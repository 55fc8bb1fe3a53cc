"""DSQG attention as a PyTorch operator over the native C ABI.

Mirrors the operator layer of the DWARF reference:
``_DSQGFn`` / ``_DSQGFnV3`` (kernels/dsqg_attention_v2.py:337-414,
kernels/dsqg_attention_v3.py:359-442) and their functional wrappers
(:417-427, :445-456).  PyTorch is used for device memory and streams only; all
arithmetic happens in libdsqg_b200.so, and the steps around it (checks, allocation, autograd
nodes) in _dsqg_torch.so.
"""
from __future__ import annotations

from typing import Sequence

import torch

from . import _lib

SPARSE_TAPS = (48, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536)
#: The reference's 44-offset set (kernels/dsqg_attention_v3.py:47-49): dense 0..32 + 11 taps.
ALL_OFFSETS = tuple(range(33)) + SPARSE_TAPS
#: Dense 0..31 + the same 11 taps: the 43-offset set the benchmark configurations name.
OFFSETS_43 = tuple(range(32)) + SPARSE_TAPS
#: 43-set extended for N = 4096.
OFFSETS_45 = OFFSETS_43 + (2048, 3072)


def _dtype_code(t: torch.Tensor) -> int:
    if t.dtype == torch.bfloat16:
        return _lib.DSQG_DTYPE_BF16
    if t.dtype == torch.float32:
        return _lib.DSQG_DTYPE_F32
    raise TypeError(f"dsqg: q/k/v must be bfloat16 or float32, got {t.dtype}")


class DSQGFunction:
    """out = DSQG(q, k, v; pos_bias, head_gain, scale_embed, offsets) with autograd (an autograd node in native code,
    csrc/dsqg_torch.cpp).

    Saves (q, k, v, pos_bias, head_gain, scale_embed, out, lse) like the reference
    (kernels/dsqg_attention_v3.py:384) and returns gradients for the six tensors.
    """

    @staticmethod
    def apply(q, k, v, pos_bias, head_gain, scale_embed, offsets):
        return _lib.native().attention(q, k, v, pos_bias, head_gain, scale_embed, _lib.offsets_handle(offsets))


def causal_mean(x):
    """Causal running mean over the sequence dimension of x [B,N,D] (bf16 or fp32; other dtypes are
    computed in fp32 and cast back): the pooling of the reference's interference block,
    `x.cumsum(dim=1) / counts` (train/train_2048_condU.py:289-292), as one kernel; its backward is the
    kernel's reverse mode."""
    if x.dtype in (torch.bfloat16, torch.float32):
        return _lib.native().causal_mean(x)
    return _lib.native().causal_mean(x.float()).to(x.dtype)


class DSQGPackedFunction:
    """DSQG on the un-permuted output of a fused qkv projection, with a token-major result (an autograd node in
    native code, csrc/dsqg_torch.cpp).

    qkv [B,N,3,H,HD] bf16 (a view of the [B,N,3*H*HD] projection output; q, k, v are read in place
    through strides), gate [B,N,H*HD] bf16 or None -> y [B,N,H*HD] = DSQG(q,k,v) (* sigmoid(gate)).
    Replaces the three `.permute(0,2,1,3).contiguous()` copies, the output permute and the gate
    multiply of the reference's attention modules (train/train_2048_condU.py:171-175,189-191) and
    their autograd backward; the gradient comes back as one dqkv tensor in the layout of qkv."""

    @staticmethod
    def apply(qkv, gate, pos_bias, head_gain, offsets, scale_embed=None):
        return _lib.native().attention_packed(qkv, gate, pos_bias, head_gain, scale_embed, _lib.offsets_handle(offsets))


class InjectKVFunction(torch.autograd.Function):
    """k += k_delta; v += v_delta (train/train_2048_condU.py:178-181) applied IN PLACE to the key
    and value thirds of a fused projection output qkv [B,N,3*D] (a non-leaf tensor that is not a
    view, e.g. what nn.Linear returned), so the packed operator can go on reading q, k, v in place.
    k_delta, v_delta: [B,N,D] token-major.  Backward: the deltas' gradients are the key and value
    thirds of qkv's gradient (views, no copy)."""

    @staticmethod
    def forward(ctx, qkv, k_delta, v_delta):
        B, N, D3 = qkv.shape
        if D3 % 3 or tuple(k_delta.shape) != (B, N, D3 // 3) or tuple(v_delta.shape) != (B, N, D3 // 3):
            raise ValueError("dsqg inject: qkv must be [B,N,3*D] and the deltas [B,N,D]")
        thirds = qkv.view(B, N, 3, D3 // 3)
        thirds[:, :, 1].add_(k_delta)
        thirds[:, :, 2].add_(v_delta)
        ctx.mark_dirty(qkv)
        ctx.delta_dtypes = (k_delta.dtype, v_delta.dtype)
        return qkv

    @staticmethod
    def backward(ctx, g):
        B, N, D3 = g.shape
        thirds = g.view(B, N, 3, D3 // 3) if g.is_contiguous() else g.reshape(B, N, 3, D3 // 3)
        kdt, vdt = ctx.delta_dtypes
        return g, thirds[:, :, 1].to(kdt), thirds[:, :, 2].to(vdt)


def packed_path_available(head_dim: int, offsets: Sequence[int], scale_embed: bool = False) -> bool:
    """True when dsqg_attention_packed can take this head width and offset set (the bf16 tensor-core
    kernels; with scale_embed head widths up to 64); otherwise callers use dsqg_attention on
    permuted copies."""
    off, J = _lib.offsets_array(offsets)
    return bool(_lib.load().dsqg_tensor_core_path(_lib.DSQG_DTYPE_BF16, int(head_dim), off, J, 1 if scale_embed else 0))


def dsqg_attention_packed(qkv, pos_bias, head_gain=None, gate=None, offsets: Sequence[int] = ALL_OFFSETS,
                          scale_embed=None):
    """DSQG straight on the fused projection output.  qkv: [B,N,3,H,HD] bf16 contiguous; gate: None
    or [B,N,H*HD] bf16 (pre-sigmoid); scale_embed: None or [J,HD] (the reference's v3 op).  Returns
    [B,N,H*HD] bf16, already multiplied by sigmoid(gate) when a gate is given."""
    return _lib.native().attention_packed(qkv, gate, pos_bias, head_gain, scale_embed, _lib.offsets_handle(offsets))


def dsqg_attention(q, k, v, pos_bias, head_gain=None, scale_embed=None,
                   offsets: Sequence[int] = ALL_OFFSETS):
    """General DSQG entry: any ascending offset set, optional per-head output gain and
    Q-weighted scale embedding.  q, k, v: [B,H,N,HD] bf16 (fast path) or fp32; fp16 inputs
    are computed in bf16 as the reference does (kernels/dsqg_attention_v3.py:452-456) and
    the result is returned in the caller's dtype."""
    orig_dtype = q.dtype
    if orig_dtype is torch.bfloat16 or orig_dtype is torch.float32:
        return _lib.native().attention(q, k, v, pos_bias, head_gain, scale_embed, _lib.offsets_handle(offsets))
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    return _lib.native().attention(q, k, v, pos_bias, head_gain, scale_embed, _lib.offsets_handle(offsets)).to(orig_dtype)


def dsqg_forward_lse(q, k, v, pos_bias, head_gain=None, scale_embed=None,
                     offsets: Sequence[int] = ALL_OFFSETS):
    """Forward without autograd; returns (out, lse).  lse is the natural-log softmax
    denominator per row, the tensor the reference saves for backward."""
    return _lib.native().forward_lse(q, k, v, pos_bias, head_gain, scale_embed, _lib.offsets_handle(offsets))
