"""Single-token DSQG decode over per-layer circular K/V ring buffers.

The DWARF reference has no decode path (README.md:175-179 describes the O(1) cache in
prose; its generate() re-runs the whole prefix, train/train_2048_condU.py:463-487).
This module provides that cache: a ring of R = max(offsets)+1 slots per (sequence, head),
a write head per sequence, and one kernel launch per layer per token.
"""
from __future__ import annotations

from typing import Sequence

import torch

from . import _lib
from .ops import OFFSETS_43, _dtype_code


def dsqg_decode_step(q, k_new, v_new, k_ring, v_ring, head, pos_bias, head_gain=None,
                     scale_embed=None, offsets: Sequence[int] = OFFSETS_43, fill=None, out=None, overlap=False):
    """One decode step for one layer.

    q, k_new, v_new [S,H,D]; k_ring, v_ring [S,H,R,D] (updated in place at slot head[s]);
    head int32 [S] on the device; fill int32 [S] (valid tokens incl. the new one) or None
    for a full ring.  Returns out [S,H,D].

    overlap=True launches the kernel so that its ring gather runs while the kernel ahead of it
    in the stream is still finishing (`dsqg_decode_overlapped`): allowed only when that kernel
    writes none of this call's head, fill, k_ring, v_ring.
    """
    return _lib.native().decode_step(q, k_new, v_new, k_ring, v_ring, head, pos_bias, head_gain, scale_embed,
                                     _lib.offsets_handle(offsets), fill, out, overlap)


def dsqg_decode_step_kv(q, k_new, v_new, kv_ring, head, pos_bias, head_gain=None, scale_embed=None,
                        offsets: Sequence[int] = OFFSETS_43, fill=None, out=None, overlap=False):
    """dsqg_decode_step over one ring that holds key and value of a slot side by side:
    kv_ring [S,H,R,2,D] (updated in place).  A tap is one contiguous read of 2*D elements."""
    return _lib.native().decode_step_kv(q, k_new, v_new, kv_ring, None, head, pos_bias, head_gain, scale_embed,
                                        _lib.offsets_handle(offsets), fill, out, overlap)


class DSQGRingCache:
    """K/V rings for L layers, one shared write head per sequence.  interleaved=True (default) keeps
    key and value of a slot side by side in one tensor kv [L,S,H,R,2,D] (a tap is one contiguous
    read; `k` and `v` are strided views of it); interleaved=False keeps two tensors k, v [L,S,H,R,D]."""

    def __init__(self, layers, sequences, heads, head_dim, offsets: Sequence[int] = OFFSETS_43,
                 dtype=torch.bfloat16, device="cuda", interleaved=True):
        self.offsets = offsets
        self.R = max(self.offsets) + 1
        self.interleaved = interleaved
        if interleaved:
            self.kv = torch.zeros(layers, sequences, heads, self.R, 2, head_dim, dtype=dtype, device=device)
            self.k, self.v = self.kv[..., 0, :], self.kv[..., 1, :]
        else:
            self.kv = None
            self.k = torch.zeros(layers, sequences, heads, self.R, head_dim, dtype=dtype, device=device)
            self.v = torch.zeros_like(self.k)
        self.head = torch.full((sequences,), -1, dtype=torch.int32, device=device)
        self.fill = torch.zeros(sequences, dtype=torch.int32, device=device)

    # The native form of the offsets is kept beside them: looking it up hashes all of them, 0.3 us of a step of 5.5 us on the host.
    # It belongs to this process and is left out of copies and pickles.
    @property
    def offsets(self):
        return self._offsets

    @offsets.setter
    def offsets(self, offsets):
        self._offsets, self._handle = tuple(int(o) for o in offsets), None

    def __getstate__(self):
        state = dict(self.__dict__)
        state["offsets"] = state.pop("_offsets")
        del state["_handle"]
        return state

    def __setstate__(self, state):
        for name, value in state.items():
            setattr(self, name, value)

    def prefill(self, layer, k, v):
        """Load the rings of `layer` from a prefix in training layout: k, v [S,H,N,D].  Sets head
        and fill for the whole cache (call it with the same N for every layer)."""
        lib = _lib.load()
        S, H, N, D = k.shape
        if tuple(self.k[layer].shape) != (S, H, self.R, D) or k.dtype != self.k.dtype or v.shape != k.shape:
            raise ValueError("dsqg ring prefill: k, v must be [S,H,N,D] matching the cache")
        k, v = k.contiguous(), v.contiguous()
        with torch.cuda.device(k.device):
            stream = torch.cuda.current_stream(k.device).cuda_stream
            if self.interleaved:
                _lib.check(lib.dsqg_ring_prefill_kv(k.data_ptr(), v.data_ptr(), self.kv[layer].data_ptr(),
                                                    self.head.data_ptr(), self.fill.data_ptr(),
                                                    S, H, N, D, self.R, _dtype_code(k), stream), "dsqg_ring_prefill_kv")
                return
            _lib.check(lib.dsqg_ring_prefill(k.data_ptr(), v.data_ptr(), self.k[layer].data_ptr(),
                                             self.v[layer].data_ptr(), self.head.data_ptr(), self.fill.data_ptr(),
                                             S, H, N, D, self.R, _dtype_code(k), stream), "dsqg_ring_prefill")

    def advance(self):
        """Move every write head to the next slot; call once per token before the layers run."""
        self.head, self.fill = _lib.native().ring_advance(self.head, self.fill, self.R)

    def step(self, layer, q, k_new, v_new, pos_bias, head_gain=None, scale_embed=None, out=None, overlap=False):
        """Decode step of `layer`.  overlap=True is safe from the second layer of a token on (the
        kernel ahead is then another layer's step or a projection, never `advance`/`prefill`)."""
        if self.interleaved:
            handle = self._handle
            if handle is None:
                handle = self._handle = _lib.offsets_handle(self._offsets)
            return _lib.native().decode_step_kv(q, k_new, v_new, self.kv, layer, self.head, pos_bias, head_gain, scale_embed,
                                                handle, self.fill, out, overlap)
        return dsqg_decode_step(q, k_new, v_new, self.k[layer], self.v[layer], self.head, pos_bias,
                                head_gain, scale_embed, self.offsets, self.fill, out, overlap)
