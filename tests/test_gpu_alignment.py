"""Head widths whose rows are read in 32-byte pieces (D = 64, 128): tensors that start on a multiple of 16 bytes only take the
variant with 16-byte pieces, with the same arithmetic in the same order."""
import pytest
import torch

import dwarf_b200
from dwarf_b200 import synth

pytestmark = pytest.mark.gpu


def _at(x, offset):
    """x in fresh memory, its first element `offset` elements after an aligned address."""
    buf = torch.empty(x.numel() + 64, dtype=x.dtype, device=x.device)
    return buf[offset:offset + x.numel()].view(x.shape).copy_(x).requires_grad_(True)


@pytest.mark.parametrize("D,with_se", [(64, False), (64, True), (128, False)])
@pytest.mark.parametrize("shape", [(1, 2, 1), (2, 3, 101), (1, 2, 560)])
def test_16_byte_aligned_tensors_give_the_same_bits(D, with_se, shape):
    B, H, N = shape
    off = dwarf_b200.OFFSETS_43
    g = torch.Generator(device="cuda").manual_seed(D + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    q, k, v, dy = ((rnd(B, H, N, D) * 0.5).bfloat16() for _ in range(4))
    pb = synth.log_linear_pos_bias(off, H).cuda() + rnd(len(off), H) * 0.05
    se = (rnd(len(off), D) * 0.1).requires_grad_(True) if with_se else None
    res = []
    for offset in (0, 8):
        x = [_at(t, offset) for t in (q, k, v)]
        p = pb.clone().requires_grad_(True)
        y = dwarf_b200.dsqg_attention(*x, p, None, se, off)
        res.append([y.detach(), *torch.autograd.grad(y, [*x, p] + ([se] if with_se else []), _at(dy, offset).detach())])
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("gated", [False, True])
def test_16_byte_aligned_packed_projection_gives_the_same_bits(gated):
    B, N, H, D = 2, 77, 2, 64
    off = dwarf_b200.OFFSETS_43
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    qkv, gate, dy, pb = rnd(B, N, 3, H, D), rnd(B, N, H * D), rnd(B, N, H * D), synth.log_linear_pos_bias(off, H).cuda()
    res = []
    for offset in (0, 8):
        x, gt = _at(qkv, offset), _at(gate, offset) if gated else None
        y = dwarf_b200.dsqg_attention_packed(x, pb, None, gt, off)
        res.append([y.detach(), *torch.autograd.grad(y, [x] + ([gt] if gated else []), _at(dy, offset).detach())])
    for a, b in zip(*res):
        assert torch.equal(a, b)
