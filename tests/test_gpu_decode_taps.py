"""Decode at the tap counts where the kernel's number of rounds (a warp's groups of lanes over all taps) changes."""
import pytest
import torch

import dwarf_b200
from oracle import dsqg_oracle as O
from tests.gpu_util import assert_bf16_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,J", [(64, J) for J in (1, 24, 25, 44, 45, 48, 49)] + [(32, J) for J in (48, 49, 88, 89, 96, 97)])
def test_tap_counts(D, J):
    g = torch.Generator().manual_seed(J)
    offsets = tuple(range(0, 2 * J, 2))
    S, H, R = 4, 3, 2 * J
    v16 = lambda *s: torch.randn(*s, generator=g).bfloat16().float()  # noqa: E731
    kr, vr, q, kn, vn = v16(S, H, R, D), v16(S, H, R, D), v16(S, H, D), v16(S, H, D), v16(S, H, D)
    pb, gain = torch.randn(J, H, generator=g) * 0.5, torch.rand(H, generator=g) + 0.5
    head = torch.tensor([0, J // 2, R - 2, R - 1], dtype=torch.int32)
    fill = torch.tensor([1, J // 2 + 1, R - 1, R], dtype=torch.int32)
    dev = lambda t: t.cuda().to(torch.bfloat16)  # noqa: E731
    kv = torch.stack([dev(kr), dev(vr)], dim=-2).contiguous()
    out = dwarf_b200.dsqg_decode_step_kv(dev(q), dev(kn), dev(vn), kv, head.cuda(), pb.cuda(), gain.cuda(), None, offsets, fill.cuda())
    ref, kref, _ = O.decode_reference_direct(q, kn, vn, kr, vr, head, pb, gain, offsets, fill=fill)
    assert_bf16_close(out.float().cpu(), ref, "out")
    assert torch.equal(kv[..., 0, :].float().cpu(), kref)
