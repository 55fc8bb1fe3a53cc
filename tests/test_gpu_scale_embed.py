"""scale_embed on the tensor-core kernels: tap sets at the edges of the kernels' tables (8-tap steps of the sparse part, 16-column
steps of the dscale_embed products, the three window widths), and the choice of tiles per warp in the forward."""
import pytest
import torch

import dwarf_b200
from dwarf_b200 import synth

from tests.gpu_util import PARAM_REL_TOL_BF16, assert_bf16_close, assert_param_grad_close, cuda_fwd_bwd, oracle_fwd_bwd

pytestmark = pytest.mark.gpu


def _taps(lo, hi, sparse):
    return tuple(range(lo, hi + 1)) + tuple(hi + 3 + 5 * i for i in range(sparse))


@pytest.mark.parametrize("shape", [(1, 2, 203, 32), (2, 1, 64, 64), (1, 1, 17, 32)])
@pytest.mark.parametrize("lo,hi,sparse", [(0, 32, 0), (0, 32, 15), (0, 32, 16), (0, 31, 8), (3, 20, 9), (0, 40, 7), (0, 48, 1), (1, 64, 63), (0, 63, 64)])
def test_tap_sets_vs_oracle(shape, lo, hi, sparse):
    B, H, N, D = shape
    offsets = _taps(lo, hi, sparse)
    g = torch.Generator().manual_seed(N + hi + sparse)
    q, k, v, dout = (torch.randn(B, H, N, D, generator=g).mul(s).bfloat16().float() for s in (0.5, 0.5, 0.5, 1.0))
    pb = torch.randn(len(offsets), H, generator=g) * 0.3
    gain = torch.rand(H, generator=g) * 0.4 + 0.8
    se = torch.randn(len(offsets), D, generator=g) * 0.1
    ref = oracle_fwd_bwd(q, k, v, pb, dout, se, gain, offsets)
    r = cuda_fwd_bwd(q, k, v, pb, dout, se, gain, offsets, torch.bfloat16)
    for nm in ("out", "dq", "dk", "dv"):
        assert_bf16_close(r[nm], ref[nm], nm)
    for nm in ("dpb", "dse", "dgain"):
        assert_param_grad_close(r[nm], ref[nm], nm, PARAM_REL_TOL_BF16)


@pytest.mark.parametrize("B,H,N,D", [(24, 8, 2047, 32), (8, 8, 2047, 32), (7, 12, 1000, 64), (9, 12, 2001, 64)])
def test_forward_does_not_depend_on_the_tiles_per_warp(B, H, N, D):
    """The last sequence of a large batch (two or three tiles per warp) against the same sequence alone (one tile)."""
    off = dwarf_b200.ALL_OFFSETS
    g = torch.Generator(device="cuda").manual_seed(N)
    q, k, v = ((torch.randn(B, H, N, D, generator=g, device="cuda") * 0.5).bfloat16() for _ in range(3))
    pb, se = synth.log_linear_pos_bias(off, H).cuda(), torch.randn(len(off), D, generator=g, device="cuda") * 0.1
    with torch.no_grad():
        whole = dwarf_b200.dsqg_attention(q, k, v, pb, None, se, off)
        alone = dwarf_b200.dsqg_attention(q[-1:], k[-1:], v[-1:], pb, None, se, off)
    assert torch.equal(whole[-1:], alone)
