"""fp32 forward: the taps are taken eight at a time, four or less at the end as a chunk of four."""
import pytest
import torch

import dwarf_b200
from tests.gpu_util import FP32_REL_TOL, oracle_fwd_bwd, rel_inf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dense,sparse", [(1, 0), (3, 0), (4, 0), (5, 0), (8, 0), (9, 0), (12, 1), (8, 4), (16, 5), (7, 6), (0, 3), (33, 3)])
@pytest.mark.parametrize("N,D", [(1, 32), (37, 8), (90, 32), (61, 64), (40, 80), (77, 128)])
def test_every_number_of_taps_in_the_last_chunk(dense, sparse, N, D):
    """FP32_REL_TOL: sums of at most D products and of J weighted values in fp32, far below it."""
    offsets = tuple(range(dense)) + tuple(range(dense + 1, dense + 1 + 6 * sparse, 6))
    g = torch.Generator().manual_seed(100 * dense + sparse)
    q, k, v = (torch.randn(1, 3, N, D, generator=g) for _ in range(3))
    pb, gain = torch.randn(len(offsets), 3, generator=g) * 0.3, torch.rand(3, generator=g) + 0.5
    se = torch.randn(len(offsets), D, generator=g) * 0.1 if D == 32 else None
    out = dwarf_b200.dsqg_attention(*(t.cuda() for t in (q, k, v, pb, gain)), None if se is None else se.cuda(), offsets).cpu()
    ref = oracle_fwd_bwd(q, k, v, pb, scale_embed=se, head_gain=gain, offsets=offsets)["out"]
    assert rel_inf(out, ref) < FP32_REL_TOL
