"""Non-finite values reach the rows that attend to them and no others."""
import pytest
import torch

import dwarf_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 40, 64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_fp32_forward_keeps_a_bad_first_row_to_its_own(D, bad):
    """Taps before the start of the sequence have weight zero; 0 * inf must not come of it."""
    N, offsets = 700, dwarf_b200.OFFSETS_43
    g = torch.Generator(device="cuda").manual_seed(0)
    q, k, v = (torch.randn(1, 2, N, D, generator=g, device="cuda") for _ in range(3))
    v[:, :, 0] = bad
    out = dwarf_b200.dsqg_attention(q, k, v, torch.zeros(len(offsets), 2, device="cuda"), None, None, offsets)
    attends = torch.zeros(N, dtype=torch.bool)
    attends[[o for o in offsets if o < N]] = True
    finite = torch.isfinite(out).all(-1).all(1).all(0).cpu()
    assert finite[~attends].all() and not finite[attends].any()


@pytest.mark.parametrize("D", [32, 64])
def test_decode_ignores_parameters_of_taps_that_do_not_exist(D):
    """Five tokens in: the scale_embed and pos_bias rows of the other taps do not count, whatever they hold."""
    S, H, offsets = 3, 4, dwarf_b200.OFFSETS_43
    outs = []
    for bad in (0.0, float("nan"), float("inf")):
        g = torch.Generator(device="cuda").manual_seed(D)
        rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
        se, bias = rnd(len(offsets), D), rnd(len(offsets), H)
        se[5:], bias[5:] = bad, bad
        cache = dwarf_b200.DSQGRingCache(1, S, H, D)
        for _ in range(5):
            cache.advance()
            out = cache.step(0, *(rnd(S, H, D).bfloat16() for _ in range(3)), bias, None, se)
        outs.append(out)
    assert torch.isfinite(outs[0]).all() and all(torch.equal(o, outs[0]) for o in outs[1:])
