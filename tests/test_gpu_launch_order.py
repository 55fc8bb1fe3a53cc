"""Kernels are scheduled while the kernel ahead of them ends; their results have to be those of one after the other."""
import pytest
import torch

import dwarf_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,dtype", [(32, torch.bfloat16), (64, torch.bfloat16), (80, torch.bfloat16), (32, torch.float32)])
def test_inputs_written_and_rewritten_in_place_between_calls(D, dtype):
    """Inputs at one address that a kernel ahead has just changed, results that the next call reads: no stale line, no early read."""
    B, H, N, J = 2, 4, 300, len(dwarf_b200.OFFSETS_43)
    g = torch.Generator(device="cuda").manual_seed(D)
    data = [torch.randn(4, B, H, N, D, generator=g, device="cuda").to(dtype) for _ in range(6)]
    pb = torch.randn(J, H, generator=g, device="cuda") * 0.1

    def step(x):
        q, k, v = (t.detach().requires_grad_(True) for t in x[:3])
        bias = pb.detach().requires_grad_(True)
        out = dwarf_b200.dsqg_attention(q, k, v, bias, None, None, dwarf_b200.OFFSETS_43)
        chained = dwarf_b200.dsqg_attention(out.detach(), q.detach(), out.detach(), pb, None, None, dwarf_b200.OFFSETS_43)
        return [out.detach(), chained, *torch.autograd.grad(out, [q, k, v, bias], x[3])]

    apart = []
    for d in data:
        torch.cuda.synchronize()
        apart.append([t.clone() for t in step(d)])
        torch.cuda.synchronize()
    buf = torch.empty_like(data[0])
    for _ in range(10):
        got = []
        for d in data:                                   # nothing waits in between
            buf.copy_(d)
            got.append(step(buf))
        for a, b in zip(apart, got):
            for x, y in zip(a, b):
                assert torch.equal(x, y)


def test_decode_after_calls_that_write_its_rings():
    """advance, prefill and the first layer's step run one after the other, overlapped steps behind them."""
    S, H, D, L = 8, 4, 64, 3
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    bias = torch.randn(len(dwarf_b200.OFFSETS_43), H, generator=g, device="cuda") * 0.1
    prompt = [(rnd(S, H, 200, D), rnd(S, H, 200, D)) for _ in range(L)]
    toks = [[(rnd(S, H, D), rnd(S, H, D), rnd(S, H, D)) for _ in range(L)] for _ in range(5)]

    def run(wait):
        cache, outs = dwarf_b200.DSQGRingCache(L, S, H, D), []
        for layer, (k, v) in enumerate(prompt):
            cache.prefill(layer, k, v)
        for tok in toks:
            cache.advance()
            wait()
            for layer, qkv in enumerate(tok):
                outs.append(cache.step(layer, *qkv, bias, overlap=layer > 0))
                wait()
        return outs + [cache.kv]

    apart = run(torch.cuda.synchronize)
    for _ in range(5):
        for a, b in zip(apart, run(lambda: None)):
            assert torch.equal(a, b)
