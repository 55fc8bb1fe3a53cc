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


def test_two_streams_that_join_eager_and_captured():
    """A call behind two streams' calls reads both results: events and graph edges hold for kernels that may start early."""
    B, H, N, D, J = 4, 8, 1000, 32, len(dwarf_b200.OFFSETS_43)
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(B, H, N, D, generator=g, device="cuda").bfloat16() for _ in range(3))
    pb = torch.randn(J, H, generator=g, device="cuda") * 0.1
    op = lambda a, b, c: dwarf_b200.dsqg_attention(a, b, c, pb, None, None, dwarf_b200.OFFSETS_43)  # noqa: E731
    want = [op(q, k, v), op(v, q, k)]
    want.append(op(want[0], want[1], want[0]))
    want.append(op(want[2], want[1], want[0]))
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def work():
        side.wait_stream(main)
        with torch.cuda.stream(side):
            two = op(v, q, k)
        one = op(q, k, v)
        main.wait_stream(side)
        three = op(one, two, one)
        side.wait_stream(main)
        with torch.cuda.stream(side):
            four = op(three, two, one)
        main.wait_stream(side)
        return [one, two, three, four]

    with torch.cuda.stream(main):
        for _ in range(5):
            got = work()
            torch.cuda.synchronize()                    # before a tensor of one stream is given back while the other may read it
            assert all(torch.equal(a, b) for a, b in zip(want, got))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            got = work()
        for _ in range(5):
            for t in got:
                t.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(want, got))


@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("writer", ["step", "prefill"])
def test_overlapped_steps_two_behind_a_kernel_that_writes_their_ring(writer, D):
    """A writes a ring, an overlapped step on other rings follows, then an overlapped step on the ring that A wrote, its write heads known ahead:
    the promise (the kernel just ahead writes none of them) is kept, so that step sees everything A wrote."""
    S, H, N = 64, 8, 1800
    offsets = dwarf_b200.OFFSETS_43
    R = max(offsets) + 1
    g = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    bias = torch.randn(len(offsets), H, generator=g, device="cuda") * 0.1
    prefix, toks = (rnd(S, H, N, D), rnd(S, H, N, D)), [[rnd(S, H, D) for _ in range(3)] for _ in range(3)]
    small = [t[:2].contiguous() for t in toks[1]]                    # the step in between: few blocks, over at once
    heads = [torch.full((S,), (N + i) % R, dtype=torch.int32, device="cuda") for i in range(2)]
    old = [rnd(S, H, R, 2, D), rnd(2, H, R, 2, D)]
    caches = [dwarf_b200.DSQGRingCache(1, S, H, D), dwarf_b200.DSQGRingCache(1, 2, H, D)]
    out = [torch.empty_like(toks[0][0]), torch.empty_like(small[0]), torch.empty_like(toks[2][0])]

    def work(wait):
        rings = [c.kv[0] for c in caches]
        for ring, x in zip(rings, old):
            ring.copy_(x)
        wait()
        step = lambda t, ring, head, o, overlap: dwarf_b200.dsqg_decode_step_kv(*t, ring, head, bias, offsets=offsets, out=o, overlap=overlap)  # noqa: E731
        if writer == "step":
            step(toks[0], rings[0], heads[0], out[0], False)
        else:
            caches[0].prefill(0, *prefix)
        wait()
        step(small, rings[1], heads[0][:2], out[1], True)
        wait()
        step(toks[2], rings[0], heads[1 if writer == "step" else 0], out[2], True)
        wait()
        return [*out[1:], *rings]

    apart = [t.clone() for t in work(torch.cuda.synchronize)]
    same = lambda got: all(torch.equal(a, b) for a, b in zip(apart, got))  # noqa: E731
    for _ in range(20):
        assert same(work(lambda: None))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = work(lambda: None)
        for _ in range(20):
            for t in got:
                t.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert same(got)
