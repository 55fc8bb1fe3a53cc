"""The layer around the operator in native code: its elementwise and reduction kernels against fp32 PyTorch, and the two autograd
nodes (attention layer, interference block) against the same modules in fp32."""
import ctypes

import pytest
import torch
import torch.nn.functional as F

import dwarf_b200
from dwarf_b200 import _lib

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _close(x, ref, rel, name):
    x, ref = x.double(), ref.double()
    assert torch.isfinite(x).all() and (x - ref).norm() <= rel * ref.norm() + 1e-6, (name, (x - ref).norm().item(), ref.norm().item())


@pytest.mark.parametrize("rows,D", [(1, 8), (3, 40), (8, 256), (301, 264), (2400, 512), (33, 1024)])
def test_layer_norm_and_column_sums(rows, D):
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, w, b, dy, dyb = rnd(rows, D) * 2 + 0.5, rnd(D), rnd(D), rnd(rows, D), rnd(rows, D).bfloat16()
    y, yb, stat = torch.empty_like(x), torch.empty_like(dyb), torch.empty(rows, 2, device="cuda")
    _lib.check(lib.dsqg_layer_norm_fwd(x.data_ptr(), w.data_ptr(), b.data_ptr(), 1e-5, y.data_ptr(), yb.data_ptr(), stat.data_ptr(), rows, D, _stream()), "fwd")
    xr, wr, br = (t.double().requires_grad_(True) for t in (x, w, b))
    ref = F.layer_norm(xr, (D,), wr, br, 1e-5)
    _close(y, ref.detach(), 1e-5, "y")
    assert torch.equal(yb, y.bfloat16())
    dx, dwb = torch.empty_like(x), torch.empty(2, D, device="cuda")
    n = lib.dsqg_layer_norm_bwd_scratch_bytes(rows, D)
    sc = torch.empty(n, dtype=torch.uint8, device="cuda")
    _lib.check(lib.dsqg_layer_norm_bwd(x.data_ptr(), stat.data_ptr(), w.data_ptr(), dy.data_ptr(), dyb.data_ptr(), dx.data_ptr(), dwb.data_ptr(),
                                       sc.data_ptr(), n, rows, D, _stream()), "bwd")
    grads = torch.autograd.grad(ref, [xr, wr, br], dy.double() + dyb.double())
    for got, want, nm in zip((dx, dwb[0], dwb[1]), grads, ("dx", "dgamma", "dbeta")):
        _close(got, want, 1e-5, nm)
    # two matrices at once, the second a block of columns of a wider one
    wide = rnd(rows, D + 72).bfloat16()
    out = torch.empty(D + 64, device="cuda")
    arr = lambda t, v: (t * 2)(*v)  # noqa: E731
    _lib.check(lib.dsqg_column_sums(arr(ctypes.c_void_p, [dyb.data_ptr(), wide.data_ptr() + 16]), arr(ctypes.c_longlong, [D, D + 72]), arr(ctypes.c_int, [D, 64]),
                                    arr(ctypes.c_void_p, [out.data_ptr(), out.data_ptr() + 4 * D]), 2, rows, _stream()), "sums")
    _close(out, torch.cat([dyb.double().sum(0), wide[:, 8:72].double().sum(0)]), 1e-5, "sums")


@pytest.mark.parametrize("B,N,D", [(1, 1, 8), (2, 31, 72), (1, 33, 64), (3, 257, 40), (1, 1025, 256), (1, 5000, 64)])
def test_gated_mean(B, N, D):
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(N)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, gate, dinter = rnd(B, N, D), rnd(B, N, D).bfloat16(), rnd(B, N, D).bfloat16()
    pool, inter = torch.empty_like(x), torch.empty_like(gate)
    _lib.check(lib.dsqg_gated_mean(x.data_ptr(), gate.data_ptr(), pool.data_ptr(), inter.data_ptr(), B, N, D, _stream()), "fwd")
    xr, gr = x.double().requires_grad_(True), gate.double().requires_grad_(True)
    pr = xr.cumsum(1) / torch.arange(1, N + 1, device="cuda")[None, :, None]
    ref = torch.sigmoid(gr) * pr
    _close(pool, pr.detach(), 1e-5, "pool")
    _close(inter, ref.detach(), 4e-3, "inter")
    dg, dx = torch.empty_like(gate), torch.empty_like(x)
    _lib.check(lib.dsqg_gated_mean_bwd(dinter.data_ptr(), gate.data_ptr(), pool.data_ptr(), dg.data_ptr(), dx.data_ptr(), B, N, D, _stream()), "bwd")
    want = torch.autograd.grad(ref, [xr, gr], dinter.double())
    _close(dx, want[0], 1e-2, "dx")
    _close(dg, want[1], 1e-2, "dg")


@pytest.mark.parametrize("B,N,dim,H", [(1, 1, 64, 2), (2, 33, 256, 8), (1, 300, 128, 2), (3, 129, 96, 3), (8, 2048, 256, 8)])
@pytest.mark.parametrize("inject", [False, True])
def test_layer_under_autocast_vs_fp32(B, N, dim, H, inject):
    torch.manual_seed(N)
    attn = dwarf_b200.DSQGAttentionQW(dim, H, dropout=0.0).cuda()
    block = dwarf_b200.InterferenceInjection(dim, H).cuda()
    torch.nn.init.normal_(attn.scale_embed, 0, 0.1)
    x = torch.randn(B, N, dim, device="cuda", requires_grad=True)
    dy = torch.randn(B, N, dim, device="cuda").bfloat16()
    named = [("x", x), *attn.named_parameters()] + (list(block.named_parameters()) if inject else [])

    def run(autocast):
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=autocast):
            deltas = block(x) if inject else None
            y = attn(x, kv_inject=deltas)
        extra = [deltas[0]] if inject else []
        return [y.detach()] + list(torch.autograd.grad(y, [p for _, p in named] + extra, dy.to(y.dtype)))
    got, want = run(True), run(False)
    dk = want[-1].double().norm()
    for (name, _), a, b in zip([("y", None)] + named, got, want):
        assert a.shape == b.shape
        a, b = a.double(), b.double()
        if name == "inter_k_proj.bias":
            # a bias on every key moves all scores of a query alike: zero but for the rounding to bf16 of dk's rows, of the ds they are summed
            # from and of the output that delta is formed from, each about 2^-9 of dk and of either sign
            assert a.norm() <= 6 * 2.0 ** -9 * dk + 2.0 ** -8 * (N == 1) * a.numel() ** 0.5, (name, a.norm().item(), dk.item())
        elif not b.any():
            # one tap: ds = dP - delta, two forms of one number of size one, the second from an output rounded to bf16
            assert N == 1 and a.norm() <= 2.0 ** -8 * a.numel() ** 0.5, (name, a.norm().item())
        else:
            assert (a - b).norm() <= 3e-2 * b.norm(), (name, (a - b).norm().item(), b.norm().item())


@pytest.mark.parametrize("B,N,dim,H", [(1, 1, 64, 2), (3, 701, 256, 8), (2, 97, 96, 3), (1, 300, 1024, 16), (8, 2048, 256, 8)])
def test_native_layer_gives_what_its_modules_give(B, N, dim, H):
    """A hook on one projection sends the layer and the interference block through their modules.  The forward rounds at the same places: deltas and output
    bit for bit.  With them the key gradients agree, and so does even the gradient of the bias on every key, a sum of nothing but their rounding errors;
    the other gradients are rounded to bf16 at different places on the way (weights: once more in the modules)."""
    torch.manual_seed(N)
    attn = dwarf_b200.DSQGAttentionQW(dim, H, dropout=0.0).cuda()
    block = dwarf_b200.InterferenceInjection(dim, H).cuda()
    torch.nn.init.normal_(attn.scale_embed, 0, 0.1)
    x = torch.randn(B, N, dim, device="cuda", requires_grad=True)
    dy = torch.randn(B, N, dim, device="cuda").bfloat16()
    named = [("x", x), *attn.named_parameters(), *block.named_parameters()]

    def run(modules):
        hooks = [m.register_forward_hook(lambda *a: None) for m in (attn.qkv_proj, block.inter_gate)] if modules else []
        with torch.autocast("cuda", dtype=torch.bfloat16):
            kd, vd = block(x)
            y = attn(x, kv_inject=(kd, vd))
        for h in hooks:
            h.remove()
        return [kd.detach(), vd.detach(), y.detach()], torch.autograd.grad(y, [p for _, p in named], dy)
    (fwd, got), (fwd_m, want) = run(False), run(True)
    for a, b, n in zip(fwd, fwd_m, ("k_delta", "v_delta", "y")):
        assert torch.equal(a, b), n
    for (n, _), a, b in zip(named, got, want):
        a, b = a.double(), b.double()
        assert (a - b).norm() <= 1e-2 * b.norm(), (n, (a - b).norm().item(), b.norm().item())


def _off_by_one(t):
    """The same values one element off an aligned address (a view of a flat buffer)."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    view = flat[1:].view(t.shape)
    view.copy_(t)
    assert view.data_ptr() % 16 and view.is_contiguous()
    return view


@pytest.mark.parametrize("x_type", [torch.float32, torch.bfloat16])
def test_layer_takes_tensors_at_any_address(x_type):
    """Parameters, inputs, deltas and the upstream gradient that do not start on 16 bytes give what aligned ones give."""
    B, N, dim, H = 2, 65, 128, 4
    torch.manual_seed(1)
    attn = dwarf_b200.DSQGAttentionQW(dim, H, dropout=0.0).cuda()
    block = dwarf_b200.InterferenceInjection(dim, H).cuda()
    x0 = torch.randn(B, N, dim, device="cuda", dtype=x_type)
    dy0 = torch.randn(B, N, dim, device="cuda").bfloat16()
    d0 = torch.randn(B, N, dim, device="cuda").bfloat16()
    # scale_embed has to be aligned for the operator itself, with or without a layer around it
    moved = [(m, n) for mod in (attn, block) for m in mod.modules() for n, _ in m.named_parameters(recurse=False) if n != "scale_embed"]
    results = []
    for off in (False, True):
        place = _off_by_one if off else torch.clone
        for m, n in moved:
            setattr(m, n, torch.nn.Parameter(place(getattr(m, n).detach())))
        x, delta = place(x0).requires_grad_(True), place(d0)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = attn(x, kv_inject=block(x))
            y2 = attn(x, kv_inject=(delta.view(B, N, H, dim // H).transpose(1, 2),) * 2)
        wrt = [x, *attn.parameters(), *block.parameters()]
        results.append([y.detach(), y2.detach(), *torch.autograd.grad(y, wrt, place(dy0))])
    for a, b in zip(*results):
        assert torch.equal(a, b)


def test_frozen_parameters_get_no_gradient_and_cost_none():
    """Each gradient on its own equals its part of the full set, and a backward for the input alone makes no weight gradients."""
    B, N, dim, H = 1, 65, 1024, 16
    torch.manual_seed(3)
    attn = dwarf_b200.DSQGAttentionQW(dim, H, dropout=0.0).cuda()
    block = dwarf_b200.InterferenceInjection(dim, H).cuda()
    torch.nn.init.normal_(attn.scale_embed, 0, 0.1)
    x = torch.randn(B, N, dim, device="cuda", requires_grad=True)
    dy = torch.randn(B, N, dim, device="cuda").bfloat16()
    params = [x, *attn.parameters(), *block.parameters()]

    def run():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return attn(x, kv_inject=block(x))
    want = torch.autograd.grad(run(), params, dy)
    for i, p in enumerate(params):
        for q in params:
            q.requires_grad_(q is p)
        got = torch.autograd.grad(run(), [p], dy)[0]
        # one product over fewer columns may be cut up in another way
        assert got.dtype == want[i].dtype and (got - want[i]).norm() <= 1e-5 * want[i].norm(), i
        y = run()
        y.backward(dy)
        assert all((q.grad is not None) == (q is p) for q in params)
        p.grad = None
    for q in params:
        q.requires_grad_(q is x)
    y = run()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    torch.autograd.grad(y, [x], dy)
    # scratch and activations of 65 rows against 32 MB of weight gradients
    assert torch.cuda.max_memory_allocated() - before < 16 << 20


@pytest.mark.parametrize("dim,H", [(256, 8), (256, 4)])
def test_what_a_layer_keeps_for_its_backward(dim, H):
    """Between forward and backward: x and the result of the operator in bf16, and once q, k, v and the gate (head width 32: as copies
    that stand in for the projection's output), row statistics, weights in bf16; the layer's output besides."""
    B, N = 4, 2048
    attn = dwarf_b200.DSQGAttentionQW(dim, H, dropout=0.0).cuda()
    x = torch.randn(B, N, dim, device="cuda", requires_grad=True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        attn(x).sum().backward()                          # workspaces of the first call
        x.grad = None
        attn.zero_grad(set_to_none=True)
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        y = attn(x)
    torch.cuda.synchronize()
    unit = B * N * dim * 2
    most = (1 + 1 + 4 + 1) * unit + B * H * N * 4 + (5 * dim * dim + 5 * dim) * 2
    assert torch.cuda.memory_allocated() - before <= most + (1 << 20), (torch.cuda.memory_allocated() - before) / unit
    y.float().sum().backward()


def test_results_may_be_changed_in_place():
    """As those of the modules: the layer's output and the deltas are tensors of their own to autograd."""
    torch.manual_seed(4)
    attn = dwarf_b200.DSQGAttentionQW(64, 2, dropout=0.0).cuda()
    block = dwarf_b200.InterferenceInjection(64, 2).cuda()
    x = torch.randn(2, 40, 64, device="cuda", requires_grad=True)
    params = [x, *attn.parameters(), *block.parameters()]

    def run(in_place):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            kd, vd = block(x)
            kd = kd.mul_(2) if in_place else kd * 2
            y = attn(x, kv_inject=(kd, vd))
        y = y.mul_(4) if in_place else y * 4
        return torch.autograd.grad(y, params, torch.ones_like(y))
    for a, b in zip(run(True), run(False)):
        assert torch.equal(a, b)


def test_a_subclass_may_bring_its_own_attend():
    class Scaled(dwarf_b200.DSQGAttentionQW):
        def attend(self, x, kv_inject=None):
            y, k, v = super().attend(x, kv_inject)
            return y * 2, k, v
    torch.manual_seed(0)
    a, b = dwarf_b200.DSQGAttentionQW(64, 2, dropout=0.0).cuda(), Scaled(64, 2, dropout=0.0).cuda()
    b.load_state_dict(a.state_dict())
    x = torch.randn(2, 20, 64, device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert torch.equal(b(x), a(x) * 2)


def test_tensors_elsewhere_are_refused_on_the_host():
    """A parameter or delta on the CPU raises before anything is launched."""
    q = torch.randn(1, 2, 40, 32, device="cuda").bfloat16()
    offsets = dwarf_b200.OFFSETS_43
    pb, gain = torch.zeros(len(offsets), 2), torch.ones(2)
    for p, g in ((pb, None), (pb.cuda(), gain)):
        with pytest.raises(ValueError, match="cuda:0"):
            dwarf_b200.dsqg_attention(q, q, q, p, g, None, offsets)
        with pytest.raises(ValueError, match="cuda:0"):
            dwarf_b200.dsqg_attention_packed(torch.randn(1, 40, 3, 2, 32, device="cuda").bfloat16(), p, g, None, offsets)
        cache = dwarf_b200.DSQGRingCache(1, 3, 2, 32)
        cache.advance()
        with pytest.raises(ValueError, match="cuda:0"):
            cache.step(0, *(torch.zeros(3, 2, 32, device="cuda", dtype=torch.bfloat16) for _ in range(3)), p, g)
    attn = dwarf_b200.DSQGAttentionQW(64, 2, dropout=0.0).cuda()
    delta = torch.zeros(1, 2, 40, 32)
    with torch.autocast("cuda", dtype=torch.bfloat16), pytest.raises(RuntimeError):
        attn(torch.randn(1, 40, 64, device="cuda"), kv_inject=(delta, delta))


# rows: less than a stage, its edges, more blocks than steps, all eight blocks of a cluster with a ragged end; cols and D: tiles half empty,
# two widths, several across.  dy is a block of columns of a wider matrix; the second job may lack its sums.
@pytest.mark.parametrize("rows,D,cols", [(1, 64, (64,)), (63, 64, (128, 64)), (65, 128, (192, 128)), (511, 192, (576, 192)), (513, 256, (1024, 256)),
                                         (300, 512, (2048, 512)), (4099, 256, (512, 256)), (777, 320, (64, 704))])
def test_weight_grads(rows, D, cols):
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    wide = [rnd(rows, c + 24) for c in cols]
    dy, x = [w[:, 8:8 + c] for w, c in zip(wide, cols)], [rnd(rows, D) for _ in cols]
    dw = [torch.full((c + 1, D), 7.0, device="cuda") for c in cols]
    sums = [torch.full((c + 1,), 7.0, device="cuda") for c in cols]
    arr = lambda t, v: (t * len(v))(*v)  # noqa: E731
    ptrs = lambda ts: arr(ctypes.c_void_p, [t.data_ptr() for t in ts])  # noqa: E731

    def call(sum_ptrs, D=D, cols=cols, rows=rows):
        return lib.dsqg_weight_grads(ptrs(dy), arr(ctypes.c_longlong, [w.stride(0) for w in wide]), arr(ctypes.c_int, list(cols)), ptrs(x), ptrs(dw), sum_ptrs,
                                     len(cols), rows, D, _stream())
    _lib.check(call(ptrs(sums)), "weight_grads")
    first = [w.clone() for w in dw]
    # one tensor-core step takes 16 products and rounds once: at most rows / 16 roundings of 2^-23 of the running sum
    rel = 2.0 ** -23 * max(8, rows / 16)
    for d, xx, w, s, c in zip(dy, x, dw, sums, cols):
        _close(w[:c], d.double().t() @ xx.double(), rel, "dw")
        _close(s[:c], d.double().sum(0), rel, "sums")
        assert (w[c] == 7).all() and s[c] == 7                       # nothing past the end
    for w in dw:
        w.zero_()
    _lib.check(call(arr(ctypes.c_void_p, [0] * len(cols))), "weight_grads without sums")
    assert all(torch.equal(a[:c], b[:c]) for a, b, c in zip(first, dw, cols))      # the same bits on every call
    assert all(s[c] == 7 for s, c in zip(sums, cols))
    assert call(ptrs(sums), D=D + 8) == call(ptrs(sums), cols=[c + 8 for c in cols]) == call(ptrs(sums), rows=0) == -2


@pytest.mark.parametrize("dim,N", [(128, 97), (256, 300)])
def test_weight_gradients_of_a_layer_with_and_without_split_sums(dim, N):
    """A caller who allows no split of a sum gets one GEMM per weight; the gradients are those of the one launch."""
    torch.manual_seed(dim)
    with torch.device("cuda"):
        attn, inject = dwarf_b200.DSQGAttentionQW(dim, dim // 32, seq_len=N, dropout=0.0), dwarf_b200.InterferenceInjection(dim, dim // 32)
    x, dy = torch.randn(2, N, dim, device="cuda"), torch.randn(2, N, dim, device="cuda").bfloat16()
    wrt = [*attn.parameters(), *inject.parameters()]

    def grads():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = attn(x, kv_inject=inject(x))
        return torch.autograd.grad(y, wrt, dy)
    was = torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction
    one = grads()
    try:
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = (False, False)
        many = grads()
    finally:
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = was
    for a, b in zip(one, many):
        _close(a, b, 2e-3, "gradient")        # the projections' GEMMs may round other bf16 values when they may not split


_NO_TENSOR_MAPS = """
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)         # ahead of the library's own symbol
import torch
from tests.test_gpu_layer import _layer_gradients
torch.save([t.cpu() for t in _layer_gradients(128, 97)], sys.argv[2])
assert fake.fake_calls() == 2
"""


def _layer_gradients(dim, N):
    torch.manual_seed(dim)
    with torch.device("cuda"):
        attn, inject = dwarf_b200.DSQGAttentionQW(dim, dim // 32, seq_len=N, dropout=0.0), dwarf_b200.InterferenceInjection(dim, dim // 32)
        x, dy = torch.randn(2, N, dim, requires_grad=True), torch.randn(2, N, dim).bfloat16()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = attn(x, kv_inject=inject(x))
    return torch.autograd.grad(y, [x, *attn.parameters(), *inject.parameters()], dy)


def test_a_layer_without_tensor_maps_takes_its_gemms(tmp_path):
    """Where the driver makes no tensor maps dsqg_weight_grads is refused, and the backward has GEMMs for the same gradients.  The refusal comes
    from a stand-in for the entry that a child process loads first."""
    import subprocess
    import sys
    from tests.conftest import ROOT
    src, lib, out = tmp_path / "fake.c", tmp_path / "fake.so", tmp_path / "grads.pt"
    src.write_text("static int calls; int dsqg_weight_grads(void) { ++calls; return -8; } int fake_calls(void) { return calls; }")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    subprocess.run([sys.executable, "-c", _NO_TENSOR_MAPS, str(lib), str(out)], check=True, cwd=ROOT, timeout=300)
    for a, b in zip(torch.load(out), _layer_gradients(128, 97)):
        _close(a.cuda(), b, 2e-3, "gradient")         # the sums are formed in another order; one of them nearly cancels


def test_a_wait_that_gave_up_is_reported_by_the_next_backward():
    """Gradients of a kernel whose wait ran out are NaN; whoever goes on training on them hears of it, and can go on once the word is cleared."""
    lib = _lib.load()
    want = _layer_gradients(128, 97)
    assert lib.dsqg_device_error(1) == 0
    _lib.check(lib.dsqg_test_wait_timeout(20000, _stream()), "wait")
    torch.cuda.synchronize()
    for _ in range(2):                                               # until it is cleared
        with pytest.raises(_lib.DSQGError, match="status -10: .* gave up"):
            _layer_gradients(128, 97)
    assert lib.dsqg_device_error(1) == 0x7e57 and lib.dsqg_device_error(0) == 0
    assert all(torch.equal(a, b) for a, b in zip(want, _layer_gradients(128, 97)))


@pytest.mark.parametrize("rows,D,cols", [(64, 128, (128,)), (700, 192, (320, 64)), (4099, 256, (1024, 256))])
def test_weight_grads_whose_waits_run_out_are_nan_throughout(rows, D, cols):
    """A block that never gets the second half of its rows: every weight gradient and every column sum is NaN, the words say so, and the next call is as before."""
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(rows)
    dy, x = ([torch.randn(rows, c, generator=g, device="cuda").bfloat16() for c in cs] for cs in (cols, [D] * len(cols)))
    dw, sums = [torch.empty(c + 1, D, device="cuda") for c in cols], [torch.empty(c + 1, device="cuda") for c in cols]
    arr = lambda t, v: (t * len(v))(*v)  # noqa: E731
    ptrs = lambda ts: arr(ctypes.c_void_p, [t.data_ptr() for t in ts])  # noqa: E731
    args = (ptrs(dy), arr(ctypes.c_longlong, cols), arr(ctypes.c_int, cols), ptrs(x), ptrs(dw), ptrs(sums), len(cols), rows, D)

    def call(timeout):
        for t in (*dw, *sums):
            t.fill_(7.0)
        _lib.check(lib.dsqg_test_weight_grads_timeout(*args, 1000000, _stream()) if timeout else lib.dsqg_weight_grads(*args, _stream()), "weight_grads")
        torch.cuda.synchronize()
        return [t.clone() for t in (*dw, *sums)]
    want = call(False)
    for t in call(True):
        assert t[:-1].isnan().all() and (t[-1] == 7).all()               # and nothing past the end
    assert lib.dsqg_weight_grads(*args, _stream()) == -10
    assert lib.dsqg_device_error(1) & ~0xf == 0x500 and lib.dsqg_device_error(0) == 0
    assert all(torch.equal(a, b) for a, b in zip(want, call(False)))
