"""The work whose speed is measured: what programs built on this package have it do.

A case is a dict of plain values with a "kind":

  infer   `dsqg_attention` without gradients (prompt processing, evaluation)
  train   `dsqg_attention` forward and backward through autograd (the operator in a training step)
  packed  `dsqg_attention_packed` forward and backward: q, k, v in the projection output, gated token-major result
  layer   a condU attention layer with K/V injection (`DSQGAttentionQW` + `InterferenceInjection`) under bf16
          autocast, forward and backward, parameter gradients included
  decode  one token for every sequence through all DSQG layers of a model (`DSQGRingCache.advance` + `.step`)

Values and distributions are those of the benchmark configurations (`dwarf_b200.synth`): q, k, v ~ N(0, 0.25), upstream
gradients ~ N(0, 1), position bias -alpha_h log(1 + delta) plus noise, head gains in [0.8, 1.2], full rings ~ N(0, 1).
"""
import torch

import dwarf_b200
from dwarf_b200.synth import log_linear_pos_bias

_DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
# 43: dense 0..31 and eleven sparse taps up to 1536; 44: the reference's own set (dense 0..32); 45: 43 extended for N = 4096
_OFFSETS = {43: dwarf_b200.OFFSETS_43, 44: dwarf_b200.ALL_OFFSETS, 45: dwarf_b200.OFFSETS_45}


def _op(kind, B, H, N, D, offsets=43, dtype="bf16", gain=True, scale_embed=False, **more):
    return dict(kind=kind, B=B, H=H, N=N, D=D, offsets=offsets, dtype=dtype, gain=gain, scale_embed=scale_embed, **more)


def listed():
    return [
        # one short prompt of odd length through one layer: launches and host time count
        _op("infer", 1, 8, 300, 32, name="prompt 1x8x300x32"),
        # a training step of a small or debugging run, ragged length
        _op("train", 2, 8, 777, 32, name="train 2x8x777x32"),
        # fp32 parity / evaluation runs of the op (benchmark configuration 0)
        _op("infer", 2, 8, 2048, 32, dtype="fp32", gain=False, name="fp32 infer 2x8x2048x32"),
        # the 13M-model training shape (benchmark configuration 1)
        _op("train", 32, 8, 2048, 32, name="train 32x8x2048x32"),
        # the same shape with the condU operator: reference offset set, scale_embed
        _op("train", 32, 8, 2048, 32, offsets=44, scale_embed=True, name="train condU 32x8x2048x32"),
        # the 85M-model training shape at head width 64 (benchmark configuration 2), and its long-sequence form
        _op("train", 16, 12, 2048, 64, name="train 16x12x2048x64"),
        _op("train", 16, 12, 4096, 64, offsets=45, name="train 16x12x4096x64"),
        # the reference's 85M condM model: head width 80
        _op("train", 8, 8, 2048, 80, offsets=44, gain=False, name="train 8x8x2048x80"),
        # what a condM layer calls in a training step: packed projection output, sigmoid gate
        _op("packed", 32, 8, 2048, 32, gain=False, name="packed 32x8x2048x32"),
        # one condU layer of a training step with the interference block's K/V injection
        _op("layer", 8, 8, 2048, 32, offsets=44, scale_embed=True, name="layer condU 8x2048x256"),
        # serving: 256 sequences, ten layers, full rings (benchmark configuration 3), and a few sequences after a prompt
        dict(kind="decode", S=256, H=12, D=64, layers=10, prompt=0, name="decode 256x12x64 10 layers"),
        dict(kind="decode", S=4, H=8, D=32, layers=5, prompt=500, name="decode 4x8x32 5 layers"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["infer", "train", "train", "packed", "layer", "decode"])
    if kind == "decode":
        return dict(kind="decode", S=_log_uniform(rng, 1, 256), H=rng.choice([8, 12]), D=rng.choice([32, 64]),
                    layers=rng.randint(1, 10), prompt=rng.choice([0, 0, rng.randint(1, 2000)]))
    H = rng.choice([8, 12])
    long = rng.random() < 0.2
    N = rng.randint(2049, 4096) if long else rng.choice([2048, _log_uniform(rng, 64, 2047), _log_uniform(rng, 64, 2047)])
    offsets = 45 if long else rng.choice([43, 44])
    if kind == "layer":
        B = _log_uniform(rng, 1, max(1, 65536 // N))
        return _op("layer", B, 8, min(N, 2048), 32, offsets=44, scale_embed=True)
    D = rng.choice([32, 32, 64, 64, 80, 128] if kind != "packed" else [32, 64])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp32"]) if kind == "infer" else "bf16"
    most = 50_000_000 if D <= 64 and dtype == "bf16" else 8_000_000
    B = _log_uniform(rng, 1, min(64, max(1, most // (H * N * D))))
    scale_embed = D <= 64 and dtype == "bf16" and rng.random() < 0.3
    return _op(kind, B, H, N, D, offsets=offsets, dtype=dtype, gain=rng.random() < 0.7, scale_embed=scale_embed)


def _prepare_decode(c, g):
    S, H, D, L = c["S"], c["H"], c["D"], c["layers"]
    cache = dwarf_b200.DSQGRingCache(L, S, H, D)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    if c["prompt"]:
        for layer in range(L):
            cache.prefill(layer, rand(S, H, c["prompt"], D), rand(S, H, c["prompt"], D))
    else:
        cache.kv.normal_(generator=g)
        cache.head = torch.randint(0, cache.R, (S,), generator=g, device="cuda", dtype=torch.int32)
        cache.fill = torch.full((S,), cache.R, dtype=torch.int32, device="cuda")
    bias = log_linear_pos_bias(cache.offsets, H).cuda()
    return {"cache": cache, "qkv": [(rand(S, H, D), rand(S, H, D), rand(S, H, D)) for _ in range(L)],
            "bias": [bias + torch.randn(bias.shape, generator=g, device="cuda") * 0.05 for _ in range(L)],
            "gain": torch.rand(H, generator=g, device="cuda") * 0.4 + 0.8, "rings": [cache.kv[i] for i in range(L)]}


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(seed)
    if c["kind"] == "decode":
        return {"case": c, **_prepare_decode(c, g)}
    B, H, N, D = c["B"], c["H"], c["N"], c["D"]
    dtype, offsets = _DTYPES[c["dtype"]], _OFFSETS[c["offsets"]]
    J, grad = len(offsets), c["kind"] != "infer"
    rand = lambda *shape, std=1.0, dt=torch.float32: (torch.randn(*shape, generator=g, device="cuda", dtype=dt) * std)  # noqa: E731
    st = {"case": c, "offsets": offsets}
    if c["kind"] == "layer":
        dim = H * D
        with torch.random.fork_rng(devices=[0]):
            torch.manual_seed(seed)
            with torch.device("cuda"):
                attn = dwarf_b200.DSQGAttentionQW(dim, H, seq_len=N, dropout=0.0, offsets=offsets)
                inject = dwarf_b200.InterferenceInjection(dim, H)
        with torch.no_grad():
            attn.scale_embed.copy_(rand(J, D, std=0.1))
            attn.if_gain.copy_(torch.rand(H, generator=g, device="cuda") * 0.4 + 0.8)
        st.update(attn=attn, inject=inject, x=rand(B, N, dim).requires_grad_(True), dy=rand(B, N, dim, dt=torch.bfloat16))
        st["wrt"] = [st["x"], *attn.parameters(), *inject.parameters()]
        return st
    st["bias"] = (log_linear_pos_bias(offsets, H).cuda() + rand(J, H, std=0.05)).requires_grad_(grad)
    st["gain"] = (torch.rand(H, generator=g, device="cuda") * 0.4 + 0.8).requires_grad_(grad) if c["gain"] else None
    st["scale_embed"] = rand(J, D, std=0.1).requires_grad_(grad) if c["scale_embed"] else None
    if c["kind"] == "packed":
        st["qkv"] = rand(B, N, 3, H, D, std=0.5, dt=dtype).requires_grad_(True)
        st["gate"] = (rand(B, N, H * D, dt=dtype) + 2.0).requires_grad_(True)
        st["dy"] = rand(B, N, H * D, dt=dtype)
        wrt = [st["qkv"], st["gate"]]
    else:
        st["qkv"] = [rand(B, H, N, D, std=0.5, dt=dtype).requires_grad_(grad) for _ in range(3)]
        st["dy"] = rand(B, H, N, D, dt=dtype) if grad else None
        wrt = list(st["qkv"])
    st["wrt"] = wrt + [t for t in (st["bias"], st["gain"], st["scale_embed"]) if t is not None]
    return st


def run(st):
    c = st["case"]
    if c["kind"] == "decode":
        cache, outs = st["cache"], []
        cache.advance()
        for layer, (q, k, v) in enumerate(st["qkv"]):
            # from the second layer on, the kernel ahead in the stream writes neither write heads nor this layer's ring
            outs.append(cache.step(layer, q, k, v, st["bias"][layer], st["gain"], overlap=layer > 0))
        return {"out": outs, "head": cache.head, "fill": cache.fill, "rings": st["rings"]}
    if c["kind"] == "infer":
        with torch.no_grad():
            return dwarf_b200.dsqg_attention(*st["qkv"], st["bias"], st["gain"], st["scale_embed"], st["offsets"])
    if c["kind"] == "train":
        y = dwarf_b200.dsqg_attention(*st["qkv"], st["bias"], st["gain"], st["scale_embed"], st["offsets"])
    elif c["kind"] == "packed":
        y = dwarf_b200.dsqg_attention_packed(st["qkv"], st["bias"], st["gain"], st["gate"], st["offsets"], st["scale_embed"])
    else:
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = st["attn"](st["x"], kv_inject=st["inject"](st["x"]))
    return [y.detach(), *torch.autograd.grad(y, st["wrt"], st["dy"])]


def work(case):
    """Inputs once, outputs once; multiply-adds of the taps that exist (forward q.k and p.v; backward five products)."""
    c = case
    if c["kind"] == "decode":
        pairs, J = c["S"] * c["H"] * c["layers"], len(dwarf_b200.OFFSETS_43)
        fill = c["prompt"] + 1 if c["prompt"] else max(dwarf_b200.OFFSETS_43) + 1
        taps = sum(o < fill for o in dwarf_b200.OFFSETS_43)
        # key and value rows of the older taps; q, k, v in, the slot and the result out; biases and gains
        return {"bytes": pairs * (2 * (taps - 1) + 6) * c["D"] * 2 + c["layers"] * (J + 1) * c["H"] * 4 + c["S"] * 16,
                "flops": pairs * taps * 4 * c["D"]}
    B, H, N, D = c["B"], c["H"], c["N"], c["D"]
    offsets, size = _OFFSETS[c["offsets"]], 2 if c["dtype"] == "bf16" else 4
    tensor = B * H * N * D * size
    pairs = B * H * sum(max(0, N - o) for o in offsets)
    params = 4 * (len(offsets) * H + (H if c["gain"] else 0) + (len(offsets) * D if c["scale_embed"] else 0))
    if c["kind"] == "infer":
        return {"bytes": 4 * tensor + params, "flops": pairs * 4 * D}
    flops = pairs * 14 * D
    if c["kind"] == "layer":
        dim = H * D
        weights = 8 * dim * dim + 10 * dim + len(offsets) * (H + D) + H      # qkv, gate, out and the injection's three projections
        # x (fp32) and dy in, y and dx out, every weight read and its gradient written
        return {"bytes": B * N * dim * (4 + 2 + 2 + 4) + 8 * weights, "flops": flops + 6 * B * N * dim * dim * 8}
    tensors = 8 if c["kind"] == "train" else 10                                # the packed form also has the gate and its gradient
    return {"bytes": tensors * tensor + 2 * params, "flops": flops}


def tolerance(case):
    # fp32: sums of at most 43 * D products in another order; bf16: stored values carry eight bits
    if case.get("dtype") == "fp32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 1e-2, "max": 0.1}
