"""The work a user of this package has it do, as a list of measurable cases.

A case is one call through the public entry points with operands already on the GPU: the plain `matmul`, the
W8A8 `matmul_scaled` / `matmul_blockwise` on operands that were quantised before, and `Int8Linear`, which quantises
its activations on the fly (that is where the activation quantisers and the Hadamard rotation are met in use).  The
path is inference only, so there is no backward direction; decode is small M, prefill large M.

Fields of a case:
    kind      "plain" | "scaled" | "blockwise" | "linear"
    M, N, K   tokens, output features, input features
    alpha     plain: the scalar of the epilogue
    mode      linear: "channel" (per-token x per-channel scales) or "blockwise" (128-wide blocks)
    hadamard  linear, blockwise: rotation block (0: none)
    bias      linear: whether the layer has one
    act       linear: dtype of the activations, "bf16" or "fp32"
"""
from __future__ import annotations

import math

import torch

import gemm_int8_b200 as g

_COST_LIMIT = 2 * 16384 * 57344 * 8192  # operations of the largest listed case
_SIZE_LIMIT = 2_600_000_000             # bytes of operands and result of the largest listed case


def _case(name, kind, M, N, K, **more):
    c = {"name": name, "kind": kind, "M": M, "N": N, "K": K, "alpha": 1.0, "mode": "", "hadamard": 0, "bias": False, "act": ""}
    c.update(more)
    return c


def listed():
    return [
        # One decoded token through a square projection: the smallest call, where launches and host time count.
        _case("decode1_channel", "linear", 1, 4096, 4096, mode="channel", act="bf16"),
        # A decode batch through an up-projection with a bias; the weights are most of the bytes.
        _case("decode16_channel_bias", "linear", 16, 14336, 4096, mode="channel", act="bf16", bias=True),
        # A larger decode batch through a down-projection; the caller quantised the activations itself.
        _case("decode64_scaled", "scaled", 64, 4096, 14336),
        # A decode batch of a model whose weights carry 128 x 128 block scales.
        _case("decode16_blockwise", "linear", 16, 8192, 8192, mode="blockwise", act="bf16"),
        # The README's example of the plain product.
        _case("plain_1024x4096x4096", "plain", 1024, 4096, 4096),
        # A ragged plain product: no dimension is a whole number of tiles, output rows are not 16-byte aligned.
        _case("plain_ragged", "plain", 777, 5003, 3088, alpha=-0.37),
        # A large square product, bound by the tensor cores.
        _case("plain_8192", "plain", 8192, 8192, 8192),
        # Prefill with per-channel weights, a batch of prompts, bias.
        _case("prefill_channel_bias", "linear", 4096, 4096, 14336, mode="channel", act="bf16", bias=True),
        # Prefill with block scales (2048 tokens, up-projection).
        _case("prefill_blockwise", "linear", 2048, 11008, 4096, mode="blockwise", act="bf16"),
        # A short prompt of odd length through a fused qkv projection, rotated fp32 activations, bias.
        _case("prompt_hadamard_fp32", "linear", 499, 10240, 8192, mode="blockwise", act="fp32", hadamard=8192, bias=True),
        # Prefill of a long down-projection with rotated activations.
        _case("prefill_hadamard", "linear", 2048, 8192, 28672, mode="blockwise", act="bf16", hadamard=4096),
        # The largest single-GPU product: a whole batch of prompts through an up-projection, operands quantised before.
        _case("large_blockwise", "blockwise", 16384, 57344, 8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(["plain", "scaled", "blockwise", "linear", "linear", "linear"])
        M = _log_int(rng, 1, 64) if rng.random() < 0.35 else _log_int(rng, 64, 16384)
        N = _log_int(rng, 1024, 57344)
        if rng.random() < 0.7:
            N = max(128, N // 128 * 128)          # layers are usually wide multiples; the rest is as drawn, odd ones too
        K = max(16, _log_int(rng, 1024, 28672) // 16 * 16)
        c = _case("", kind, M, N, K)
        del c["name"]
        if kind == "plain":
            c["alpha"] = rng.choice([1.0, round(rng.uniform(-2.0, 2.0), 3)])
        if kind == "linear":
            c["mode"] = rng.choice(["channel", "blockwise"])
            c["bias"] = rng.random() < 0.5
            c["act"] = rng.choice(["bf16", "bf16", "fp32"])
            if c["mode"] == "blockwise" and rng.random() < 0.6:
                block = rng.choice([128, 256, 512, 1024, 2048, 4096, 8192])
                c["K"] = K = max(block, K // block * block)
                c["hadamard"] = block
        if 2 * M * N * K <= _COST_LIMIT and work(c)["bytes"] <= _SIZE_LIMIT:
            return c


def _activations(M, K, gen, dtype):
    """Gaussian activations with a thousandth of the channels twenty times as large, as layer inputs have them."""
    a = torch.randn(M, K, generator=gen, device="cuda")
    a[:, torch.randperm(K, generator=gen, device="cuda")[: max(1, round(0.001 * K))]] *= 20.0
    return a.to(dtype)


def _inputs(case, seed):
    """The tensors of a case: operands and scales, or a layer's float weight, bias and activations."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    M, N, K = case["M"], case["N"], case["K"]

    def int8(rows):
        return torch.randint(-128, 127, (rows, K), dtype=torch.int8, device="cuda", generator=gen)

    def scales(*shape):
        return torch.rand(*shape, device="cuda", generator=gen) * 0.02 + 0.001

    if case["kind"] == "plain":
        return dict(x=int8(M), y=int8(N))
    if case["kind"] == "scaled":
        return dict(x=int8(M), y=int8(N), sx=scales(M), sw=scales(N))
    if case["kind"] == "blockwise":
        kb = -(-K // 128)
        return dict(x=int8(M), y=int8(N), sx=scales(M, kb), sw=scales(-(-N // 128), kb))
    w = torch.randn(N, K, generator=gen, device="cuda") * 0.02
    bias = (torch.randn(N, generator=gen, device="cuda") * 0.1).to(torch.bfloat16) if case["bias"] else None
    return dict(w=w, bias=bias, x=_activations(M, K, gen, torch.bfloat16 if case["act"] == "bf16" else torch.float32))


def prepare(case, seed):
    t = _inputs(case, seed)
    if case["kind"] != "linear":
        return dict(t, kind=case["kind"], alpha=case["alpha"])
    layer = g.Int8Linear.from_float(t["w"], t["bias"], mode=case["mode"], hadamard_block=case["hadamard"] or None)
    return {"kind": "linear", "layer": layer, "x": t["x"]}


def run(state):
    kind = state["kind"]
    if kind == "plain":
        return g.matmul(state["x"], state["y"], state["alpha"])
    if kind == "scaled":
        return g.matmul_scaled(state["x"], state["y"], state["sx"], state["sw"])
    if kind == "blockwise":
        return g.matmul_blockwise(state["x"], state["y"], state["sx"], state["sw"])
    return state["layer"](state["x"])


def work(case):
    """Each operand read once, the bf16 result written once; two integer operations per multiply-add."""
    M, N, K = case["M"], case["N"], case["K"]
    kb, nb = -(-K // 128), -(-N // 128)
    nbytes = N * K + 2 * M * N
    if case["kind"] == "linear":
        nbytes += M * K * (2 if case["act"] == "bf16" else 4) + 4 * (N if case["mode"] == "channel" else nb * kb)
        nbytes += 2 * N if case["bias"] else 0
    else:
        nbytes += M * K + {"plain": 0, "scaled": 4 * (M + N), "blockwise": 4 * kb * (M + nb)}[case["kind"]]
    return {"bytes": nbytes, "flops": 2 * M * N * K}


def tolerance(case):
    """Four times what one bf16 rounding of a result evaluated in 64 bits was seen to give (2-norm 1.65e-3, largest
    3.9e-3 of the value; the integer sums are exact and the fp32 sums over K blocks add 1e-7); a bias is added in bf16
    after the first rounding and rounds once more (2-norm 2.3e-3, largest 7.6e-3 of the larger of value and rms)."""
    if case["bias"]:
        return {"rel": 9.5e-3, "max": 3.0e-2}
    return {"rel": 6.6e-3, "max": 1.6e-2}


def _rotate64(a, block):
    """Normalised Walsh-Hadamard transform of the rows in blocks of `block`, as a product with the matrix."""
    h = torch.ones(1, 1, dtype=torch.float64, device=a.device)
    while h.shape[0] < block:
        h = torch.cat((torch.cat((h, h), 1), torch.cat((h, -h), 1)), 0)
    return ((a.reshape(-1, block) @ h) * block ** -0.5).reshape(a.shape)


def _rounded(a, rows, cols):
    """What symmetric int8 quantisation leaves of `a`, one scale per rows x cols tile, in the precision of `a`."""
    R, C = a.shape
    p = torch.nn.functional.pad(a, (0, -C % cols, 0, -R % rows))
    t = p.reshape(p.shape[0] // rows, rows, p.shape[1] // cols, cols)
    s = t.abs().amax(dim=(1, 3), keepdim=True) / 127.0
    s = torch.where(s > 0, s, torch.ones_like(s))
    return (torch.round(t / s).clamp(-127, 127) * s).reshape(p.shape)[:R, :C]


def exact(case, seed):
    """The result in 64 bits.  Quantisation is part of what a layer computes and is carried out in 64 bits as well."""
    t = _inputs(case, seed)
    M, N, K = case["M"], case["N"], case["K"]
    x = t.pop("x").double()
    if case["kind"] == "linear":
        w = t.pop("w").double()
        if case["hadamard"]:
            x, w = _rotate64(x, case["hadamard"]), _rotate64(w, case["hadamard"])
        blocks = case["mode"] == "blockwise"
        x = _rounded(x, 1, 128 if blocks else K)
        w = _rounded(w, 128 if blocks else 1, 128 if blocks else K)
        out = x @ w.t()
        return out if t["bias"] is None else out + t["bias"].double()
    y = t.pop("y").double()
    if case["kind"] == "blockwise":
        x *= t["sx"].double().repeat_interleave(128, dim=1)[:, :K]
        y *= t["sw"].double().repeat_interleave(128, dim=1)[:, :K].repeat_interleave(128, dim=0)[:N]
    out = x @ y.t()
    if case["kind"] == "scaled":
        out *= t["sx"].double()[:, None] * t["sw"].double()[None, :]
    return out * case["alpha"] if case["kind"] == "plain" else out
