"""GEMM_INT8_STATIC_WEIGHTS=1 promises that the weight operand of the scaled product is not written by the work directly in front of
it.  What the promise does not cover must be ordered as without it: the second operand of the plain product, and weights that a
kernel further back in the stream writes.  The writers here are the library's own quantisers, which let the next kernel start before
they have written anything; the data alternate, so that a read that came too early would see the other set.  All checks are
bit comparisons with the oracle."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def g(monkeypatch):
    import gemm_int8_b200

    monkeypatch.setenv("GEMM_INT8_STATIC_WEIGHTS", "1")
    gemm_int8_b200.reload_env()
    yield gemm_int8_b200
    monkeypatch.delenv("GEMM_INT8_STATIC_WEIGHTS")
    gemm_int8_b200.reload_env()
    assert gemm_int8_b200.device_status() == 0


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _quantise_into(g, a, q, s):
    """Per-row quantiser into fixed buffers (the operators allocate theirs)."""
    rc = g._C.gi8_quantize_token(_p(a), 1, _p(q), _p(s), a.shape[0], a.shape[1], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, g._C.gi8_last_error()


def _pair(M, K, gen):
    return [torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2)]


@pytest.mark.parametrize("M, N, K", [(1, 4096, 4096), (16, 8192, 1024), (64, 2048, 8192), (16, 1001, 272)])
def test_plain_product_of_an_operand_quantised_in_front(g, oracle, M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(N)
    assert g.pick_variant(0, M, N, K) == "smallm_cluster"
    sources = _pair(N, K, gen)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    want = [oracle.c_matmul(x.cpu(), g.quantize_per_token(a)[0].cpu(), -0.37) for a in sources]
    y, s = torch.empty(N, K, dtype=torch.int8, device="cuda"), torch.empty(N, device="cuda")
    outs = []
    for i in range(40):
        _quantise_into(g, sources[i % 2], y, s)
        outs.append(g.matmul(x, y, -0.37))
    for i, out in enumerate(outs):
        assert np.array_equal(oracle.bf16_bits(out), want[i % 2]), i


def _product_in_front(g, form, gen):
    """A call of this library that stands between the writer of the weights and their reader."""
    M = 16
    if form in ("smallm", "smallm_split", "dense"):
        M, N, K = (200, 2048, 1024) if form == "dense" else (16, 16384, 512) if form == "smallm" else (16, 1024, 8192)
        x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
        w = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
        sx, sw = torch.rand(M, device="cuda", generator=gen), torch.rand(N, device="cuda", generator=gen)
        return lambda: g.matmul_scaled(x, w, sx, sw)
    layer = g.Int8Linear.from_float(torch.randn(1024, 1024, device="cuda", generator=gen), mode=form)
    x = torch.randn(M, 1024, device="cuda", generator=gen).to(torch.bfloat16)
    return lambda: layer(x)


@pytest.mark.parametrize("form", ["smallm", "smallm_split", "dense", "channel", "blockwise"])
@pytest.mark.parametrize("captured", [False, True])
def test_weights_written_two_calls_back(g, oracle, form, captured):
    """writer of w -> another product -> product with w: w is not written by the work directly in front, so the promise holds."""
    gen = torch.Generator(device="cuda").manual_seed(7)
    M, N, K = 16, 8192, 1024
    sources = _pair(N, K, gen)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    sx = torch.rand(M, device="cuda", generator=gen)
    quantised = [g.quantize_per_token(a) for a in sources]
    want = [oracle.c_matmul_scaled(x.cpu(), q.cpu(), sx.cpu(), s.cpu()) for q, s in quantised]
    between = _product_in_front(g, form, gen)
    first = between().clone()
    w, sw = torch.empty(N, K, dtype=torch.int8, device="cuda"), torch.empty(N, device="cuda")

    def step(i):
        _quantise_into(g, sources[i % 2], w, sw)
        other = between()
        return g.matmul_scaled(x, w, sx, sw), other

    if captured:
        step(0)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = [step(i) for i in range(4)]
        for _ in range(10):
            graph.replay()
    else:
        outs = [step(i) for i in range(40)]
    for i, (out, other) in enumerate(outs):
        assert np.array_equal(oracle.bf16_bits(out), want[i % 2]), i
        assert torch.equal(other.view(torch.int16), first.view(torch.int16)), i


@pytest.mark.parametrize("blockwise, M", [(1, 128), (0, 64), (0, 200)])
def test_weights_written_by_the_quantiser_of_the_layer_in_front(g, oracle, blockwise, M):
    """The quantised activations of a layer are the weights of the product behind it: the layer's own product, which may request
    its weights under its quantiser, stands between their writer and their reader."""
    gen = torch.Generator(device="cuda").manual_seed(13)
    N, K = 2048, 1024
    if blockwise:
        assert g.pick_variant(2, M, N, K) in ("blockwise_bn64", "blockwise_bn128")
    sources = _pair(M, K, gen)
    layer = g.Int8Linear.from_float(torch.randn(N, K, device="cuda", generator=gen), mode="blockwise" if blockwise else "channel")
    a = torch.randint(-128, 128, (16, K), dtype=torch.int8, device="cuda", generator=gen)
    sx, sw = torch.rand(16, device="cuda", generator=gen), torch.rand(M, device="cuda", generator=gen)
    quantise = g.quantize_per_token_block if blockwise else g.quantize_per_token
    want = [(oracle.c_matmul_scaled(a.cpu(), quantise(x)[0].cpu(), sx.cpu(), sw.cpu()), layer(x)) for x in sources]
    xq, xs = torch.empty(M, K, dtype=torch.int8, device="cuda"), torch.empty(M, 8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    outs = []
    for i in range(40):
        out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        rc = g._C.gi8_linear(_p(sources[i % 2]), 1, _p(layer.weight_q), _p(layer.weight_scale), K // 128, None, blockwise, 0, _p(xq), _p(xs), _p(out),
                             M, N, K, stream)
        assert rc == 0, g._C.gi8_last_error()
        outs.append((g.matmul_scaled(a, xq, sx, sw), out))
    for i, (scaled, out) in enumerate(outs):
        assert np.array_equal(oracle.bf16_bits(scaled), want[i % 2][0]), i
        assert torch.equal(out.view(torch.int16), want[i % 2][1].view(torch.int16)), i
