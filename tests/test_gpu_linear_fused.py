"""Int8Linear runs quantiser and product as one operator with the bias in the product's epilogue.  The result must be that of
the quantiser, the product and a bf16 addition called one after the other, bit for bit, on every kernel the product can
take: small M with and without K splits, narrow and wide tiles, two launches, ragged rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    import gemm_int8_b200

    return gemm_int8_b200


def _composed(g, layer, x):
    if layer.mode == "blockwise":
        xq, xs = g.quantize_per_token_block(x) if layer.hadamard_block is None else g.hadamard_quantize_per_token_block(x, layer.hadamard_block)
        out = g.matmul_blockwise(xq, layer.weight_q, xs, layer.weight_scale)
    else:
        out = g.matmul_scaled(*_swap(g.quantize_per_token(x), layer))
    return out if layer.bias is None else out + layer.bias.to(out.dtype)


def _swap(q, layer):
    return q[0], layer.weight_q, q[1], layer.weight_scale


def _layer(g, N, K, mode, had, bias, gen):
    w = torch.randn(N, K, device="cuda", generator=gen) * 0.02
    b = torch.randn(N, device="cuda", generator=gen).to(torch.bfloat16) if bias else None
    return g.Int8Linear.from_float(w, b, mode=mode, hadamard_block=had)


@pytest.mark.parametrize("mode, had", [("channel", None), ("blockwise", None), ("blockwise", 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_fused_equals_composed(g, mode, had, dtype):
    gen = torch.Generator(device="cuda").manual_seed(3)
    for M, N, K in [(1, 520, 512), (16, 4096, 1024), (33, 1001, 768), (64, 264, 2048), (65, 264, 256), (129, 777, 512), (300, 1000, 512),
                    (256, 512, 16384), (512, 10240, 2048)]:
        for bias in (False, True):
            layer = _layer(g, N, K, mode, had, bias, gen)
            for _ in range(2):
                x = (torch.randn(M, K, device="cuda", generator=gen) * 2).to(dtype)
                out = layer(x)
                assert torch.equal(out.view(torch.int16), _composed(g, layer, x).view(torch.int16)), (M, N, K, bias)
    assert g.device_status() == 0


@pytest.mark.parametrize("variant", ["dense_bn256", "dense_bn128", "dense_bn64", "pair", "smallm", "smallm_cluster"])
def test_fused_forced_variants(g, variant):
    gen = torch.Generator(device="cuda").manual_seed(5)
    g.force_variant(variant)
    try:
        for mode in ("channel", "blockwise"):
            for M, N, K in [(7, 520, 1040), (130, 300, 640)]:
                layer = _layer(g, N, K, mode, None, True, gen)
                x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
                assert torch.equal(layer(x).view(torch.int16), _composed(g, layer, x).view(torch.int16)), (mode, M, N, K)
    finally:
        g.force_variant(None)


def test_what_is_not_fused_and_what_is_refused(g):
    gen = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(2, 3, 256, device="cuda", generator=gen).to(torch.bfloat16)
    layer = _layer(g, 136, 256, "channel", None, True, gen)
    want = _composed(g, layer, x.reshape(6, 256)).reshape(2, 3, 136)
    assert torch.equal(layer(x), want)
    assert torch.equal(layer(x.transpose(0, 1)), want.transpose(0, 1))     # not contiguous
    layer.bias = layer.bias.float().reshape(1, 136)                        # broadcasts, another dtype
    assert torch.equal(layer(x), want)
    layer.bias = layer.bias.reshape(136).clone().requires_grad_()          # differentiated: stays a tensor addition
    layer(x).sum().backward()
    assert torch.equal(layer.bias.grad, torch.full((136,), 6.0, device="cuda"))
    assert layer(x[:0]).shape == (0, 3, 136)
    with pytest.raises(RuntimeError):
        layer(x[..., :128])
    with pytest.raises(RuntimeError):
        layer(x.cpu())
    rot = g.Int8Linear(layer.weight_q, torch.ones(2, 2, device="cuda"), mode="blockwise", hadamard_block=384)
    with pytest.raises(RuntimeError):
        rot(x)
    rot.hadamard_block = 0
    with pytest.raises(RuntimeError):
        rot(x)


@pytest.mark.parametrize("mode", ["channel", "blockwise"])
def test_fused_sees_what_was_just_written(g, mode):
    """Weights, scales, bias and activations replaced by device copies between the calls, on a side stream and in a captured graph.
    (Copies order what follows them, so this is about nothing being kept from one call to the next; the order behind kernels that
    let the next one start early is tested in test_gpu_launch_ordering.py.)"""
    gen = torch.Generator(device="cuda").manual_seed(11)
    a, b = (_layer(g, 2048, 4096, mode, None, True, gen) for _ in range(2))
    live = _layer(g, 2048, 4096, mode, None, True, gen)
    xs = [torch.randn(16, 4096, device="cuda", generator=gen).to(torch.bfloat16) for _ in range(2)]
    want = [_composed(g, l, x) for l, x in zip((a, b), xs)]
    x = torch.empty_like(xs[0])
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())

    def step(i):
        for dst, src in zip((live.weight_q, live.weight_scale, live.bias, x), ((a, b)[i].weight_q, (a, b)[i].weight_scale, (a, b)[i].bias, xs[i])):
            dst.copy_(src)
        return live(x)

    with torch.cuda.stream(stream):
        outs = [step(k % 2) for k in range(20)]
    stream.synchronize()
    for k, out in enumerate(outs):
        assert torch.equal(out, want[k % 2]), k
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        o0, o1 = step(0), step(1)
    for _ in range(5):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(o0, want[0]) and torch.equal(o1, want[1])
    assert g.device_status() == 0
