"""Order of the library's launches in a stream.  Every launch is a programmatic dependent: it may be resident while the kernel in
front of it runs, products behind a quantiser request their weights early, and the second launch of a split product reads its
operands without waiting.  Here the library's own kernels, which let the next one start before they have ended, follow one another
directly (no copies or torch kernels between them, which would order everything); data alternate, so that a read that came too
early, or a write that overtook its reader, would show.  The bits must be those of ordinary launches (GEMM_INT8_PDL=0)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

# mode, M, N, K, what the product runs on (kind as in pick_variant: 1 scaled, 2 blockwise)
FORMS = [
    ("channel", 16, 8192, 1024, "smallm_cluster"),
    ("channel", 16, 1024, 8192, "smallm_cluster"),            # K splits
    ("channel", 100, 5008, 1040, "dense_bn64"),
    ("channel", 300, 28672, 1040, "dense_bn256"),             # waves over ragged rows: the quantiser releases as it ends
    ("channel", 777, 4096, 1024, "pair"),
    ("channel", 130, 1024, 16384, "splitk8"),                 # 64 CTAs
    ("channel", 100, 13952, 14336, "splitk2"),                # 110 CTAs
    ("channel", 1024, 14336, 8192, "pair+splitk8"),           # two launches
    ("blockwise", 16, 2048, 1024, "blockwise_bn64"),
    ("blockwise", 100, 5008, 1040, "blockwise_bn64"),
    ("blockwise", 300, 8192, 1024, "blockwise_bn256"),
    ("blockwise", 300, 16384, 1040, "blockwise_bn256"),       # waves over ragged rows
    ("blockwise", 512, 10240, 8192, "blockwise_bn256+columns_bn64"),   # two launches
    ("blockwise", 700, 8192, 12288, "blockwise_pair"),
]


@pytest.fixture(scope="module")
def g():
    import gemm_int8_b200

    yield gemm_int8_b200
    assert gemm_int8_b200.device_status() == 0


@pytest.fixture()
def ordinary(g, monkeypatch):
    """Runs a function with ordinary, fully ordered launches."""
    def run(fn):
        monkeypatch.setenv("GEMM_INT8_PDL", "0")
        g.reload_env()
        try:
            out = fn()
            torch.cuda.synchronize()
            return out
        finally:
            monkeypatch.delenv("GEMM_INT8_PDL")
            g.reload_env()

    return run


def _layer(g, mode, N, K, gen, bias=True):
    w = torch.randint(-127, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    scale = torch.rand(*((-(-N // 128), -(-K // 128)) if mode == "blockwise" else (N,)), device="cuda", generator=gen) * 0.01
    b = torch.randn(N, device="cuda", generator=gen).to(torch.bfloat16) if bias else None
    return g.Int8Linear(w, scale, b, mode=mode)


def _inputs(M, K, gen):
    return [torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16) * (i + 1) for i in range(2)]


def _same(outs, want):
    for i, out in enumerate(outs):
        assert torch.equal(out.view(torch.int16), want[i % 2].view(torch.int16)), i


def _run(step, captured, n=12):
    """Outputs of step(0), step(1), step(0), ... launched back to back, or of two steps captured and replayed."""
    if not captured:
        return [step(i % 2) for i in range(n)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        step(0)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        outs = [step(0), step(1)]
    for _ in range(n):
        graph.replay()
    torch.cuda.synchronize()
    return outs


@pytest.mark.parametrize("mode, M, N, K, form", FORMS)
@pytest.mark.parametrize("captured", [False, True])
def test_layer_behind_layer(g, ordinary, mode, M, N, K, form, captured):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    assert g.pick_variant(2 if mode == "blockwise" else 1, M, N, K) == form
    first = _layer(g, mode, N, K, gen)
    seconds = [_layer(g, m, 512, N, gen) for m in ("channel", "blockwise")]
    xs = _inputs(M, K, gen)
    for second in seconds:
        step = lambda i: second(first(xs[i]))
        _same(_run(step, captured), ordinary(lambda: [step(0), step(1)]))


@pytest.mark.parametrize("kind, M, N, K", [(0, 100, 4096, 1040), (2, 100, 4096, 1040),      # let the next launch start when they have waited
                                           (0, 100, 5008, 1040), (2, 100, 5008, 1040), (2, 300, 16384, 1040),   # as they end
                                           (0, 70, 14336, 16400)])                          # an ordinary launch
@pytest.mark.parametrize("captured", [False, True])
def test_product_quantiser_product(g, ordinary, kind, M, N, K, captured):
    """Products on quantised operands, with the readers of their results directly behind."""
    gen = torch.Generator(device="cuda").manual_seed(N)
    i8 = lambda *shape: torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=gen)
    xs, w, w2, sw2 = [i8(M, K), i8(M, K)], i8(N, K), i8(512, N), torch.rand(512, device="cuda", generator=gen)
    scales = torch.rand(M, -(-K // 128), device="cuda", generator=gen), torch.rand(-(-N // 128), -(-K // 128), device="cuda", generator=gen)

    def step(i):
        y = g.matmul(xs[i], w, 0.01) if kind == 0 else g.matmul_blockwise(xs[i], w, *scales)
        q, s = g.quantize_per_token(y)
        return g.matmul_scaled(q, w2, s, sw2)

    _same(_run(step, captured), ordinary(lambda: [step(0), step(1)]))


def _quantise_into(g, mode, a, q, s):
    fn = g._C.gi8_quantize_token_block if mode == "blockwise" else g._C.gi8_quantize_token
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = fn(p(a), 1, p(q), p(s), a.shape[0], a.shape[1], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, g._C.gi8_last_error()


@pytest.mark.parametrize("mode, M, N, K, form", [f for f in FORMS if f[2] * f[3] < 2**24])
@pytest.mark.parametrize("between", [False, True])
@pytest.mark.parametrize("captured", [False, True])
def test_layer_behind_the_quantiser_of_its_weights(g, ordinary, mode, M, N, K, form, between, captured):
    """The kernel in front of the layer, or one small-M product further back, writes its weights (and per-row scales)."""
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    layer = _layer(g, mode, N, K, gen)
    sources = _inputs(N, K, gen)
    scales = layer.weight_scale if mode == "channel" else torch.empty(N, -(-K // 128), device="cuda")
    other = (torch.randint(-128, 128, (16, 1024), dtype=torch.int8, device="cuda", generator=gen),
             torch.randint(-128, 128, (8192, 1024), dtype=torch.int8, device="cuda", generator=gen),
             torch.rand(16, device="cuda", generator=gen), torch.rand(8192, device="cuda", generator=gen))
    x = _inputs(M, K, gen)[0]

    def step(i):
        _quantise_into(g, mode, sources[i], layer.weight_q, scales)
        if between:
            g.matmul_scaled(*other)
        return layer(x)

    _same(_run(step, captured), ordinary(lambda: [step(0), step(1)]))


@pytest.mark.parametrize("captured", [False, True])
def test_operand_written_on_another_stream(g, ordinary, captured):
    """A product whose stream joins another one directly in front of it: the event orders it behind the writer there, although its own
    launch need not wait for the end of the kernel in front."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    M, N, K = 16, 8192, 1024
    sources = _inputs(N, K, gen)
    w, s = torch.empty(N, K, dtype=torch.int8, device="cuda"), torch.empty(N, device="cuda")
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    sx = torch.rand(M, device="cuda", generator=gen)
    side = torch.cuda.Stream()

    def step(i):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            _quantise_into(g, "channel", sources[i], w, s)
        g.matmul(x, x)               # the kernel in front in this stream
        main.wait_stream(side)
        return g.matmul_scaled(x, w, sx, s)

    _same(_run(step, captured), ordinary(lambda: [step(0), step(1)]))
