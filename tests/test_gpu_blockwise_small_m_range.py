"""What the small-M blockwise kernel has to take as the tiles do: strided scale rows, scales up to infinities and NaN, outputs that are two-byte aligned
(with their neighbours untouched), launches of the library directly behind it; and that the dispatch reaches it, by the name of the kernel that ran."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, seed=1):
    gen = torch.Generator().manual_seed(seed)
    kb, nb = -(-K // 128), -(-N // 128)
    return (torch.randint(-128, 128, (M, K), generator=gen, dtype=torch.int8), torch.randint(-128, 128, (N, K), generator=gen, dtype=torch.int8),
            torch.rand(M, kb, generator=gen) + 0.5, torch.rand(nb, kb, generator=gen) - 0.5)


@pytest.mark.parametrize("M, N, K", [(1, 264, 512), (16, 264, 1168), (7, 9601, 400)])
@pytest.mark.parametrize("pad_a, pad_w", [(5, 3), (0, 1), (3, 0)])
def test_strided_scales(oracle, M, N, K, pad_a, pad_w):
    import gemm_int8_b200 as g

    x, y, sa, sw = _operands(M, N, K)
    kb = sa.shape[1]
    big_a, big_w = torch.full((M, kb + pad_a), float("nan")).cuda(), torch.full((sw.shape[0], kb + pad_w), float("nan")).cuda()
    big_a[:, :kb], big_w[:, :kb] = sa.cuda(), sw.cuda()
    got = g.matmul_blockwise(x.cuda(), y.cuda(), big_a[:, :kb], big_w[:, :kb])
    assert np.array_equal(oracle.bf16_bits(got), oracle.c_matmul_blockwise(x, y, sa, sw))


@pytest.mark.parametrize("sa_factor, sw_factor", [(1e-30, 1e-12), (1e-20, 1e-18), (2.0**60, 2.0**46), (-1e33, 1.0), (1e30, 1e30), (float("inf"), 1.0),
                                                  (1.0, float("-inf")), (float("nan"), 1.0), (1.0, float("nan")), (float("inf"), 0.0)])
def test_scale_range(oracle, sa_factor, sw_factor):
    import gemm_int8_b200 as g

    for M, N, K in [(5, 264, 144), (16, 70, 512), (1, 130, 1024)]:
        x, y, sa, sw = _operands(M, N, K, M)
        x[: M // 2], y[: N // 4] = -128, 127
        y[-1] = 0                      # zero partials against infinite scales
        sa[::3] *= sa_factor
        sw[:, 1:] *= sw_factor
        if M > 1:
            sa[1, 0] = 0.0
        want = oracle.c_matmul_blockwise(x, y, sa, sw)
        got = oracle.bf16_bits(g.matmul_blockwise(x.cuda(), y.cuda(), sa.cuda(), sw.cuda()))
        nan = (want & 0x7FFF) > 0x7F80
        assert np.array_equal((got & 0x7FFF) > 0x7F80, nan) and np.array_equal(got[~nan], want[~nan]), (M, N, K)


@pytest.mark.parametrize("M, N, K", [(1, 130, 272), (16, 65, 512), (3, 128, 128)])
@pytest.mark.parametrize("offset", [1, 2, 3, 7])
def test_output_alignment(oracle, M, N, K, offset):
    import gemm_int8_b200 as g

    x, y, sa, sw = _operands(M, N, K)
    out = torch.full((M * N + 32,), 12345, dtype=torch.int16, device="cuda")
    args = [t.cuda() for t in (x, y, sa, sw)]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = g._C.gi8_matmul_blockwise(p(args[0]), p(args[1]), p(args[2]), sa.shape[1], p(args[3]), sw.shape[1], ctypes.c_void_p(out.data_ptr() + 2 * offset),
                                   M, N, K, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, g._C.gi8_last_error()
    got = out.cpu().numpy()
    assert np.array_equal(got[offset:offset + M * N].view(np.uint16).reshape(M, N), oracle.c_matmul_blockwise(x, y, sa, sw))
    assert (got[:offset] == 12345).all() and (got[offset + M * N:] == 12345).all()


@pytest.mark.parametrize("N, K", [(14336, 1040), (4096, 1040)])   # four and six stages behind the quantiser
def test_layer_behind_layer(monkeypatch, N, K):
    """Alternating inputs through two layers, launched without anything between them: the bits of ordinary, fully ordered launches."""
    import gemm_int8_b200 as g

    gen = torch.Generator(device="cuda").manual_seed(N)
    make = lambda n, k: g.Int8Linear.from_float(torch.randn(n, k, device="cuda", generator=gen), torch.randn(n, device="cuda", generator=gen).to(torch.bfloat16), mode="blockwise")
    first, second = make(N, K), make(9600, N)
    xs = [torch.randn(16, K, device="cuda", generator=gen).to(torch.bfloat16) * (i + 1) for i in range(2)]
    monkeypatch.setenv("GEMM_INT8_PDL", "0")
    g.reload_env()
    try:
        want = [second(first(x)) for x in xs]
        torch.cuda.synchronize()
    finally:
        monkeypatch.delenv("GEMM_INT8_PDL")
        g.reload_env()
    for i, out in enumerate([second(first(xs[i % 2])) for i in range(12)]):
        assert torch.equal(out.view(torch.int16), want[i % 2].view(torch.int16)), i


def _kernels_of(fn):
    from torch.profiler import ProfilerActivity, profile

    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    return [e.name for e in p.events() if "gi8::" in e.name]


@pytest.mark.parametrize("M, N, K, small", [(1, 264, 512, "<4>"), (16, 264, 512, "<4>"), (16, 8192, 8192, "<6>"), (16, 9473, 8192, "<4>"), (17, 264, 512, None)])
def test_kernel_that_runs(M, N, K, small):
    import gemm_int8_b200 as g

    args = [t.cuda() for t in _operands(M, N, K)]
    names = _kernels_of(lambda: g.matmul_blockwise(*args))
    if not names:
        pytest.skip("no kernel records from the profiler")
    assert len(names) == 1
    assert ("blockwise_smallm_kernel" + small in names[0]) if small else ("blockwise_gemm_kernel" in names[0])
    assert g.pick_variant(2, M, N, K) == "blockwise_bn64"
