"""The small-M blockwise kernel with four and with six stages (grids of more and of fewer CTAs than SMs, short and long K, alone and behind a
layer's quantiser, with and without a bias), against the 64-wide tiles (the same bits; those are compared with the oracle elsewhere)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# four stages; six (128 and 148 CTAs, long K, the second with an odd count of K blocks); four (one CTA more than SMs)
@pytest.mark.parametrize("M, N, K", [(16, 7552, 8192), (16, 8192, 8192), (3, 9472, 8208), (16, 9473, 8192), (16, 8192, 8176), (1, 512, 16400)])
def test_product(M, N, K):
    import gemm_int8_b200 as g

    gen = torch.Generator(device="cuda").manual_seed(N + K)
    kb = -(-K // 128)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    y = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    sa, sw = torch.rand(M, kb, device="cuda", generator=gen), torch.rand(-(-N // 128), kb, device="cuda", generator=gen)
    out = g.matmul_blockwise(x, y, sa, sw)
    try:
        g.force_variant("dense_bn64")
        assert torch.equal(out, g.matmul_blockwise(x, y, sa, sw))
    finally:
        g.force_variant(None)
    assert g.device_status() == 0


@pytest.mark.parametrize("M, N, K", [(1, 264, 16), (16, 4096, 1040), (9, 9472, 1664), (16, 9473, 1040), (16, 14336, 1040), (5, 14344, 2048)])
@pytest.mark.parametrize("bias", [False, True])
def test_layer(M, N, K, bias):
    import gemm_int8_b200 as g

    gen = torch.Generator(device="cuda").manual_seed(N + K)
    layer = g.Int8Linear.from_float(torch.randn(N, K, device="cuda", generator=gen), torch.randn(N, device="cuda", generator=gen).to(torch.bfloat16) if bias else None,
                                    mode="blockwise")
    for _ in range(4):  # back to back: the next call's CTAs start beside this one's
        x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
        out = layer(x)
        try:
            g.force_variant("dense_bn64")
            assert torch.equal(out, layer(x))
        finally:
            g.force_variant(None)
    assert g.device_status() == 0
