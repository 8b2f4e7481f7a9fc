"""The two-CTA blockwise tile on grids of few waves: taken for long K, unless a column split promises more."""
import pytest
import torch


def test_long_k_takes_the_two_cta_tile():
    import gemm_int8_b200 as g

    pv = g.pick_variant
    assert pv(2, 2048, 8192, 28672) == "blockwise_pair" and pv(2, 700, 9001, 12288) == "blockwise_pair"
    assert pv(2, 700, 9000, 12272) == "blockwise_pair"            # 96 K blocks, the last one ragged
    assert pv(2, 700, 9000, 12160) == "blockwise_bn256"           # 95 K blocks
    assert "+columns_bn" in pv(2, 512, 10240, 28672)              # one full wave and twelve tiles
    assert pv(2, 2048, 28672, 14336) == "blockwise_pair"          # twelve waves and sixteen tiles
    assert pv(2, 16, 8192, 28672) == "blockwise_bn64"


@pytest.mark.gpu
@pytest.mark.parametrize("M, N, K", [(2000, 4800, 12288), (700, 9001, 12272), (512, 10240, 12416)])
def test_long_k_matches_one_cta_tiles(M, N, K):
    """(The one-CTA tiles are compared with the oracle elsewhere; same operation order, so the bits are equal.)"""
    import gemm_int8_b200 as g

    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    y = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    kb = -(-K // 128)
    sa, sw = torch.rand(M, kb, device="cuda", generator=gen), torch.rand(-(-N // 128), kb, device="cuda", generator=gen)
    out = g.matmul_blockwise(x, y, sa, sw)
    g.force_variant("dense_bn128")
    try:
        assert torch.equal(out, g.matmul_blockwise(x, y, sa, sw))
    finally:
        g.force_variant(None)
