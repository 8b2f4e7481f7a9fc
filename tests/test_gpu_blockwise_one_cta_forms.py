"""256-wide one-CTA blockwise tiles: grids of up to two waves run the form whose partial buffers share their barriers with the stages, longer ones
the decoupled form.  Both sides of the line, at counts of K blocks that leave stages and buffers in every relation, against the 128-wide
tiles (the same bits; those are compared with the oracle elsewhere)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [16, 128, 272, 384, 512, 640, 1152, 1536])
@pytest.mark.parametrize("tiles", [1, 148, 149, 296, 297, 445])
def test_forms(tiles, K):
    import gemm_int8_b200 as g

    M, N = 100, 256 * tiles - 56
    gen = torch.Generator(device="cuda").manual_seed(tiles + K)
    kb = -(-K // 128)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    y = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    sa, sw = torch.rand(M, kb, device="cuda", generator=gen), torch.rand(-(-N // 128), kb, device="cuda", generator=gen)
    try:
        g.force_variant("dense_bn256")
        out = g.matmul_blockwise(x, y, sa, sw)
        g.force_variant("dense_bn128")
        assert torch.equal(out, g.matmul_blockwise(x, y, sa, sw))
    finally:
        g.force_variant(None)
    assert g.device_status() == 0


@pytest.mark.parametrize("tiles, K", [(149, 640), (296, 384), (297, 640), (445, 512)])
def test_forms_with_bias(tiles, K):
    import gemm_int8_b200 as g

    M, N = 100, 256 * tiles
    gen = torch.Generator(device="cuda").manual_seed(tiles + K)
    layer = g.Int8Linear.from_float(torch.randn(N, K, device="cuda", generator=gen), torch.randn(N, device="cuda", generator=gen).to(torch.bfloat16),
                                    mode="blockwise")
    x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    try:
        g.force_variant("dense_bn256")
        out = layer(x)
        g.force_variant("dense_bn128")
        assert torch.equal(out, layer(x))
    finally:
        g.force_variant(None)
    assert g.device_status() == 0
