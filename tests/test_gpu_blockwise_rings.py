"""256-wide blockwise tiles: the partial buffers restart with every tile while the operand stages run on, so that tiles of an odd count of
K blocks leave the two rings in every relation to each other.  Several tiles per CTA, against the narrow tiles (the same bits; those
are compared with the oracle elsewhere)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [16, 128, 256, 272, 384, 512, 640, 896, 1040, 1408])
@pytest.mark.parametrize("variant", ["dense_bn256", "pair"])
def test_rings(variant, K):
    import gemm_int8_b200 as g

    M, N = 900, 12040   # 376 or 192 tiles on 148 or 74 slots
    gen = torch.Generator(device="cuda").manual_seed(K)
    kb = -(-K // 128)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    y = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    sa, sw = torch.rand(M, kb, device="cuda", generator=gen), torch.rand(-(-N // 128), kb, device="cuda", generator=gen)
    try:
        g.force_variant(variant)
        out = g.matmul_blockwise(x, y, sa, sw)
        g.force_variant("dense_bn128")
        assert torch.equal(out, g.matmul_blockwise(x, y, sa, sw))
    finally:
        g.force_variant(None)
    assert g.device_status() == 0
