"""Dense products with four and with eight epilogue warps: grids of one tile, of exactly one wave, of one tile more, and of two and three waves, with
rows that TMA can and cannot address, against the integer product (bit for bit)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant, M, N", [("pair", 256, 256), ("pair", 256, 74 * 256), ("pair", 256, 75 * 256), ("pair", 250, 74 * 256 - 5), ("pair", 250, 149 * 256 - 5),
                                           ("dense_bn256", 128, 148 * 256), ("dense_bn256", 128, 148 * 256 + 1), ("dense_bn256", 100, 297 * 256 - 3),
                                           ("dense_bn128", 128, 148 * 128), ("dense_bn128", 128, 149 * 128), ("dense_bn64", 37, 148 * 64), ("dense_bn64", 37, 149 * 64 + 9)])
def test_epilogue_warps(variant, M, N):
    import gemm_int8_b200 as g

    K = 144
    gen = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    y = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    want = x.float() @ y.float().t()   # exact: |sum| <= 144 * 2^14 < 2^24
    try:
        g.force_variant(variant)
        assert torch.equal(g.matmul(x, y), want.to(torch.bfloat16))
        sx, sw = torch.rand(M, device="cuda", generator=gen), torch.rand(N, device="cuda", generator=gen)
        assert torch.equal(g.matmul_scaled(x, y, sx, sw), (want * (sx[:, None] * sw[None, :])).to(torch.bfloat16))
    finally:
        g.force_variant(None)
    assert g.device_status() == 0
