"""Dense epilogue: a warp's two staging blocks alternate from store to store, also across tiles that hold an odd number of 32-column chunks (the
last column tile where N % 64 is 8 to 32, and 64-wide tiles under eight epilogue warps).  Many tiles per CTA and a short K, so that
stores follow one another closely, against the integer product (bit for bit)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant, M, N", [("pair", 56832, 32), ("pair", 37888, 288), ("pair", 19000, 352), ("dense_bn256", 56832, 24), ("dense_bn256", 28416, 608),
                                           ("dense_bn128", 56832, 96), ("dense_bn128", 28416, 160), ("dense_bn64", 56832, 32), ("dense_bn64", 28416, 96),
                                           ("dense_bn64", 18944, 64), ("dense_bn64", 148 * 128, 24)])
@pytest.mark.parametrize("K", [16, 256])
def test_blocks_alternate(variant, M, N, K):
    import gemm_int8_b200 as g

    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    y = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    want = (x.float() @ y.float().t()).to(torch.bfloat16)   # exact: |sum| <= 256 * 2^14 = 2^22
    try:
        g.force_variant(variant)
        for _ in range(8):
            assert torch.equal(g.matmul(x, y), want)
    finally:
        g.force_variant(None)
    assert g.device_status() == 0
