"""Column splits of even and of odd counts of row blocks (the first launch runs on one-CTA tiles for both), against the 128-wide tiles (the same
bits; those are compared with the oracle elsewhere)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, N, K", [(512, 10240, 512), (385, 10240, 272), (256, 19200, 640), (130, 19200, 144), (128, 38400, 384), (100, 38408, 512)])
def test_column_split_pairs(monkeypatch, M, N, K):
    import gemm_int8_b200 as g

    gen = torch.Generator(device="cuda").manual_seed(M)
    kb = -(-K // 128)
    x = torch.randint(-128, 128, (M, K), dtype=torch.int8, device="cuda", generator=gen)
    y = torch.randint(-128, 128, (N, K), dtype=torch.int8, device="cuda", generator=gen)
    sa, sw = torch.rand(M, kb, device="cuda", generator=gen), torch.rand(-(-N // 128), kb, device="cuda", generator=gen)
    monkeypatch.setenv("GEMM_INT8_TAIL_SPLIT", "2")
    g.reload_env()
    try:
        assert "+columns_bn" in g.pick_variant(2, M, N, K)
        out = g.matmul_blockwise(x, y, sa, sw)
        g.force_variant("dense_bn128")
        assert torch.equal(out, g.matmul_blockwise(x, y, sa, sw))
    finally:
        g.force_variant(None)
        monkeypatch.delenv("GEMM_INT8_TAIL_SPLIT", raising=False)
        g.reload_env()
    assert g.device_status() == 0
