"""Thin dense grids with a long K: split over K where the split-K kernel can write the rows, narrow tiles where it cannot."""
import numpy as np
import pytest
import torch


def test_rows_the_split_kernel_cannot_write_keep_narrow_tiles():
    import gemm_int8_b200 as g

    pv = g.pick_variant
    for kind in (0, 1):
        assert pv(kind, 200, 4096, 28672) == "splitk4" and pv(kind, 200, 4104, 28672).startswith("splitk")
        assert pv(kind, 200, 4097, 28672) == "dense_bn64" and pv(kind, 200, 4100, 28672) == "dense_bn64"
        assert pv(kind, 128, 1000, 28672) == "splitk8" and pv(kind, 128, 1001, 28672) == "dense_bn64"
        assert pv(kind, 1024, 14336, 16384) == "pair+splitk8" and pv(kind, 1024, 14335, 16384) == "pair"


@pytest.mark.gpu
@pytest.mark.parametrize("M, N, K", [(200, 1001, 8192), (100, 1004, 12304), (130, 257, 16384), (500, 1001, 4112)])
def test_ragged_thin_grids_match_oracle(oracle, M, N, K):
    import gemm_int8_b200 as g

    gen = torch.Generator().manual_seed(N)
    x = torch.randint(-128, 128, (M, K), generator=gen, dtype=torch.int8)
    y = torch.randint(-128, 128, (N, K), generator=gen, dtype=torch.int8)
    sx, sw = torch.rand(M, generator=gen), torch.rand(N, generator=gen)
    xd, yd = x.cuda(), y.cuda()
    assert np.array_equal(oracle.bf16_bits(g.matmul(xd, yd, -0.37)), oracle.c_matmul(x, y, -0.37))
    assert np.array_equal(oracle.bf16_bits(g.matmul_scaled(xd, yd, sx.cuda(), sw.cuda())), oracle.c_matmul_scaled(x, y, sx, sw))
    assert np.array_equal(g.matmul_i32(xd, yd).cpu().numpy(), oracle.c_matmul_i32(x, y))
