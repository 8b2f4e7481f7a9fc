"""Block-scaled products of up to sixteen tokens run on a kernel of their own (64 weight rows against 16 tokens): bit equality with the oracle
at the edges of its tiles, at odd counts of K blocks, around the depth of its rings (four stages of two K blocks; six: see the test of the stages), for scales
whose products overflow or vanish, and for outputs of odd width; the seventeenth token is another kernel's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, N, K", [(1, 8, 16), (1, 1000, 1024), (16, 64, 128), (16, 65, 272), (9, 129, 1296), (5, 14337, 144), (16, 2048, 8192),
                                     (8, 63, 256), (7, 264, 1040), (15, 9472, 1664), (15, 9473, 1664), (2, 9600, 1040), (16, 4096, 4112), (17, 264, 1040)])
def test_small_m(oracle, M, N, K):
    import gemm_int8_b200 as g

    gen = torch.Generator().manual_seed(M + N)
    KB, NB = -(-K // 128), -(-N // 128)
    x = torch.randint(-128, 128, (M, K), generator=gen, dtype=torch.int8)
    y = torch.randint(-128, 128, (N, K), generator=gen, dtype=torch.int8)
    x[0], y[0] = -128, -128
    sa, sw = torch.rand(M, KB, generator=gen) + 0.5, torch.rand(NB, KB, generator=gen) - 0.5
    for factor in (1.0, 1e-38, 2.0**110):
        want = oracle.c_matmul_blockwise(x, y, sa * factor, sw)
        got = g.matmul_blockwise(x.cuda(), y.cuda(), (sa * factor).cuda(), sw.cuda())
        assert np.array_equal(oracle.bf16_bits(got), want), factor
    assert g.device_status() == 0
