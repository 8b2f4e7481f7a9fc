"""The plain product of few tokens runs on the small-M kernel with scales 1 and alpha; bit equality with the oracle at the edges of
its token tiles, K splits and dispatch, and for alphas whose product with a scale of 1 must stay what it is."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M, N, K", [(1, 1, 16), (1, 1000, 1024), (16, 4096, 4096), (16, 129, 272), (9, 14337, 144), (17, 1000, 4096), (64, 264, 4112),
                                     (33, 1001, 8192), (64, 520, 4080), (65, 264, 4096)])
@pytest.mark.parametrize("alpha", [1.0, -0.37, 0.0, 3e38])
def test_plain_small_m(oracle, M, N, K, alpha):
    import gemm_int8_b200 as g

    gen = torch.Generator().manual_seed(M + N)
    x = torch.randint(-128, 128, (M, K), generator=gen, dtype=torch.int8)
    y = torch.randint(-128, 128, (N, K), generator=gen, dtype=torch.int8)
    small = M <= 16 or (M <= 64 and N <= 4096 and K >= 4096)
    assert (g.pick_variant(0, M, N, K) == "smallm_cluster") == small
    got = g.matmul(x.cuda(), y.cuda(), alpha)
    assert np.array_equal(oracle.bf16_bits(got), oracle.c_matmul(x, y, alpha))
