"""Blockwise scales over the whole fp32 range.  The 256-wide tiles promote partials through a factor 2^22 of the scale product,
and recompute what that factor overflows; every scale must still give the one rounding per K block that the oracle has (bit
equality).  Integer extremes (all -128, all 127) are among the operands: they bound the bias the partials carry."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    import gemm_int8_b200

    return gemm_int8_b200


@pytest.mark.parametrize("variant", ["dense_bn256", "pair", "dense_bn128", "dense_bn64"])
@pytest.mark.parametrize("sa_factor, sw_factor", [(1.0, 1.0), (1e-30, 1e-12), (1e-20, 1e-18), (2.0**60, 2.0**45.9), (2.0**60, 2.0**46), (1e36, 1.0),
                                                  (-1e33, 1.0), (1e30, 1e30)])
def test_scale_range(g, oracle, variant, sa_factor, sw_factor):
    gen = torch.Generator().manual_seed(17)
    g.force_variant(variant)
    try:
        for M, N, K in [(130, 300, 640), (5, 264, 144), (40, 17, 512)]:
            x = torch.randint(-128, 128, (M, K), generator=gen, dtype=torch.int8)
            y = torch.randint(-128, 128, (N, K), generator=gen, dtype=torch.int8)
            x[: M // 4] = -128
            y[: N // 4] = 127
            y[N // 4 : N // 2] = -128
            KB, NB = -(-K // 128), -(-N // 128)
            sa, sw = torch.rand(M, KB, generator=gen) + 0.5, torch.rand(NB, KB, generator=gen) + 0.5
            sa[::3] *= sa_factor   # some rows only: a warp holds both kinds
            sw[:, 1:] *= sw_factor
            sa[1, 0] = 0.0
            want = oracle.c_matmul_blockwise(x, y, sa, sw)
            got = oracle.bf16_bits(g.matmul_blockwise(x.cuda(), y.cuda(), sa.cuda(), sw.cuda()))
            nan = (want & 0x7FFF) > 0x7F80
            assert np.array_equal((got & 0x7FFF) > 0x7F80, nan) and np.array_equal(got[~nan], want[~nan]), (M, N, K)
            f = g.matmul_blockwise_f32(x.cuda(), y.cuda(), sa.cuda(), sw.cuda())
            assert np.array_equal(oracle.bf16_bits(f.to(torch.bfloat16))[~nan], want[~nan]), (M, N, K)
    finally:
        g.force_variant(None)
