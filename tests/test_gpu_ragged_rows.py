"""Outputs whose rows TMA cannot address (N not a multiple of 8, or a base off 16 bytes): they leave through shared memory row
by row, two columns or one per lane.  Bit equality with the oracle (integer sums, one rounding), and nothing written beside
the matrix."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    import gemm_int8_b200

    return gemm_int8_b200


def _p(t, offset=0):
    return ctypes.c_void_p(t.data_ptr() + offset)


@pytest.mark.parametrize("variant", ["dense_bn256", "dense_bn128", "dense_bn64", "pair", None])
@pytest.mark.parametrize("offset", [0, 1])
def test_ragged_rows_match_oracle(g, oracle, variant, offset):
    gen = torch.Generator().manual_seed(31)
    K = 272
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    g.force_variant(variant)
    try:
        for M, N in [(1, 1), (33, 31), (32, 66), (129, 129), (257, 259), (70, 520)]:
            x = torch.randint(-128, 128, (M, K), generator=gen, dtype=torch.int8)
            y = torch.randint(-128, 128, (N, K), generator=gen, dtype=torch.int8)
            sx, sw = torch.rand(M, generator=gen), torch.rand(N, generator=gen)
            sa, sb = torch.rand(M, 3, generator=gen), torch.rand(-(-N // 128), 3, generator=gen)
            xd, yd, sxd, swd, sad, sbd = (t.cuda() for t in (x, y, sx, sw, sa, sb))
            for kind in ("plain", "scaled", "blockwise"):
                out = torch.full((M * N + 16,), 7.0, dtype=torch.bfloat16, device="cuda")
                o = _p(out, 2 * offset)
                if kind == "plain":
                    rc = g._C.gi8_matmul(_p(xd), _p(yd), o, M, N, K, -0.37, stream)
                    want = oracle.c_matmul(x, y, -0.37)
                elif kind == "scaled":
                    rc = g._C.gi8_matmul_scaled(_p(xd), _p(yd), _p(sxd), _p(swd), o, M, N, K, None, 0, stream)
                    want = oracle.c_matmul_scaled(x, y, sx, sw)
                else:
                    rc = g._C.gi8_matmul_blockwise(_p(xd), _p(yd), _p(sad), 3, _p(sbd), 3, o, M, N, K, stream)
                    want = oracle.c_matmul_blockwise(x, y, sa, sb)
                assert rc == 0, g._C.gi8_last_error()
                got = out.cpu()
                assert np.array_equal(oracle.bf16_bits(got[offset : offset + M * N].reshape(M, N)), want), (kind, M, N)
                assert bool((got[:offset] == 7).all()) and bool((got[offset + M * N :] == 7).all()), (kind, M, N)
    finally:
        g.force_variant(None)
