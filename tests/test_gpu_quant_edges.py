"""The quantisers where their work is cut up: rows that just fit, or just do not fit, the 2, 4 or 8 loads a thread keeps in
registers, and rotation blocks whose last unit of 2048 (times four warps), 4096 or 8192 elements is not full.  Integers and
scales must equal the oracle's bit for bit (they are defined operation by operation, so there is no tolerance)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    import gemm_int8_b200

    return gemm_int8_b200


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_row_quantiser_register_edges(g, oracle, dtype):
    gen = torch.Generator().manual_seed(7)
    per_load = 256 * (16 // dtype.itemsize)
    step = 16 // dtype.itemsize
    for loads in (2, 4, 8):
        for K in (loads * per_load - step, loads * per_load, loads * per_load + step):
            a = torch.randn(3, K, generator=gen)
            a[1] *= 1e-20
            a[2, -1] = 50.0  # the largest element is the last one
            a = a.to(dtype)
            q, s = g.quantize_per_token(a.cuda())
            qr, sr = oracle.c_quantize_blocks(a.float(), 1, K)
            assert np.array_equal(q.cpu().numpy(), qr) and np.array_equal(s.cpu().numpy(), sr.reshape(-1)), (K, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [128, 256, 512, 1024, 2048, 4096, 8192])
def test_rotation_partial_units(g, oracle, dtype, H):
    gen = torch.Generator().manual_seed(H)
    for M, blocks in [(1, 1), (3, 1), (5, 3), (1, 17), (37, 2)]:
        K = blocks * H
        a = torch.randn(M, K, generator=gen) * torch.exp(torch.randn(M, 1, generator=gen) * 5)
        a[:, 0] *= 30
        a = a.to(dtype)
        q, s = g.hadamard_quantize_per_token_block(a.cuda(), H)
        qr, sr = oracle.c_quantize_blocks(oracle.c_hadamard_rotate(a.float(), H), 1, 128)
        assert np.array_equal(s.cpu().numpy(), sr), (M, K, H)
        assert np.array_equal(q.cpu().numpy(), qr), (M, K, H)
