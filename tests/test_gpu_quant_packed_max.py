"""bf16 activations: the maxima are taken on packed bf16 pairs.  Signs, zeros of both signs, infinities, NaN (ignored by the maximum) and
subnormals in either half of a pair must give what the same values give as fp32, bit for bit (scales that are NaN or infinite included)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [16, 128, 1040, 4096, 8200, 16384, 20480])
def test_bf16_like_fp32(K):
    import gemm_int8_b200 as g

    gen = torch.Generator().manual_seed(K)
    rows = [torch.randn(K, generator=gen) * s for s in (1.0, -1e-38, 1e38, 1e-41)]
    rows += [torch.full((K,), v) for v in (0.0, -0.0, -3.0, float("nan"), float("inf"))]
    for v in (float("nan"), float("inf"), float("-inf"), -200.0, 200.0):
        for at in (0, 1, K // 2, K - 2, K - 1):
            r = torch.randn(K, generator=gen)
            r[at] = v
            rows.append(r)
    a = torch.stack(rows).to(torch.bfloat16).cuda()
    for fn in (g.quantize_per_token, g.quantize_per_token_block):
        q, s = fn(a)
        qf, sf = fn(a.float())
        assert torch.equal(q, qf) and torch.equal(s.view(torch.int32), sf.view(torch.int32))
