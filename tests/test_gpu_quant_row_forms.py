"""The row quantiser at the edges of its forms (two, four and eight 16-byte loads held in registers, and rows longer than that), for both types, against
torch: s = amax / 127, q = the fp32 quotient rounded half to even."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loads, extra", [(1, 0), (2, 0), (2, 1), (4, 0), (4, 1), (8, 0), (8, 1), (16, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_forms(dtype, loads, extra):
    import gemm_int8_b200 as g

    per = 16 // dtype.itemsize               # elements of a load
    K = 256 * per * loads + per * extra      # the last of `loads` passes of 256 threads is full, `extra` threads take another
    gen = torch.Generator(device="cuda").manual_seed(K)
    a = torch.randn(1300, K, generator=gen, device="cuda").to(dtype)   # more rows than CTAs
    a[0], a[1, -1], a[2, 0] = 0.0, 50.0, -50.0
    a[3] = torch.arange(K, device="cuda") % 255 - 127                  # exact quotients
    a[4] = (torch.arange(K, device="cuda") % 127 + 0.5).to(dtype)      # half-integers against a scale of one (and bf16's nearest to them)
    a[4, 0] = 127.0
    q, s = g.quantize_per_token(a)
    v = a.float()
    amax = v.abs().amax(dim=1)
    want_s = torch.where(amax > 0, amax / torch.full_like(amax, 127.0), torch.ones_like(amax))
    assert torch.equal(s.flatten(), want_s)
    want = torch.round(v / want_s[:, None]).clamp(-127, 127).to(torch.int8)
    assert torch.equal(q, want)
