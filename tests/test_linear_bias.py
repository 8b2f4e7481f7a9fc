"""Which addition the bias of an Int8Linear takes: the epilogue of the product, or a tensor operation behind it.  A layer made from
a torch.nn.Linear hands its bias over as a Parameter, which is differentiated only while gradients are recorded."""
import contextlib

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.utils._python_dispatch import TorchDispatchMode


class _Ops(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.calls = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.calls.append((func._schema.name, args))
        return func(*args, **(kwargs or {}))


def _calls(mode, bias, context):
    """Operators of one forward pass, on fake tensors (no device needed)."""
    import gemm_int8_b200 as g

    K, N = 256, 136
    scale = torch.empty(2, 2) if mode == "blockwise" else torch.empty(N)
    layer = g.Int8Linear(torch.empty(N, K, dtype=torch.int8), scale, bias, mode=mode)
    with context(), _Ops() as ops:
        out = layer(torch.empty(6, K, dtype=torch.bfloat16))
    assert out.shape == (6, N)
    linear = [a for n, a in ops.calls if n == "gemm_int8_CUDA::int8_linear"]
    assert len(linear) == 1
    return linear[0][3] is not None, any(n.startswith("aten::add") for n, _ in ops.calls), out


@pytest.mark.parametrize("mode", ["channel", "blockwise"])
def test_parameter_bias_is_fused_unless_gradients_are_recorded(mode):
    with FakeTensorMode():
        plain, parameter = torch.empty(136, dtype=torch.bfloat16), torch.nn.Parameter(torch.empty(136, dtype=torch.bfloat16))
        for context in (torch.no_grad, torch.inference_mode):
            fused, added, out = _calls(mode, parameter, context)
            assert fused and not added and not out.requires_grad
        fused, added, out = _calls(mode, parameter, contextlib.nullcontext)
        assert not fused and added and out.requires_grad
        for context in (torch.no_grad, contextlib.nullcontext):
            fused, added, _ = _calls(mode, plain, context)
            assert fused and not added


@pytest.mark.gpu
@pytest.mark.parametrize("mode, M", [("channel", 16), ("channel", 130), ("blockwise", 16), ("blockwise", 300)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_parameter_bias_gives_the_same_bits(mode, M, dtype):
    import gemm_int8_b200 as g

    gen = torch.Generator(device="cuda").manual_seed(M)
    linear = torch.nn.Linear(512, 264, device="cuda", dtype=dtype)
    layer = g.Int8Linear.from_float(linear.weight, linear.bias, mode=mode)
    x = torch.randn(M, 512, device="cuda", generator=gen).to(torch.bfloat16)
    recorded = layer(x)                       # the tensor addition
    assert recorded.requires_grad
    for context in (torch.no_grad, torch.inference_mode):
        with context():
            assert torch.equal(layer(x).view(torch.int16), recorded.detach().view(torch.int16))
    recorded.sum().backward()
    assert torch.equal(linear.bias.grad, torch.full_like(linear.bias, float(M)))
    assert g.device_status() == 0
