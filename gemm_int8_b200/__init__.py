"""B200-native INT8 GEMM behind the reference's Python/PyTorch operator surface.

Mirrors gemm_int8/__init__.py of the reference:

* ``matmul(x, y, alpha=1.0)`` -> bf16 ``(x @ y.T) * alpha``            (gemm_int8/__init__.py:28-37)
* torch op ``gemm_int8_CUDA::int8_matmul(Tensor A, Tensor B, float alpha) -> Tensor`` with a CUDA
  implementation and a fake (meta) kernel                          (csrc/kernels/bindings.cpp:30-38,
                                                                     gemm_int8/__init__.py:16-25)

and adds the W8A8 entry points the reference lacks: ``matmul_scaled`` (per-token x per-channel scales)
and ``matmul_blockwise`` (per-token-per-128-K activation scales, per-128x128 weight scales).

The schemas and fake kernels of the torch ops are defined here; their CUDA implementations are a thin C++ layer
(csrc/torch_ops.cpp) over the C ABI of ``libgemm_int8_b200.so`` (raw device pointers and the current CUDA stream).  Importing this package without the compiled
library raises ImportError, as the reference does (gemm_int8/__init__.py:9-10); there is no CPU path.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib

_C = _lib.load()

KBLOCK = 128

# --------------------------------------------------------------------------------------------------
# op schemas.  Namespace, name and schema of int8_matmul are the reference's (bindings.cpp:30-33).
# --------------------------------------------------------------------------------------------------
_NS = "gemm_int8_CUDA"
_libdef = torch.library.Library(_NS, "DEF")
_libdef.define("int8_matmul(Tensor A, Tensor B, float alpha) -> Tensor")
_libdef.define("int8_matmul_i32(Tensor A, Tensor B) -> Tensor")
_libdef.define("int8_matmul_scaled(Tensor A, Tensor B, Tensor a_scale, Tensor b_scale) -> Tensor")
_libdef.define("int8_matmul_blockwise(Tensor A, Tensor B, Tensor A_scale, Tensor B_scale) -> Tensor")
_libdef.define("int8_matmul_blockwise_f32(Tensor A, Tensor B, Tensor A_scale, Tensor B_scale) -> Tensor")
_libdef.define("quantize_token_block(Tensor a) -> (Tensor, Tensor)")
_libdef.define("quantize_token(Tensor a) -> (Tensor, Tensor)")
_libdef.define("hadamard_quantize_token_block(Tensor a, int block) -> (Tensor, Tensor)")
_libdef.define("int8_linear(Tensor x, Tensor weight_q, Tensor weight_scale, Tensor? bias, bool blockwise, int? hadamard) -> Tensor")


def _stream_ptr(device: torch.device) -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)


class _on_device:
    """Makes `device` current for the duration of a launch (no-op when it already is)."""

    __slots__ = ("idx", "prev")

    def __init__(self, device: torch.device):
        self.idx = device.index if device.index is not None else torch.cuda.current_device()
        self.prev = -1

    def __enter__(self):
        cur = torch.cuda.current_device()
        if cur != self.idx:
            self.prev = cur
            torch.cuda.set_device(self.idx)

    def __exit__(self, *exc):
        if self.prev >= 0:
            torch.cuda.set_device(self.prev)
        return False


def _ptr(t: torch.Tensor) -> ctypes.c_void_p:
    return ctypes.c_void_p(t.data_ptr())


# The CUDA implementations (csrc/torch_ops.cpp) register themselves when their library is loaded.
_lib.load_ops()


# --------------------------------------------------------------------------------------------------
# fake (meta) kernels: shape/dtype propagation for torch.compile, as gemm_int8/__init__.py:16-25
# --------------------------------------------------------------------------------------------------
def _fake_common(x: torch.Tensor, y: torch.Tensor) -> None:
    torch._check(x.device.type == "cuda", lambda: "x must be a CUDA tensor")
    torch._check(y.device.type == "cuda", lambda: "y must be a CUDA tensor")
    torch._check(x.dtype == torch.int8, lambda: "x must be an int8 tensor")
    torch._check(y.dtype == torch.int8, lambda: "y must be an int8 tensor")
    torch._check(len(x.shape) == 2, lambda: "x must be a 2D tensor")
    torch._check(len(y.shape) == 2, lambda: "y must be a 2D tensor")
    torch._check(x.shape[1] == y.shape[1], lambda: "x.shape[1] must be equal to y.shape[1]")


@torch.library.register_fake(f"{_NS}::int8_matmul")
def _(x: torch.Tensor, y: torch.Tensor, alpha: float = 1.0):
    _fake_common(x, y)
    return torch.empty(x.shape[0], y.shape[0], device=x.device, dtype=torch.bfloat16)


@torch.library.register_fake(f"{_NS}::int8_matmul_i32")
def _(x: torch.Tensor, y: torch.Tensor):
    _fake_common(x, y)
    return torch.empty(x.shape[0], y.shape[0], device=x.device, dtype=torch.int32)


@torch.library.register_fake(f"{_NS}::int8_matmul_scaled")
def _(x: torch.Tensor, y: torch.Tensor, a_scale: torch.Tensor, b_scale: torch.Tensor):
    _fake_common(x, y)
    torch._check(a_scale.dtype == torch.float32 and b_scale.dtype == torch.float32, lambda: "scales must be float32")
    return torch.empty(x.shape[0], y.shape[0], device=x.device, dtype=torch.bfloat16)


@torch.library.register_fake(f"{_NS}::int8_matmul_blockwise")
def _(x: torch.Tensor, y: torch.Tensor, A_scale: torch.Tensor, B_scale: torch.Tensor):
    _fake_common(x, y)
    torch._check(A_scale.dtype == torch.float32 and B_scale.dtype == torch.float32, lambda: "scales must be float32")
    torch._check(len(A_scale.shape) == 2 and len(B_scale.shape) == 2, lambda: "scales must be 2D tensors")
    return torch.empty(x.shape[0], y.shape[0], device=x.device, dtype=torch.bfloat16)


@torch.library.register_fake(f"{_NS}::int8_matmul_blockwise_f32")
def _(x: torch.Tensor, y: torch.Tensor, A_scale: torch.Tensor, B_scale: torch.Tensor):
    _fake_common(x, y)
    torch._check(A_scale.dtype == torch.float32 and B_scale.dtype == torch.float32, lambda: "scales must be float32")
    torch._check(len(A_scale.shape) == 2 and len(B_scale.shape) == 2, lambda: "scales must be 2D tensors")
    return torch.empty(x.shape[0], y.shape[0], device=x.device, dtype=torch.float32)


# --------------------------------------------------------------------------------------------------
# public functions
# --------------------------------------------------------------------------------------------------
def matmul(x: torch.Tensor, y: torch.Tensor, alpha: float = 1.0) -> torch.Tensor:
    """INT8 matrix product ``(x @ y.t()) * alpha`` returned as bf16.

    Same call as the reference's ``gemm_int8.matmul`` (gemm_int8/__init__.py:28-37).

    Arguments:
        x: int8 CUDA tensor of shape (M, K), contiguous
        y: int8 CUDA tensor of shape (N, K), contiguous
        alpha: scalar multiplied into the fp32-converted int32 accumulator before the bf16 cast
    """
    return torch.ops.gemm_int8_CUDA.int8_matmul(x, y, alpha)


def matmul_i32(x: torch.Tensor, y: torch.Tensor) -> torch.Tensor:
    """Raw int32 accumulators ``x @ y.t()`` (bit-exact verification of the integer main loop)."""
    return torch.ops.gemm_int8_CUDA.int8_matmul_i32(x, y)


def matmul_scaled(x_q: torch.Tensor, w_q: torch.Tensor, x_scale: torch.Tensor, w_scale: torch.Tensor) -> torch.Tensor:
    """W8A8 GEMM with per-token and per-output-channel scales.

    ``out[m, n] = bf16( fp32(acc[m, n]) * (x_scale[m] * w_scale[n]) )`` with ``acc = x_q @ w_q.t()`` in int32.
    x_q (M, K) int8, w_q (N, K) int8, x_scale (M,) fp32, w_scale (N,) fp32.
    """
    return torch.ops.gemm_int8_CUDA.int8_matmul_scaled(x_q, w_q, x_scale, w_scale)


def matmul_blockwise(x_q: torch.Tensor, w_q: torch.Tensor, x_scale: torch.Tensor, w_scale: torch.Tensor) -> torch.Tensor:
    """Blockwise-dequantised W8A8 GEMM.

    ``out[m, n] = bf16( sum_kb fp32(P[m, n, kb]) * (x_scale[m, kb] * w_scale[n // 128, kb]) )`` where ``P`` is
    the exact int32 dot product over the kb-th 128-wide K block, accumulated in fp32 with one fused
    multiply-add per block in ascending kb order.
    x_q (M, K) int8, w_q (N, K) int8, x_scale (M, ceil(K/128)) fp32, w_scale (ceil(N/128), ceil(K/128)) fp32.
    """
    return torch.ops.gemm_int8_CUDA.int8_matmul_blockwise(x_q, w_q, x_scale, w_scale)


def matmul_blockwise_f32(x_q: torch.Tensor, w_q: torch.Tensor, x_scale: torch.Tensor, w_scale: torch.Tensor) -> torch.Tensor:
    """`matmul_blockwise` before its bf16 cast: the fp32 accumulators (one fused multiply-add per 128-wide K block,
    ascending).  The partial result of a K-sharded GEMM (see `dist.matmul_blockwise_ksharded`)."""
    return torch.ops.gemm_int8_CUDA.int8_matmul_blockwise_f32(x_q, w_q, x_scale, w_scale)


def sum_parts_bf16(parts: torch.Tensor) -> torch.Tensor:
    """parts fp32 [P, ...] (contiguous) -> bf16 [...]: ((parts[0] + parts[1]) + parts[2]) + ... in fp32, cast once."""
    if not parts.is_cuda or parts.dtype != torch.float32 or parts.dim() < 2:
        raise RuntimeError("sum_parts_bf16: a CUDA float32 tensor [P, ...] is expected")
    parts = parts.contiguous()
    P = parts.shape[0]
    count = parts[0].numel()
    out = torch.empty(parts.shape[1:], dtype=torch.bfloat16, device=parts.device)
    with _on_device(parts.device):
        rc = _C.gi8_sum_parts_bf16(_ptr(parts), P, count, _ptr(out), count, _stream_ptr(parts.device))
    _lib.check(_C, rc)
    return out


@torch.library.register_fake(f"{_NS}::quantize_token_block")
def _(a: torch.Tensor):
    torch._check(len(a.shape) == 2, lambda: "a must be a 2D tensor")
    kb = (a.shape[1] + KBLOCK - 1) // KBLOCK
    return (torch.empty(a.shape[0], a.shape[1], device=a.device, dtype=torch.int8),
            torch.empty(a.shape[0], kb, device=a.device, dtype=torch.float32))


@torch.library.register_fake(f"{_NS}::hadamard_quantize_token_block")
def _(a: torch.Tensor, block: int):
    torch._check(len(a.shape) == 2, lambda: "a must be a 2D tensor")
    kb = (a.shape[1] + KBLOCK - 1) // KBLOCK
    return (torch.empty(a.shape[0], a.shape[1], device=a.device, dtype=torch.int8),
            torch.empty(a.shape[0], kb, device=a.device, dtype=torch.float32))


@torch.library.register_fake(f"{_NS}::int8_linear")
def _(x: torch.Tensor, weight_q: torch.Tensor, weight_scale: torch.Tensor, bias: torch.Tensor | None, blockwise: bool, hadamard: int | None):
    torch._check(len(x.shape) == 2 and len(weight_q.shape) == 2, lambda: "x and weight_q must be 2D tensors")
    torch._check(weight_q.dtype == torch.int8, lambda: "weight_q must be an int8 tensor")
    torch._check(x.shape[1] == weight_q.shape[1], lambda: "x.shape[1] must be equal to weight_q.shape[1]")
    return torch.empty(x.shape[0], weight_q.shape[0], device=x.device, dtype=torch.bfloat16)


@torch.library.register_fake(f"{_NS}::quantize_token")
def _(a: torch.Tensor):
    torch._check(len(a.shape) == 2, lambda: "a must be a 2D tensor")
    return (torch.empty(a.shape[0], a.shape[1], device=a.device, dtype=torch.int8),
            torch.empty(a.shape[0], device=a.device, dtype=torch.float32))


def quantize_per_token_block(a: torch.Tensor):
    """Fused activation quantiser for `matmul_blockwise`: a [M, K] fp32/bf16 (CUDA) -> (q int8 [M, K],
    scales fp32 [M, ceil(K/128)]), one symmetric scale per token per 128-wide K block (amax / 127, round half
    even, clamp to +-127) -- bit-identical to `quant.quantize_per_token_block`."""
    return torch.ops.gemm_int8_CUDA.quantize_token_block(a)


def hadamard_quantize_per_token_block(a: torch.Tensor, block: int | None = None):
    """Walsh-Hadamard rotation along K in blocks of `block` (default: the largest power of two dividing K, at most
    8192) fused with `quantize_per_token_block` in one pass over the activations -- bit-identical to
    `quant.quantize_per_token_block(quant.hadamard_rotate(a.float(), block))`.  The weights must have been rotated
    the same way before they were quantised (offline)."""
    K = a.shape[-1]
    if block is None:
        block = min(K & -K, 8192)
    return torch.ops.gemm_int8_CUDA.hadamard_quantize_token_block(a, block)


def quantize_per_token(a: torch.Tensor):
    """Fused per-token quantiser for `matmul_scaled`: a [M, K] -> (q int8 [M, K], scales fp32 [M])."""
    return torch.ops.gemm_int8_CUDA.quantize_token(a)


def force_variant(name: str | None) -> None:
    """Force a kernel variant ("dense_bn256", "dense_bn128", "dense_bn64", "pair", "smallm", "smallm_cluster");
    None = fitted dispatch."""
    _lib.check(_C, _C.gi8_force_variant(name.encode() if name else None))


def pick_variant(kind: int, M: int, N: int, K: int) -> str:
    """Variant the dispatch selects for a shape; kind 0 plain, 1 scaled, 2 blockwise."""
    return _C.gi8_pick_variant(kind, M, N, K).decode()


def device_status() -> int:
    """Synchronises the current device and returns (then clears) its kernel status word; 0 = healthy.

    A non-zero word means a kernel gave up a bounded wait; the results of that launch are invalid."""
    code = ctypes.c_uint32(0)
    _lib.check(_C, _C.gi8_device_status(ctypes.byref(code)))
    return int(code.value)


def check_device() -> None:
    """Synchronises the current device and raises GemmInt8Error (GI8_ERR_DEVICE_TIMEOUT) if a kernel since the
    last check gave up a bounded wait -- the counterpart of the reference's exception on a failed launch
    (csrc/kernels/gemm.cu:108-121)."""
    _lib.check(_C, _C.gi8_device_check())


def reload_env() -> None:
    """Re-reads the GEMM_INT8_* tuning variables (they are otherwise read once, at first use)."""
    _lib.check(_C, _C.gi8_reload_env())


# GEMM_INT8_KERNEL=<variant> forces a kernel variant for the whole process (tuning and profiling).
import os as _os

if _os.environ.get("GEMM_INT8_KERNEL"):
    force_variant(_os.environ["GEMM_INT8_KERNEL"])


from .linear import Int8Linear  # noqa: E402

__all__ = ["matmul", "matmul_i32", "matmul_scaled", "matmul_blockwise", "matmul_blockwise_f32", "sum_parts_bf16",
           "quantize_per_token_block",
           "quantize_per_token", "Int8Linear", "force_variant", "pick_variant", "device_status", "check_device", "reload_env"]
