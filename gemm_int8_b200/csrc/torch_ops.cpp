// CUDA implementations of the torch operators of the namespace gemm_int8_CUDA (their schemas and fake kernels are defined in
// Python): operand checks, allocation of the results, and one call into the C ABI on the current stream.
//
// The reference binds its operator in C++ as well (csrc/kernels/bindings.cpp:10-38).  What bounds a decode step is host
// time: with these bodies in Python, a linear layer of one token (4096 x 4096) took 25.4 us a call, with them here 12.2 us.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/pybind11.h>
#include <torch/library.h>

#include <tuple>

#include "../../include/gemm_int8_b200.h"

// The torch and Python this library was compiled against; _build.py compares it with what is installed.
extern "C" {
extern const char gi8_torch_ops_built_for[];
const char gi8_torch_ops_built_for[] = GI8_BUILT_FOR;
}

namespace {

constexpr int64_t kBlock = 128;

int64_t blocks_of(int64_t n) { return (n + kBlock - 1) / kBlock; }

// A non-zero status of the C ABI becomes the package's Python exception, with its status code.
void check(int status)
{
    if (status == GI8_OK) return;
    const std::string message = gi8_last_error();
    pybind11::gil_scoped_acquire gil;
    pybind11::object type = pybind11::module_::import("gemm_int8_b200._lib").attr("GemmInt8Error");
    pybind11::object value = type(status, message);
    PyErr_SetObject(type.ptr(), value.ptr());
    throw pybind11::error_already_set();
}

struct Sizes {
    int64_t M, N, K;
};

// The reference checks contiguity, device type and same-GPU (bindings.cpp:15-20) and leaves dtype, rank and the K match
// to its fake kernel (gemm_int8/__init__.py:18-24); here the real kernel checks them all.
Sizes check_operands(const char* name, const at::Tensor& A, const at::Tensor& B)
{
    TORCH_CHECK(A.is_cuda() && B.is_cuda(), name, ": A and B must be CUDA tensors");
    TORCH_CHECK(A.device() == B.device(), name, ": A and B must be on the same GPU, got ", A.device(), " and ", B.device());
    TORCH_CHECK(A.scalar_type() == at::kChar && B.scalar_type() == at::kChar, name, ": A and B must be int8, got ", A.scalar_type(),
                " and ", B.scalar_type());
    TORCH_CHECK(A.dim() == 2 && B.dim() == 2, name, ": A and B must be 2-D");
    TORCH_CHECK(A.size(1) == B.size(1), name, ": A.shape[1] (", A.size(1), ") must equal B.shape[1] (", B.size(1), ")");
    TORCH_CHECK(A.is_contiguous() && B.is_contiguous(), name, ": A and B must be contiguous");
    return {A.size(0), B.size(0), A.size(1)};
}

void check_scale(const char* name, const char* what, const at::Tensor& t, at::IntArrayRef shape, const at::Device& device)
{
    TORCH_CHECK(t.device() == device, name, ": ", what, " must be on ", device, ", got ", t.device());
    TORCH_CHECK(t.scalar_type() == at::kFloat, name, ": ", what, " must be float32, got ", t.scalar_type());
    TORCH_CHECK(t.sizes() == shape, name, ": ", what, " must have shape ", shape, ", got ", t.sizes());
}

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

at::Tensor new_tensor(at::IntArrayRef shape, at::ScalarType dtype, const at::Tensor& like)
{
    return at::empty(shape, at::TensorOptions().dtype(dtype).device(like.device()));
}

const int8_t* i8(const at::Tensor& t) { return static_cast<const int8_t*>(t.data_ptr()); }
const float* f32(const at::Tensor& t) { return static_cast<const float*>(t.data_ptr()); }

at::Tensor int8_matmul(const at::Tensor& A, const at::Tensor& B, double alpha)
{
    const Sizes n = check_operands("int8_matmul", A, B);
    const c10::cuda::CUDAGuard guard(A.device());
    at::Tensor out = new_tensor({n.M, n.N}, at::kBFloat16, A);
    check(gi8_matmul(i8(A), i8(B), out.data_ptr(), n.M, n.N, n.K, static_cast<float>(alpha), stream_of(A)));
    return out;
}

at::Tensor int8_matmul_i32(const at::Tensor& A, const at::Tensor& B)
{
    const Sizes n = check_operands("int8_matmul_i32", A, B);
    const c10::cuda::CUDAGuard guard(A.device());
    at::Tensor out = new_tensor({n.M, n.N}, at::kInt, A);
    check(gi8_matmul_i32(i8(A), i8(B), static_cast<int32_t*>(out.data_ptr()), n.M, n.N, n.K, stream_of(A)));
    return out;
}

// Per-row scales: [R] or [R, 1].
at::Tensor row_scale(const char* name, const char* what, const at::Tensor& t, int64_t rows, const at::Device& device)
{
    const at::Tensor flat = t.dim() == 2 && t.size(1) == 1 ? t.reshape({-1}) : t;
    check_scale(name, what, flat, {rows}, device);
    return flat.contiguous();
}

at::Tensor int8_matmul_scaled(const at::Tensor& A, const at::Tensor& B, const at::Tensor& a_scale, const at::Tensor& b_scale)
{
    const char* name = "int8_matmul_scaled";
    const Sizes n = check_operands(name, A, B);
    const at::Tensor sa = row_scale(name, "a_scale", a_scale, n.M, A.device());
    const at::Tensor sb = row_scale(name, "b_scale", b_scale, n.N, A.device());
    const c10::cuda::CUDAGuard guard(A.device());
    at::Tensor out = new_tensor({n.M, n.N}, at::kBFloat16, A);
    // (only a forced scratch variant asks for a workspace)
    const int64_t bytes = gi8_matmul_scaled_workspace_bytes(n.M, n.N, n.K);
    at::Tensor ws;
    if (bytes > 0) ws = at::zeros({bytes}, at::TensorOptions().dtype(at::kByte).device(A.device()));
    check(gi8_matmul_scaled(i8(A), i8(B), f32(sa), f32(sb), out.data_ptr(), n.M, n.N, n.K, bytes > 0 ? ws.data_ptr() : nullptr, bytes,
                            stream_of(A)));
    return out;
}

// Block scales [rows, cols] and their row stride; copied where the kernels could not walk them.
at::Tensor block_scale(const at::Tensor& t, int64_t& ld)
{
    const int64_t rows = t.size(0), cols = t.size(1);
    at::Tensor s = t.stride(1) != 1 && cols > 1 ? t.contiguous() : t;
    ld = rows > 1 ? s.stride(0) : cols;
    if (ld < cols) s = s.contiguous(), ld = cols;
    return s;
}

at::Tensor blockwise(const char* name, const at::Tensor& A, const at::Tensor& B, const at::Tensor& A_scale, const at::Tensor& B_scale,
                     bool as_f32)
{
    const Sizes n = check_operands(name, A, B);
    check_scale(name, "A_scale", A_scale, {n.M, blocks_of(n.K)}, A.device());
    check_scale(name, "B_scale", B_scale, {blocks_of(n.N), blocks_of(n.K)}, A.device());
    const c10::cuda::CUDAGuard guard(A.device());
    int64_t ld_sa, ld_sb;
    const at::Tensor sa = block_scale(A_scale, ld_sa), sb = block_scale(B_scale, ld_sb);
    at::Tensor out = new_tensor({n.M, n.N}, as_f32 ? at::kFloat : at::kBFloat16, A);
    if (as_f32)
        check(gi8_matmul_blockwise_f32(i8(A), i8(B), f32(sa), ld_sa, f32(sb), ld_sb, static_cast<float*>(out.data_ptr()), n.M, n.N, n.K,
                                       stream_of(A)));
    else
        check(gi8_matmul_blockwise(i8(A), i8(B), f32(sa), ld_sa, f32(sb), ld_sb, out.data_ptr(), n.M, n.N, n.K, stream_of(A)));
    return out;
}

at::Tensor int8_matmul_blockwise(const at::Tensor& A, const at::Tensor& B, const at::Tensor& A_scale, const at::Tensor& B_scale)
{
    return blockwise("int8_matmul_blockwise", A, B, A_scale, B_scale, false);
}

at::Tensor int8_matmul_blockwise_f32(const at::Tensor& A, const at::Tensor& B, const at::Tensor& A_scale, const at::Tensor& B_scale)
{
    return blockwise("int8_matmul_blockwise_f32", A, B, A_scale, B_scale, true);
}

// ------------------------------------------------------------------------------------------------ quantisers
void check_activations(const char* name, const at::Tensor& a)
{
    TORCH_CHECK(a.is_cuda(), name, ": input must be a CUDA tensor (the torch reference lives in gemm_int8_b200.quant)");
    TORCH_CHECK(a.dim() == 2, name, ": input must be 2-D [tokens, features]");
    TORCH_CHECK(a.scalar_type() == at::kFloat || a.scalar_type() == at::kBFloat16, name, ": input must be float32 or bfloat16, got ",
                a.scalar_type());
}

enum class Quantiser { kRow, kBlock, kHadamard };

std::tuple<at::Tensor, at::Tensor> quantise(const char* name, const at::Tensor& a, Quantiser kind, int64_t had)
{
    check_activations(name, a);
    const c10::cuda::CUDAGuard guard(a.device());
    const at::Tensor c = a.contiguous();
    const int64_t M = c.size(0), K = c.size(1);
    at::Tensor q = new_tensor({M, K}, at::kChar, c);
    at::Tensor s = kind == Quantiser::kRow ? new_tensor({M}, at::kFloat, c) : new_tensor({M, blocks_of(K)}, at::kFloat, c);
    const int dtype = c.scalar_type() == at::kFloat ? 0 : 1;
    int8_t* qp = static_cast<int8_t*>(q.data_ptr());
    float* sp = static_cast<float*>(s.data_ptr());
    if (kind == Quantiser::kRow) check(gi8_quantize_token(c.data_ptr(), dtype, qp, sp, M, K, stream_of(c)));
    else if (kind == Quantiser::kBlock) check(gi8_quantize_token_block(c.data_ptr(), dtype, qp, sp, M, K, stream_of(c)));
    else check(gi8_hadamard_quantize_token_block(c.data_ptr(), dtype, qp, sp, M, K, had, stream_of(c)));
    return {q, s};
}

std::tuple<at::Tensor, at::Tensor> quantize_token_block(const at::Tensor& a) { return quantise("quantize", a, Quantiser::kBlock, 0); }
std::tuple<at::Tensor, at::Tensor> quantize_token(const at::Tensor& a) { return quantise("quantize", a, Quantiser::kRow, 0); }
std::tuple<at::Tensor, at::Tensor> hadamard_quantize_token_block(const at::Tensor& a, int64_t block)
{
    return quantise("hadamard_quantize", a, Quantiser::kHadamard, block);
}

// ------------------------------------------------------------------------------------------------ linear layer
// Quantiser and product with one call into the library, which launches the second as a programmatic dependent of the
// first; the quantised activations live in one scratch tensor.  hadamard: rotation block, or none.
at::Tensor int8_linear(const at::Tensor& x, const at::Tensor& w, const at::Tensor& w_scale, const std::optional<at::Tensor>& bias, bool blocks,
                       std::optional<int64_t> hadamard)
{
    const char* name = "int8_linear";
    TORCH_CHECK(!hadamard.has_value() || *hadamard > 0, name, ": rotation block ", *hadamard);
    check_activations(name, x);
    TORCH_CHECK(w.device() == x.device(), name, ": the weight must be on ", x.device(), ", got ", w.device());
    TORCH_CHECK(w.scalar_type() == at::kChar && w.dim() == 2 && w.is_contiguous(), name, ": the weight must be a contiguous 2-D int8 tensor");
    TORCH_CHECK(x.size(1) == w.size(1), name, ": x has ", x.size(1), " features, the weight ", w.size(1));
    const int64_t M = x.size(0), N = w.size(0), K = x.size(1);
    const c10::cuda::CUDAGuard guard(x.device());
    at::Tensor ws;
    int64_t ld = 0;
    if (blocks) {
        check_scale(name, "weight_scale", w_scale, {blocks_of(N), blocks_of(K)}, x.device());
        ws = block_scale(w_scale, ld);
    } else {
        ws = row_scale(name, "weight_scale", w_scale, N, x.device());
    }
    at::Tensor b;
    if (bias.has_value()) {
        TORCH_CHECK(bias->device() == x.device() && bias->dim() == 1 && bias->size(0) == N, name, ": bias must have shape [", N, "] on ", x.device());
        b = bias->to(at::kBFloat16).contiguous();
    }
    const at::Tensor c = x.contiguous();
    at::Tensor out = new_tensor({M, N}, at::kBFloat16, x);
    const int64_t q_bytes = (M * K + 255) / 256 * 256;
    at::Tensor scratch = new_tensor({q_bytes + 4 * M * (blocks ? blocks_of(K) : 1)}, at::kByte, x);
    uint8_t* q = static_cast<uint8_t*>(scratch.data_ptr());
    const int status = gi8_linear(c.data_ptr(), c.scalar_type() == at::kFloat ? 0 : 1, i8(w), f32(ws), ld, b.defined() ? b.data_ptr() : nullptr,
                                  blocks, hadamard.value_or(0), reinterpret_cast<int8_t*>(q), reinterpret_cast<float*>(q + q_bytes), out.data_ptr(), M, N, K,
                                  stream_of(x));
    if (status == GI8_ERR_WORKSPACE && !blocks) {  // a forced variant that the single call does not have
        auto [xq, xs] = quantize_token(c);
        out = int8_matmul_scaled(xq, w, xs, ws);
        return b.defined() ? out + b : out;
    }
    check(status);
    return out;
}

}  // namespace

TORCH_LIBRARY_IMPL(gemm_int8_CUDA, CUDA, m)
{
    m.impl("int8_matmul", &int8_matmul);
    m.impl("int8_matmul_i32", &int8_matmul_i32);
    m.impl("int8_matmul_scaled", &int8_matmul_scaled);
    m.impl("int8_matmul_blockwise", &int8_matmul_blockwise);
    m.impl("int8_matmul_blockwise_f32", &int8_matmul_blockwise_f32);
    m.impl("quantize_token_block", &quantize_token_block);
    m.impl("quantize_token", &quantize_token);
    m.impl("hadamard_quantize_token_block", &hadamard_quantize_token_block);
    m.impl("int8_linear", &int8_linear);
}
