// Python extension `_native`: the host path between the Python functions and libbi8.so.
//
// Every public operation is one call into this module: it validates its operands, allocates the results and the scratch from
// torch's caching allocator, and enqueues the kernels through the C ABI of include/bi8.h on torch's current stream.  Written
// against the CPython call protocol (METH_FASTCALL) without a binding layer, because a decode-sized layer is 9 us of device
// time: the same steps in Python (tensor views, torch.empty, attribute look-ups, one ctypes call with twenty converted
// arguments) took 40 us per call and were what bounded every call below about 50 us.
//
// Nothing here computes: the operations' meaning, shapes and layouts are described in triton_functions.py, and there is no
// path for tensors that are not on a CUDA device.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <mutex>
#include <optional>
#include <string>

#include "../../include/bi8.h"

namespace {

using at::Tensor;

// ---- errors: the Python exception types that the functions have always raised ------------------------------------------
struct PyFail {
    PyObject* type;          // borrowed: a builtin exception class or g_error_class
    std::string text;
};
PyObject* g_error_class = nullptr;       // blockwise_int8_linear_b200._lib.Bi8Error, set when the module is loaded

[[noreturn]] void value_error(std::string text) { throw PyFail{PyExc_ValueError, std::move(text)}; }
[[noreturn]] void assertion(const char* text) { throw PyFail{PyExc_AssertionError, text}; }

void check(int status, const char* what) {
    if (status != BI8_OK)
        throw PyFail{g_error_class ? g_error_class : PyExc_RuntimeError,
                     std::string(what) + " failed with status " + std::to_string(status) + ": " + bi8_last_error_string()};
}

std::string shape_of(const Tensor& t) {
    std::string s = "[";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + "]";
}
std::string shape_of(int64_t a, int64_t b) { return "[" + std::to_string(a) + ", " + std::to_string(b) + "]"; }

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kBFloat16: return BI8_BF16;
        case at::kHalf: return BI8_F16;
        case at::kFloat: return BI8_F32;
        default: value_error(std::string("unsupported dtype ") + c10::toString(t) + ": expected bfloat16, float16 or float32");
    }
}

// ---- allocation and streams ---------------------------------------------------------------------------------------------
// the allocator behind torch.empty, without the dispatcher in front of it
Tensor empty_on(const Tensor& like, at::IntArrayRef sizes, at::ScalarType type) {
    return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}

// Sizes of the buffers that one call carves out of a single allocation.
struct Carve {
    int64_t bytes = 0;
    int64_t take(int64_t n) {
        const int64_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    }
};

// Scratch of one call: partial results of divided tiles, quantized activations that no caller sees.  A call is several launches, and
// the interpreter lock is not held while they are enqueued, so two threads that share a stream may enqueue theirs
// alternately, and calls on forked streams of one capture become branches of a graph that may run at the same time: scratch
// belongs to the call, not to its stream or capture.  The allocator gives the memory to others only behind what the
// call has enqueued on its stream (the returned tensor is held until then), and while a stream is captured it takes it
// from the capture's memory pool, which stays reserved for the graph's lifetime.
Tensor scratch(const Tensor& like, int64_t bytes) { return bytes > 0 ? empty_on(like, {bytes}, at::kByte) : Tensor(); }

// Makes the operand's device current for a call and names its current stream.
struct OnDevice {
    c10::cuda::CUDAGuard guard;
    c10::cuda::CUDAStream stream;
    explicit OnDevice(const Tensor& t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index())) {}
    void* raw() const { return stream.stream(); }
};

// ---- matrices -----------------------------------------------------------------------------------------------------------
// A matrix with contiguous rows: where it lies, its row pitch in elements, and the tensor that owns it.
struct Mat {
    Tensor owner;
    const void* ptr = nullptr;
    int64_t rows = 0, cols = 0, ld = 0;
};

bool rows_contiguous(int64_t rows, int64_t cols, int64_t s0, int64_t s1) {
    return (cols == 1 || s1 == 1) && (rows <= 1 || s0 >= cols);
}

Mat mat(const Tensor& t, int64_t rows, int64_t cols, int64_t s0, int64_t s1, bool transposed) {
    Mat m;
    m.rows = rows;
    m.cols = cols;
    if (rows_contiguous(rows, cols, s0, s1)) {
        m.owner = t;
        m.ld = rows > 1 ? s0 : std::max<int64_t>(cols, 1);
    } else {
        m.owner = (transposed ? t.t() : t).contiguous();
        m.ld = std::max<int64_t>(cols, 1);
    }
    m.ptr = m.owner.data_ptr();
    return m;
}

Mat mat2d(const Tensor& t) {
    if (t.dim() != 2) value_error("expected a 2-D tensor, got " + shape_of(t));
    return mat(t, t.size(0), t.size(1), t.stride(0), t.stride(1), false);
}

Mat mat2d_t(const Tensor& t) {          // the transpose of a 2-D tensor
    return mat(t, t.size(1), t.size(0), t.stride(1), t.stride(0), true);
}

// [..., K] as [rows, K]
Mat mat_rows(const Tensor& t) {
    if (t.dim() == 2) return mat2d(t);
    if (t.dim() == 0) value_error("expected a tensor with a feature dimension, got a scalar");
    const int64_t k = t.size(-1), rows = k ? t.numel() / k : t.numel();
    if (t.is_contiguous()) return mat(t, rows, k, k, 1, false);
    return mat2d(t.reshape({-1, k}));
}

void need_cuda(const Tensor& t) {
    if (!t.is_cuda()) assertion("x.is_cuda");
}

// Row pitch of a quantized matrix: the next multiple of 16 bytes, which is what the wide kernels and the tensor-core GEMM take.
int64_t pitch16(int64_t n) { return (n + 15) / 16 * 16; }

// int8 [rows, cols], dense, or (`pitched`) with rows that begin on 16-byte boundaries: a view of a wider buffer where cols is not
// a multiple of 16
Tensor empty_q(const Tensor& like, int64_t rows, int64_t cols, bool pitched) {
    const int64_t ld = pitched ? pitch16(cols) : cols;
    Tensor t = empty_on(like, {rows, ld}, at::kChar);
    return ld == cols ? t : t.narrow(1, 0, cols);
}

// Copy with a 16-byte aligned row pitch of an int8 operand that has none; the bytes between K and the pitch are never read.  What
// is copied is the matrix that `m` describes, at its address and with its pitch: the owner itself may be that matrix or
// its transpose, which its shape does not tell where both have the same.
bool on_boundaries(const Mat& m) { return m.ld % 16 == 0 && reinterpret_cast<uintptr_t>(m.ptr) % 16 == 0; }
Mat repitch(const Mat& m, const OnDevice& on) {
    if (on_boundaries(m)) return m;
    Mat out = m;
    out.ld = pitch16(m.cols);
    out.owner = empty_on(m.owner, {m.rows, out.ld}, at::kChar);
    out.ptr = out.owner.data_ptr();
    check(bi8_copy_rows(static_cast<const int8_t*>(m.ptr), m.ld, static_cast<int8_t*>(out.owner.data_ptr()), out.ld, m.rows, m.cols, on.raw()),
          "bi8_copy_rows");
    return out;
}

// Whether that is worth its launches.  Without it the GEMM is the CUDA-core kernel's, whose time grows with K for any output: against copy
// and tensor cores 4.5 and 5 us at K = 65 (1 to 40 rows, 64 to 4000 columns), 7 and 5 at 129, 11 and 6 at 257, 20 and 7 at 513, 36
// and 8 at 1001; and with the output for any K: 1024 x 2000 takes 11 and 7 us at K = 17, 19 and 7 at 65, 29 and 8 at 129, 8192 x 4096
// takes 126 and 24, 260 and 28, 407 and 35.  A launch is 2.5 us of host time: the lines are where it is paid for.
bool worth_repitch(int64_t m, int64_t n, int64_t k) { return k % 16 != 0 && (k >= 256 || m * n >= (1ll << 27) / (k + 64)); }

// ---- quantizers ---------------------------------------------------------------------------------------------------------
struct Quantized {
    Tensor q, s;
    int64_t ld() const { return std::max(q.stride(0), q.size(1)); }      // of what empty_q gives, a single row's too
};

// Whether a quantized tensor that a caller gets has a row pitch of 16 bytes.  Callers may view, save or hand on what they get, so it
// is dense, except for large 16-bit matrices: there the re-pitching copy that the GEMM would make of it costs more than a
// launch, and such callers have always got a view.
bool pitched_result(const Tensor& x, int64_t block) {
    const int64_t r = x.size(0), c = x.size(1);
    return x.element_size() == 2 && block % 16 == 0 && r * c >= (1 << 22) && std::min(r, c) >= 256;
}

// `operand`: the result goes into a GEMM and to nobody else, so it gets the pitch that the GEMM wants
Quantized quantize_rowwise(const Tensor& x, int64_t block, bool operand) {
    need_cuda(x);
    OnDevice on(x);
    const Mat m = mat2d(x);
    const int code = dtype_code(x.scalar_type());
    Quantized r{empty_q(x, m.rows, m.cols, operand || pitched_result(x, block)), empty_on(x, {ceil_div(m.cols, block), m.rows}, at::kFloat)};
    check(bi8_quantize_rowwise_pitched(m.ptr, code, m.ld, r.q.mutable_data_ptr<int8_t>(), r.ld(), r.s.mutable_data_ptr<float>(), m.rows, m.cols,
                                       (int)block, on.raw()),
          "bi8_quantize_rowwise");
    return r;
}

Quantized quantize_colwise(const Tensor& x, int64_t block, bool operand) {
    need_cuda(x);
    OnDevice on(x);
    const Mat m = mat2d(x);
    const int code = dtype_code(x.scalar_type());
    Quantized r{empty_q(x, m.cols, m.rows, operand || pitched_result(x, block)), empty_on(x, {ceil_div(m.rows, block), m.cols}, at::kFloat)};
    check(bi8_quantize_colwise_pitched(m.ptr, code, m.ld, r.q.mutable_data_ptr<int8_t>(), r.ld(), r.s.mutable_data_ptr<float>(), m.rows, m.cols,
                                       (int)block, on.raw()),
          "bi8_quantize_colwise");
    return r;
}

struct Dual {
    Quantized row, col;
};

Dual quantize_dual(const Tensor& x, int64_t block) {
    need_cuda(x);
    OnDevice on(x);
    const Mat m = mat2d(x);
    const int code = dtype_code(x.scalar_type());
    const bool pitched = pitched_result(x, block);
    Dual d{{empty_q(x, m.rows, m.cols, pitched), empty_on(x, {ceil_div(m.cols, block), m.rows}, at::kFloat)},
           {empty_q(x, m.cols, m.rows, pitched), empty_on(x, {ceil_div(m.rows, block), m.cols}, at::kFloat)}};
    check(bi8_quantize_dual_pitched(m.ptr, code, m.ld, d.row.q.mutable_data_ptr<int8_t>(), d.row.ld(), d.row.s.mutable_data_ptr<float>(),
                                    d.col.q.mutable_data_ptr<int8_t>(), d.col.ld(), d.col.s.mutable_data_ptr<float>(), m.rows, m.cols,
                                    (int)block, on.raw()),
          "bi8_quantize_dual");
    return d;
}

void check_scales(const Tensor& s, int64_t nb, int64_t rows, int64_t block, const char* name) {
    if (s.dim() != 2 || s.size(0) != nb || s.size(1) != rows || s.scalar_type() != at::kFloat)
        value_error(std::string(name) + " must be float32 " + shape_of(nb, rows) + " for block " + std::to_string(block) + ", got " +
                    c10::toString(s.scalar_type()) + " " + shape_of(s));
}

Tensor dequantize(const Tensor& q, const Tensor& state, int64_t block, at::ScalarType out_type) {
    need_cuda(q);
    if (q.dim() != 2) value_error("expected a 2-D tensor, got " + shape_of(q));
    if (q.scalar_type() != at::kChar) value_error(std::string("expected an int8 tensor, got ") + c10::toString(q.scalar_type()));
    const int64_t m = q.size(0), k = q.size(1);
    check_scales(state, ceil_div(k, block), m, block, "state");
    OnDevice on(q);
    const Mat x = mat2d(q);
    const Tensor s = state.contiguous();
    Tensor out = empty_on(q, {m, k}, out_type);
    check(bi8_dequantize_rowwise_pitched(static_cast<const int8_t*>(x.ptr), x.ld, s.const_data_ptr<float>(), out.data_ptr(), dtype_code(out_type), m, k, (int)block, on.raw()),
          "bi8_dequantize_rowwise");
    return out;
}

// ---- GEMM ---------------------------------------------------------------------------------------------------------------
// Bias operand: a contiguous vector of a type the kernels read, or nothing.
struct Bias {
    Tensor owner;
    const void* ptr = nullptr;
    int code = 0;
    Bias(const Tensor& b, int64_t n) {
        if (!b.defined()) return;
        if (b.numel() != n) value_error("bias must have " + std::to_string(n) + " elements, got " + std::to_string(b.numel()));
        owner = (b.dim() == 1 ? b : b.reshape({n})).contiguous();
        const at::ScalarType t = owner.scalar_type();
        if (t != at::kBFloat16 && t != at::kHalf && t != at::kFloat) owner = owner.to(at::kFloat);
        ptr = owner.data_ptr();
        code = dtype_code(owner.scalar_type());
    }
};

// Workspace of a GEMM call: without seeds no parts of a tile meet in a cluster, and those that would have take one.
size_t gemm_workspace(int64_t m, int64_t n, int64_t k, int64_t block, int flags) {
    return flags & BI8_GEMM_NO_SEED ? bi8_gemm_workspace_bytes(m, n, k, (int)block) : bi8_gemm_workspace_used(m, n, k, (int)block);
}

struct Operands {
    Mat a, bt;
};

// Brings both int8 operands to the form the library takes: a [M, K] and b^T [N, K] with contiguous rows.
Operands gemm_operands(const Tensor& a, const Tensor& b, const OnDevice& on) {
    need_cuda(a);
    if (a.dim() != 2 || b.dim() != 2) value_error("expected 2-D operands, got " + shape_of(a) + " and " + shape_of(b));
    if (a.size(1) != b.size(0)) assertion("incompatible dimensions");
    if (a.scalar_type() != at::kChar || b.scalar_type() != at::kChar)
        value_error(std::string("operands must be int8, got ") + c10::toString(a.scalar_type()) + " and " + c10::toString(b.scalar_type()));
    Operands o{mat2d(a), mat2d_t(b)};
    // The tensor-core kernels need 16-byte aligned operand rows: where it is worth it both operands are re-pitched once.  Not for
    // a narrow output of more rows than the decode kernel takes: callers get the reference's order of operations there,
    // from the CUDA cores.
    const int64_t m = o.a.rows, n = o.bt.rows;
    if (worth_repitch(m, n, a.size(1)) && (m <= 64 || m * n >= 128 * 128)) {
        o.a = repitch(o.a, on);
        o.bt = repitch(o.bt, on);
    }
    return o;
}

Tensor gemm(const Tensor& a_in, const Tensor& b_in, const Tensor& state_x, const Tensor& state_w, const Tensor& bias_in, int64_t block,
            at::ScalarType out_type, int flags) {
    need_cuda(a_in);
    OnDevice on(a_in);
    const Operands o = gemm_operands(a_in, b_in, on);
    const int64_t m = o.a.rows, n = o.bt.rows, k = o.a.cols, nb = ceil_div(k, block);
    check_scales(state_x, nb, m, block, "state_x");
    check_scales(state_w, nb, n, block, "state_w");
    const Tensor sx = state_x.contiguous(), sw = state_w.contiguous();
    Tensor c = empty_on(a_in, {m, n}, out_type);
    const Bias bias(bias_in, n);
    const size_t ws_bytes = gemm_workspace(m, n, k, block, flags);
    const Tensor ws = scratch(a_in, (int64_t)ws_bytes);
    check(bi8_gemm_dequant(static_cast<const int8_t*>(o.a.ptr), o.a.ld, static_cast<const int8_t*>(o.bt.ptr), o.bt.ld, sx.const_data_ptr<float>(),
                           sw.const_data_ptr<float>(), bias.ptr, bias.code, c.data_ptr(), n, dtype_code(out_type), m, n, k, (int)block,
                           ws.defined() ? ws.data_ptr() : nullptr, ws_bytes, flags, on.raw()),
          "bi8_gemm_dequant");
    return c;
}

Tensor block_partials(const Tensor& a, const Tensor& b, int64_t block, int flags) {
    need_cuda(a);
    OnDevice on(a);
    const Operands o = gemm_operands(a, b, on);
    const int64_t m = o.a.rows, n = o.bt.rows, k = o.a.cols;
    Tensor out = at::zeros({ceil_div(k, block), m, n}, at::TensorOptions().dtype(at::kInt).device(a.device()));
    check(bi8_gemm_block_partials(static_cast<const int8_t*>(o.a.ptr), o.a.ld, static_cast<const int8_t*>(o.bt.ptr), o.bt.ld,
                                  out.mutable_data_ptr<int32_t>(), m, n, k, (int)block, flags, on.raw()),
          "bi8_gemm_block_partials");
    return out;
}

// ---- producer step + quantizer + GEMM + residual ------------------------------------------------------------------------
// Operands of a fused producer step with a shared row pitch.
struct Pre {
    int op;
    Mat x, x2;
    Tensor weight;
    Pre(int op_, const Tensor& x_in, const Tensor& x2_in, const Tensor& w_in) : op(op_), x(mat_rows(x_in)) {
        if (op == BI8_PRE_SILU_MUL) {
            if (!x2_in.defined() || x2_in.sizes() != x_in.sizes() || x2_in.scalar_type() != x_in.scalar_type() || x2_in.device() != x_in.device())
                value_error("silu_mul needs a second operand with x's shape, dtype and device");
            x2 = mat_rows(x2_in);
            if (x2.ld != x.ld) {           // e.g. one of the two was copied: give both the same row pitch
                x = mat_rows(x_in.contiguous());
                x2 = mat_rows(x2_in.contiguous());
            }
        }
        if (op == BI8_PRE_RMSNORM && w_in.defined()) {
            if (w_in.numel() != x.cols) value_error("norm weight must have " + std::to_string(x.cols) + " elements, got " + std::to_string(w_in.numel()));
            weight = (w_in.dim() == 1 ? w_in : w_in.reshape({-1})).to(x_in.scalar_type()).contiguous();
        }
    }
    const void* weight_ptr() const { return weight.defined() ? weight.data_ptr() : nullptr; }
};

Quantized quantize_pre(int op, const Tensor& x_in, const Tensor& x2, const Tensor& weight, double eps, int64_t block) {
    need_cuda(x_in);
    if (x_in.dim() != 2) value_error("expected a 2-D tensor, got " + shape_of(x_in));
    OnDevice on(x_in);
    const Pre pre(op, x_in, x2, weight);
    const int64_t m = pre.x.rows, k = pre.x.cols;
    Quantized r{empty_q(x_in, m, k, false), empty_on(x_in, {ceil_div(k, block), m}, at::kFloat)};
    check(bi8_quantize_rowwise_pre_pitched(op, pre.x.ptr, pre.x2.ptr, dtype_code(x_in.scalar_type()), pre.x.ld, pre.weight_ptr(), (float)eps,
                                   r.q.mutable_data_ptr<int8_t>(), r.ld(), r.s.mutable_data_ptr<float>(), m, k, (int)block, on.raw()),
          "bi8_quantize_rowwise_pre");
    return r;
}

// y = pre(x) W^T (+ bias) (+ residual) for x [..., K] and the int8 weights as `w` = [N, K] (or, with `w_transposed`, its [K, N] view)
Tensor linear(int op, const Tensor& x_in, const Tensor& w, bool w_transposed, const Tensor& state_w, const Tensor& bias_in, const Tensor& x2,
              const Tensor& norm_weight, double eps, const Tensor& residual, const Tensor& out_in, int64_t block, at::ScalarType out_type, int flags) {
    need_cuda(x_in);
    if (w.dim() != 2) value_error("expected 2-D weights, got " + shape_of(w));
    if (x_in.dim() == 0 || x_in.size(-1) != w.size(w_transposed ? 0 : 1)) assertion("incompatible dimensions");
    if (w.scalar_type() != at::kChar) value_error(std::string("weights must be int8, got ") + c10::toString(w.scalar_type()));
    OnDevice on(x_in);
    const Pre pre(op, x_in, x2, norm_weight);
    Mat bt = w_transposed ? mat2d_t(w) : mat2d(w);
    const int64_t m = pre.x.rows, k = pre.x.cols, n = bt.rows, nb = ceil_div(k, block);
    check_scales(state_w, nb, n, block, "state_w");
    const Tensor sw = state_w.contiguous();
    c10::SmallVector<int64_t, 6> shape(x_in.sizes().begin(), x_in.sizes().end());
    shape.back() = n;
    Tensor out = out_in, res = residual;
    int64_t ldc = n, ldr = 0;
    auto check_2d = [&](const Tensor& t, const char* name) {
        if (t.dim() != 2 || t.size(0) != m || t.size(1) != n || t.scalar_type() != out_type || t.stride(1) != 1 || t.device() != x_in.device())
            value_error(std::string(name) + " must be " + c10::toString(out_type) + " " + shape_of(m, n) + " with contiguous rows on " + x_in.device().str());
        return m > 1 ? t.stride(0) : std::max<int64_t>(n, 1);
    };
    if (out.defined()) ldc = check_2d(out, "out");
    else out = empty_on(x_in, shape, out_type);
    if (res.defined()) {
        if (res.dim() != 2 && n > 0) res = res.reshape({-1, n});
        ldr = check_2d(res, "residual");
    }
    const Bias bias(bias_in, n);
    Tensor target = out;
    if (res.defined() && out.data_ptr() == res.data_ptr() && !(m <= 64 && bias.ptr == nullptr && n % 4 == 0 && k % 16 == 0 && ldc == ldr)) {
        target = empty_on(x_in, {m, n}, out_type);          // not the path that may update in place
        ldc = n;
    }
    const int x_code = dtype_code(x_in.scalar_type());
    const void* res_ptr = res.defined() ? res.data_ptr() : nullptr;
    auto fused = [&](int8_t* xq, float* sx, void* ws, size_t ws_bytes) {
        return bi8_gemm_dequant_fused_pre(op, pre.x.ptr, pre.x2.ptr, x_code, pre.x.ld, pre.weight_ptr(), (float)eps, xq, sx,
                                          static_cast<const int8_t*>(bt.ptr), bt.ld, sw.const_data_ptr<float>(), bias.ptr, bias.code, res_ptr, ldr,
                                          target.data_ptr(), ldc, dtype_code(out_type), m, n, k, (int)block, ws, ws_bytes, flags, on.raw());
    };
    auto finish = [&] {
        if (!target.is_same(out)) out.copy_(target);
        return out;
    };
    // The form that quantizes inside the GEMM needs no scratch, whose allocation is 0.6 us of such a call (one token through
    // 4096 x 4096: 8.8 us with it, 8.2 without).  Where that form does not apply nothing has been launched.
    if (m <= 16 && m * k <= BI8_ONE_LAUNCH_VALUES && k % 16 == 0) {
        const int rc = fused(nullptr, nullptr, nullptr, 0);
        if (rc != BI8_ERR_WORKSPACE) {
            check(rc, "bi8_gemm_dequant_fused_pre");
            return finish();
        }
    }
    const size_t ws_bytes = gemm_workspace(m, n, k, block, flags);
    // the quantized activations live in the call's scratch behind the GEMM's workspace
    Carve carve;
    carve.take((int64_t)ws_bytes);
    const int64_t xq_at = carve.take(m * pitch16(k)), sx_at = carve.take(nb * m * 4);
    // Weights whose rows are not 16-byte aligned (of a layer, a checkpoint's dense copy) are copied to rows that are where the GEMM is
    // long enough to gain from it.
    const bool copy_w = k % 16 != 0 && worth_repitch(m, n, k) && !on_boundaries(bt);
    const int64_t w_at = copy_w ? carve.take(n * pitch16(k)) : 0;
    const Tensor ws = scratch(x_in, carve.bytes);
    char* ws_ptr = ws.defined() ? static_cast<char*>(ws.data_ptr()) : nullptr;
    int8_t* xq = reinterpret_cast<int8_t*>(ws_ptr + xq_at);
    float* sx = reinterpret_cast<float*>(ws_ptr + sx_at);
    void* gemm_ws = ws_bytes ? ws_ptr : nullptr;
    if (k % 16 != 0) {
        // rows that are not 16-byte aligned: the activations are quantized into rows that are, with the copy in one launch if they are few
        // (one after another it is the copy first: the GEMM starts early behind the short quantizer)
        bi8_quantize_task tasks[2] = {};
        bi8_quantize_task &tw = tasks[0], &tx = tasks[1];
        if (copy_w) {
            tw.x = bt.ptr;
            tw.x_dtype = BI8_I8;
            tw.ldx = bt.ld;
            tw.rows = n;
            tw.cols = k;
            tw.q_row = reinterpret_cast<int8_t*>(ws_ptr + w_at);
            tw.ldq_row = pitch16(k);
            bt.ptr = tw.q_row;
            bt.ld = tw.ldq_row;
        }
        if (op == BI8_PRE_NONE) {
            tx.x = pre.x.ptr;
            tx.x_dtype = x_code;
            tx.ldx = pre.x.ld;
            tx.rows = m;
            tx.cols = k;
            tx.q_row = xq;
            tx.ldq_row = pitch16(k);
            tx.s_row = sx;
            check(bi8_quantize_many(copy_w ? tasks : &tx, copy_w ? 2 : 1, (int)block, on.raw()), "bi8_quantize_many");
        } else {
            if (copy_w) check(bi8_quantize_many(&tw, 1, (int)block, on.raw()), "bi8_quantize_many");
            check(bi8_quantize_rowwise_pre_pitched(op, pre.x.ptr, pre.x2.ptr, x_code, pre.x.ld, pre.weight_ptr(), (float)eps, xq, pitch16(k), sx, m, k,
                                                   (int)block, on.raw()),
                  "bi8_quantize_rowwise_pre");
        }
        check(bi8_gemm_dequant_residual(xq, pitch16(k), static_cast<const int8_t*>(bt.ptr), bt.ld, sx, sw.const_data_ptr<float>(), bias.ptr, bias.code,
                                        res_ptr, ldr, target.data_ptr(), ldc, dtype_code(out_type), m, n, k, (int)block, gemm_ws, ws_bytes,
                                        flags & ~BI8_GEMM_QUANT_IN_KERNEL, on.raw()),
              "bi8_gemm_dequant_residual");
        return finish();
    }
    check(fused(xq, sx, gemm_ws, ws_bytes), "bi8_gemm_dequant_fused_pre");
    return finish();
}

// ---- training: forward and backward as one autograd node ----------------------------------------------------------------
// What the Python side knows at call time; the backward pass looks it up again (block size and result type are module-level
// knobs, and the cache of quantized weights is a dict on the weight).
PyObject* g_config = nullptr;            // the module blockwise_int8_linear_b200.block_linear_config

int64_t config_block() {                 // with the interpreter lock
    PyObject* v = PyObject_GetAttrString(g_config, "GROUP_SIZE");
    if (!v) throw python_error();
    const long long b = PyLong_AsLongLong(v);
    Py_DECREF(v);
    if (b == -1 && PyErr_Occurred()) throw python_error();
    if (b < 1 || b > 0x7fffffff) value_error("block size must be positive, got " + std::to_string(b));
    return b;
}
at::ScalarType config_dtype() {          // with the interpreter lock
    PyObject* v = PyObject_GetAttrString(g_config, "INPUT_OUTPUT_TORCH_TYPE");
    if (!v) throw python_error();
    const bool is_dtype = THPDtype_Check(v);
    const at::ScalarType t = is_dtype ? reinterpret_cast<THPDtype*>(v)->scalar_type : at::kFloat;
    Py_DECREF(v);
    if (!is_dtype) throw PyFail{PyExc_TypeError, "INPUT_OUTPUT_TORCH_TYPE must be a torch.dtype"};
    (void)dtype_code(t);
    return t;
}

// A quantized matrix as the kernels see it: int8 rows with pitch ld, block scales [blocks, rows].
struct QRef {
    int8_t* q = nullptr;
    float* s = nullptr;
    int64_t rows = 0, cols = 0, ld = 0;
};

// Where a quantized [rows, cols] lies in one allocation of the call, and the reference to it once that exists.  The training
// passes keep no tensor of an intermediate result: one allocation per pass instead of two per quantization.
struct QPlan {
    int64_t rows = 0, cols = 0, q_at = 0, s_at = 0;
    QPlan() = default;
    QPlan(Carve& c, int64_t rows_, int64_t cols_, int64_t block) : rows(rows_), cols(cols_) {
        q_at = c.take(rows * pitch16(cols));
        s_at = c.take(ceil_div(cols, block) * rows * 4);
    }
    QRef in(void* mem) const {
        char* m = static_cast<char*>(mem);
        return {reinterpret_cast<int8_t*>(m + q_at), reinterpret_cast<float*>(m + s_at), rows, cols, pitch16(cols)};
    }
};

QRef ref_of(const Quantized& r) {
    return {static_cast<int8_t*>(r.q.data_ptr()), static_cast<float*>(r.s.data_ptr()), r.q.size(0), r.q.size(1),
            r.ld()};
}

// The quantizations of a pass, which share a launch where they are small.
struct Tasks {
    bi8_quantize_task list[4];
    int n = 0;
    // x row-wise and / or column-wise
    void add(const Mat& m, int code, const QRef* row, const QRef* col) {
        bi8_quantize_task t{};
        t.x = m.ptr;
        t.x_dtype = code;
        t.ldx = m.ld;
        t.rows = m.rows;
        t.cols = m.cols;
        if (row) {
            t.q_row = row->q;
            t.ldq_row = row->ld;
            t.s_row = row->s;
        }
        if (col) {
            t.q_col = col->q;
            t.ldq_col = col->ld;
            t.s_col = col->s;
        }
        list[n++] = t;
    }
    bool fits(int64_t block) const { return n > 0 && bi8_quantize_many_fits(list, n, (int)block) != 0; }
    void run(int64_t block, void* stream) const {
        if (n > 0) check(bi8_quantize_many(list, n, (int)block, stream), "bi8_quantize_many");
    }
};
// out = a b^T (+ bias); `ws` of at least bi8_gemm_workspace_used
void gemm_into(const QRef& a, const QRef& b, const Bias* bias, int64_t block, const Tensor& out, void* ws, size_t ws_bytes, void* stream) {
    check(bi8_gemm_dequant(a.q, a.ld, b.q, b.ld, a.s, b.s, bias ? bias->ptr : nullptr, bias ? bias->code : 0, out.data_ptr(), b.rows,
                           dtype_code(out.scalar_type()), a.rows, b.rows, a.cols, (int)block, ws_bytes ? ws : nullptr, ws_bytes, 0, stream),
          "bi8_gemm_dequant");
}

// One blocking of a weight from the cache dict under `key`, or undefined tensors.
Quantized cache_get(PyObject* cache, const char* key) {
    if (!cache) return {};
    pybind11::gil_scoped_acquire gil;
    PyObject* hit = PyDict_GetItemString(cache, key);
    if (hit && PyTuple_Check(hit) && PyTuple_GET_SIZE(hit) == 2)
        return {THPVariable_Unpack(PyTuple_GET_ITEM(hit, 0)), THPVariable_Unpack(PyTuple_GET_ITEM(hit, 1))};
    return {};
}
void cache_put(PyObject* cache, const char* key, const Quantized& r) {
    pybind11::gil_scoped_acquire gil;
    PyObject* pair = PyTuple_New(2);
    if (!pair) throw python_error();
    PyTuple_SET_ITEM(pair, 0, THPVariable_Wrap(r.q));
    PyTuple_SET_ITEM(pair, 1, THPVariable_Wrap(r.s));
    const int rc = PyDict_SetItemString(cache, key, pair);
    Py_DECREF(pair);
    if (rc != 0) throw python_error();
}

Tensor as_bytes(const Tensor& like, int64_t bytes) { return empty_on(like, {std::max<int64_t>(bytes, 1)}, at::kByte); }

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// Backward of y = x W^T + bias with both GEMMs in blockwise int8 (block_linear.py:85-112 in the reference).
struct LinearBackward : public Node {
    SavedVariable x;                     // x itself, or (x_quantized) the bytes of its column-wise int8 copy and scales
    SavedVariable weight;
    bool x_quantized = false, has_bias = false, fuse_dual = true;
    int64_t block = 0;
    std::vector<int64_t> x_sizes;
    PyObject* cache = nullptr;           // owned reference to the weight's cache dict, or null

    ~LinearBackward() override {
        if (cache && Py_IsInitialized()) {
            pybind11::gil_scoped_acquire gil;
            Py_DECREF(cache);
        }
    }
    std::string name() const override { return "blockwise_int8_linearBackward"; }
    void release_variables() override {
        std::lock_guard<std::mutex> lock(mutex_);
        x.reset_data();
        weight.reset_data();
    }
    variable_list apply(variable_list&& grads) override;
};

variable_list LinearBackward::apply(variable_list&& grads) {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    // A backward pass that is itself recorded: the bias gradient is a sum of G that can be differentiated again.  The two products
    // of quantized operands cannot.
    const bool want_b = has_bias && task_should_compute_output(2), recorded = at::GradMode::is_enabled() && grads[0].requires_grad();
    int64_t b = 0;
    at::ScalarType type;
    try {
        {
            pybind11::gil_scoped_acquire gil;
            b = config_block();
            type = config_dtype();
        }
        if (x_quantized && b != block)
            throw std::runtime_error("GROUP_SIZE changed between the forward and the backward pass of a BlockInt8Linear");
        std::lock_guard<std::mutex> lock(mutex_);
        auto self = getptr();
        const Tensor saved_x = x.unpack(self), w = weight.unpack(self);
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        const bool need_x = task_should_compute_output(0), need_w = task_should_compute_output(1), need_b = want_b && !recorded;
        need_cuda(grads[0]);
        OnDevice on(grads[0]);
        const Mat g = mat_rows(grads[0]), wm = mat2d(w);
        const int g_code = dtype_code(grads[0].scalar_type()), w_code = dtype_code(w.scalar_type());
        const int64_t m = g.rows, n = g.cols, k = wm.cols;
        Mat xm;
        if (need_w && !x_quantized) xm = mat_rows(saved_x);

        // every intermediate result of this pass lies in one allocation
        const Quantized cached = need_x ? cache_get(cache, "col") : Quantized{};
        Quantized fresh;                                     // the weight's other blocking, where the cache is to keep it
        const size_t ws_x = need_x ? bi8_gemm_workspace_used(m, k, n, (int)b) : 0, ws_w = need_w ? bi8_gemm_workspace_used(n, k, m, (int)b) : 0,
                     ws_b = need_b ? bi8_column_sum_workspace_bytes(m, n) : 0,
                     ws_d = need_b && need_x && need_w && fuse_dual ? bi8_quantize_dual_sum_workspace_bytes(g_code, m, n, (int)b) : 0;
        Carve carve;
        const int64_t ws_at = carve.take((int64_t)std::max({ws_x, ws_w, ws_b, ws_d}));
        QPlan g_row, g_col, w_col, x_col;
        if (need_x) g_row = QPlan(carve, m, n, b);
        if (need_w) g_col = QPlan(carve, n, m, b);
        if (need_x && !cached.q.defined() && !cache) w_col = QPlan(carve, k, n, b);
        if (need_w && x_quantized) {
            Carve kept;
            x_col = QPlan(kept, k, m, b);                    // the layout in which train_linear saved it
        } else if (need_w) {
            x_col = QPlan(carve, k, m, b);
        }
        const Tensor mem = as_bytes(grads[0], carve.bytes);
        void* const base = mem.data_ptr();
        void* const ws = static_cast<char*>(base) + ws_at;
        void* const st = on.raw();

        // All operands first: G (in both blockings with one read, where the layer fuses them), the weight along N and the tokens of x.
        const QRef gr = need_x ? g_row.in(base) : QRef{}, gc = need_w ? g_col.in(base) : QRef{};
        Tasks tasks;
        if (need_x && need_w && fuse_dual) {
            tasks.add(g, g_code, &gr, &gc);
        } else {
            if (need_x) tasks.add(g, g_code, &gr, nullptr);
            if (need_w) tasks.add(g, g_code, nullptr, &gc);
        }
        QRef wt, xt;
        if (need_x) {
            // A cached blocking is still valid: unpacking the weight raised if it was modified since the forward pass.
            if (cached.q.defined()) wt = ref_of(cached);
            else {
                if (cache) {
                    fresh = Quantized{empty_q(w, k, n, true), empty_on(w, {ceil_div(n, b), k}, at::kFloat)};
                    wt = ref_of(fresh);
                } else {
                    wt = w_col.in(base);
                }
                tasks.add(wm, w_code, nullptr, &wt);
            }
        }
        if (need_w) {
            xt = x_col.in(x_quantized ? saved_x.data_ptr() : base);
            if (!x_quantized) tasks.add(xm, dtype_code(saved_x.scalar_type()), nullptr, &xt);
        }
        // small passes: the bias gradient rides in the same launch
        bool summed = false;
        if (need_b) {
            out[2] = empty_on(grads[0], {n}, grads[0].scalar_type());
            if (tasks.n > 0 && tasks.list[0].x == g.ptr) {
                tasks.list[0].sum = out[2].data_ptr();
                summed = tasks.fits(b);
                if (!summed) tasks.list[0].sum = nullptr;
            }
            if (!summed && ws_d && m > 0 && n > 0) {
                // larger ones: from the read that makes both blockings
                check(bi8_quantize_dual_sum(g.ptr, g_code, g.ld, gr.q, gr.ld, gr.s, gc.q, gc.ld, gc.s, out[2].data_ptr(), m, n, (int)b, ws, ws_d, st),
                      "bi8_quantize_dual_sum");
                for (int i = 1; i < tasks.n; ++i) tasks.list[i - 1] = tasks.list[i];
                --tasks.n;
                summed = true;
            }
        }
        tasks.run(b, st);
        if (fresh.q.defined()) cache_put(cache, "col", fresh);
        if (need_x) {
            // contraction over N, both operands blocked along N (block_linear.py:92-95)
            out[0] = empty_on(grads[0], x_sizes, type);
            gemm_into(gr, wt, nullptr, b, out[0], ws, ws_x, st);
        }
        if (need_w) {
            // contraction over the tokens, both operands blocked along M (block_linear.py:100-104)
            out[1] = empty_on(grads[0], {n, k}, type);
            gemm_into(gc, xt, nullptr, b, out[1], ws, ws_w, st);
        }
        if (need_b && !summed) {
            check(bi8_column_sum(g.ptr, g_code, g.ld, out[2].data_ptr(), m, n, ws_b ? ws : nullptr, ws_b, st), "bi8_column_sum");
        }
    } catch (const PyFail& e) {
        pybind11::gil_scoped_acquire gil;
        PyErr_SetString(e.type, e.text.c_str());
        python_error err;
        err.persist();
        throw err;
    }
    if (want_b && recorded) out[2] = grads[0].reshape({-1, grads[0].size(-1)}).sum(0);
    return out;
}

// y = x W^T (+ bias), every operand quantized on the fly, recorded for backward when a gradient is wanted.  With `fuse_dual`
// a layer whose weight is trained reads x once for both of its blockings and keeps the int8 transposed copy instead of x.
Tensor train_linear(const Tensor& x_in, const Tensor& w, const Tensor& bias_in, int64_t block, at::ScalarType type, bool fuse_dual, PyObject* cache) {
    need_cuda(x_in);
    if (x_in.dim() == 0 || w.dim() != 2 || x_in.size(-1) != w.size(1)) assertion("incompatible dimensions");
    const bool grad = at::GradMode::is_enabled() && (x_in.requires_grad() || w.requires_grad() || (bias_in.defined() && bias_in.requires_grad()));
    std::shared_ptr<LinearBackward> node;
    if (grad) {
        node = std::shared_ptr<LinearBackward>(new LinearBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(x_in, w, bias_in));
    }
    Tensor out;
    {
        at::AutoDispatchBelowADInplaceOrView below_autograd;
        OnDevice on(x_in);
        const Mat x = mat_rows(x_in), wm = mat2d(w);
        const int x_code = dtype_code(x_in.scalar_type()), w_code = dtype_code(w.scalar_type());
        const int64_t m = x.rows, n = wm.rows, k = wm.cols;
        const bool keep = node && w.requires_grad() && fuse_dual;
        const Quantized cached = cache_get(cache, "row");
        Quantized fresh;
        const size_t ws_bytes = bi8_gemm_workspace_used(m, n, k, (int)block);
        Carve carve, kept;
        const int64_t ws_at = carve.take((int64_t)ws_bytes);
        const QPlan x_row(carve, m, k, block), x_col = keep ? QPlan(kept, k, m, block) : QPlan();
        const QPlan w_row = !cached.q.defined() && !cache ? QPlan(carve, n, k, block) : QPlan();
        const Tensor mem = as_bytes(x_in, carve.bytes);
        void* const base = mem.data_ptr();
        void* const st = on.raw();
        const QRef xq = x_row.in(base);
        Tasks tasks;
        if (keep) {
            const Tensor saved = as_bytes(x_in, kept.bytes);
            const QRef xt = x_col.in(saved.data_ptr());
            tasks.add(x, x_code, &xq, &xt);
            node->x = SavedVariable(saved, false);
            node->x_quantized = true;
        } else {
            tasks.add(x, x_code, &xq, nullptr);
        }
        QRef wq;
        if (cached.q.defined()) {
            wq = ref_of(cached);
        } else if (cache) {
            fresh = Quantized{empty_q(w, n, k, true), empty_on(w, {ceil_div(k, block), n}, at::kFloat)};
            wq = ref_of(fresh);
            tasks.add(wm, w_code, &wq, nullptr);
        } else {
            wq = w_row.in(base);
            tasks.add(wm, w_code, &wq, nullptr);
        }
        tasks.run(block, st);
        if (fresh.q.defined()) cache_put(cache, "row", fresh);
        const Bias bias(bias_in, n);
        c10::SmallVector<int64_t, 6> shape(x_in.sizes().begin(), x_in.sizes().end());
        shape.back() = n;
        out = empty_on(x_in, shape, type);
        gemm_into(xq, wq, bias.ptr ? &bias : nullptr, block, out, static_cast<char*>(base) + ws_at, ws_bytes, st);
    }
    if (node) {
        if (!node->x_quantized) node->x = SavedVariable(x_in, false);
        node->weight = SavedVariable(w, false);
        node->has_bias = bias_in.defined();
        node->fuse_dual = fuse_dual;
        node->block = block;
        node->x_sizes = x_in.sizes().vec();
        if (cache) {
            pybind11::gil_scoped_acquire gil;
            Py_INCREF(cache);
            node->cache = cache;
        }
        torch::autograd::set_history(out, node);
    }
    return out;
}

// ---- decode step: rotary embedding and cache append ---------------------------------------------------------------------
Tensor rope_cache_append(const Tensor& qkv_in, const Tensor& cis_in, const Tensor& pos, const Tensor& kcache, const Tensor& vcache) {
    need_cuda(qkv_in);
    if (qkv_in.dim() != 4 || qkv_in.size(1) != 3 || qkv_in.size(3) % 2 != 0) value_error("expected [B, 3, H, D] with even D, got " + shape_of(qkv_in));
    const int64_t b = qkv_in.size(0), h = qkv_in.size(2), d = qkv_in.size(3);
    OnDevice on(qkv_in);
    const Tensor qkv = qkv_in.contiguous();
    // complex64 [D/2] or float32 (cos, sin) pairs: the same bytes
    const bool cplx = cis_in.scalar_type() == at::kComplexFloat;
    if ((!cplx && cis_in.scalar_type() != at::kFloat) || cis_in.numel() * (cplx ? 2 : 1) != d || !cis_in.is_contiguous())
        value_error("cis must hold " + std::to_string(d / 2) + " contiguous (cos, sin) float32 pairs");
    if (pos.scalar_type() != at::kLong || pos.numel() != 1 || pos.device() != qkv.device())
        value_error("pos must be an int64 tensor with one element on the activations' device");
    if (kcache.dim() != 4) value_error("caches must be 4-D, got " + shape_of(kcache));
    const int64_t max_len = kcache.size(2);
    for (const Tensor* c : {&kcache, &vcache})
        if (c->dim() != 4 || c->size(0) != b || c->size(1) != h || c->size(2) != max_len || c->size(3) != d || c->scalar_type() != qkv.scalar_type() ||
            !c->is_contiguous() || c->device() != qkv.device())
            value_error(std::string("caches must be contiguous ") + c10::toString(qkv.scalar_type()) + " [" + std::to_string(b) + ", " + std::to_string(h) +
                        ", max_len, " + std::to_string(d) + "] on " + qkv.device().str());
    Tensor q = empty_on(qkv, {b, h, 1, d}, qkv.scalar_type());
    check(bi8_rope_cache_append(qkv.data_ptr(), dtype_code(qkv.scalar_type()), static_cast<const float*>(cis_in.data_ptr()),
                                static_cast<const long long*>(pos.data_ptr()), q.data_ptr(), kcache.data_ptr(), vcache.data_ptr(), b, h, d, max_len, on.raw()),
          "bi8_rope_cache_append");
    return q;
}

// ---- bindings -----------------------------------------------------------------------------------------------------------
struct Args {
    PyObject* const* a;
    Py_ssize_t n;
    const Tensor& tensor(int i) const {
        if (!THPVariable_Check(a[i])) throw PyFail{PyExc_TypeError, std::string("expected a tensor, got ") + Py_TYPE(a[i])->tp_name};
        return THPVariable_Unpack(a[i]);
    }
    Tensor optional(int i) const { return a[i] == Py_None ? Tensor() : tensor(i); }
    int64_t integer(int i) const {
        const long long v = PyLong_AsLongLong(a[i]);
        if (v == -1 && PyErr_Occurred()) throw python_error();
        return v;
    }
    double number(int i) const {
        const double v = PyFloat_AsDouble(a[i]);
        if (v == -1.0 && PyErr_Occurred()) throw python_error();
        return v;
    }
    at::ScalarType dtype(int i) const {
        if (!THPDtype_Check(a[i])) throw PyFail{PyExc_TypeError, "expected a torch.dtype"};
        const at::ScalarType t = reinterpret_cast<THPDtype*>(a[i])->scalar_type;
        (void)dtype_code(t);
        return t;
    }
    int64_t block(int i) const {
        const int64_t b = integer(i);
        if (b < 1 || b > 0x7fffffff) value_error("block size must be positive, got " + std::to_string(b));
        return b;
    }
};

PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap(const Quantized& r) {
    PyObject* t = PyTuple_New(2);
    PyTuple_SET_ITEM(t, 0, wrap(r.q));
    PyTuple_SET_ITEM(t, 1, wrap(r.s));
    return t;
}
PyObject* wrap(const Dual& d) {
    PyObject* t = PyTuple_New(4);
    PyTuple_SET_ITEM(t, 0, wrap(d.row.q));
    PyTuple_SET_ITEM(t, 1, wrap(d.row.s));
    PyTuple_SET_ITEM(t, 2, wrap(d.col.q));
    PyTuple_SET_ITEM(t, 3, wrap(d.col.s));
    return t;
}

// Runs `body` without the interpreter lock (kernel launches can block when the launch queue is full) and turns its exceptions into Python's.
template <typename Body>
PyObject* call(const char* name, const Args& args, Py_ssize_t want, Body body, bool records_history = false) {
    try {
        if (args.n != want) throw PyFail{PyExc_TypeError, std::string(name) + " takes " + std::to_string(want) + " arguments, got " + std::to_string(args.n)};
        auto result = [&] {
            auto work = body(args);            // reads the arguments with the lock held
            pybind11::gil_scoped_release no_gil;
            std::optional<at::AutoDispatchBelowADInplaceOrView> below_autograd;
            if (!records_history) below_autograd.emplace();
            return work();
        }();
        return wrap(result);
    } catch (const PyFail& e) {
        PyErr_SetString(e.type, e.text.c_str());
        return nullptr;
    } catch (...) {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

#define BI8_METHOD(name) PyObject* name##_py(PyObject*, PyObject* const* a, Py_ssize_t n)

BI8_METHOD(quantize_rowwise) {   // x, block, whether the result is only a GEMM operand
    return call("quantize_rowwise", {a, n}, 3, [](const Args& g) {
        return [x = g.tensor(0), b = g.block(1), operand = g.integer(2) != 0] { return quantize_rowwise(x, b, operand); };
    });
}
BI8_METHOD(quantize_colwise) {   // x, block, whether the result is only a GEMM operand
    return call("quantize_colwise", {a, n}, 3, [](const Args& g) {
        return [x = g.tensor(0), b = g.block(1), operand = g.integer(2) != 0] { return quantize_colwise(x, b, operand); };
    });
}
BI8_METHOD(quantize_dual) {
    return call("quantize_dual", {a, n}, 2, [](const Args& g) { return [x = g.tensor(0), b = g.block(1)] { return quantize_dual(x, b); }; });
}
BI8_METHOD(quantize_pre) {       // op, x, x2, weight, eps, block
    return call("quantize_pre", {a, n}, 6, [](const Args& g) {
        return [op = (int)g.integer(0), x = g.tensor(1), x2 = g.optional(2), w = g.optional(3), eps = g.number(4), b = g.block(5)] {
            return quantize_pre(op, x, x2, w, eps, b);
        };
    });
}
BI8_METHOD(dequantize) {         // q, state, block, dtype
    return call("dequantize", {a, n}, 4, [](const Args& g) {
        return [q = g.tensor(0), s = g.tensor(1), b = g.block(2), t = g.dtype(3)] { return dequantize(q, s, b, t); };
    });
}
BI8_METHOD(gemm) {               // a, b, state_x, state_w, bias, block, dtype, flags
    return call("gemm", {a, n}, 8, [](const Args& g) {
        return [x = g.tensor(0), y = g.tensor(1), sx = g.tensor(2), sw = g.tensor(3), bias = g.optional(4), b = g.block(5), t = g.dtype(6),
                f = (int)g.integer(7)] { return gemm(x, y, sx, sw, bias, b, t, f); };
    });
}
BI8_METHOD(block_partials) {     // a, b, block, flags
    return call("block_partials", {a, n}, 4, [](const Args& g) {
        return [x = g.tensor(0), y = g.tensor(1), b = g.block(2), f = (int)g.integer(3)] { return block_partials(x, y, b, f); };
    });
}
BI8_METHOD(matmul) {             // op, x [M, K], b [K, N], state_w, bias, x2, norm_weight, eps, residual, out, block, dtype, flags
    return call("matmul", {a, n}, 13, [](const Args& g) {
        if (g.tensor(1).dim() != 2) {
            need_cuda(g.tensor(1));
            value_error("expected a 2-D tensor, got " + shape_of(g.tensor(1)));
        }
        return [op = (int)g.integer(0), x = g.tensor(1), w = g.tensor(2), sw = g.tensor(3), bias = g.optional(4), x2 = g.optional(5), nw = g.optional(6),
                eps = g.number(7), res = g.optional(8), out = g.optional(9), b = g.block(10), t = g.dtype(11), f = (int)g.integer(12)] {
            return linear(op, x, w, true, sw, bias, x2, nw, eps, res, out, b, t, f);
        };
    });
}
BI8_METHOD(linear) {             // op, x [..., K], W int8 [N, K], state_w, bias, x2, norm_weight, eps, residual, block, dtype
    return call("linear", {a, n}, 11, [](const Args& g) {
        return [op = (int)g.integer(0), x = g.tensor(1), w = g.tensor(2), sw = g.tensor(3), bias = g.optional(4), x2 = g.optional(5), nw = g.optional(6),
                eps = g.number(7), res = g.optional(8), b = g.block(9), t = g.dtype(10)] {
            return linear(op, x, w, false, sw, bias, x2, nw, eps, res, Tensor(), b, t, 0);
        };
    });
}
BI8_METHOD(train_linear) {       // x [..., K], W [N, K], bias, fuse_dual, cache dict or None: block size and type from the config module
    return call("train_linear", {a, n}, 5, [](const Args& g) {
        PyObject* cache = g.a[4] == Py_None ? nullptr : g.a[4];
        if (cache && !PyDict_Check(cache)) throw PyFail{PyExc_TypeError, "the weight cache must be a dict"};
        return [x = g.tensor(0), w = g.tensor(1), bias = g.optional(2), fuse = PyObject_IsTrue(g.a[3]) == 1, b = config_block(), t = config_dtype(), cache] {
            return train_linear(x, w, bias, b, t, fuse, cache);
        };
    }, true);
}
BI8_METHOD(rope_cache_append) {  // qkv, cis, pos, kcache, vcache
    return call("rope_cache_append", {a, n}, 5, [](const Args& g) {
        return [q = g.tensor(0), c = g.tensor(1), p = g.tensor(2), k = g.tensor(3), v = g.tensor(4)] { return rope_cache_append(q, c, p, k, v); };
    });
}
BI8_METHOD(bind) {               // the exception class of failed library calls, the configuration module
    if (n != 2) {
        PyErr_SetString(PyExc_TypeError, "bind takes 2 arguments");
        return nullptr;
    }
    g_error_class = Py_NewRef(a[0]);
    g_config = Py_NewRef(a[1]);
    Py_RETURN_NONE;
}

#define BI8_ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name##_py)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {BI8_ENTRY(quantize_rowwise), BI8_ENTRY(quantize_colwise), BI8_ENTRY(quantize_dual), BI8_ENTRY(quantize_pre),
                         BI8_ENTRY(dequantize), BI8_ENTRY(gemm), BI8_ENTRY(block_partials), BI8_ENTRY(matmul), BI8_ENTRY(linear),
                         BI8_ENTRY(train_linear), BI8_ENTRY(rope_cache_append), BI8_ENTRY(bind),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Host path of the blockwise-int8 operations.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
