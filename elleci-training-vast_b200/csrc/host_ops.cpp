// The operator calls of a layer step as one native call each: argument checks, output allocation on the caching allocator,
// the current stream, and the C-ABI call, for the functions of int2_tc_ops.py that every forward, backward and decode call
// goes through.  Same checks in the same order, same messages and same results as the Python statements they replace;
// what is gone is their cost: a small step (1024 tokens, 1536 -> 1536) is 59 us of kernels and was 275 us of host time, most of
// it in torch.cuda.current_stream(), torch.empty, tensor methods and ctypes conversions, a dozen per operator.
// Host time of a pass through the module API, before -> now: training step of that layer 275 -> 145 us, decode of one token 57 -> 19 us,
// feed-forward block with 4 tokens 177 -> 56 us.
//
// No state of its own but the handles that set_hooks hands over: the status word of each device, the function that turns a status
// into an exception and the one that checks the device's status word.  Scratch that a call needs and leaves is allocated per call.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <dlfcn.h>

#include <cstdlib>

#include "../../include/elleci_int2.h"

namespace {

using at::Tensor;

PyObject* g_check = nullptr;            // _lib.check(name, status): raises ElleciError
PyObject* g_status_of = nullptr;        // int2_tc_ops.device_status(device) -> int32 tensor
PyObject* g_check_status = nullptr;     // int2_tc_ops.check_device_status(device)

// The library's entry points, taken from the very file that the Python binding has loaded.
#define EL_FUNCTIONS(X)                                                                                                   \
    X(el_quantize_rows) X(el_zero) X(el_quantize_grad) X(el_quantize_tensor) X(el_rmsnorm_quantize_rows)                          \
    X(el_rmsnorm_backward) X(el_rmsnorm_backward_workspace_bytes) X(el_swiglu_quantize_rows) X(el_swiglu_backward)     \
    X(el_swiglu_backward_workspace_bytes) X(el_prelinear_rows) X(el_gemm_workspace_bytes) X(el_gemm_fwd_ws)            \
    X(el_gemm_dx_ws) X(el_dw_hysteresis) X(el_gemm_dw) X(el_hysteresis_from_dw) X(el_linear_decode) X(el_prelinear_decode) X(el_decode_workspace_bytes)
struct Library {
#define X(name) decltype(&::name) name = nullptr;
    EL_FUNCTIONS(X)
#undef X
} g_lib;

struct PyError {};                      // a Python exception is already set

[[noreturn]] void raise(const char* msg) {
    PyErr_SetString(PyExc_RuntimeError, msg);
    throw PyError();
}
[[noreturn]] void raise(const std::string& msg) { raise(msg.c_str()); }
#define EL_REQUIRE(cond, msg) do { if (!(cond)) raise(msg); } while (0)

bool is_none(PyObject* o) { return o == nullptr || o == Py_None; }

// an argument that has to be a CUDA tensor (the message names it as the Python functions do)
const Tensor& cuda_arg(PyObject* o, const char* name) {
    if (!THPVariable_Check(o) || !THPVariable_Unpack(o).is_cuda()) raise(std::string(name) + " must be a CUDA tensor");
    return THPVariable_Unpack(o);
}
const Tensor& tensor_arg(PyObject* o, const char* name) {
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s must be a tensor", name);
        throw PyError();
    }
    return THPVariable_Unpack(o);
}
double float_arg(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyError();
    return v;
}
long long int_arg(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw PyError();
    return v;
}
at::ScalarType dtype_arg(PyObject* o) {
    if (!THPDtype_Check(o)) {
        PyErr_SetString(PyExc_TypeError, "a torch.dtype is expected");
        throw PyError();
    }
    return reinterpret_cast<THPDtype*>(o)->scalar_type;
}
bool float_type(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16 || t == at::kFloat; }
int code_of(at::ScalarType t) {
    switch (t) {
        case at::kHalf: return EL_F16;
        case at::kBFloat16: return EL_BF16;
        case at::kFloat: return EL_F32;
        case at::kInt: return EL_I32;
        default:
            PyErr_Format(PyExc_KeyError, "torch.%s", c10::toString(t));
            throw PyError();
    }
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// A tensor's data pointer, null for an undefined one.  Throws for a tensor without storage (a functorch wrapper, a fake tensor),
// so the operators read the pointers of their inputs first: nothing has then been allocated or cached.
template <typename T = void> T* ptr(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }

struct ReleasedGil {                    // gives the GIL up and takes it back on every way out of the scope
    PyThreadState* state = PyEval_SaveThread();
    ReleasedGil() = default;
    ReleasedGil(const ReleasedGil&) = delete;
    ~ReleasedGil() noexcept(false) { PyEval_RestoreThread(state); }      // ends the thread if the interpreter is shutting down
};

// Makes a C-ABI call without the GIL (a full launch queue may block in it) and raises for a status other than 0.  The arguments
// are values by then: nothing that can throw or touches Python runs without the GIL.
template <typename... P, typename... A>
void call(const char* name, int (*fn)(P...), A... args) {
    int status;
    {
        const ReleasedGil released;
        status = fn(static_cast<P>(args)...);
    }
    if (status != EL_OK) {
        PyObject* r = PyObject_CallFunction(g_check, "si", name, status);
        Py_XDECREF(r);
        if (r != nullptr) PyErr_SetString(PyExc_RuntimeError, name);
        throw PyError();
    }
}

PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* none() { Py_RETURN_NONE; }

template <typename... A>
PyObject* tuple_of(A... items) {
    PyObject* objs[] = {items...};
    PyObject* t = PyTuple_New(sizeof...(items));
    for (size_t i = 0; i < sizeof...(items); ++i) {
        if (objs[i] == nullptr) { Py_XDECREF(t); throw PyError(); }
        PyTuple_SET_ITEM(t, (Py_ssize_t)i, objs[i]);
    }
    return t;
}

// The status word of x's device: the one tensor that the Python function hands to every caller, kept here for the life of the
// process (the reference is never given back, so the address stays good whatever becomes of the Python module's dict).
int32_t* status_word(const Tensor& x) {
    static int32_t* words[64] = {};
    const int dev = x.device().index();
    if (dev < 0 || dev >= 64) raise("device index out of range");
    if (words[dev] == nullptr) {
        PyObject* d = PyObject_CallFunction(g_status_of, "N", THPDevice_New(x.device()));
        if (d == nullptr) throw PyError();
        int32_t* word = THPVariable_Unpack(d).data_ptr<int32_t>();
        if (words[dev] == nullptr) words[dev] = word;       // another thread may have come first; it holds the same tensor
    }
    return words[dev];
}
void maybe_check(const Tensor& x) {
    const char* v = std::getenv("ELLECI_CHECK_STATUS");
    if (v == nullptr || v[0] != '1' || v[1] != 0) return;
    PyObject* r = PyObject_CallFunction(g_check_status, "N", THPDevice_New(x.device()));
    if (r == nullptr) throw PyError();
    Py_DECREF(r);
}

// A 2-D view whose rows are contiguous is read in place (a column window of a wider matrix qualifies); anything else is made
// contiguous and its leading dimensions flattened.
struct Rows {
    Tensor t;
    int64_t M, cols, ld;
};
Rows rows_view(const Tensor& t) {
    if (t.dim() == 2 && t.stride(1) == 1 && t.stride(0) >= t.size(1)) return {t, t.size(0), t.size(1), t.stride(0)};
    Tensor c = t.contiguous();
    int64_t M = 1;
    for (int64_t i = 0; i + 1 < c.dim(); ++i) M *= c.size(i);
    const int64_t cols = c.size(-1);
    return {c, M, cols, cols};
}
Tensor like_rows(const Tensor& x, int64_t cols, at::ScalarType dt) {      // x's leading dimensions, `cols` columns
    auto sizes = x.sizes().vec();
    sizes.back() = cols;
    return at::empty(sizes, x.options().dtype(dt).requires_grad(false).memory_format(at::MemoryFormat::Contiguous));
}
Tensor new_empty(const Tensor& x, at::IntArrayRef sizes, at::ScalarType dt) {
    return at::empty(sizes, at::TensorOptions().device(x.device()).dtype(dt));
}

// ---- quantisers ---------------------------------------------------------------------------------------------------------
PyObject* quantize_rows(PyObject* const* a) {
    const Tensor& x = cuda_arg(a[0], "x");
    EL_REQUIRE(float_type(x.scalar_type()), "x must be float16, bfloat16 or float32");
    const float eps = (float)float_arg(a[1]);
    const Rows v = rows_view(x);
    const void* xp = ptr(v.t);
    Tensor q, amax, fold_max, fold;
    if (is_none(a[4])) {
        q = like_rows(x, v.cols, at::kChar);
    } else {
        const Tensor& out = tensor_arg(a[4], "out");
        EL_REQUIRE(out.is_cuda() && out.scalar_type() == at::kChar && out.is_contiguous() && out.numel() == v.M * v.cols,
                   "out must be a contiguous int8 CUDA tensor of M*K elements");
        q = out;
    }
    int mode = EL_QUANT_FULL;
    if (is_none(a[3])) {
        amax = new_empty(x, {v.M}, at::kFloat);
    } else {
        amax = tensor_arg(a[3], "raw_absmax");
        EL_REQUIRE(amax.scalar_type() == at::kFloat && amax.numel() == v.M && amax.is_contiguous(), "raw_absmax must be a contiguous float32 [M]");
        mode = EL_QUANT_WITH_ABSMAX;
    }
    if (!is_none(a[2])) {
        fold = tensor_arg(a[2], "fold_absmax");
        EL_REQUIRE(fold.scalar_type() == at::kFloat && fold.numel() == v.M, "fold_absmax must be float32 [M]");
        fold_max = new_empty(x, {1}, at::kFloat);
        call("el_zero", g_lib.el_zero, ptr(fold_max), sizeof(float), stream());
    }
    call("el_quantize_rows", g_lib.el_quantize_rows, xp, code_of(x.scalar_type()), v.ld, ptr<int8_t>(q), ptr<float>(amax), v.M, v.cols, eps,
         mode, ptr<float>(fold), ptr<float>(fold_max), stream());
    if (fold.defined()) return tuple_of(wrap(q), wrap(amax), wrap(fold_max));
    return tuple_of(wrap(q), wrap(amax));
}

PyObject* quantize_grad(PyObject* const* a) {
    const Tensor& dY = cuda_arg(a[0], "dY");
    const Rows v = rows_view(dY);
    const Tensor &xa = tensor_arg(a[1], "x_absmax"), &ga = tensor_arg(a[2], "g_absmax");
    EL_REQUIRE(xa.scalar_type() == at::kFloat && xa.numel() == v.M, "x_absmax must be float32 [M]");
    EL_REQUIRE(ga.scalar_type() == at::kFloat && ga.numel() == 1, "g_absmax must be float32 [1]");
    const int dt = code_of(dY.scalar_type());
    const void* yp = ptr(v.t);
    const float *xap = ptr<float>(xa), *gap = ptr<float>(ga);
    Tensor Gq = like_rows(dY, v.cols, at::kChar);
    call("el_quantize_grad", g_lib.el_quantize_grad, yp, dt, v.ld, xap, gap, ptr<int8_t>(Gq), v.M, v.cols, stream());
    return wrap(Gq);
}

PyObject* quantize_tensor(PyObject* const* a) {
    const Tensor& in = cuda_arg(a[0], "Input");
    cuda_arg(a[1], "d_global_max");
    EL_REQUIRE(float_type(in.scalar_type()), "Input must be float16");
    Tensor x = in.contiguous();
    const void* xp = ptr(x);
    Tensor out = new_empty(x, x.sizes(), at::kChar), scale = new_empty(x, {1}, at::kFloat);
    call("el_quantize_tensor", g_lib.el_quantize_tensor, xp, code_of(x.scalar_type()), ptr<int8_t>(out), ptr<float>(scale), x.numel(), stream());
    return tuple_of(wrap(out), wrap(scale));
}

// ---- norm and gate ------------------------------------------------------------------------------------------------------
PyObject* rmsnorm_quantize_rows(PyObject* const* a) {
    const Tensor &x = cuda_arg(a[0], "x"), &w = cuda_arg(a[1], "weight");
    const float neps = (float)float_arg(a[2]), qeps = (float)float_arg(a[3]);
    EL_REQUIRE(float_type(x.scalar_type()), "x must be float16, bfloat16 or float32");
    const Rows v = rows_view(x);
    EL_REQUIRE(w.scalar_type() == at::kFloat && w.numel() == v.cols && w.is_contiguous(), "weight must be a contiguous float32 [K]");
    const void* xp = ptr(v.t);
    const float* wp = ptr<float>(w);
    Tensor q = like_rows(x, v.cols, at::kChar), amax = new_empty(x, {v.M}, at::kFloat), rstd = new_empty(x, {v.M}, at::kFloat);
    call("el_rmsnorm_quantize_rows", g_lib.el_rmsnorm_quantize_rows, xp, code_of(x.scalar_type()), v.ld, wp, neps, ptr<int8_t>(q), ptr<float>(amax),
         ptr<float>(rstd), v.M, v.cols, qeps, stream());
    return tuple_of(wrap(q), wrap(amax), wrap(rstd));
}

PyObject* rmsnorm_backward(PyObject* const* a) {
    const Tensor &g = cuda_arg(a[0], "g"), &x = cuda_arg(a[1], "x");
    const Tensor &w = tensor_arg(a[2], "weight"), &rstd = tensor_arg(a[3], "rstd");
    EL_REQUIRE(g.scalar_type() == x.scalar_type() && g.sizes() == x.sizes(), "g and x must have the same shape and dtype");
    const int64_t K = x.size(-1);
    Tensor gc = g.contiguous(), xc = x.contiguous();
    const int64_t M = K ? xc.numel() / K : 0;
    EL_REQUIRE(w.scalar_type() == at::kFloat && w.numel() == K, "weight must be float32 [K]");
    EL_REQUIRE(rstd.scalar_type() == at::kFloat && rstd.numel() == M, "rstd must be float32 [M]");
    const int dt = code_of(xc.scalar_type());
    Tensor wc = w.contiguous();
    const void *gp = ptr(gc), *xp = ptr(xc);
    const float *wp = ptr<float>(wc), *rp = ptr<float>(rstd);
    const size_t need = g_lib.el_rmsnorm_backward_workspace_bytes((int)K);
    Tensor ws = new_empty(x, {(int64_t)need}, at::kByte);
    Tensor dx = new_empty(x, xc.sizes(), xc.scalar_type()), dw = new_empty(x, {K}, at::kFloat);
    call("el_rmsnorm_backward", g_lib.el_rmsnorm_backward, gp, xp, dt, wp, rp, ptr(dx), ptr<float>(dw), ptr(ws), need, M, K, stream());
    return tuple_of(wrap(dx), wrap(dw));
}

// 2-D views of gate and up with one common row pitch (the two halves of a [M, 2H] matrix qualify)
void gate_up(const Tensor& gate, const Tensor& up, Rows& g, Rows& u) {
    EL_REQUIRE(gate.scalar_type() == up.scalar_type() && gate.sizes() == up.sizes(), "gate and up must have the same shape and dtype");
    EL_REQUIRE(float_type(gate.scalar_type()), "gate and up must be float16, bfloat16 or float32");
    g = rows_view(gate);
    u = rows_view(up);
    if (u.ld != g.ld) {
        g.t = g.t.contiguous();
        u.t = u.t.contiguous();
        g.ld = u.ld = g.cols;
    }
}

PyObject* swiglu_quantize_rows(PyObject* const* a) {
    const Tensor &gate = cuda_arg(a[0], "gate"), &up = cuda_arg(a[1], "up");
    const float neps = (float)float_arg(a[3]), qeps = (float)float_arg(a[4]);
    Rows g, u;
    gate_up(gate, up, g, u);
    Tensor w, rstd;
    if (!is_none(a[2])) {
        w = tensor_arg(a[2], "norm_weight");
        EL_REQUIRE(w.scalar_type() == at::kFloat && w.numel() == g.cols && w.is_contiguous(), "norm_weight must be a contiguous float32 [H]");
    }
    const void *gp = ptr(g.t), *up_p = ptr(u.t);
    const float* wp = ptr<float>(w);
    if (w.defined()) rstd = new_empty(gate, {g.M}, at::kFloat);
    Tensor q = like_rows(gate, g.cols, at::kChar), amax = new_empty(gate, {g.M}, at::kFloat);
    call("el_swiglu_quantize_rows", g_lib.el_swiglu_quantize_rows, gp, up_p, code_of(gate.scalar_type()), g.ld, wp, neps, ptr<int8_t>(q),
         ptr<float>(amax), ptr<float>(rstd), g.M, g.cols, qeps, stream());
    return tuple_of(wrap(q), wrap(amax), w.defined() ? wrap(rstd) : none());
}

PyObject* swiglu_backward(PyObject* const* a) {
    const Tensor &gy = cuda_arg(a[0], "gy"), &gate = cuda_arg(a[1], "gate"), &up = cuda_arg(a[2], "up");
    Rows g, u;
    gate_up(gate, up, g, u);
    const int64_t M = g.M, H = g.cols;
    EL_REQUIRE(gy.scalar_type() == gate.scalar_type() && gy.numel() == M * H, "gy must have the shape and dtype of gate");
    Tensor gyc = gy.contiguous(), dg, du, dw, ws, w, rstd;
    const void *yp = ptr(gyc), *gp = ptr(g.t), *up_p = ptr(u.t);
    int64_t ld_d = H;
    const bool own = is_none(a[5]);
    if (own) {
        dg = new_empty(gate, gate.sizes(), gate.scalar_type());
        du = new_empty(gate, gate.sizes(), gate.scalar_type());
    } else {
        const Tensor& out = tensor_arg(a[5], "out");
        EL_REQUIRE(out.scalar_type() == gate.scalar_type() && out.dim() == 2 && out.size(0) == M && out.size(1) == 2 * H && out.is_contiguous(),
                   "out must be a contiguous [M, 2H] tensor");
        dg = out.narrow(1, 0, H);
        du = out.narrow(1, H, H);
        ld_d = 2 * H;
    }
    size_t need = 0;
    if (!is_none(a[3])) {
        w = tensor_arg(a[3], "norm_weight");
        EL_REQUIRE(w.scalar_type() == at::kFloat && w.numel() == H, "norm_weight must be float32 [H]");
        EL_REQUIRE(!is_none(a[4]), "rstd must be float32 [M]");
        rstd = tensor_arg(a[4], "rstd");
        EL_REQUIRE(rstd.scalar_type() == at::kFloat && rstd.numel() == M, "rstd must be float32 [M]");
        need = g_lib.el_swiglu_backward_workspace_bytes((int)H);
        ws = new_empty(gate, {(int64_t)need}, at::kByte);
        dw = new_empty(gate, {H}, at::kFloat);
        w = w.contiguous();
    }
    const bool norm = w.defined();
    if (!norm && !is_none(a[4])) rstd = tensor_arg(a[4], "rstd");
    call("el_swiglu_backward", g_lib.el_swiglu_backward, yp, gp, up_p, code_of(gate.scalar_type()), g.ld, ptr<float>(w), ptr<float>(rstd), ptr(dg),
         ptr(du), ld_d, ptr<float>(dw), ptr(ws), need, M, H, stream());
    return tuple_of(wrap(dg), wrap(du), norm ? wrap(dw) : none());
}

PyObject* prelinear_rows(PyObject* const* a) {
    const Tensor& x = cuda_arg(a[0], "x");
    const float neps = (float)float_arg(a[3]);
    Rows v, u;
    const bool gated = !is_none(a[1]);
    if (gated) {
        gate_up(x, cuda_arg(a[1], "up"), v, u);
    } else {
        EL_REQUIRE(float_type(x.scalar_type()), "x must be float16, bfloat16 or float32");
        v = rows_view(x);
    }
    Tensor w;
    if (!is_none(a[2])) {
        w = tensor_arg(a[2], "norm_weight");
        EL_REQUIRE(w.scalar_type() == at::kFloat && w.numel() == v.cols && w.is_contiguous(), "norm_weight must be a contiguous float32 [K]");
    }
    const void *xp = ptr(v.t), *up_p = ptr(u.t);
    const float* wp = ptr<float>(w);
    Tensor y = like_rows(x, v.cols, x.scalar_type());
    call("el_prelinear_rows", g_lib.el_prelinear_rows, xp, up_p, code_of(x.scalar_type()), v.ld, wp, neps, ptr(y), v.M, v.cols, stream());
    return wrap(y);
}

// ---- GEMMs --------------------------------------------------------------------------------------------------------------
// Scratch of a GEMM that splits its reduction over idle CTA pairs (few output tiles): the caching allocator hands it out in
// stream order.
Tensor gemm_scratch(const Tensor& x, int mode, int64_t M, int64_t N, int64_t K, int path) {
    const int p = path & ~EL_FLAG_LEAN;
    if (p != EL_PATH_AUTO && p != EL_PATH_TC) return Tensor();
    const size_t need = g_lib.el_gemm_workspace_bytes(mode, (int)M, (int)N, (int)K);
    return need ? new_empty(x, {(int64_t)need}, at::kByte) : Tensor();
}

PyObject* gemm_fwd(PyObject* const* a) {
    const Tensor &Xq = cuda_arg(a[0], "X_int8"), &W = cuda_arg(a[1], "W_packed"), &amax = cuda_arg(a[2], "d_scale_x");
    const int stride = (int)int_arg(a[3]), path = (int)int_arg(a[6]);
    const float gamma = (float)float_arg(a[4]);
    const at::ScalarType out_dt = dtype_arg(a[5]);
    EL_REQUIRE(Xq.scalar_type() == at::kChar, "X_int8 must be int8");
    EL_REQUIRE(W.scalar_type() == at::kByte, "W_packed must be uint8");
    EL_REQUIRE(amax.scalar_type() == at::kFloat, "d_scale_x must be float32");
    EL_REQUIRE(W.dim() == 2, "W_packed must be 2-D [N, ceil(K/4)]");
    const int64_t N = W.size(0), pK = W.size(1), K = Xq.size(-1);
    if ((K + 3) / 4 != pK)
        raise("Dimension mismatch: X has " + std::to_string(K) + " features but W_packed has packed_K=" + std::to_string(pK) +
              " (expected ceil(K/4)=" + std::to_string((K + 3) / 4) + ")");
    Tensor Xf = Xq.contiguous(), Wc = W.contiguous();
    const int64_t M = K ? Xf.numel() / K : Xf.reshape({-1, K}).size(0);
    EL_REQUIRE(stride == 0 || amax.numel() == M, "one absmax per token expected");
    const int dt = code_of(out_dt);
    const int8_t* xp = ptr<int8_t>(Xf);
    const uint8_t* wp = ptr<uint8_t>(Wc);
    const float* ap = ptr<float>(amax);
    Tensor Y = like_rows(Xq, N, out_dt), ws = gemm_scratch(Xq, 0, M, N, K, path);
    call("el_gemm_fwd_ws", g_lib.el_gemm_fwd_ws, xp, wp, ptr(Y), dt, ap, stride, gamma, M, N, K, path, ptr(ws), ws.defined() ? ws.numel() : 0,
         status_word(Xq), stream());
    maybe_check(Xq);
    return wrap(Y);
}

PyObject* gemm_dx(PyObject* const* a) {
    const Tensor &dYq = cuda_arg(a[0], "dY_int8"), &W = cuda_arg(a[1], "W_packed"), &amax = cuda_arg(a[2], "d_scale_dy");
    const int stride = (int)int_arg(a[3]), path = (int)int_arg(a[7]);
    const float gamma = (float)float_arg(a[4]);
    const int64_t K = int_arg(a[5]);
    const at::ScalarType out_dt = dtype_arg(a[6]);
    EL_REQUIRE(dYq.scalar_type() == at::kChar, "dY_int8 must be int8");
    EL_REQUIRE(W.scalar_type() == at::kByte, "W_packed must be uint8");
    EL_REQUIRE(amax.scalar_type() == at::kFloat, "d_scale_dy must be float32");
    if (W.dim() != 2) {
        PyErr_SetString(PyExc_ValueError, "W_packed must be 2-D [N, ceil(K/4)]");
        throw PyError();
    }
    const int64_t N = W.size(0), pK = W.size(1);
    if (dYq.size(-1) != N) raise("dY has " + std::to_string(dYq.size(-1)) + " features but W_packed has " + std::to_string(N) + " rows");
    if ((K + 3) / 4 != pK) raise("K=" + std::to_string(K) + " does not match W_packed's packed_K=" + std::to_string(pK));
    Tensor Yf = dYq.contiguous(), Wc = W.contiguous();
    const int64_t M = N ? Yf.numel() / N : Yf.reshape({-1, N}).size(0);
    EL_REQUIRE(stride == 0 || amax.numel() == M, "one absmax per token expected");
    const int dt = code_of(out_dt);
    const int8_t* yp = ptr<int8_t>(Yf);
    const uint8_t* wp = ptr<uint8_t>(Wc);
    const float* ap = ptr<float>(amax);
    Tensor dX = like_rows(dYq, K, out_dt), ws = gemm_scratch(dYq, 1, M, N, K, path);
    call("el_gemm_dx_ws", g_lib.el_gemm_dx_ws, yp, wp, ptr(dX), dt, ap, stride, gamma, M, N, K, path, ptr(ws), ws.defined() ? ws.numel() : 0,
         status_word(dYq), stream());
    maybe_check(dYq);
    return wrap(dX);
}

PyObject* dw_hysteresis(PyObject* const* a) {
    const Tensor &Gq = cuda_arg(a[0], "Gq"), &Xq = cuda_arg(a[1], "Xq");
    EL_REQUIRE(Gq.scalar_type() == at::kChar && Xq.scalar_type() == at::kChar, "Gq and Xq must be int8");
    const Tensor &ga = tensor_arg(a[2], "g_absmax"), &W = tensor_arg(a[3], "W_packed"), &H = tensor_arg(a[4], "H_packed");
    const int64_t N = Gq.size(-1), K = Xq.size(-1);
    Tensor G2 = Gq.contiguous(), X2 = Xq.contiguous();
    const int64_t M = N ? G2.numel() / N : 0;
    EL_REQUIRE((K ? X2.numel() / K : 0) == M, "Gq and Xq must have the same number of tokens");
    EL_REQUIRE(W.dim() == 2 && W.size(0) == N && W.size(1) == (K + 3) / 4 && H.dim() == 2 && H.size(0) == N && H.size(1) == (K + 1) / 2,
               "W_packed / H_packed shape mismatch");
    EL_REQUIRE(W.is_contiguous() && H.is_contiguous(), "W_packed/H_packed must be contiguous");
    const float lr = (float)float_arg(a[5]), lr_scale = (float)float_arg(a[6]), decay = (float)float_arg(a[8]);
    const int threshold = (int)int_arg(a[7]);
    const int step = (int)(uint32_t)int_arg(a[9]);
    const uint32_t idx_base = (uint32_t)int_arg(a[10]);
    const int8_t *gp = ptr<int8_t>(G2), *xp = ptr<int8_t>(X2);
    const float* gap = ptr<float>(ga);
    uint8_t *wp = ptr<uint8_t>(W), *hp = ptr<uint8_t>(H);
    call("el_dw_hysteresis", g_lib.el_dw_hysteresis, gp, xp, gap, wp, hp, lr, lr_scale, threshold, decay, step, idx_base, M, N, K, status_word(Gq),
         stream());
    maybe_check(Gq);
    return none();
}

// The weight update of a layer's step in one call: quantise_rows with the fold, quantise_grad and the fused weight gradient and
// hysteresis update (or, for widths that it does not take, weight gradient and update as two calls), with the conversions and
// checks that the layer made around them.  Host time of the update, separate calls -> this one: 34 -> 17 us (1024 tokens, 1536 -> 1536),
// 68 -> 20 us where the fused kernel does not fit (2048 tokens, 16 -> 8192); of the whole step 152 -> 120 and 229 -> 154 us, in both the
// attribute writes that went through nn.Module among it.
// weight_update(dY, x_absmax, Xq, W_packed, H_packed, half, lr, lr_scale, threshold, decay, step, idx_base, g_absmax) -> (dYq, its row
// maxima), or None where the caller has the folded maximum already (g_absmax): quantise_rows is then left out.
// dY is any shape of M*N elements when `half`; else its last dimension has to be N, as the dX GEMM takes dYq in dY's shape.
PyObject* weight_update(PyObject* const* a) {
    const Tensor& dY = cuda_arg(a[0], "dY");
    const Tensor &ax = tensor_arg(a[1], "x_absmax"), &Xq = cuda_arg(a[2], "Xq");
    const Tensor &W = tensor_arg(a[3], "W_packed"), &H = tensor_arg(a[4], "H_packed");
    const bool half = PyObject_IsTrue(a[5]) == 1;
    const float lr = (float)float_arg(a[6]), lr_scale = (float)float_arg(a[7]), decay = (float)float_arg(a[9]);
    const int threshold = (int)int_arg(a[8]);
    const int step = (int)(uint32_t)int_arg(a[10]);
    const uint32_t idx_base = (uint32_t)int_arg(a[11]);
    EL_REQUIRE(Xq.scalar_type() == at::kChar, "Gq and Xq must be int8");
    EL_REQUIRE(W.dim() == 2, "W_packed / H_packed shape mismatch");
    const int64_t N = W.size(0), K = Xq.size(-1);
    // the gradient as float rows: the caller's own tensor where it is one already
    Tensor d = dY.dim() == 2 && dY.size(1) == N ? dY : dY.reshape({-1, N});
    if (!float_type(d.scalar_type())) d = d.to(at::kFloat);
    if (half && d.scalar_type() != at::kHalf) d = d.to(at::kHalf);
    d = d.contiguous();
    const int64_t M = d.size(0);
    // dYq has dY's leading dimensions where these count the M rows, and [M, N] where not
    auto q_sizes = dY.sizes().vec();
    if (q_sizes.empty()) q_sizes.push_back(N);
    q_sizes.back() = N;
    int64_t q_rows = 1;
    for (size_t i = 0; i + 1 < q_sizes.size(); ++i) q_rows *= q_sizes[i];
    if (q_rows != M) {
        EL_REQUIRE(half, "dY's last dimension must be the number of rows of W_packed");
        q_sizes = {M, N};
    }
    Tensor X2 = Xq.contiguous();
    EL_REQUIRE((K ? X2.numel() / K : 0) == M, "Gq and Xq must have the same number of tokens");
    EL_REQUIRE(W.size(1) == (K + 3) / 4 && H.dim() == 2 && H.size(0) == N && H.size(1) == (K + 1) / 2, "W_packed / H_packed shape mismatch");
    EL_REQUIRE(W.is_contiguous() && H.is_contiguous(), "W_packed/H_packed must be contiguous");
    EL_REQUIRE(W.is_cuda() && H.is_cuda() && W.scalar_type() == at::kByte && H.scalar_type() == at::kByte, "W_packed/H_packed must be uint8");
    EL_REQUIRE(ax.scalar_type() == at::kFloat && (ax.numel() == M || ax.numel() == 1), "fold_absmax must be float32 [M]");
    Tensor rows = ax.numel() == M ? ax.contiguous() : ax.expand({M}).contiguous();
    const bool fused = N % 16 == 0 && K % 32 == 0;
    const int dt = code_of(d.scalar_type());
    const void* dp = ptr(d);
    const int8_t* xp = ptr<int8_t>(X2);
    const float* ap = ptr<float>(rows);
    uint8_t *wp = ptr<uint8_t>(W), *hp = ptr<uint8_t>(H);
    Tensor dYq, ady, folded;
    if (!is_none(a[12])) {
        folded = cuda_arg(a[12], "g_absmax");
        EL_REQUIRE(folded.scalar_type() == at::kFloat && folded.numel() == 1, "g_absmax must be float32 [1]");
    } else {
        dYq = new_empty(d, q_sizes, at::kChar);
        ady = new_empty(d, {M}, at::kFloat);
    }
    // dYq and its maxima go back to the caller (the dX GEMM reads them); the folded gradient, its maximum and, unfused, the weight
    // gradient are this call's own, in one block, each on a 256-byte boundary
    const int64_t g_bytes = (M * N + 255) & ~(int64_t)255;
    Tensor own = new_empty(d, {256 + g_bytes + (fused ? 0 : N * K * 4)}, at::kByte);
    float* gmax = folded.defined() ? ptr<float>(folded) : ptr<float>(own);
    int8_t* gq = ptr<int8_t>(own) + 256;
    float* dw = reinterpret_cast<float*>(gq + g_bytes);
    int32_t* word = status_word(d);
    void* st = stream();
    if (!folded.defined()) {
        call("el_zero", g_lib.el_zero, gmax, sizeof(float), st);
        call("el_quantize_rows", g_lib.el_quantize_rows, dp, dt, N, ptr<int8_t>(dYq), ptr<float>(ady), M, N, 1e-30f, EL_QUANT_FULL, ap, gmax, st);
    }
    call("el_quantize_grad", g_lib.el_quantize_grad, dp, dt, N, ap, gmax, gq, M, N, st);
    if (fused) {
        call("el_dw_hysteresis", g_lib.el_dw_hysteresis, gq, xp, gmax, wp, hp, lr, lr_scale, threshold, decay, step, idx_base, M, N, K, word, st);
    } else {
        call("el_gemm_dw", g_lib.el_gemm_dw, gq, xp, dw, EL_F32, gmax, M, N, K, EL_PATH_AUTO, word, st);
        call("el_hysteresis_from_dw", g_lib.el_hysteresis_from_dw, dw, wp, hp, lr, lr_scale, threshold, decay, step, N, K, idx_base, 1, st);
    }
    maybe_check(d);
    if (folded.defined()) return none();
    return tuple_of(wrap(dYq), wrap(ady));
}

// ---- decode -------------------------------------------------------------------------------------------------------------
// linear_decode(x, W_packed, gamma, out_dtype, workspace, up, norm_weight, norm_eps)
PyObject* linear_decode(PyObject* const* a) {
    const Tensor &x = cuda_arg(a[0], "x"), &W = cuda_arg(a[1], "W_packed");
    const float gamma = (float)float_arg(a[2]), neps = (float)float_arg(a[7]);
    EL_REQUIRE(float_type(x.scalar_type()), "x must be float16, bfloat16 or float32");
    EL_REQUIRE(W.scalar_type() == at::kByte && W.dim() == 2, "W_packed must be uint8 [N, ceil(K/4)]");
    const int64_t N = W.size(0), pK = W.size(1), K = x.size(-1);
    if ((K + 3) / 4 != pK) raise("x has " + std::to_string(K) + " features but W_packed has packed_K=" + std::to_string(pK));
    const bool gated = !is_none(a[5]), normed = !is_none(a[6]);
    Rows v, u;
    Tensor w;
    if (gated) {
        gate_up(x, cuda_arg(a[5], "up"), v, u);
    } else if (normed) {
        v = rows_view(x);
    } else {
        Tensor xc = x.contiguous();
        v = {xc, K ? xc.numel() / K : 0, K, K};
    }
    if (normed) {
        w = tensor_arg(a[6], "norm_weight");
        EL_REQUIRE(w.scalar_type() == at::kFloat && w.numel() == K && w.is_contiguous(), "norm_weight must be a contiguous float32 [K]");
    }
    const int64_t M = v.M;
    Tensor Wc = W.contiguous();
    EL_REQUIRE(M >= 1 && M <= 64, "linear_decode takes 1..64 tokens; use quantize_rows + matmul_rows beyond that");
    const at::ScalarType out_dt = is_none(a[3]) ? x.scalar_type() : dtype_arg(a[3]);
    const int dt = code_of(out_dt);
    const void *xp = ptr(v.t), *up_p = ptr(u.t);
    const float* nwp = ptr<float>(w);
    const uint8_t* wp = ptr<uint8_t>(Wc);
    void* st = stream();
    Tensor ws;                      // the kernels need none; what a caller passes has to be large enough all the same
    size_t have = 0;
    if (!is_none(a[4])) {
        ws = tensor_arg(a[4], "workspace");
        have = (size_t)ws.numel() * ws.element_size();
        EL_REQUIRE(ws.is_cuda() && have >= g_lib.el_decode_workspace_bytes((int)N), "workspace too small");
    }
    // one allocation for the quantised tokens and, on a 16-byte boundary behind them, their maxima
    const int64_t xq_bytes = (M * K + 15) & ~(int64_t)15;
    Tensor scratch = new_empty(x, {xq_bytes + M * 4}, at::kByte), Y = like_rows(x, N, out_dt);
    int8_t* xq = ptr<int8_t>(scratch);
    float* amax = reinterpret_cast<float*>(xq + xq_bytes);
    int32_t* word = status_word(x);
    if (gated || normed)
        call("el_prelinear_decode", g_lib.el_prelinear_decode, xp, up_p, code_of(x.scalar_type()), v.ld, nwp, neps, wp, ptr(Y), dt, gamma, xq, amax,
             ptr(ws), have, M, N, K, word, st);
    else
        call("el_linear_decode", g_lib.el_linear_decode, xp, code_of(x.scalar_type()), wp, ptr(Y), dt, gamma, xq, amax, ptr(ws), have, M, N, K, word, st);
    maybe_check(x);
    return wrap(Y);
}

// ---- module -------------------------------------------------------------------------------------------------------------
template <PyObject* (*F)(PyObject* const*), int NARGS>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != NARGS) {
        PyErr_Format(PyExc_TypeError, "expected %d positional arguments, got %d", NARGS, (int)n);
        return nullptr;
    }
    try {
        return F(args);
    } catch (const PyError&) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// set_hooks(check, device_status, check_device_status, path of the loaded library)
PyObject* set_hooks(PyObject* const* a) {
    const char* path = PyUnicode_AsUTF8(a[3]);
    if (path == nullptr) throw PyError();
    void* handle = dlopen(path, RTLD_NOW | RTLD_NOLOAD);
    EL_REQUIRE(handle != nullptr, "the library is not loaded");
    bool all = true;
#define X(name) all = (g_lib.name = reinterpret_cast<decltype(&::name)>(dlsym(handle, #name))) != nullptr && all;
    EL_FUNCTIONS(X)
#undef X
    EL_REQUIRE(all, "the library lacks an entry point");
    PyObject** dst[] = {&g_check, &g_status_of, &g_check_status};
    for (int i = 0; i < 3; ++i) {
        Py_INCREF(a[i]);
        Py_XSETREF(*dst[i], a[i]);
    }
    return none();
}

#define EL_ENTRY(name, n) {#name, (PyCFunction)(void (*)(void))entry<name, n>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    EL_ENTRY(quantize_rows, 5), EL_ENTRY(quantize_grad, 3), EL_ENTRY(quantize_tensor, 2), EL_ENTRY(rmsnorm_quantize_rows, 4),
    EL_ENTRY(rmsnorm_backward, 4), EL_ENTRY(swiglu_quantize_rows, 5), EL_ENTRY(swiglu_backward, 6), EL_ENTRY(prelinear_rows, 4),
    EL_ENTRY(gemm_fwd, 7), EL_ENTRY(gemm_dx, 8), EL_ENTRY(dw_hysteresis, 11), EL_ENTRY(weight_update, 13), EL_ENTRY(linear_decode, 8), EL_ENTRY(set_hooks, 4),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "elleci_host_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_elleci_host_ops(void) { return PyModule_Create(&module_def); }
