// Native call path of the torch operator: what a call of RWKVKernelOperator / wkv6() does between Python and the C ABI
// (include/wkv6_b200.h), as one C++ function per call.
//
// Small calls are bound by the host, not by the GPU: one decode step is 2.5 us of kernel, the parity-size training call
// 90 us, and the same steps in Python (argument checks, a ctypes struct, tensor allocation through the dispatcher, a
// Python autograd node with zero-filled gradients for the checkpoint buffer) took 27 us and 300 us.  Every function
// here returns None when the call is not the plain one it handles - other tensor types, a tracing or dispatch mode,
// layouts or arguments that need a conversion or an error message - and the Python path then runs instead.
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/grad_mode.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/Exceptions.h>
#include <ATen/ATen.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>

#include "../../include/wkv6_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// The library is the one the Python side loaded (WKV6_B200_LIB may select another build of it).
struct Api {
    decltype(&::wkv6_forward) forward = nullptr;
    decltype(&::wkv6_backward) backward = nullptr;
    decltype(&::wkv6_decode) decode = nullptr;
    decltype(&::wkv6_ckpt_bytes) ckpt_bytes = nullptr;
    decltype(&::wkv6_backward_workspace_bytes) backward_workspace_bytes = nullptr;
    decltype(&::wkv6_sum_rows) sum_rows = nullptr;
    decltype(&::wkv6_split_segments) split_segments = nullptr;
    decltype(&::wkv6_split_state_bytes) split_state_bytes = nullptr;
    decltype(&::wkv6_split_workspace_bytes) split_workspace_bytes = nullptr;
    decltype(&::wkv6_forward_split) forward_split = nullptr;
    decltype(&::wkv6_backward_split) backward_split = nullptr;
    decltype(&::wkv6_resolve_variant) resolve_variant = nullptr;
    decltype(&::wkv6_last_error) last_error = nullptr;
    bool bound = false;
} api;

int dtype_code(at::ScalarType t) {
    switch (t) {
        case at::kBFloat16: return WKV6_BF16;
        case at::kHalf: return WKV6_F16;
        case at::kFloat: return WKV6_F32;
        default: return -1;
    }
}

// fp16 inputs give fp32 outputs and gradients, as in the reference operator
at::ScalarType result_type(at::ScalarType x) { return x == at::kHalf ? at::kFloat : x; }

bool plain_mode() {
    return api.bound && !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::impl::torch_function_mode_enabled() &&
           !torch::jit::tracer::isTracing();
}

// A strided CUDA tensor that is what its memory holds: not wrapped by a transform, no lazy negation.
bool plain_storage(const Tensor &t) {
    constexpr c10::DispatchKeySet odd({c10::DispatchKey::Python, c10::DispatchKey::Batched, c10::DispatchKey::FuncTorchBatched,
                                       c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize,
                                       c10::DispatchKey::Conjugate, c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
    return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.has_storage() && (t.key_set() & odd).empty();
}

// ... and of the exact class Tensor (or Parameter).
bool plain_tensor(PyObject *o) { return THPVariable_CheckExact(o) && plain_storage(THPVariable_Unpack(o)); }

struct Call {
    wkv6_problem p{};
    at::ScalarType xt{}, yt{};
    int64_t B = 0, T = 0, C = 0, H = 0;
    bool dense = false, chunked = false;
    int G = 1;               // segments the library cuts the sequences into
    int backward_G() const { return xt == at::kHalf ? 1 : G; }   // the backward of fp16 inputs is not split
};

// Fills the problem from the operator's five tensors; false when they are not what the native path handles.  cut: the
// library may cut the sequences into segments.
bool make_call(const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u, int64_t N, int64_t variant,
               bool cut, Call &c) {
    if (r.dim() != 3 || N <= 0) return false;
    c.B = r.size(0); c.T = r.size(1); c.C = r.size(2);
    if (c.B == 0 || c.T == 0 || c.C == 0 || c.C % N != 0) return false;
    c.H = c.C / N;
    c.xt = r.scalar_type();
    c.yt = result_type(c.xt);
    const auto dev = r.device();
    for (const Tensor *t : {&r, &k, &v, &w})
        if (reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 != 0) return false;
    for (const Tensor *t : {&k, &v, &w})
        if (t->scalar_type() != c.xt || t->device() != dev || t->sizes() != r.sizes() || t->strides() != r.strides()) return false;
    if (u.device() != dev || (u.scalar_type() != c.xt && u.scalar_type() != at::kFloat) || u.numel() != c.C || !u.is_contiguous())
        return false;
    if (dtype_code(c.xt) < 0 || r.stride(2) != 1) return false;
    // rows that overlap (broadcast inputs, windows): outputs have the inputs' strides, and the C ABI takes a stride of 0 for "dense"
    const int64_t ld = c.T > 1 ? r.stride(1) : c.C, bs = c.B > 1 ? r.stride(0) : c.T * ld;
    if (c.T > 1 && ld < c.C) return false;
    if (c.B > 1 && bs < (c.T - 1) * ld + c.C && (bs < c.C || (c.T > 1 && ld < (c.B - 1) * bs + c.C))) return false;
    c.dense = r.is_contiguous();
    wkv6_problem &p = c.p;
    p.B = (int32_t)c.B; p.T = (int32_t)c.T; p.H = (int32_t)c.H; p.N = (int32_t)N;
    p.x_dtype = dtype_code(c.xt); p.y_dtype = dtype_code(c.yt); p.u_dtype = dtype_code(u.scalar_type());
    p.gu_dtype = WKV6_F32; p.s_dtype = WKV6_F32; p.variant = (int32_t)variant;
    p.row_stride = ld;
    p.batch_stride = bs;
    const int variant_of = api.resolve_variant(&p);
    if (variant_of < 0) return false;
    c.chunked = variant_of == WKV6_VARIANT_CHUNK;
    c.G = cut ? api.split_segments(&p) : 1;
    return true;
}

Tensor like(const Tensor &r, at::ScalarType t, bool dense) {   // one stride set serves inputs and outputs
    return dense ? at::detail::empty_cuda(r.sizes(), t, r.device(), std::nullopt)
                 : at::detail::empty_strided_cuda(r.sizes(), r.strides(), t, r.device());
}

Tensor bytes(size_t n, const Tensor &r) { return at::detail::empty_cuda({(int64_t)n}, at::kByte, r.device(), std::nullopt); }

void *stream_of(const Tensor &r) { return c10::cuda::getCurrentCUDAStream(r.device().index()).stream(); }

// The forward without a checkpoint, split where the library says so; `states` receives the segments' entering states.
int run_forward(const Call &c, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w, const Tensor &u, Tensor &y,
                const void *s_in, int32_t kinds, void *s_out, Tensor *states) {
    if (c.G == 1)
        return api.forward(&c.p, r.data_ptr(), k.data_ptr(), v.data_ptr(), w.data_ptr(), u.data_ptr(), y.data_ptr(), s_in, nullptr,
                           kinds, s_out, nullptr, stream_of(r));
    Tensor st;   // the chunked variant needs it for a backward only
    if (states || !c.chunked) st = bytes(api.split_state_bytes(&c.p), r);
    const size_t nws = api.split_workspace_bytes(&c.p, 0);
    Tensor ws = bytes(nws, r);
    if (states) *states = st;
    return api.forward_split(&c.p, r.data_ptr(), k.data_ptr(), v.data_ptr(), w.data_ptr(), u.data_ptr(), y.data_ptr(), s_in, nullptr,
                             kinds, s_out, st.defined() ? static_cast<float *>(st.data_ptr()) : nullptr, ws.data_ptr(), nws, stream_of(r));
}

void ok(int rc) { TORCH_CHECK(rc == 0, "wkv6_b200 error ", rc, ": ", api.last_error()); }

struct WKV6Function : public torch::autograd::Function<WKV6Function> {
    static Tensor forward(AutogradContext *ctx, const Tensor &r, const Tensor &k, const Tensor &v, const Tensor &w,
                          const Tensor &u, int64_t N, int64_t variant, bool cut) {
        Call c;
        TORCH_CHECK(make_call(r, k, v, w, u, N, variant, cut, c), "wkv6: unsupported call");   // checked by the caller
        Tensor y = like(r, c.yt, c.dense);
        // what the backward needs beside the inputs: the chunk checkpoints, or the segments' entering states
        Tensor kept;
        if (c.G > 1) {
            ok(run_forward(c, r, k, v, w, u, y, nullptr, 0, nullptr, &kept));
            if (c.backward_G() == 1) kept = bytes(0, r);
        } else {
            const size_t nckpt = api.ckpt_bytes(&c.p);
            kept = bytes(nckpt, r);
            ok(api.forward(&c.p, r.data_ptr(), k.data_ptr(), v.data_ptr(), w.data_ptr(), u.data_ptr(), y.data_ptr(), nullptr, nullptr,
                           0, nullptr, nckpt ? kept.data_ptr() : nullptr, stream_of(r)));
        }
        ctx->save_for_backward({r, k, v, w, u, kept});
        ctx->saved_data["N"] = N;
        ctx->saved_data["variant"] = variant;
        ctx->saved_data["cut"] = cut;
        return y;
    }

    // Gradients that are batched (is_grads_batched, vectorised Jacobians), lazily negated or of another class: the registered
    // operator, whose dispatch takes them apart.  The chunked variant's kept states are the checkpoints it expects; its sequential
    // variant expects none.
    static variable_list through_dispatcher(const Call &c, const variable_list &s, const Tensor &gy) {
        static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("wkv6_b200::backward", "").typed<std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>(
            const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &, const Tensor &, int64_t, int64_t)>();
        const Tensor &r = s[0], &u = s[4];
        auto [gr, gk, gv, gw, rows] = op.call(r, s[1], s[2], s[3], u, gy, c.chunked ? s[5] : bytes(0, r), c.p.N, c.p.variant);
        const auto xt = r.scalar_type();
        variable_list out{gr.to(xt), gk.to(xt), gv.to(xt), gw.to(xt), rows.sum(0).to(u.scalar_type()).reshape(u.sizes())};
        out.resize(8);
        return out;
    }

    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        variable_list s = ctx->get_saved_variables();
        const Tensor &r = s[0], &k = s[1], &v = s[2], &w = s[3], &u = s[4], &kept = s[5];
        const bool twice = at::GradMode::is_enabled();
        Tensor gr, gk, gv, gw, gu;
        {
            at::NoGradGuard no_grad;
            c10::cuda::CUDAGuard guard(r.device());
            Call c;
            TORCH_CHECK(make_call(r, k, v, w, u, ctx->saved_data["N"].toInt(), ctx->saved_data["variant"].toInt(),
                                  ctx->saved_data["cut"].toBool(), c),
                        "wkv6: unsupported call");
            Tensor gy = grads[0];
            if (!plain_storage(gy)) return through_dispatcher(c, s, gy);
            if (gy.strides() != r.strides() || reinterpret_cast<uintptr_t>(gy.data_ptr()) % 16 != 0)
                gy = like(r, c.yt, c.dense).copy_(gy);
            gr = like(r, c.yt, c.dense); gk = like(r, c.yt, c.dense);
            gv = like(r, c.yt, c.dense); gw = like(r, c.yt, c.dense);
            const int G = c.backward_G();
            const int64_t nrows = c.B * G;
            Tensor rows = at::detail::empty_cuda({nrows, c.C}, at::kFloat, r.device(), std::nullopt);
            const bool have = kept.numel() > 0;
            const size_t nws = G > 1 ? api.split_workspace_bytes(&c.p, 1) : api.backward_workspace_bytes(&c.p, have ? 1 : 0);
            Tensor ws;
            if (nws) ws = bytes(nws, r);
            void *pws = nws ? ws.data_ptr() : nullptr, *st = stream_of(r);
            if (G > 1)
                ok(api.backward_split(&c.p, r.data_ptr(), k.data_ptr(), v.data_ptr(), w.data_ptr(), u.data_ptr(), gy.data_ptr(),
                                      gr.data_ptr(), gk.data_ptr(), gv.data_ptr(), gw.data_ptr(), rows.data_ptr<float>(),
                                      static_cast<const float *>(kept.data_ptr()), pws, nws, st));
            else
                ok(api.backward(&c.p, r.data_ptr(), k.data_ptr(), v.data_ptr(), w.data_ptr(), u.data_ptr(), gy.data_ptr(), gr.data_ptr(),
                                gk.data_ptr(), gv.data_ptr(), gw.data_ptr(), rows.data_ptr(), have ? kept.data_ptr() : nullptr, pws,
                                nws, st));
            if (nrows == 1) {
                gu = rows;
            } else {
                gu = at::detail::empty_cuda({c.C}, at::kFloat, r.device(), std::nullopt);
                ok(api.sum_rows(rows.data_ptr<float>(), nrows, c.C, gu.data_ptr<float>(), st));
            }
            gu = gu.view(u.sizes());
            if (gu.scalar_type() != u.scalar_type()) gu = gu.to(u.scalar_type());
            if (c.yt != c.xt) { gr = gr.to(c.xt); gk = gk.to(c.xt); gv = gv.to(c.xt); gw = gw.to(c.xt); }
        }
        variable_list out{gr, gk, gv, gw, gu};
        if (twice) {   // a gradient of the gradient is not available: say so when it is asked for
            auto err = std::make_shared<torch::autograd::DelayedError>("the WKV6 backward is not differentiable", 5);
            for (auto &t : out) t = t.detach().requires_grad_(true);
            out = (*err)(std::move(out));
        }
        out.resize(8);
        return out;
    }
};

PyObject *none() { Py_RETURN_NONE; }

#define ARG(i) THPVariable_Unpack(args[i])

// wkv6(r, k, v, w, u, head_size, variant, cut = True) -> y or None
PyObject *py_wkv6(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if ((n != 7 && n != 8) || !plain_mode()) return none();
    for (int i = 0; i < 5; ++i)
        if (!plain_tensor(args[i])) return none();
    const int64_t N = PyLong_AsLongLong(args[5]), variant = PyLong_AsLongLong(args[6]);
    const bool cut = n < 8 || PyObject_IsTrue(args[7]) == 1;
    if (PyErr_Occurred()) return nullptr;
    const Tensor &r = ARG(0), &k = ARG(1), &v = ARG(2), &w = ARG(3), &u = ARG(4);
    Call c;
    if (!make_call(r, k, v, w, u, N, variant, cut, c)) return none();
    const bool grad = at::GradMode::is_enabled() && (r.requires_grad() || k.requires_grad() || v.requires_grad() ||
                                                     w.requires_grad() || u.requires_grad());
    Tensor y;
    {
        pybind11::gil_scoped_release no_gil;
        c10::cuda::CUDAGuard guard(r.device());
        if (grad) {
            y = WKV6Function::apply(r, k, v, w, u, N, variant, cut);
        } else {
            y = like(r, c.yt, c.dense);
            if (run_forward(c, r, k, v, w, u, y, nullptr, 0, nullptr, nullptr) != 0)
                y.reset();
        }
    }
    if (!y.defined()) return none();   // the Python path raises the library's error
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// with_state(r, k, v, w, u, init_state or None, head_size, variant, cut = True) -> (y, state) or None
PyObject *py_with_state(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if ((n != 8 && n != 9) || !plain_mode()) return none();
    for (int i = 0; i < 5; ++i)
        if (!plain_tensor(args[i])) return none();
    const int64_t N = PyLong_AsLongLong(args[6]), variant = PyLong_AsLongLong(args[7]);
    const bool cut = n < 9 || PyObject_IsTrue(args[8]) == 1;
    if (PyErr_Occurred()) return nullptr;
    const Tensor &r = ARG(0), &k = ARG(1), &v = ARG(2), &w = ARG(3), &u = ARG(4);
    Call c;
    if (!make_call(r, k, v, w, u, N, variant, cut, c)) return none();
    const void *s_in = nullptr;
    int32_t kinds = 0;
    at::ScalarType st = at::kFloat;
    if (args[5] != Py_None) {
        if (!plain_tensor(args[5])) return none();
        const Tensor &s = ARG(5);
        const int64_t d = s.dim();
        if ((d != 3 && d != 4) || !s.is_contiguous() || s.device() != r.device()) return none();
        if (s.size(d - 3) != c.H || s.size(d - 2) != N || s.size(d - 1) != N) return none();
        kinds = d == 4 ? (int32_t)s.size(0) : 1;
        if (kinds != 1 && kinds != c.B) return none();
        st = s.scalar_type();
        if (st != at::kFloat && st != at::kBFloat16) return none();
        s_in = s.data_ptr();
        c.p.s_dtype = dtype_code(st);
    }
    Tensor y, out;
    int rc;
    {
        pybind11::gil_scoped_release no_gil;
        c10::cuda::CUDAGuard guard(r.device());
        y = like(r, c.yt, c.dense);
        out = at::detail::empty_cuda({c.B, c.H, N, N}, st, r.device(), std::nullopt);
        if (c.T == 1 && N == 64 && c.dense && st == at::kFloat)   // a decode step: the state-streaming kernel
            rc = api.decode(&c.p, r.data_ptr(), k.data_ptr(), v.data_ptr(), w.data_ptr(), u.data_ptr(), y.data_ptr(),
                            static_cast<const float *>(s_in), nullptr, kinds, out.data_ptr<float>(), stream_of(r));
        else
            rc = run_forward(c, r, k, v, w, u, y, s_in, kinds, out.data_ptr(), nullptr);
    }
    if (rc != 0) return none();        // the Python path raises the library's error
    PyObject *t = PyTuple_New(2);
    if (t == nullptr) return nullptr;
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(y)));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(out)));
    return t;
    END_HANDLE_TH_ERRORS
}

// bind(path): the library's entry points, from the object the Python side has loaded
PyObject *py_bind(PyObject *, PyObject *arg) {
    const char *path = PyUnicode_AsUTF8(arg);
    if (path == nullptr) return nullptr;
    void *h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (h == nullptr) return PyErr_Format(PyExc_ImportError, "%s", dlerror());
#define SYM(name)                                                                                                   \
    if ((api.name = reinterpret_cast<decltype(api.name)>(dlsym(h, "wkv6_" #name))) == nullptr)                      \
        return PyErr_Format(PyExc_ImportError, "%s lacks wkv6_" #name, path);
    SYM(forward) SYM(backward) SYM(decode) SYM(ckpt_bytes) SYM(backward_workspace_bytes) SYM(sum_rows)
    SYM(split_segments) SYM(split_state_bytes) SYM(split_workspace_bytes) SYM(forward_split) SYM(backward_split)
    SYM(resolve_variant) SYM(last_error)
#undef SYM
    api.bound = true;
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", py_bind, METH_O, nullptr},
    {"wkv6", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_wkv6)), METH_FASTCALL, nullptr},
    {"with_state", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_with_state)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
