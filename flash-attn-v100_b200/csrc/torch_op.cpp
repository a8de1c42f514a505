// The common calls of flash_attention_v100() as a native autograd operator: fp16, bf16 or fp32 tensors on one GPU as the
// kernels take them, without bias or dropout.  attention() checks whether a call is one of these and answers None where
// it is not; ops/attention.py's Function then takes the call, with its messages, its other options and its error cases.
//
// What it is for: the Python operator is 40 us of host work around a forward and 150 around a training step (argument
// checks, a ctypes block, the Python side of autograd), more than the kernels of a short call take.  B200: a prompt of
// B1 N128 H8 D64 39 -> 10 us, a training step of B32 N197 H12 D64 157 -> 95 (bound by its kernels then).
//
// Replaces, for these calls, the reference's autograd.Function (ops/attention.py:36-333).
#include <ATen/FunctionalTensorWrapper.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/PythonFallbackKernel.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>
#include <atomic>
#include <cmath>
#include <cstring>
#include "../../include/fa_b200.h"

namespace py = pybind11;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

constexpr int kMaxDevices = 64;
constexpr size_t kF32PlanesMaxBytes = (size_t)8 << 30;      // as F32_PLANES_MAX_BYTES in ops/attention.py
std::atomic<int32_t*> g_status_word[kMaxDevices];           // pinned, one per device, held by ops/attention.py

// The exception types of kernels/_cabi.py; may run in an autograd thread.
void raise_for_status(int rc, const char* what) {
    if (rc == FA_OK) return;
    const std::string msg = std::string(what) + ": " + fa_b200_strerror(rc) + ": " + fa_b200_last_error();
    py::gil_scoped_acquire gil;
    const bool value = rc == FA_EINVAL || rc == FA_EUNSUPPORTED || rc == FA_EALIGN;
    PyErr_SetString(value ? PyExc_ValueError : PyExc_RuntimeError, msg.c_str());
    python_error err;
    err.persist();
    throw err;
}

// Unit stride on the head dimension, 16-byte rows: what utils.py passes to the kernels untouched.
bool rows_fit(const at::Tensor& t) {
    uintptr_t bits = (uintptr_t)t.const_data_ptr();
    for (int i = 0; i < 3; ++i) bits |= (uintptr_t)(t.stride(i) * t.element_size());
    return t.stride(3) == 1 && (bits & 15u) == 0;
}

fa_b200_tensor operand(const at::Tensor& t) { return {const_cast<void*>(t.const_data_ptr()), t.stride(0), t.stride(1), t.stride(2)}; }

struct Call {
    double scale;
    bool causal, fast;
    int64_t shift;
    at::Tensor lengths;         // may be undefined
};

fa_b200_params params_of(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, const at::Tensor& lse, const Call& c) {
    fa_b200_params p;
    memset(&p, 0, sizeof(p));
    p.struct_bytes = sizeof(p);
    p.q = operand(q); p.k = operand(k); p.v = operand(v); p.o = operand(o);
    p.lse = lse.mutable_data_ptr<float>();
    const int device = q.device().index();
    p.status_word = g_status_word[device].load(std::memory_order_acquire);
    p.stream = c10::cuda::getCurrentCUDAStream(device).stream();
    p.B = (int32_t)q.size(0); p.Nq = (int32_t)q.size(1); p.Nk = (int32_t)k.size(1);
    p.H = (int32_t)q.size(2); p.Hkv = (int32_t)k.size(2); p.D = (int32_t)q.size(3);
    p.dtype = q.scalar_type() == at::kHalf ? FA_B200_F16 : (q.scalar_type() == at::kBFloat16 ? FA_B200_BF16 : FA_B200_F32);
    p.causal = c.causal;
    p.variant = FA_B200_VARIANT_AUTO;
    p.device = device;
    p.scale = (float)c.scale;
    p.causal_shift = c.causal ? (int32_t)c.shift : 0;
    if (c.lengths.defined()) p.kv_lengths = c.lengths.const_data_ptr<int32_t>();
    return p;
}

at::Tensor bytes_like(const at::Tensor& q, size_t n) { return at::empty({(int64_t)n}, q.options().dtype(at::kByte)); }

// o, lse and, for a bf16 call whose gradients will be asked for, what rounding o dropped.  `split`: the keys of a call with
// few queries may be shared out over the SMs (calls whose inputs want gradients keep whole pairs of tiles).
void forward(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const Call& c, bool split, bool residual, at::Tensor& o, at::Tensor& lse,
             at::Tensor& o_lo) {
    o = at::empty(q.sizes(), q.options());
    lse = at::empty({q.size(0), q.size(2), q.size(1)}, q.options().dtype(at::kFloat));
    fa_b200_params p = params_of(q, k, v, o, lse, c);
    if (residual) { o_lo = at::empty(q.sizes(), q.options()); p.o_lo = operand(o_lo); }
    const size_t n = split ? fa_b200_fwd_workspace_bytes(&p) : 0;
    if (n) {
        const at::Tensor ws = bytes_like(q, n);
        raise_for_status(fa_b200_fwd_with_workspace(&p, ws.mutable_data_ptr(), n), "fa_b200_fwd");
    } else {
        raise_for_status(fa_b200_fwd(&p), "fa_b200_fwd");
    }
}

void backward(at::Tensor d_o, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& o, const at::Tensor& lse,
              const at::Tensor& o_lo, const Call& c, at::Tensor& dq, at::Tensor& dk, at::Tensor& dv) {
    if (!rows_fit(d_o)) d_o = d_o.contiguous();
    dq = at::empty(q.sizes(), q.options()); dk = at::empty(k.sizes(), k.options()); dv = at::empty(v.sizes(), v.options());
    fa_b200_params p = params_of(q, k, v, o, lse, c);
    p.d_o = operand(d_o); p.dq = operand(dq); p.dk = operand(dk); p.dv = operand(dv);
    const bool f32 = q.scalar_type() == at::kFloat;
    if (c.fast && !f32 && q.size(3) == 64) p.variant = FA_B200_VARIANT_TCGEN05;
    if (o_lo.defined()) p.o_lo = operand(o_lo);
    if (f32) {
        // planes for the tensor-core kernels, up to a limit and as far as the allocator goes
        const size_t n = fa_b200_bwd_scratch_bytes(&p);
        at::Tensor ws;
        if (n && n <= kF32PlanesMaxBytes) {
            try { ws = bytes_like(q, n); } catch (const c10::OutOfMemoryError&) {}
        }
        if (ws.defined()) { raise_for_status(fa_b200_bwd_with_scratch(&p, ws.mutable_data_ptr(), n), "fa_b200_bwd"); return; }
    }
    const size_t n = fa_b200_bwd_workspace_bytes(&p);
    const at::Tensor ws = bytes_like(q, n);
    p.workspace = ws.mutable_data_ptr();
    p.workspace_bytes = n;
    raise_for_status(fa_b200_bwd(&p), "fa_b200_bwd");
}

struct Attention : torch::autograd::Function<Attention> {
    static variable_list forward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const Call& c) {
        at::Tensor o, lse, o_lo;
        ::forward(q, k, v, c, false, q.scalar_type() == at::kBFloat16, o, lse, o_lo);
        variable_list kept{q, k, v, o, lse};
        if (o_lo.defined()) kept.push_back(o_lo);
        ctx->save_for_backward(std::move(kept));
        ctx->saved_data["scale"] = c.scale;
        ctx->saved_data["flags"] = (int64_t)c.causal | ((int64_t)c.fast << 1) | (c.shift << 2);
        if (c.lengths.defined()) ctx->saved_data["lengths"] = c.lengths;
        ctx->mark_non_differentiable({lse});
        ctx->set_materialize_grads(false);             // (lse's would be a launch of zeros)
        return {o, lse};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list kept = ctx->get_saved_variables();
        const int64_t flags = ctx->saved_data["flags"].toInt();
        const auto lengths = ctx->saved_data.find("lengths");
        const Call c{ctx->saved_data["scale"].toDouble(), (flags & 1) != 0, (flags & 2) != 0, flags >> 2,
                     lengths == ctx->saved_data.end() ? at::Tensor() : lengths->second.toTensor()};
        at::Tensor d[3];
        at::AutoDispatchBelowADInplaceOrView below;          // (allocations and a copy: nothing of this is recorded)
        if (!grads[0].defined()) grads[0] = at::zeros_like(kept[3]);
        ::backward(grads[0], kept[0], kept[1], kept[2], kept[3], kept[4], kept.size() > 5 ? kept[5] : at::Tensor(), c, d[0], d[1], d[2]);
        variable_list out(4);
        for (int i = 0; i < 3; ++i)
            if (ctx->needs_input_grad(i)) out[i] = d[i];
        return out;
    }
};

// A plain tensor on a GPU: no subclass, no wrapper, no dual number, no bits to be resolved first.
bool plain(PyObject* obj, const at::Tensor*& t) {
    if (!THPVariable_CheckExact(obj)) return false;
    t = &THPVariable_Unpack(obj);
    const auto keys = t->key_set();
    return t->is_cuda() && t->layout() == at::kStrided && !t->is_conj() && !t->is_neg() && !t->_is_zerotensor() &&
           !keys.has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::Functionalize, c10::DispatchKey::FuncTorchBatched,
                                              c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched})) &&
           !t->_fw_grad(0).defined();
}

// Whether something else wants to see the call's operators: a transform, a tracer, a mode.
bool watched() {
    return c10::impl::TorchDispatchModeTLS::any_modes_set() || at::impl::torch_function_mode_enabled() ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchVmapMode) ||
           c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Functionalize) || at::tracer::impl::is_dispatch_enabled();
}

// (o, lse), or None where the call is not one of those served here.
py::object attention(py::handle q_, py::handle k_, py::handle v_, py::handle scale_, bool causal, bool bottom_right, py::handle lengths_, bool fast) {
    const at::Tensor *qp, *kp, *vp, *lp = nullptr;
    if (watched() || !plain(q_.ptr(), qp) || !plain(k_.ptr(), kp) || !plain(v_.ptr(), vp)) return py::none();
    const at::Tensor q = *qp, k = *kp, v = *vp;          // (own references: other threads run during the call)
    const auto type = q.scalar_type();
    if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || k.sizes() != v.sizes() || q.size(0) != k.size(0) || q.size(3) != k.size(3) ||
        k.size(2) == 0 || q.size(2) % k.size(2) != 0 || q.numel() == 0 || k.numel() == 0 || q.size(3) > 128 ||
        (type != at::kHalf && type != at::kBFloat16 && type != at::kFloat) || k.scalar_type() != type || v.scalar_type() != type ||
        k.device() != q.device() || v.device() != q.device() || !rows_fit(q) || !rows_fit(k) || !rows_fit(v))
        return py::none();
    for (const at::Tensor* t : {&q, &k})
        if (t->size(0) > INT32_MAX || t->size(1) > INT32_MAX || t->size(2) > INT32_MAX) return py::none();
    const int device = q.device().index();
    if (device >= kMaxDevices || !g_status_word[device].load(std::memory_order_acquire)) return py::none();
    Call c{std::pow((double)q.size(3), -0.5), causal, fast, 0, {}};
    if (!scale_.is_none()) {
        if (!PyFloat_CheckExact(scale_.ptr())) return py::none();
        c.scale = PyFloat_AS_DOUBLE(scale_.ptr());
    }
    if (!lengths_.is_none()) {
        if (!plain(lengths_.ptr(), lp) || lp->scalar_type() != at::kInt || lp->device() != q.device() || lp->dim() != 1 || lp->size(0) != q.size(0) ||
            !lp->is_contiguous())
            return py::none();
        c.lengths = lp->detach();
    }
    if (causal && bottom_right) {
        if (k.size(1) < q.size(1) || lp) return py::none();
        c.shift = k.size(1) - q.size(1);
    }
    const bool wants = q.requires_grad() || k.requires_grad() || v.requires_grad();
    at::Tensor o, lse, o_lo;
    try {
        // Allocation and launches may have to wait (for memory, for room in the launch queue): other Python threads, which
        // may be what the GPU waits for, run meanwhile.
        py::gil_scoped_release others_run;
        if (wants && at::GradMode::is_enabled()) {
            variable_list out = Attention::apply(q, k, v, c);
            o = std::move(out[0]); lse = std::move(out[1]);
        } else {
            at::AutoDispatchBelowADInplaceOrView below;
            forward(q, k, v, c, !wants, false, o, lse, o_lo);
        }
    } catch (python_error& e) {
        e.restore();
        throw py::error_already_set();
    }
    return py::make_tuple(py::reinterpret_steal<py::object>(THPVariable_Wrap(std::move(o))), py::reinterpret_steal<py::object>(THPVariable_Wrap(std::move(lse))));
}

}  // namespace

#ifndef FA_TORCH_VERSION
#error "the build names the torch whose headers these are (FA_TORCH_VERSION)"
#endif
// Read by kernels/_cabi.py before Python imports the module: what stands above is laid out for this torch and no other.
extern "C" __attribute__((visibility("default"))) const char* fa_b200_torch_built_for() { return FA_TORCH_VERSION; }

PYBIND11_MODULE(fa_b200_torch, m) {
    m.def("attention", &attention);
    m.def("set_status_word", [](int device, uintptr_t word) {
        if (device >= 0 && device < kMaxDevices) g_status_word[device].store((int32_t*)word, std::memory_order_release);
    });
}
